// Device memory that a call needs between its own kernels (the activation planes of the batch kernels).
//
// Outside a capture every stream has one buffer, which grows: the calls of a stream follow each other, so the next call's
// first kernel starts after the previous call's last one has read it.  A handful of streams is remembered; a further one
// takes the place of the longest unused, whose work is waited for first.
//
// A captured call may be replayed at any time and on any stream, so a capture gets memory of its own: one buffer per stream
// that takes part in it and size (calls captured on one stream follow each other in the graph, those on streams that the capture
// forked to may run beside them), tied to the graph by a user object.  When the graph and everything instantiated from it are
// gone the buffer goes to a free list that the next capture or the next growing stream takes from.
//
// Streams are told apart by their ids, which are never given out twice: a handle is reused once its stream is destroyed (while
// that stream's last work may still be running), and the per-thread default stream has one handle for every thread.  (A stream
// that is being captured must not be asked for its id and cannot be destroyed: there the handle, and the thread.)  The id is
// asked for once for each stream that a caller binds, and each time for the per-thread one: 0.25 us of a batch call.
//
// Callers hold the library's lock.
#include "kernels.h"

#include <mutex>
#include <vector>

namespace weft {

namespace {

struct Buffer { uint8_t *base; size_t bytes; int device; };
struct StreamBuffer { unsigned long long stream; int device; Buffer buffer; unsigned long long used; };
struct CaptureBuffer { unsigned long long id; const void *stream; Buffer buffer; };
thread_local char t_thread;                 // its address tells threads apart

constexpr size_t kStreams = 8, kFree = 8;
std::vector<StreamBuffer> g_streams;
std::vector<CaptureBuffer> g_captures;      // of the captures still being recorded, newest last
unsigned long long g_clock = 0, g_generation = 0;

std::mutex g_returned_lock;                 // the user object's callback runs on a thread of the driver's
std::vector<Buffer> g_returned;

void give_back(void *p) {                   // no CUDA calls are allowed here
    Buffer *b = static_cast<Buffer *>(p);
    std::lock_guard<std::mutex> guard(g_returned_lock);
    g_returned.push_back(*b);
    delete b;
}

// In this mode a thread may allocate, free and wait while it or another thread captures.
class Relaxed {
  public:
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode_); }

  private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// A buffer of at least `bytes`: a returned one that fits without being four times too large, or a new allocation.
cudaError_t obtain(size_t bytes, int device, Buffer *out) {
    {
        std::lock_guard<std::mutex> guard(g_returned_lock);
        for (size_t i = 0; i < g_returned.size(); ++i)
            if (g_returned[i].device == device && g_returned[i].bytes >= bytes && g_returned[i].bytes / 4 <= bytes) {
                *out = g_returned[i];
                g_returned.erase(g_returned.begin() + i);
                return cudaSuccess;
            }
    }
    const size_t want = (bytes + bytes / 4 + 65535) & ~size_t(65535);
    uint8_t *base = nullptr;
    const cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&base), want);
    if (e != cudaSuccess) return e;
    *out = Buffer{base, want, device};
    return cudaSuccess;
}

void drop_surplus() {                       // outside a capture: keep a few returned buffers, free the rest
    std::vector<Buffer> surplus;
    {
        std::lock_guard<std::mutex> guard(g_returned_lock);
        while (g_returned.size() > kFree) { surplus.push_back(g_returned.front()); g_returned.erase(g_returned.begin()); }
    }
    if (surplus.empty()) return;
    Relaxed relaxed;
    for (const Buffer &b : surplus) cudaFree(b.base);
}

}  // namespace

unsigned long long workspace_generation() { return g_generation; }

cudaError_t workspace(size_t bytes, cudaStream_t stream, unsigned long long *stream_id, uint8_t **out) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    cudaGraph_t graph = nullptr;
    e = cudaStreamGetCaptureInfo(stream, &status, &id, &graph);
    if (e != cudaSuccess) return e;
    if (status == cudaStreamCaptureStatusActive) {
        const void *who = stream == cudaStreamPerThread ? static_cast<const void *>(&t_thread) : stream;
        for (const CaptureBuffer &c : g_captures)
            if (c.id == id && c.stream == who && c.buffer.bytes >= bytes) { *out = c.buffer.base; return cudaSuccess; }
        Relaxed relaxed;
        Buffer b;
        e = obtain(bytes, device, &b);
        if (e != cudaSuccess) return e;
        cudaUserObject_t object;
        Buffer *owned = new Buffer(b);
        e = cudaUserObjectCreate(&object, owned, give_back, 1, cudaUserObjectNoDestructorSync);
        if (e != cudaSuccess) { give_back(owned); return e; }
        e = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
        if (e != cudaSuccess) { cudaUserObjectRelease(object, 1); return e; }
        if (g_captures.size() >= kStreams) g_captures.erase(g_captures.begin());
        g_captures.push_back(CaptureBuffer{id, who, b});
        *out = b.base;
        return cudaSuccess;
    }
    if (!*stream_id || stream == cudaStreamPerThread) {
        e = cudaStreamGetId(stream, stream_id);
        if (e != cudaSuccess) { *stream_id = 0; return e; }
    }
    drop_surplus();
    StreamBuffer *mine = nullptr;
    for (StreamBuffer &s : g_streams)
        if (s.stream == *stream_id && s.device == device) mine = &s;
    if (mine && mine->buffer.bytes >= bytes) {
        mine->used = ++g_clock;
        *out = mine->buffer.base;
        return cudaSuccess;
    }
    Relaxed relaxed;
    if (!mine) {
        if (g_streams.size() >= kStreams) {
            size_t oldest = 0;
            for (size_t i = 1; i < g_streams.size(); ++i)
                if (g_streams[i].used < g_streams[oldest].used) oldest = i;
            e = cudaDeviceSynchronize();    // its stream may be gone by now; what it left behind is not
            if (e != cudaSuccess) return e;
            cudaFree(g_streams[oldest].buffer.base);
            g_streams.erase(g_streams.begin() + oldest);
            ++g_generation;
        }
        g_streams.push_back(StreamBuffer{*stream_id, device, Buffer{nullptr, 0, device}, 0});
        mine = &g_streams.back();
    }
    mine->used = ++g_clock;
    if (mine->buffer.bytes < bytes) {
        if (mine->buffer.base) {            // the stream's earlier work may still read the old one
            e = cudaStreamSynchronize(stream);
            if (e != cudaSuccess) return e;
            cudaFree(mine->buffer.base);
            mine->buffer = Buffer{nullptr, 0, device};
            ++g_generation;
        }
        e = obtain(bytes, device, &mine->buffer);
        if (e != cudaSuccess) return e;
    }
    *out = mine->buffer.base;
    return cudaSuccess;
}

}  // namespace weft
