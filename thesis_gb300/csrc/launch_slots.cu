// launch_slots.cu -- the memory that persistent launches need while they run
// (launch_slots.hpp): grid-barrier counters, words of a device array of fixed
// size, and the 2-D engine's exchange buffers.
#include "launch_slots.hpp"

#include "host.hpp"

namespace st {

namespace {

// Calls that a capture in another thread (or on this one) would refuse: asking
// for an event, allocating.  None of them becomes part of a capture.
struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

constexpr int kBarrierWords = 256;
__device__ unsigned g_grid_bar[kBarrierWords];

void CUDART_CB graph_gone(void *flag) { static_cast<std::atomic<bool> *>(flag)->store(false); }

struct Cuda {
    typedef cudaStream_t Stream;
    typedef cudaEvent_t Event;
    struct Capture {
        unsigned long long id = 0;
        cudaGraph_t graph = nullptr;
    };
    bool words;  // slots are words of g_grid_bar as long as there are any
    unsigned *base = nullptr;
    std::vector<int> free_words;

    explicit Cuda(bool w) : words(w) {}

    int alloc(size_t bytes, void **mem) {
        Relaxed r;
        if (words && !base) {
            ST_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&base), g_grid_bar));
            for (int k = kBarrierWords; k-- > 0;) free_words.push_back(k);
        }
        if (words && !free_words.empty()) {
            *mem = base + free_words.back();
            free_words.pop_back();
            return STENCIL_OK;
        }
        ST_CUDA(cudaMalloc(mem, bytes));
        return STENCIL_OK;
    }
    void dealloc(void *mem) {
        Relaxed r;
        unsigned *w = static_cast<unsigned *>(mem);
        if (base && w >= base && w < base + kBarrierWords) free_words.push_back((int)(w - base));
        else cudaFree(mem);
    }
    int make_event(Event *e) {
        ST_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
        return STENCIL_OK;
    }
    void drop_event(Event e) { cudaEventDestroy(e); }
    int record(Event e, Stream s) {
        ST_CUDA(cudaEventRecord(e, s));
        return STENCIL_OK;
    }
    bool happened(Event e) {
        Relaxed r;
        if (cudaEventQuery(e) == cudaSuccess) return true;
        cudaGetLastError();
        return false;
    }
    int wait(Stream s, Event e) {
        ST_CUDA(cudaStreamWaitEvent(s, e, 0));
        return STENCIL_OK;
    }
    void sync(Event e) {
        Relaxed r;
        cudaEventSynchronize(e);
    }
    // the array's address may be another one after a device reset
    void emptied() {
        base = nullptr;
        free_words.clear();
    }
    int hold(cudaGraph_t graph, std::atomic<bool> *flag) {
        cudaUserObject_t obj = nullptr;
        ST_CUDA(cudaUserObjectCreate(&obj, flag, graph_gone, 1, cudaUserObjectNoDestructorSync));
        if (cudaError_t e = cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove)) {
            cudaUserObjectRelease(obj, 1);
            return cuda_fail(e, "cudaGraphRetainUserObject");
        }
        return STENCIL_OK;
    }
};

// One of each kind per device, made on first use and kept until the process
// ends (a graph's callback may come late).  At most as many barrier words as
// the array has, and 16 exchange buffers (the largest is 20 MB), beside those
// that graphs hold.
struct DevicePools {
    Cuda words{true}, buffers{false};
    SlotPool<Cuda> barriers{&words, kBarrierWords}, exchanges{&buffers, 16};
    std::mutex mu;
    size_t largest = 0;  // bytes of the largest exchange asked for outside a capture
};

DevicePools *pools() {
    static std::mutex mu;
    static DevicePools *p[64] = {};
    const int dev = current_device();
    if (dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!p[dev]) p[dev] = new DevicePools;
    return p[dev];
}

int take_slot(SlotPool<Cuda> &pool, cudaStream_t s, const Cuda::Capture &cap, size_t bytes, LaunchSlot *slot) {
    // the calling thread's default stream: one handle for many streams; a
    // capturing stream cannot be asked for its id, but its handle is its own
    // until the capture ends
    unsigned long long id = 0;
    if (s != cudaStreamPerThread) {
        if (cap.id) id = (unsigned long long)reinterpret_cast<uintptr_t>(s);
        else ST_CUDA(cudaStreamGetId(s, &id));
    }
    SlotPool<Cuda>::Slot *x = nullptr;
    const int rc = pool.take(s, id, cap, bytes, &x);
    if (rc) return rc;
    slot->pool = &pool;
    slot->slot = x;
    slot->stream = s;
    ST_CUDA(cudaMemsetAsync(x->mem, 0, bytes, s));
    return STENCIL_OK;
}

int capture_of(cudaStream_t s, Cuda::Capture *cap) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    ST_CUDA(cudaStreamGetCaptureInfo(s, &st, &cap->id, &cap->graph));
    if (st == cudaStreamCaptureStatusNone) *cap = Cuda::Capture();
    else if (st != cudaStreamCaptureStatusActive) return fail(STENCIL_ECUDA, "the stream's capture is invalid");
    return STENCIL_OK;
}

}  // namespace

LaunchSlot::~LaunchSlot() {
    if (slot) static_cast<SlotPool<Cuda> *>(pool)->ended(static_cast<SlotPool<Cuda>::Slot *>(slot), stream);
}

void *LaunchSlot::mem() const { return static_cast<SlotPool<Cuda>::Slot *>(slot)->mem; }

int take_barrier(cudaStream_t s, LaunchSlot *slot) {
    DevicePools *p = pools();
    if (!p) return fail(STENCIL_ECUDA, "no current device");
    Cuda::Capture cap;
    const int rc = capture_of(s, &cap);
    return rc ? rc : take_slot(p->barriers, s, cap, sizeof(unsigned), slot);
}

int take_exchange(cudaStream_t s, size_t bytes, LaunchSlot *slot) {
    DevicePools *p = pools();
    if (!p) return fail(STENCIL_ECUDA, "no current device");
    Cuda::Capture cap;
    const int rc = capture_of(s, &cap);
    if (rc) return rc;
    {
        std::lock_guard<std::mutex> lock(p->mu);
        if (cap.id && bytes > p->largest)
            return fail(STENCIL_EUNSUPPORTED,
                        "2-D temporal blocking: run the dispatch once outside the graph capture "
                        "(its exchange buffer is allocated then)");
        p->largest = std::max(p->largest, bytes);
    }
    return take_slot(p->exchanges, s, cap, bytes, slot);
}

void release_slots() {
    DevicePools *p = pools();
    if (!p) return;
    p->barriers.release();
    p->exchanges.release();
    std::lock_guard<std::mutex> lock(p->mu);
    p->largest = 0;
}

}  // namespace st
