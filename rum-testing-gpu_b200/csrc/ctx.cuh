// The library context: one device, one stream, cached lattice tables and workspaces.
#pragma once
#include <atomic>
#include <map>
#include <memory>
#include <mutex>

#include "common.cuh"

struct rumb_ctx;

namespace rumb {

struct BmWorkBase {
    virtual ~BmWorkBase() {}
    // what outlives a call only to save the next one's allocation: freed, counted
    virtual bool give_back() { return false; }
    virtual size_t spare_bytes() const { return 0; }
};

struct Ctx : public Spare {
    int device = 0;
    cudaStream_t own = nullptr;       // the context's stream (work always runs here)
    cudaStream_t user = nullptr;      // optional caller stream, joined by events
    cudaEvent_t ev_a = nullptr, ev_b = nullptr;
    std::atomic<int> cancel{0};
    // popcount-ordered node ids per n (int32, ascending inside a layer) and layer bounds
    std::map<int, std::shared_ptr<DevBuf>> layers;
    std::map<int, std::vector<ll>> layer_bounds;
    std::unique_ptr<BmWorkBase> bm64, bm32;     // BM-ADMM workspaces
    std::unique_ptr<BmWorkBase> batch64, batch32;  // batched-draw workspaces
    std::unique_ptr<BmWorkBase> cert;           // float64 certificate workspace
    std::unique_ptr<BmWorkBase> batch_cert;     // a batch's, of several slots
    const BmWorkBase *batch_now = nullptr;      // the running batch's workspace: its draws and slots are in use
    // A batch's certificate slots and uploaded draws stay for the next batch, until another call needs their memory.
    bool give_back() override {
        bool any = !batch_now && batch_cert;
        if (!batch_now) batch_cert.reset();
        for (BmWorkBase *w : {batch64.get(), batch32.get()})
            if (w && w != batch_now && w->give_back()) any = true;
        return any;
    }
    size_t bytes() const override {
        size_t b = batch_cert ? batch_cert->spare_bytes() : 0;
        for (const BmWorkBase *w : {batch64.get(), batch32.get()})
            if (w) b += w->spare_bytes();
        return b;
    }
    std::unique_ptr<BmWorkBase> scratch;        // primitive calls' scratch
    // the captured iteration and check graphs of the last solve of each kind (bm.cu; released before the
    // workspaces they launch on)
    std::unique_ptr<BmWorkBase> graphs64, graphs32, batch_graphs64, batch_graphs32;
    cudaEvent_t ev_t0 = nullptr, ev_t1 = nullptr;   // a call's device time (made on first use)
    // overlapped checks: a second stream and its two events; a check's pinned result words (made on first use)
    cudaStream_t aux = nullptr;
    cudaEvent_t ev_snap = nullptr, ev_done = nullptr;
    double *res_host = nullptr;
    void ensure_aux() {
        if (aux) return;
        RUMB_CUDA(cudaStreamCreateWithFlags(&aux, cudaStreamNonBlocking));
        RUMB_CUDA(cudaEventCreateWithFlags(&ev_snap, cudaEventDisableTiming));
        RUMB_CUDA(cudaEventCreateWithFlags(&ev_done, cudaEventDisableTiming));
    }
    // pinned words for a check's results and the timing events
    void ensure_host() {
        if (!res_host) RUMB_CUDA(cudaMallocHost(&res_host, 64 * sizeof(double)));
        if (!ev_t0) RUMB_CUDA(cudaEventCreate(&ev_t0));
        if (!ev_t1) RUMB_CUDA(cudaEventCreate(&ev_t1));
    }

    // Make the context's stream wait for the caller's stream (call start) ...
    void join_in() {
        if (user) {
            RUMB_CUDA(cudaEventRecord(ev_a, user));
            RUMB_CUDA(cudaStreamWaitEvent(own, ev_a, 0));
        }
    }
    // ... and the caller's stream wait for the context's (call end).
    void join_out() {
        if (user) {
            RUMB_CUDA(cudaEventRecord(ev_b, own));
            RUMB_CUDA(cudaStreamWaitEvent(user, ev_b, 0));
        }
    }
    const int *layer_table(int n, std::vector<ll> &bounds);
};

// RAII: the context whose spare memory a call may take
struct SpareGuard {
    Spare *prev;
    explicit SpareGuard(Spare *s) : prev(g_spare) { g_spare = s; }
    ~SpareGuard() { g_spare = prev; }
};

// RAII: make ctx's device current for the duration of a call
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) RUMB_CUDA(cudaSetDevice(dev));
    }
    ~DeviceGuard() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

}  // namespace rumb

struct rumb_ctx {
    rumb::Ctx c;
};

// A kept ADMM state (x2, s, y, z) on the device.
struct rumb_bm_state {
    int n = 0;
    int dtype = RUMB_F64;   // element type of the slabs (RUMB_F64 or RUMB_F32)
    int device = 0;
    rumb::DevBuf x2, s, y, z;
};
