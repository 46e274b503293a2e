// Copies between host buffers and the device through pinned staging
// (HostStage, lqg_host.h).
#include <cstring>

#include "lqg_host.h"

namespace lqg_host {

namespace {

// The staging at a size for copies of n bytes; replacing it waits for the
// copies that still use it.
lqg_status ready(HostStage& g, size_t n) {
    const size_t slot = n <= HostStage::kSmall ? HostStage::kSmall : HostStage::kLarge;
    if (g.slot >= slot) return LQG_OK;
    for (int i = 0; i < HostStage::kSlots; ++i) {
        if (g.busy[i]) LQG_CUDA(cudaEventSynchronize(g.ev[i]));
        g.busy[i] = false;
        if (!g.ev[i]) LQG_CUDA(cudaEventCreateWithFlags(&g.ev[i], cudaEventDisableTiming));
    }
    if (g.p) cudaFreeHost(g.p);
    g.p = nullptr;
    g.slot = 0;
    if (cudaHostAlloc(&g.p, HostStage::kSlots * slot + kCtlWords * sizeof(uint32_t),
                      cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        g.p = nullptr;
        return fail(LQG_ERR_NOMEM, "pinned staging allocation failed");
    }
    g.slot = slot;
    return LQG_OK;
}

// Whether the driver can copy from or to p without staging of its own.
bool registered(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

}  // namespace

lqg_status copy_in(Workspace& w, void* dst, const void* src, size_t n, cudaStream_t st) {
    if (n == 0) return LQG_OK;
    if (registered(src)) {
        LQG_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st));
        return LQG_OK;
    }
    HostStage& g = w.stage;
    lqg_status s = ready(g, n);
    if (s != LQG_OK) return s;
    const size_t slot = g.slot;
    for (size_t o = 0; o < n; o += slot) {
        const size_t c = n - o < slot ? n - o : slot;
        const int i = g.next;
        g.next = (g.next + 1) % HostStage::kSlots;
        unsigned char* h = g.p + i * slot;
        if (g.busy[i]) LQG_CUDA(cudaEventSynchronize(g.ev[i]));
        g.busy[i] = false;
        std::memcpy(h, static_cast<const unsigned char*>(src) + o, c);
        LQG_CUDA(cudaMemcpyAsync(static_cast<unsigned char*>(dst) + o, h, c, cudaMemcpyHostToDevice, st));
        LQG_CUDA(cudaEventRecord(g.ev[i], st));
        g.busy[i] = true;
    }
    return LQG_OK;
}

lqg_status copy_out(Workspace& w, void* dst, const void* src, size_t n, cudaStream_t st) {
    if (n == 0) {
        LQG_CUDA(cudaStreamSynchronize(st));
        return LQG_OK;
    }
    if (registered(dst)) {
        LQG_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st));
        LQG_CUDA(cudaStreamSynchronize(st));
        return LQG_OK;
    }
    HostStage& g = w.stage;
    lqg_status s = ready(g, n);
    if (s != LQG_OK) return s;
    const size_t slot = g.slot;
    const size_t chunks = (n + slot - 1) / slot;
    auto size_of = [&](size_t k) {
        const size_t o = k * slot;
        return n - o < slot ? n - o : slot;
    };
    // chunk k goes through slot k % kSlots, requested once chunk k - kSlots has
    // been copied on; copies out of the slots (copy_in) come earlier in `st`
    auto request = [&](size_t k) -> lqg_status {
        const int i = (int)(k % HostStage::kSlots);
        LQG_CUDA(cudaMemcpyAsync(g.p + i * slot,
                                 static_cast<const unsigned char*>(src) + k * slot,
                                 size_of(k), cudaMemcpyDeviceToHost, st));
        LQG_CUDA(cudaEventRecord(g.ev[i], st));
        return LQG_OK;
    };
    for (int i = 0; i < HostStage::kSlots; ++i) {
        // a slot of another stream's copy_in (every earlier call ended
        // synchronised with its own stream unless it failed)
        if (g.busy[i]) LQG_CUDA(cudaEventSynchronize(g.ev[i]));
        g.busy[i] = false;
    }
    for (size_t k = 0; k < chunks && k < HostStage::kSlots; ++k)
        if ((s = request(k)) != LQG_OK) return s;
    for (size_t k = 0; k < chunks; ++k) {
        const int i = (int)(k % HostStage::kSlots);
        LQG_CUDA(cudaEventSynchronize(g.ev[i]));
        std::memcpy(static_cast<unsigned char*>(dst) + k * slot, g.p + i * slot,
                    size_of(k));
        if (k + HostStage::kSlots < chunks && (s = request(k + HostStage::kSlots)) != LQG_OK) return s;
    }
    return LQG_OK;
}

lqg_status fetch_ctl(Workspace& w, size_t most, cudaStream_t st) {
    lqg_status s = ready(w.stage, most);
    if (s != LQG_OK) return s;
    LQG_CUDA(cudaMemcpyAsync(w.stage.ctl(), w.d_ctl, kCtlWords * sizeof(uint32_t),
                             cudaMemcpyDeviceToHost, st));
    return LQG_OK;
}

}  // namespace lqg_host
