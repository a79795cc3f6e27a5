// transfer.cu -- copies between the caller's host arrays and the device.
//
// A pageable copy runs through the driver's own staging one array at a time, and a
// copy back blocks until it is done: a call with ten small arrays waits ten times,
// and a large array moves at the speed of one core (6 GB/s with its page faults).
// Small arrays of a call are gathered in pinned slots, so that their copies queue
// behind one another and the call waits once; large ones are moved by up to four
// threads, each pipelining its share through its own slot.
//
// The slots are shared by all contexts of the process: at most MAX_SLOTS of SLOT
// bytes, taken under a mutex for the length of a call, and freed with the last
// context.  A call that finds none falls back to the plain copy.
#include <mutex>
#include <system_error>
#include <thread>

#include "common.cuh"

namespace sofia {
namespace {

constexpr size_t SLOT = 1 << 20;
constexpr int MAX_SLOTS = 16;
constexpr size_t DRIVER_SMALL = 64 << 10;  // up to here an H2D copy returns at once
constexpr size_t SHARE = 1 << 20;          // least bytes of a thread of a large copy
constexpr int MAX_THREADS = 4;

struct Pool {
    std::mutex m;
    void *free_slots[MAX_SLOTS];
    int nfree = 0, total = 0, contexts = 0;
};
Pool &pool() {
    static Pool p;
    return p;
}

char *take_slot() {
    Pool &p = pool();
    std::lock_guard<std::mutex> g(p.m);
    if (p.nfree > 0) return (char *)p.free_slots[--p.nfree];
    if (p.total >= MAX_SLOTS) return nullptr;
    void *s = nullptr;
    if (cudaHostAlloc(&s, SLOT, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    ++p.total;
    return (char *)s;
}

void give_slot(void *s) {
    Pool &p = pool();
    std::lock_guard<std::mutex> g(p.m);
    if (p.contexts > 0) {
        p.free_slots[p.nfree++] = s;
    } else {
        cudaFreeHost(s);
        --p.total;
    }
}

bool is_pinned(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// One thread's share of a large copy, half a slot at a time: the copy of one half
// overlaps the memcpy of the other.
struct Share {
    int device;
    bool out;
    char *host, *dev;
    size_t bytes;
    cudaStream_t st;
    cudaEvent_t ready;
    char *slot;
    cudaError_t err;
};
void move_share(Share *w) {
    constexpr size_t HALF = SLOT / 2;
    cudaError_t e = cudaSetDevice(w->device);
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (auto &x : ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(w->st, w->ready, 0);
    const size_t n = (w->bytes + HALF - 1) / HALF;
    auto len = [&](size_t k) { return k + 1 < n ? HALF : w->bytes - k * HALF; };
    for (size_t k = 0; k < n + (w->out ? 1 : 0) && e == cudaSuccess; ++k) {
        char *half = w->slot + (k & 1) * HALF;
        if (w->out) {
            if (k < n) {
                e = cudaMemcpyAsync(half, w->dev + k * HALF, len(k), cudaMemcpyDeviceToHost, w->st);
                if (e == cudaSuccess) e = cudaEventRecord(ev[k & 1], w->st);
            }
            if (k > 0 && e == cudaSuccess) {
                e = cudaEventSynchronize(ev[(k - 1) & 1]);
                if (e == cudaSuccess)
                    memcpy(w->host + (k - 1) * HALF, w->slot + ((k - 1) & 1) * HALF, len(k - 1));
            }
        } else {
            if (k >= 2) e = cudaEventSynchronize(ev[k & 1]);
            if (e != cudaSuccess) break;
            memcpy(half, w->host + k * HALF, len(k));
            e = cudaMemcpyAsync(w->dev + k * HALF, half, len(k), cudaMemcpyHostToDevice, w->st);
            if (e == cudaSuccess) e = cudaEventRecord(ev[k & 1], w->st);
        }
    }
    // nothing of the share is in flight when its slot goes back
    const cudaError_t s = cudaStreamSynchronize(w->st);
    if (e == cudaSuccess) e = s;
    for (auto &x : ev)
        if (x) cudaEventDestroy(x);
    w->err = e;
}

// A large copy by several threads, done when this returns.  False: not attempted.
bool move_large(sofia_nb_ctx *ctx, bool out, void *host, void *dev, size_t bytes, int *rc) {
    *rc = SOFIA_OK;
    const unsigned hc = std::thread::hardware_concurrency();
    int nt = (int)(bytes / SHARE);
    nt = nt < 1 ? 1 : (nt > MAX_THREADS ? MAX_THREADS : nt);
    if (hc > 0 && nt > (int)hc) nt = (int)hc;
    Share w[MAX_THREADS];
    int got = 0;
    while (got < nt) {
        if (!ctx->xstream[got] &&
            cudaStreamCreateWithFlags(&ctx->xstream[got], cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            ctx->xstream[got] = nullptr;
            break;
        }
        if (!(w[got].slot = take_slot())) break;
        ++got;
    }
    if (got == 0) return false;
    cudaEvent_t ready = nullptr;
    cudaError_t e = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(ready, ctx->stream);
    if (e == cudaSuccess) {
        const size_t part = ((bytes + got - 1) / got + 63) & ~(size_t)63;
        std::thread th[MAX_THREADS];
        for (int t = 0; t < got; ++t) {
            const size_t b0 = part * t < bytes ? part * t : bytes;
            const size_t b1 = part * (t + 1) < bytes ? part * (t + 1) : bytes;
            w[t] = Share{ctx->device, out, (char *)host + b0, (char *)dev + b0, b1 - b0,
                         ctx->xstream[t], ready, w[t].slot, cudaSuccess};
        }
        for (int t = 1; t < got; ++t) {
            try {
                th[t] = std::thread(move_share, &w[t]);
            } catch (const std::system_error &) {
                move_share(&w[t]);
            }
        }
        move_share(&w[0]);
        for (int t = 1; t < got; ++t)
            if (th[t].joinable()) th[t].join();
        for (int t = 0; t < got; ++t)
            if (e == cudaSuccess) e = w[t].err;
    }
    if (ready) cudaEventDestroy(ready);
    for (int t = 0; t < got; ++t) give_slot(w[t].slot);
    if (e != cudaSuccess) *rc = cuda_fail(ctx, e, out ? "copy to host" : "copy to device");
    return true;
}

}  // namespace

void transfer_open() {
    Pool &p = pool();
    std::lock_guard<std::mutex> g(p.m);
    ++p.contexts;
}

void transfer_close() {
    Pool &p = pool();
    std::lock_guard<std::mutex> g(p.m);
    if (--p.contexts > 0) return;
    while (p.nfree > 0) {
        cudaFreeHost(p.free_slots[--p.nfree]);
        --p.total;
    }
}

HostCopies::HostCopies(sofia_nb_ctx *c) : ctx(c), outer(c->copies) { c->copies = this; }

HostCopies::~HostCopies() {
    // a call that failed half-way: neither its slots nor the caller's pinned arrays may
    // be in use when it returns
    if (!idle) cudaStreamSynchronize(ctx->stream);
    for (int i = 0; i < nslot; ++i) give_slot(slots[i]);
    ctx->copies = outer;
}

// Room for a small array in the call's slots, or NULL.
char *HostCopies::reserve(size_t bytes) {
    const size_t need = (bytes + 255) & ~(size_t)255;
    if (need > SLOT) return nullptr;
    if (nslot == 0 || used + need > SLOT) {
        if (nslot == MAX) return nullptr;
        char *s = take_slot();
        if (!s) return nullptr;
        slots[nslot++] = s;
        used = 0;
    }
    char *p = slots[nslot - 1] + used;
    used += need;
    return p;
}

int HostCopies::in(void *dev, const void *host, size_t bytes) {
    if (bytes > DRIVER_SMALL && !is_pinned(host)) {
        if (bytes <= SLOT) {
            if (char *p = reserve(bytes)) {
                memcpy(p, host, bytes);
                host = p;
            }
        } else {
            int rc;
            if (move_large(ctx, false, const_cast<void *>(host), dev, bytes, &rc)) return rc;
        }
    }
    idle = false;
    SOFIA_CUDA(ctx, cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
    return SOFIA_OK;
}

int HostCopies::out(void *host, const void *dev, size_t bytes) {
    if (!is_pinned(host)) {
        if (bytes <= SLOT) {
            char *p = nout < MAX ? reserve(bytes) : nullptr;
            if (p) {
                idle = false;
                SOFIA_CUDA(ctx, cudaMemcpyAsync(p, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
                outs[nout++] = Out{host, p, bytes};
                return SOFIA_OK;
            }
        } else {
            int rc;
            if (move_large(ctx, true, host, const_cast<void *>(dev), bytes, &rc)) return rc;
        }
    }
    idle = false;
    SOFIA_CUDA(ctx, cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    return SOFIA_OK;
}

int HostCopies::sync() {
    SOFIA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int i = 0; i < nout; ++i) memcpy(outs[i].host, outs[i].pinned, outs[i].bytes);
    nout = 0;
    idle = true;
    return SOFIA_OK;
}

}  // namespace sofia
