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
// bytes and MAX_BIG of BIG bytes, taken under a mutex for the length of a call, and
// freed with the last context.  A call that finds none falls back to the plain copy.
//
// The driver pins host memory in blocks of 2 MB (1 to 3 ms each, 9 ms on some hosts)
// and hands out parts of them in microseconds.  A context's status words have opened
// one such block, and four slots of 448 KB fit beside them: a large copy of a new
// context, or the small arrays of a call, pin nothing new, where slots of 1 MB took a
// block for every two (first pass of a new context: FP64 point at 90,000 atoms 3.8 ms,
// 5.9 with those; five bonded calls 2.3 and 5.2).  Copies so large that the calls per
// slot tell (BIG_FROM: the 37 MB list of 9,000 atoms there and back 6.6 ms a pass in
// slots of 256 KB, 4.8 in 1 MB) take big slots.
#include <mutex>
#include <thread>

#include "common.cuh"

namespace sofia {
namespace {

constexpr size_t SLOT = 448 << 10, BIG = 1 << 20;
constexpr int MAX_SLOTS = 24, MAX_BIG = 4;
constexpr size_t BIG_FROM = 16 << 20;
constexpr size_t SMALL = 1 << 20;          // arrays up to here go through the call's slots
constexpr size_t PIECE = 32 << 10;         // least part of an array worth a copy of its own
constexpr int IN_BLOCK = 4;                // slots beside a context's status words
constexpr size_t DRIVER_SMALL = 64 << 10;  // up to here an H2D copy returns at once
constexpr size_t SHARE = 1 << 20;          // least bytes of a thread of a large copy
constexpr int MAX_THREADS = 4;

// The slots of one size.
struct Slots {
    size_t bytes;
    int most;
    void *free_slots[MAX_SLOTS];
    int nfree = 0, total = 0;
    Slots(size_t b, int m) : bytes(b), most(m) {}
};
struct Pool {
    std::mutex m;
    Slots slot{SLOT, MAX_SLOTS}, big{BIG, MAX_BIG};
    int contexts = 0;
};
Pool &pool() {
    static Pool p;
    return p;
}

char *take_slot(Slots &s) {
    std::lock_guard<std::mutex> g(pool().m);
    if (s.nfree > 0) return (char *)s.free_slots[--s.nfree];
    if (s.total >= s.most) return nullptr;
    void *p = nullptr;
    if (cudaHostAlloc(&p, s.bytes, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    ++s.total;
    return (char *)p;
}

void give_slot(Slots &s, void *p) {
    std::lock_guard<std::mutex> g(pool().m);
    if (pool().contexts > 0) {
        s.free_slots[s.nfree++] = p;
    } else {
        cudaFreeHost(p);
        --s.total;
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
    size_t half;  // bytes of half the slot
    cudaError_t err;
};
void move_share(Share *w) {
    const size_t HALF = w->half;
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
    Slots *from[MAX_THREADS];
    int got = 0;
    while (got < nt) {
        if (!ctx->xstream[got] &&
            cudaStreamCreateWithFlags(&ctx->xstream[got], cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            ctx->xstream[got] = nullptr;
            break;
        }
        from[got] = &pool().big;
        if (bytes < BIG_FROM || !(w[got].slot = take_slot(*from[got])))
            w[got].slot = take_slot(*(from[got] = &pool().slot));
        if (!w[got].slot) break;
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
                         ctx->xstream[t], ready, w[t].slot, from[t]->bytes / 2, cudaSuccess};
        }
        for (int t = 1; t < got; ++t) {
            try {
                th[t] = std::thread(move_share, &w[t]);
            } catch (...) {  // no thread, or no memory for one
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
    for (int t = 0; t < got; ++t) give_slot(*from[t], w[t].slot);
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
    for (Slots *s : {&p.slot, &p.big})
        while (s->nfree > 0) {
            cudaFreeHost(s->free_slots[--s->nfree]);
            --s->total;
        }
}

HostCopies::HostCopies(sofia_nb_ctx *c) : ctx(c), outer(c->copies) { c->copies = this; }

HostCopies::~HostCopies() {
    // a call that failed half-way: neither its slots nor the caller's pinned arrays may
    // be in use when it returns
    if (!idle) cudaStreamSynchronize(ctx->stream);
    for (int i = 0; i < nslot; ++i) give_slot(pool().slot, slots[i]);
    ctx->copies = outer;
}

// Room for the next part of a small array in the call's slots: whole in a slot that has
// the room, else in a new one while those are IN_BLOCK at most, then in what is left of
// the others.  *bytes comes in as what is left of the array and goes out as the part's
// size; NULL: no room.
char *HostCopies::reserve(size_t *bytes) {
    int at = 0;
    while (at < nslot && SLOT - used[at] < *bytes) ++at;
    if (at == nslot && nslot >= IN_BLOCK)
        for (at = 0; at < nslot && SLOT - used[at] < PIECE;) ++at;
    if (at == nslot) {
        if (nslot == MAX || !(slots[nslot] = take_slot(pool().slot))) return nullptr;
        used[nslot++] = 0;
    }
    if (*bytes > SLOT - used[at]) *bytes = SLOT - used[at];
    char *p = slots[at] + used[at];
    used[at] += (*bytes + 255) & ~(size_t)255;
    return p;
}

int HostCopies::in(void *dev, const void *host, size_t bytes) {
    const char *h = (const char *)host;
    char *d = (char *)dev;
    if (bytes > DRIVER_SMALL && !is_pinned(host)) {
        if (bytes > SMALL) {
            int rc;
            if (move_large(ctx, false, const_cast<void *>(host), dev, bytes, &rc)) return rc;
        }
        for (size_t part = bytes; bytes > 0 && bytes <= SMALL; part = bytes) {
            char *p = reserve(&part);
            if (!p) break;  // the rest the plain way
            memcpy(p, h, part);
            idle = false;
            SOFIA_CUDA(ctx, cudaMemcpyAsync(d, p, part, cudaMemcpyHostToDevice, ctx->stream));
            h += part;
            d += part;
            bytes -= part;
        }
        if (bytes == 0) return SOFIA_OK;
    }
    idle = false;
    SOFIA_CUDA(ctx, cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, ctx->stream));
    return SOFIA_OK;
}

int HostCopies::out(void *host, const void *dev, size_t bytes) {
    char *h = (char *)host;
    const char *d = (const char *)dev;
    if (!is_pinned(host)) {
        if (bytes > SMALL) {
            int rc;
            if (move_large(ctx, true, host, const_cast<void *>(dev), bytes, &rc)) return rc;
        }
        for (size_t part = bytes; bytes > 0 && bytes <= SMALL && nout < MAX_OUT; part = bytes) {
            char *p = reserve(&part);
            if (!p) break;  // the rest the plain way
            idle = false;
            SOFIA_CUDA(ctx, cudaMemcpyAsync(p, d, part, cudaMemcpyDeviceToHost, ctx->stream));
            outs[nout++] = Out{h, p, part};
            h += part;
            d += part;
            bytes -= part;
        }
        if (bytes == 0) return SOFIA_OK;
    }
    idle = false;
    SOFIA_CUDA(ctx, cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, ctx->stream));
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
