"""CPU test of the host copies (csrc/transfer.cu), compiled as host code against a stand-in
for the CUDA runtime in which a queued copy runs as late as the real one may: when its
stream or event is waited for.  Covers what a call leaves behind when it fails half-way,
arrays that are reused at once, every size class in both directions, a call that finds all
pinned slots taken, threads that cannot be made, what a first call pins, and the slots'
return with the last context."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SRC = r"""
#include <cmath>
#include "transfer.cu"
#include <atomic>
#include <cstdlib>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <vector>

// ---- the stand-in runtime: copies wait in their stream's queue
static std::recursive_mutex g_m;
static std::map<cudaStream_t, std::deque<std::function<void()>>> g_q;
static std::map<char *, size_t> g_pinned;      // cudaHostAlloc and the caller's pinned arrays
static std::map<cudaEvent_t, cudaStream_t> g_ev;
static size_t g_alloc = 0, g_bytes = 0, g_most = 0;  // live cudaHostAlloc blocks
static std::atomic<long> g_id{100};
static bool pinned_(const void *p) {
    auto it = g_pinned.upper_bound((char *)p);
    return it != g_pinned.begin() && (char *)p < (--it)->first + it->second;
}
static void drain(cudaStream_t s) {
    auto &q = g_q[s];
    while (!q.empty()) {
        auto f = q.front();
        q.pop_front();
        f();
    }
}
static size_t pending() {
    size_t n = 0;
    for (auto &q : g_q) n += q.second.size();
    return n;
}
// operator new fails for this thread, outside the stand-ins
static thread_local bool t_nomem = false;
struct Exempt {
    bool was = t_nomem;
    Exempt() { t_nomem = false; }
    ~Exempt() { t_nomem = was; }
};
void *operator new(size_t n) {
    void *p = t_nomem ? nullptr : malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
#define LOCK Exempt ex; std::lock_guard<std::recursive_mutex> lk(g_m)
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    LOCK; *p = malloc(n); g_pinned[(char *)*p] = n; ++g_alloc; g_bytes += n;
    if (g_bytes > g_most) g_most = g_bytes;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    LOCK; g_bytes -= g_pinned[(char *)p]; g_pinned.erase((char *)p); --g_alloc; free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    LOCK; memset(a, 0, sizeof(*a));
    a->type = pinned_(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    LOCK; *s = (cudaStream_t)(g_id++); return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { LOCK; drain(s); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    LOCK; *e = (cudaEvent_t)(g_id++); return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { LOCK; g_ev[e] = s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { LOCK; drain(g_ev[e]); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned) {
    LOCK; drain(g_ev[e]); return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    LOCK;
    if (pinned_(k == cudaMemcpyHostToDevice ? s : d)) {
        g_q[st].push_back([=] { memcpy(d, s, n); });
    } else if (k == cudaMemcpyHostToDevice && n <= (64 << 10)) {  // staged by the driver
        std::vector<char> t((const char *)s, (const char *)s + n);
        g_q[st].push_back([=] { memcpy(d, t.data(), n); });
    } else {
        drain(st);
        memcpy(d, s, n);
    }
    return cudaSuccess;
}
}

typedef std::vector<unsigned char> Bytes;
static int failures = 0;
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); ++failures; } } while (0)
static Bytes noise(size_t n, unsigned seed) {
    Bytes b(n);
    for (auto &x : b) { seed = seed * 1664525u + 1013904223u; x = (unsigned char)(seed >> 24); }
    return b;
}
struct Ctx : sofia_nb_ctx {
    Ctx() { stream = (cudaStream_t)(g_id++); sofia::transfer_open(); }
    ~Ctx() { sofia::transfer_close(); }
};
static const size_t SIZES[] = {1, 255, 256, 65536, 65537, 200000, 262143, 262144, 262145, 700001,
                               1048576, 1048577, 2097153, 9000001, 16777216, 20000003};
// one array in and back: reused as soon as in() returns, delivered by sync()
static void round_trip(sofia_nb_ctx *c, size_t n, unsigned seed) {
    const Bytes want = noise(n, seed);
    Bytes a = want, dev(n, 0), b(n, 0);
    sofia::HostCopies h(c);
    CHECK(h.in(dev.data(), a.data(), n) == SOFIA_OK);
    std::fill(a.begin(), a.end(), 0x55);
    CHECK(h.out(b.data(), dev.data(), n) == SOFIA_OK);
    CHECK(h.sync() == SOFIA_OK);
    CHECK(dev == want && b == want);
}
static void failed_calls() {
    Ctx c;
    for (size_t n : {100ul, 100000ul, 3000000ul})
        for (int pin = 0; pin < 2; ++pin)
            for (int dir = 0; dir < 2; ++dir) {
                Bytes a = noise(n, 7), dev(n);
                if (pin) g_pinned[(char *)a.data()] = n;
                {
                    sofia::HostCopies h(&c);
                    CHECK((dir ? h.out(a.data(), dev.data(), n) : h.in(dev.data(), a.data(), n)) ==
                          SOFIA_OK);
                }  // the call fails here, before sync()
                CHECK(pending() == 0);
                if (pin) g_pinned.erase((char *)a.data());
            }
}
static void sizes() {
    Ctx c;
    unsigned seed = 1;
    for (size_t n : SIZES) round_trip(&c, n, ++seed);
    // many arrays of one call, all delivered by its sync()
    std::vector<Bytes> want, dev, got;
    for (int k = 0; k < 40; ++k) {
        want.push_back(noise(40000 * (k % 9) + 1, 100 + k));
        dev.push_back(Bytes(want[k].size()));
        got.push_back(Bytes(want[k].size()));
    }
    sofia::HostCopies h(&c);
    for (int k = 0; k < 40; ++k) CHECK(h.in(dev[k].data(), want[k].data(), want[k].size()) == SOFIA_OK);
    for (int k = 0; k < 40; ++k) CHECK(h.out(got[k].data(), dev[k].data(), got[k].size()) == SOFIA_OK);
    CHECK(h.sync() == SOFIA_OK);
    CHECK(got == want);
}
static void slots_taken() {
    Ctx c, d;
    std::vector<Bytes> a, dev;
    // calls that hold every slot there is: further small arrays pin nothing more
    std::vector<sofia::HostCopies *> held;
    std::vector<Ctx *> others;
    for (size_t last = ~0ul; g_alloc != last;) {
        last = g_alloc;
        others.push_back(new Ctx);
        held.push_back(new sofia::HostCopies(others.back()));
        for (int k = 0; k < 20; ++k) {
            a.push_back(noise(250000, 3));
            dev.push_back(Bytes(250000));
            CHECK(held.back()->in(dev.back().data(), a.back().data(), 250000) == SOFIA_OK);
        }
    }
    unsigned seed = 50;
    for (size_t n : SIZES) round_trip(&d, n, ++seed);
    for (auto *h : held) { CHECK(h->sync() == SOFIA_OK); delete h; }
    for (auto *o : others) delete o;
    for (size_t k = 0; k < a.size(); ++k) CHECK(dev[k] == a[k]);
    CHECK(g_most <= (16u << 20));
}
// What a new context pins: a large array, or a call's small ones, fit in the 2 MB that the
// driver pins at least, beside the context's own few words.
static void first_use() {
    const size_t most = 7u << 18;
    { Ctx c; round_trip(&c, 9000000, 5); CHECK(g_most <= most); }
    { Ctx c; round_trip(&c, 216000, 6); CHECK(g_most <= most); }
    Ctx c;
    Bytes a = noise(540000, 8), dev(540000);
    sofia::HostCopies h(&c);
    for (size_t n : {384000, 96000, 540000, 288000}) CHECK(h.in(dev.data(), a.data(), n) == SOFIA_OK);
    CHECK(h.out(a.data(), dev.data(), 288000) == SOFIA_OK);
    CHECK(h.sync() == SOFIA_OK && g_most <= most);
}
static void threads() {
    auto work = [](unsigned seed) {
        for (int k = 0; k < 20; ++k) {
            Ctx c;
            for (size_t n : SIZES) round_trip(&c, n, seed + k);
        }
    };
    std::thread t1(work, 1000), t2(work, 2000), t3(work, 3000);
    t1.join(); t2.join(); t3.join();
}
// Threads that cannot be made: the calling one moves their shares.
static void no_memory() {
    Ctx c;
    const Bytes want = noise(9000001, 9);
    Bytes dev(want.size()), got(want.size());
    sofia::HostCopies h(&c);
    t_nomem = true;
    const int in = h.in(dev.data(), want.data(), want.size());
    const int out = h.out(got.data(), dev.data(), got.size());
    t_nomem = false;
    CHECK(in == SOFIA_OK && out == SOFIA_OK && h.sync() == SOFIA_OK && got == want);
}
int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "failed_calls") failed_calls();
    if (what == "sizes") sizes();
    if (what == "slots_taken") slots_taken();
    if (what == "threads") threads();
    if (what == "first_use") first_use();
    if (what == "no_memory") no_memory();
    CHECK(g_alloc == 0 && pending() == 0);  // the last context took the slots with it
    printf(failures ? "failed\n" : "ok\n");
    return failures != 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("copies")
    (d / "copies.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I",
                    os.path.join(ROOT, "molecular_simulation_code_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", CUDA_INC, "-o", str(d / "copies"),
                    str(d / "copies.cpp")], check=True, timeout=300)
    return str(d / "copies")


@pytest.mark.parametrize("what", ["failed_calls", "sizes", "slots_taken", "threads",
                                  "first_use", "no_memory"])
def test_host_copies(harness, what):
    r = subprocess.run([harness, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
