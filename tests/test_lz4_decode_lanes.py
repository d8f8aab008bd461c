"""The LZ4 stream decoder's kernel source run on the CPU, its 256 threads as coroutines that go on in
a random order from one barrier to the next.  Shared memory written before every thread has read it,
or a barrier that only some threads reach, shows as threads that wait at different barriers or as
wrong bytes, whatever the hardware's timing would hide.  The streams hold sequences that do not fit
a window, each thread's path through them being the decoder's branch on shared values."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_gpu_lz4_decode import CASES, _stream

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BEFORE = r"""
#include <setjmp.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <random>
#include <vector>

#define __global__
#define __device__
#define __shared__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))
#define FULLMASK 0xffffffffu
using std::max;
using std::min;
struct uint4 { uint32_t x, y, z, w; };
static uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }

namespace lanes {
constexpr int N = 256, STACK = 1 << 16;
enum { RUN, AT_BLOCK, AT_WARP, ENDED };
struct Lane { ucontext_t start; jmp_buf at; bool begun; int state, site; std::vector<char> stack; };
static Lane lane[N];
static jmp_buf home;
static int cur;
static void (*body)();
// values of a collective, by its turn: a lane is at most one collective ahead of another
static int warp_val[2][N], warp_turn[N], any_val[3], block_turn[N];

static void wait_at(int state, int site)
{
    lane[cur].state = state;
    lane[cur].site = site;
    if (!_setjmp(lane[cur].at)) _longjmp(home, 1);
}
static void entry()
{
    body();
    lane[cur].state = ENDED;
    _longjmp(home, 1);
}
static void step(int k)
{
    cur = k;
    if (_setjmp(home)) return;
    if (lane[k].begun) _longjmp(lane[k].at, 1);
    lane[k].begun = true;
    setcontext(&lane[k].start);
}
// 0: every lane ended; 1: lanes of one block (or warp) wait at different barriers
static int run(void (*f)(), uint64_t seed)
{
    std::mt19937_64 rng(seed);
    body = f;
    for (int k = 0; k < N; k++) {
        lane[k].stack.resize(STACK);
        getcontext(&lane[k].start);
        lane[k].start.uc_stack.ss_sp = lane[k].stack.data();
        lane[k].start.uc_stack.ss_size = STACK;
        lane[k].start.uc_link = nullptr;
        makecontext(&lane[k].start, entry, 0);
        lane[k].begun = false;
        lane[k].state = RUN;
        warp_turn[k] = block_turn[k] = 0;
    }
    memset(any_val, 0, sizeof any_val);
    int order[N];
    for (int k = 0; k < N; k++) order[k] = k;
    for (;;) {
        // lanes in a random order, or warps in a random order with lane 0's warp first or last
        std::shuffle(order, order + N, rng);
        if (rng() & 1) {
            int first[N / 32];
            for (int &v : first) v = (int)(rng() % 1000);
            first[0] = rng() & 1 ? -1 : 1000;
            std::stable_sort(order, order + N, [&](int a, int b) { return first[a / 32] < first[b / 32]; });
        }
        bool moved = false;
        for (int k : order)
            if (lane[k].state == RUN) { step(k); moved = true; }
        for (int w = 0; w < N; w += 32) {
            bool all = true;
            for (int k = w; k < w + 32; k++) all = all && lane[k].state == AT_WARP && lane[k].site == lane[w].site;
            for (int k = w; all && k < w + 32; k++) { lane[k].state = RUN; moved = true; }
        }
        bool all = true, ended = true;
        for (int k = 0; k < N; k++) {
            all = all && lane[k].state == AT_BLOCK && lane[k].site == lane[0].site;
            ended = ended && lane[k].state == ENDED;
        }
        if (ended) return 0;
        for (int k = 0; all && k < N; k++) { lane[k].state = RUN; moved = true; }
        if (!moved) return 1;
    }
}
static int shfl_up(int v, int o, int site)
{
    const int k = cur, turn = warp_turn[k]++ & 1;
    warp_val[turn][k] = v;
    wait_at(AT_WARP, site);
    return (k & 31) >= o ? warp_val[turn][k - o] : v;
}
static int any(int v, int site)
{
    const int turn = block_turn[cur]++ % 3;
    any_val[turn] |= v;
    any_val[(turn + 1) % 3] = 0;
    wait_at(AT_BLOCK, site);
    return any_val[turn];
}
struct Idx { int x; };
static Idx index() { return {cur}; }
}  // namespace lanes
#define threadIdx (lanes::index())
#define __syncthreads() lanes::wait_at(lanes::AT_BLOCK, __LINE__)
#define __syncthreads_or(v) lanes::any(v, __LINE__)
#define __shfl_up_sync(m, v, o) lanes::shfl_up(v, o, __LINE__)
template <typename T> static T __ldg(const T *p) { return *p; }
template <typename T> static T __ldcg(const T *p) { return *p; }
template <typename T> static T atomicAdd(T *p, T v) { const T o = *p; *p += v; return o; }
static void atomicOr(uint32_t *p, uint32_t v) { *p |= v; }
static int __ffs(int v) { return __builtin_ffs(v); }
static int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }

struct Dim { unsigned x; };
static const Dim blockIdx = {0}, gridDim = {1};

struct Lz4Job { const uint8_t *src; uint8_t *dst; int *err; int32_t csize, dlen; };
constexpr int DE_LZ4 = 3;
static void dev_fail(int *err, int code) { if (!*err) *err = code; }
"""

AFTER = r"""
alignas(16) uint8_t sm_dcta[sizeof(dcta::Smem)];
static Lz4Job job;
static int planes[8];
static unsigned next_job;
static void one() { k_lz4_decode_cta(&job, planes, 8, &next_job); }

// 0: decoded; DE_LZ4: refused; -1: threads waited at different barriers.  src and dst are followed
// and preceded by 16 bytes (the kernel reads whole 16-byte words).
extern "C" int decode(const uint8_t *src, int csize, uint8_t *dst, int dlen, uint64_t seed)
{
    int err = 0;
    job = {src, dst, &err, csize, dlen};
    memset(planes, 0, sizeof planes);
    planes[0] = 1;
    next_job = 0;
    std::mt19937_64 rng(seed ^ 77);
    for (uint8_t &b : sm_dcta) b = (uint8_t)rng();           // shared memory starts with anything
    return lanes::run(one, seed) ? -1 : err;
}
"""


@pytest.fixture(scope="module")
def decode(tmp_path_factory):
    with open(os.path.join(ROOT, "iron-array_b200", "csrc", "codec.cu")) as f:
        text = f.read()
    kernel = text[text.index("namespace dcta {"):text.index("constexpr int TILE = 1024;")]
    d = tmp_path_factory.mktemp("lanes")
    (d / "lanes.cpp").write_text(BEFORE + kernel + AFTER)
    subprocess.run(["g++", "-O1", "-w", "-std=c++17", "-fPIC", "-shared", "-U_FORTIFY_SOURCE", "-fcf-protection=none",
                    "-o", str(d / "lanes.so"), str(d / "lanes.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "lanes.so")).decode
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64]

    def run(comp, n, seed):
        src = np.zeros(len(comp) + 48, np.uint8)
        at = 16 + seed % 16
        src[at:at + len(comp)] = np.frombuffer(comp, np.uint8)
        out = np.full(n + 32, 0xA5, np.uint8)
        rc = fn(src.ctypes.data + at, len(comp), out.ctypes.data + 16, n, seed)
        assert (out[:16] == 0xA5).all() and (out[n + 16:] == 0xA5).all()
        return rc, out[16:n + 16].tobytes()

    return run


# sequences wholly in a window, and literal runs and match headers longer than one (2048 bytes),
# first in a stream, in the middle, next to short ones
STREAMS = dict(CASES, apart=([2100, 3000, 6000], [4, 9, 40], [1, 50, 2000]),
               mixed=([0, 1, 2, 2040, 2048, 2060, 4100], [4, 5, 18, 19, 300, 530000], [1, 2, 3, 700, 9000]))


@pytest.mark.parametrize("kind", sorted(STREAMS))
def test_any_order_of_threads(decode, kind):
    for seed in range(6):
        rng = np.random.default_rng(seed)
        comp, want = _stream(rng, 9000 if seed < 5 else 30000, *STREAMS[kind])
        rc, got = decode(comp, len(want), seed)
        assert rc != -1, "threads waited at different barriers"
        assert rc == 0 and got == want, (kind, seed)
