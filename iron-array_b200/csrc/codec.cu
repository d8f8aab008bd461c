// Blosc2 LZ4+SHUFFLE chunk decoder and encoder on the GPU.
//
// Replaces, for ironArray's matmul path, the Blosc2 block decode done by
// blosc2_getitem_ctx / blosc2_decompress_ctx (src/linalg/iarray_gemm.c:259-274,
// src/linalg/iarray_gemm_a.c:316, src/linalg/iarray_gemv.c:194-209, and the panel
// slices of src/iarray_container.c:628-737) and the output encode done by
// blosc2_compress_ctx (src/linalg/iarray_gemm.c:405-422, src/linalg/matmul/gemm.c:216-233),
// plus Caterva's padded blocked layout (iarray_from_buffer / iarray_to_buffer,
// src/iarray_constructor.c:218-305).
//
// Decode = parse (8 lanes per block read its stream headers and queue its LZ4 streams) -> LZ4 (one
// CTA per LZ4 stream from a job queue that may span several containers; each window of the
// stream decoded in parallel: token chain by linked segment tracks, output resolved in shared
// memory) -> unshuffle/scatter (slices of shuffled blocks staged in shared memory by bulk
// asynchronous copies, items written to the dense row-major array; a general path for the other
// blocks).  Raw and run streams are never copied before the scatter.
//
// Encode = gather/shuffle (dense -> byte-plane image) -> LZ4 -> layout (per chunk: stream
// kinds, offsets, memcpy fallback; exclusive scan of chunk sizes) -> emit (copy payloads
// into the final contiguous chunk buffer).  Two LZ4 encoders: one warp per stream
// reproducing liblz4 1.9.4 LZ4_compress_fast(acceleration 1) output byte for byte (the codec
// c-blosc2 calls for BLOSC_LZ4: 16 KiB hash table in shared memory, 32 positions at a time),
// and a parallel-parse encoder (one CTA per stream, valid LZ4 with
// different bytes).  Stream-kind selection (zero/run, raw when LZ4 does not fit, memcpyed
// chunk when the output would exceed nbytes + 32) follows c-blosc2's blosc_c rules.
#include <cuda_runtime.h>
#include <stdint.h>

#include "bytes.cuh"
#include "common.cuh"
#include "tc_common.cuh"

namespace iab {

#define FULLMASK 0xffffffffu

// 4 bytes at any address; the aligned words read hold at least one of them each.
__device__ __forceinline__ int32_t ld_s32(const uint8_t *p)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~uintptr_t(3));
    const uint32_t sh = (uint32_t)(a & 3) * 8;
    return (int32_t)__funnelshift_r(__ldg(w), sh ? __ldg(w + 1) : 0u, sh);
}

__device__ __forceinline__ void dev_fail(int *err, int code) { atomicCAS(err, 0, code); }

// q = a / b, r = a - q b for a >= 0, b > 0: 32-bit division when both fit (the usual case),
// 64-bit otherwise.
__device__ __forceinline__ void divmod(int64_t a, int64_t b, int64_t &q, int64_t &r)
{
    if (((a | b) >> 31) == 0) {
        const uint32_t q32 = (uint32_t)a / (uint32_t)b;
        q = q32;
        r = a - (int64_t)q32 * b;
    } else {
        q = a / b;
        r = a - q * b;
    }
}

// Block b of chunk c: its first logical row and column, and how many of its rows (nr) and
// columns (nc) hold logical items (the rest is chunk or array padding; 0 when none do).
struct BlockSpan {
    int64_t row0, col0;
    int nr, nc;
};
__device__ __forceinline__ BlockSpan block_span(const Geom &g, int64_t c, int64_t b)
{
    BlockSpan s;
    int64_t ci0, ci1, bi0, bi1;
    divmod(c, g.cgrid[1], ci0, ci1);
    divmod(b, g.bgrid[1], bi0, bi1);
    s.row0 = ci0 * g.chunk[0] + bi0 * g.block[0];
    s.col0 = ci1 * g.chunk[1] + bi1 * g.block[1];
    s.nr = (int)max((int64_t)0, min(min(g.block[0], g.chunk[0] - bi0 * g.block[0]), g.shape[0] - s.row0));
    s.nc = (int)max((int64_t)0, min(min(g.block[1], g.chunk[1] - bi1 * g.block[1]), g.shape[1] - s.col0));
    return s;
}

// ============================================================================ decode
// D0: parse one (chunk, block) per 8 lanes, lane j for stream j.  What bounds it is the chain of
// loads (chunk offset, header, block start, and one size word after the other, each where the
// stream before it ends) and, as every warp runs the code once, fetching the instructions: so a
// lane loads one header word and one size word, the latter at once where it lies when the streams
// before it are raw, the usual case but for the last planes; the group then goes through the
// streams in a loop of a few instructions, loading only the size words that lie elsewhere, and
// lane j stores stream j's descriptor.  (One thread per block, its loops unrolled: 16 us a
// launch for an operand of some ten blocks, timed with its events; now 12.)
// zf (optional): per (chunk, block) zero flags of the reference's block-pair products:
// bit 0 = block_is_zeros (src/linalg/iarray_gemm.c:28-77: no memcpyed or special chunk, and
// the first typesize csize words from the block's bstart are all 0: Blosc2 v5 chunks always
// carry the flag bit the reference reads as "split"), bit 1 = chunk_is_zeros (:17-26:
// special value ZERO); nzero counts the flagged blocks that hold logical items.  Blocks of padding
// only, which every ragged array has, take part in no product, so they do not call for the zero
// rule's launches (4056 x 3230 x 3712 float64 5.17 -> 4.85 ms; 4000 x 4001 float64 matrix-vector product in
// blocks of 150 x 100, whose rule needs the dense matrix, 0.487 -> 0.35).
struct ParsedStream {
    bool lz4;                  // an LZ4 stream
    bool general;              // lane 0 of a block that the fast scatter does not take
    int32_t q, cs, neblock;    // its payload's place in the chunk, its size, its output's
    const uint8_t *chunk;
};
__device__ __forceinline__ void parse_block(const Geom &g, const uint8_t *__restrict__ ch, const int64_t *__restrict__ off,
                                            const int32_t *__restrict__ len, BlockDesc *bd, StreamDesc *sd, int *err,
                                            uint8_t *zf, int *nzero, int64_t t, bool valid, ParsedStream &ps)
{
    const int j = threadIdx.x & 7;
    int64_t c = 0, b = 0, coff = 0;
    int32_t clen = 0;
    if (valid) {
        divmod(t, g.nblocks, c, b);
        coff = off[c];
        clen = len[c];
    }
    const uint8_t *p = ch + coff;
    bool ok = clen >= 32;
    const int32_t hw = ok ? ld_s32(p + 4 * j) : 0;
    const int32_t bstart = ok && 36 + 4 * b <= clen ? ld_s32(p + 32 + 4 * b) : 0;
    const uint32_t w0 = (uint32_t)__shfl_sync(FULLMASK, hw, 0, 8);
    const int32_t nbytes = __shfl_sync(FULLMASK, hw, 1, 8), bsz = __shfl_sync(FULLMASK, hw, 2, 8),
                  cbytes = __shfl_sync(FULLMASK, hw, 3, 8), w16 = __shfl_sync(FULLMASK, hw, 4, 8),
                  w20 = __shfl_sync(FULLMASK, hw, 5, 8);
    const uint32_t w28 = (uint32_t)__shfl_sync(FULLMASK, hw, 7, 8);
    const uint8_t flags = (uint8_t)(w0 >> 16), ts = (uint8_t)(w0 >> 24);
    ok = ok && (flags & 0x05) == 0x05 && nbytes == g.chunk_nbytes && cbytes >= 32 && cbytes <= clen;
    int fail = ok || !valid ? 0 : DE_HEADER;
    // the size word of stream j where the streams before it are raw
    const int32_t step = (int32_t)(g.blocksize / g.itemsize) + 4;
    int32_t pre = 0;
    {
        const int64_t at = bstart + (int64_t)j * step;
        if (ok && j < g.itemsize && bstart >= 32 && at + 4 <= cbytes) pre = ld_s32(p + at);
    }
    const int special = (int)(w28 >> 28) & 7;
    if (zf) {
        bool z = ok && !special && !(flags & 0x02) && 32 + 4 * (b + 1) <= cbytes && bstart >= 32 &&
                 bstart + 4 * (int64_t)ts <= cbytes;
        for (int i = j; z && i < ts; i += 8) z = ld_s32(p + bstart + 4 * i) == 0;
        const unsigned group = 0xffu << (threadIdx.x & 24);
        z = (__ballot_sync(FULLMASK, z) & group) == group;
        if (valid && j == 0) {
            const uint8_t zflag = ok ? (special == 1 ? 2 : 0) | (z ? 1 : 0) : 0;
            zf[t] = zflag;
            if (zflag && nzero) {
                const BlockSpan sp = block_span(g, c, b);
                if (sp.nr > 0 && sp.nc > 0) atomicAdd(nzero, 1);
            }
        }
    }
    int mode = BM_PLAIN, nstreams = 1, neblock = (int)g.blocksize;
    int64_t value_src = 0, src = 0;
    int kind = SK_RUN, slen = 0;
    bool streams = false;                          // a block of size words and payloads
    if (ok) {
        if (special) {
            if (special == 2) mode = BM_NAN;
            else if (special == 3) {
                if (cbytes < 32 + (int32_t)g.itemsize) fail = DE_HEADER;
                mode = BM_VALUE; value_src = coff + 32;
            } else if (special != 1 && special != 4) fail = DE_HEADER;
        } else if (flags & 0x02) {                 // memcpyed: raw blocked items
            if (cbytes < 32 + nbytes) fail = DE_BOUNDS;
            else if (j == 0) { kind = SK_RAW; slen = (int)g.blocksize; src = coff + 32 + b * g.blocksize; }
        } else {
            // filters: only SHUFFLE (slot 5 == 1) or none are produced on this path
            const uint8_t filter5 = (uint8_t)((uint32_t)w20 >> 8);
            const bool filt_ok = w16 == 0 && (w20 & 0xFF) == 0 && filter5 <= 1;
            const int64_t bs_end = 32 + 4 * g.nblocks;
            if (bsz != g.blocksize || ts != g.itemsize || !filt_ok) {
                fail = DE_HEADER;
            } else {
                nstreams = !(flags & 0x10) ? ts : 1;
                neblock = (int)(g.blocksize / nstreams);
                if (bs_end > cbytes || bstart < bs_end || bstart >= cbytes) fail = DE_BOUNDS;
                else {
                    streams = true;
                    if (filter5 == 1 && ts > 1) mode = BM_SHUFFLED;
                }
            }
        }
    }
    bool whole = streams;
    int32_t at = 0;
    {
        int64_t q = bstart;
#pragma unroll 1
        for (int k = 0; k < 8; k++) {
            const int32_t ahead = __shfl_sync(FULLMASK, pre, k, 8);
            if (!whole || k >= nstreams) continue;
            if (q + 4 > cbytes) { fail = DE_BOUNDS; whole = false; continue; }
            const int32_t cs = q == bstart + (int64_t)k * step ? ahead : ld_s32(p + q);
            q += 4;
            if (cs == 0) continue;
            if (cs < 0) {
                if (q + 1 > cbytes || !(p[q] & 1) || cs < -255) { fail = DE_RUN_TOKEN; whole = false; continue; }
                q += 1;
                if (k == j) slen = -cs;
                continue;
            }
            if (q + cs > cbytes || cs > neblock) { fail = DE_BOUNDS; whole = false; continue; }
            if (k == j) {
                kind = cs == neblock ? SK_RAW : SK_LZ4;
                slen = cs;
                src = coff + q;
                at = (int32_t)q;
            }
            q += cs;
        }
    }
    if (streams && !whole) { kind = SK_RUN; slen = 0; }
    if (valid) {
        if (j == 0) {
            BlockDesc d;
            d.mode = mode; d.nstreams = nstreams; d.neblock = neblock; d.pad = 0; d.value_src = value_src;
            bd[t] = d;
            if (fail) dev_fail(err, fail);
        }
        StreamDesc d;
        d.kind = kind; d.len = slen; d.src = src;
        sd[t * 8 + j] = d;
    }
    ps.lz4 = valid && kind == SK_LZ4;
    ps.general = valid && j == 0 && !(mode == BM_SHUFFLED && nstreams == g.itemsize);
    ps.q = at; ps.cs = slen; ps.neblock = neblock; ps.chunk = p;
}

// Queues the LZ4 streams of a warp's blocks (every lane calls): stream j of a block goes to region
// j of the queue, counted by njobs[j], so that the decoder gets the streams plane by plane.  (The
// first planes of smooth floats are the longest streams, the last one the shortest: handed out in
// the blocks' order instead, the decode of a 20000 x 20000 float32 matrix takes 6.45 ms, by planes 6.0.)
// The eight counters are bumped by one instruction per warp.
__device__ __forceinline__ void queue_streams(const ParsedStream &ps, uint8_t *blk_scratch, int *err, Lz4Job *jobs,
                                              int *njobs, int64_t jcap)
{
    const int lane = threadIdx.x & 31, j = lane & 7;
    const unsigned m = __ballot_sync(FULLMASK, ps.lz4) & (0x01010101u << j);   // the plane's
    if (!__any_sync(FULLMASK, ps.lz4)) return;
    int base = 0;
    if (lane < 8 && m) base = atomicAdd(njobs + j, __popc(m));
    const int64_t region = jcap / 8, k = (int64_t)__shfl_sync(FULLMASK, base, j) + __popc(m & ((1u << lane) - 1u));
    if (!ps.lz4) return;
    if (k < region) {
        Lz4Job jb;
        jb.src = ps.chunk + ps.q; jb.dst = blk_scratch + (int64_t)j * ps.neblock; jb.err = err;
        jb.csize = ps.cs; jb.dlen = ps.neblock;
        jobs[j * region + k] = jb;
    } else {
        dev_fail(err, DE_BOUNDS);                                // (a region holds a stream of every block)
    }
}

// (blockDim.x is a multiple of 32; 8 threads a block)
constexpr int PARSE_T = 128;
__global__ void __launch_bounds__(PARSE_T) k_parse(Geom g, const uint8_t *__restrict__ ch, const int64_t *__restrict__ off,
                                                   const int32_t *__restrict__ len, BlockDesc *bd, StreamDesc *sd,
                                                   Lz4Job *jobs, int *njobs, int64_t jcap, int *err, int *ngeneral,
                                                   uint8_t *scratch, uint8_t *zf, int *nzero)
{
    const int64_t total = g.nchunks * g.nblocks;
    for (int64_t t0 = (int64_t)blockIdx.x * (PARSE_T / 8); t0 < total; t0 += (int64_t)gridDim.x * (PARSE_T / 8)) {
        const int64_t t = t0 + threadIdx.x / 8;
        ParsedStream ps;
        parse_block(g, ch, off, len, bd, sd, err, zf, nzero, t, t < total, ps);
        queue_streams(ps, scratch + t * g.blocksize, err, jobs, njobs, jcap);
        const unsigned m = __ballot_sync(FULLMASK, ps.general);
        if (m && (threadIdx.x & 31) == 0) atomicAdd(ngeneral, __popc(m));
    }
}
static unsigned parse_grid(int64_t nbl, int sms)
{
    return (unsigned)std::max<int64_t>(std::min<int64_t>(ceil_div(nbl, PARSE_T / 8), (int64_t)sms * 16), 1);
}

// D1: LZ4 stream decode, one CTA (256 threads) per stream, streams handed out
// dynamically (a CTA's first is that of its own number, see stream_at) from a job queue, which may
// hold the streams of several containers: each job carries its source, destination and status
// word.  The stream is consumed in windows of up to DW compressed bytes staged in shared memory
// (the next window's loads are issued as soon as its start is known).  With many streams in flight
// the SM's issue rate bounds the kernel (1,024 of 64 KiB: 72% of the slots), so each step is chosen
// for few instructions per byte:
//  1. the chain of token positions from the window start: every thread walks the tokens of one
//     32-byte segment from one of its first four bytes, four tracks per segment.  A walk from
//     a wrong byte need not meet the true chain soon (sequences of 3 bytes keep their phase),
//     but the true chain soon runs on one of the four tracks: so a track's exit is linked to
//     the track it enters (after a few more tokens, where it is on none), and the tracks on
//     the path from the window start are marked by pointer doubling over the 256 tracks.  The
//     result is a bit per window byte;
//  2. each thread reads the lengths of the tokens of its 8 bytes, and an exclusive scan over
//     token counts and output lengths numbers the sequences and places their output;
//  3. the output is resolved in groups of at most DCAP bytes in shared memory: a literal
//     byte takes its value from the window, a match byte points at its source (a source
//     inside the same match is folded back below the match start modulo the offset); sources
//     before the group are read from the already written output (a ring of its latest bytes,
//     else global memory).  Sequences are filled by one, eight or all threads, by length;
//  4. every byte follows its sources (at most HOPS of them per sweep; a byte left open keeps
//     its place on the chain, so that the chains through it shorten) and is written;
//  5. a sequence with more than DCAP output bytes is copied straight in global memory
//     (all its sources lie before its own match start), and a sequence too long for a
//     window is decoded alone with its header read from global memory.
// Measured against the doubled chain, matches copied byte by byte from global memory where the
// ring did not reach, and separate resolving and writing sweeps: a 512 MiB float64 operand pair
// of 64 KiB planes 2.06 -> 1.25 ms, 250 KB planes of a smooth 1.6 GB float32 matrix 9.85 -> 6.1 ms.
namespace dcta {
constexpr int THREADS = 256;
constexpr int DW = 2048;                   // compressed bytes per window
constexpr int SEG = 32, NSEG = DW / SEG;   // segments of the chain walk
constexpr int TRACKS = THREADS / NSEG;
constexpr int SPAN = DW / THREADS;         // per thread of the field step (at most 3 tokens)
constexpr int MAXS = DW / 3 + 2;           // sequences per window (a non-final one takes >= 3 bytes)
constexpr int HB = 8192;                   // output history kept in shared memory for match sources
constexpr int LONGSEQ = 16, GROUP = 8;     // longer sequences are filled by GROUP threads
constexpr int VLONG = 256;                 // and longer ones by the whole CTA
constexpr int DCAP = 3584;                 // output bytes resolved in shared memory at once
constexpr int HOPS = 12;
constexpr int WALK_MAX = 32;               // chains of at most this many sequences are walked by one thread
constexpr uint16_t STOP = 0xFFFF, ENDS = 0xFFFE;
constexpr uint32_t RES = 0x80000000u;      // resolved output byte (value in the low 8 bits)
constexpr uint32_t BIAS = 65536;           // else the source's place relative to the group, plus BIAS
struct Smem {
    union {
        uint32_t st[DCAP];                 // per output byte
        struct {                           // the chain walk (before the output is resolved)
            uint32_t m[THREADS];           // a track's tokens, track-major
            uint32_t any[NSEG];            // the tokens of a segment's tracks
            uint16_t link[2][THREADS + 1]; // the track after it, then the 2nd, 4th, ... (THREADS: none)
            uint16_t entry[THREADS];       // where the path enters a track
            uint8_t on[THREADS];           // on the path
        } c;
    };
    int32_t ostart[MAXS + 1];              // output offset of each sequence in the window
    uint16_t llen[MAXS];
    int32_t mlen[MAXS];
    uint16_t lpos[MAXS];
    uint16_t off[MAXS];
    uint32_t mask[DW / 32];                // token positions
    uint4 raw[DW / 16 + 1];                // the window from its 16-byte boundary
    uint8_t hist[HB];                      // the last HB output bytes (ring, by absolute position)
    uint16_t longs[DCAP / (LONGSEQ + 1) + 1];  // sequences of a group longer than LONGSEQ bytes
    uint16_t vlongs[DCAP / (VLONG + 1) + 1];   // longer than VLONG bytes
    int32_t nlong, nvlong;
    int32_t wsum[THREADS / 32];
    int32_t scal[9];
};
}  // namespace dcta

// next[q] for a sequence starting at window offset q (n valid bytes, rem bytes left in
// the stream from the window start).
__device__ __forceinline__ uint16_t dcta_next(const uint8_t *win, int q, int n, int rem)
{
    const int tok = win[q];
    int lit = tok >> 4, r = q + 3 + lit;
    if (lit != 15 && (tok & 15) != 15 && r <= n) return (uint16_t)r;
    r = q + 1;
    if (lit == 15) {
        int b = 255;
        while (b == 255) {
            if (r >= n) return dcta::STOP;
            b = win[r++];
            lit += b;
        }
    }
    r += lit;
    if (r > n) return dcta::STOP;
    if (r == rem) return dcta::ENDS;      // literals reach the stream end: the last sequence
    if (r + 2 > n) return dcta::STOP;
    r += 2;
    if ((tok & 15) == 15) {
        int b = 255;
        while (b == 255) {
            if (r >= n) return dcta::STOP;
            b = win[r++];
        }
    }
    return (uint16_t)r;                   // r <= n; r == n: the next token starts the next window
}

__global__ void __launch_bounds__(dcta::THREADS, 6) k_lz4_decode_cta(const Lz4Job *__restrict__ jobs,
                                                                  const int *__restrict__ planes, int64_t jcap,
                                                                  unsigned *next_job)
{
    using namespace dcta;
    extern __shared__ __align__(16) uint8_t sm_dcta[];
    Smem &S = *reinterpret_cast<Smem *>(sm_dcta);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t region = jcap / 8;               // the queue's part for one plane
    if (tid == 0) S.nlong = S.nvlong = 0;          // first use follows the barriers below
    // 16 bytes of the window at p from its 16-byte boundary; every block read holds a byte of the stream
    auto fetch = [&](const uint8_t *in, int p, int isz) -> uint4 {
        const int y = tid * 16 - (int)(reinterpret_cast<uintptr_t>(in + p) & 15);
        return tid <= DW / 16 && p + y < isz && y < DW ? __ldg(reinterpret_cast<const uint4 *>(in + p + y))
                                                       : make_uint4(0u, 0u, 0u, 0u);
    };
    for (bool first = true;; first = false) {
        __syncthreads();
        if (tid == 0) S.scal[0] = (int)(first ? blockIdx.x : gridDim.x + atomicAdd(next_job, 1u));
        __syncthreads();
        int64_t jid = (unsigned)S.scal[0];
        int plane = 0;
        for (; plane < 8; plane++) {
            const int64_t n = min((int64_t)planes[plane], region);
            if (jid < n) break;
            jid -= n;
        }
        if (plane == 8) break;
        const Lz4Job jb = jobs[plane * region + jid];
        const uint8_t *__restrict__ in = jb.src;
        const int isz = jb.csize;
        uint8_t *out = jb.dst;
        const int osz = jb.dlen;
        int p = 0, op = 0;                 // window start in the input, output written so far
        int hist_from = 0;                 // S.hist holds output bytes [hist_from, written)
        bool bad = false, done = false;    // block-uniform
        bool walk = false;                 // block-uniform: one thread walks this window's chain (after a sparse window)
        uint4 pre = fetch(in, 0, isz);
        while (!done && !bad) {
            const int rem = isz - p, n = min(DW, rem);
            const uint8_t *win = reinterpret_cast<const uint8_t *>(S.raw) + (reinterpret_cast<uintptr_t>(in + p) & 15);
            __syncthreads();
            if (tid <= DW / 16) S.raw[tid] = pre;
            if (tid < DW / 32) S.mask[tid] = 0;
            __syncthreads();
            if (n <= 0) { bad = true; break; }
            // After a window of few sequences (long literal runs, long matches) one thread walks the
            // chain of token positions, at most WALK_MAX steps; when the chain does not leave the
            // window by then, and in the other windows, all threads walk tracks.  Both leave the tokens in mask, why the chain ended (n, ENDS or STOP) in
            // scal[1], the last token in scal[3].
            bool found = false;
            if (walk) {
                if (tid == 0) {
                    int q = 0, k = 0, res = 0;
                    for (;;) {
                        const uint16_t v = dcta_next(win, q, n, rem);
                        S.mask[q >> 5] |= 1u << (q & 31);
                        if (v >= n) { res = 1; S.scal[1] = v; S.scal[3] = q; break; }
                        if (++k >= WALK_MAX) break;
                        q = v;
                    }
                    S.scal[8] = res;
                }
                __syncthreads();
                found = S.scal[8] != 0;
            }
            if (!found) {
                const int seg = tid % NSEG, lo = seg * SEG, hi = min(lo + SEG, n);
                uint32_t m = 0;
                int x = lo + tid / NSEG;
                while (x < hi) {                            // positions grow: at most SEG / 3 + 1 steps
                    m |= 1u << (x - lo);
                    x = dcta_next(win, x, n, rem);
                }
                S.c.m[tid] = m;
                if (tid < DW / 32) S.mask[tid] = 0;         // (the one-thread walk's, when it gave up)
                __syncthreads();
                if (tid < NSEG) {
                    uint32_t any = 0;
#pragma unroll
                    for (int t = 0; t < TRACKS; t++) any |= S.c.m[t * NSEG + tid];
                    S.c.any[tid] = any;
                }
                __syncthreads();
                int e = x, link = THREADS;
                while (e < n && !((S.c.any[e / SEG] >> (e % SEG)) & 1u)) e = dcta_next(win, e, n, rem);
                if (e < n) {
#pragma unroll
                    for (int t = 0; t < TRACKS; t++)
                        if ((S.c.m[t * NSEG + e / SEG] >> (e % SEG)) & 1u) link = t * NSEG + e / SEG;
                }
                S.c.link[0][tid] = (uint16_t)link;
                S.c.on[tid] = tid == 0;                     // the window starts on track 0 of segment 0
                if (tid == 0) S.c.link[0][THREADS] = S.c.link[1][THREADS] = (uint16_t)THREADS;
                __syncthreads();
                int j = link;
#pragma unroll
                for (int k = 0; (1 << k) < NSEG; k++) {     // tracks fewer than 2^k links away are on
                    if (S.c.on[tid] && j < THREADS) S.c.on[j] = 1;
                    j = S.c.link[k & 1][j];
                    S.c.link[(k & 1) ^ 1][tid] = (uint16_t)j;
                    __syncthreads();
                }
                const bool on = S.c.on[tid];
                if (on) {
                    int last = lo + 31 - __clz((int)m);
                    for (int t = x; t != e; t = dcta_next(win, t, n, rem)) {   // tokens on no track
                        atomicOr(&S.mask[t >> 5], 1u << (t & 31));
                        last = t;
                    }
                    if (link < THREADS) S.c.entry[link] = (uint16_t)e;
                    else { S.scal[1] = e; S.scal[3] = last; }
                }
                __syncthreads();
                if (on) atomicOr(&S.mask[seg], m & (FULLMASK << (tid ? S.c.entry[tid] % SEG : 0)));
                __syncthreads();
            }
            const int term = S.scal[1], lastq = S.scal[3];  // term: n, ENDS or STOP
            const int pnext = p + (term == STOP ? lastq : n);
            if (term != STOP || lastq > 0) {                // at least one whole sequence
                if (term != ENDS) pre = fetch(in, pnext, isz);
                // sequence fields and validity: the tokens of this thread's SPAN bytes
                if (tid == 0) S.scal[2] = 0;
                int part = 0, num = 0;                      // output bytes, sequences
                int f_lit[3], f_ml[3], f_lp[3], f_off[3];
                uint32_t mt = (S.mask[tid * SPAN >> 5] >> (tid * SPAN & 31)) & ((1u << SPAN) - 1u);
                if (term == STOP && lastq / SPAN == tid) mt &= ~(1u << (lastq % SPAN));   // not whole
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    f_lit[k] = f_ml[k] = f_lp[k] = f_off[k] = 0;
                    if (mt) {
                        const int q = tid * SPAN + __ffs((int)mt) - 1;
                        mt &= mt - 1;
                        const int tok = win[q];
                        int r = q + 1, lit = tok >> 4;
                        if (lit == 15) {
                            int b = 255;
                            while (b == 255) { b = win[r++]; lit += b; }
                        }
                        f_lp[k] = r;
                        f_lit[k] = lit;
                        r += lit;
                        int ml = 0;
                        if (!(q == lastq && term == ENDS)) {
                            f_off[k] = win[r] | (win[r + 1] << 8);
                            r += 2;
                            ml = tok & 15;
                            if (ml == 15) {
                                int b = 255;
                                while (b == 255) { b = win[r++]; ml += b; }
                            }
                            ml += 4;
                        }
                        f_ml[k] = ml;
                        part += lit + ml;
                        num++;
                    }
                }
                // exclusive scan of counts (10 bits) and output lengths (below 255 DW < 2^20)
                static_assert(MAXS < 1024 && 255 * DW < (1 << 20), "packed scan");
                int incl = part | (num << 20);
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(FULLMASK, incl, o);
                    if (lane >= o) incl += v;
                }
                if (lane == 31) S.wsum[warp] = incl;
                __syncthreads();
                int wbase = 0;
#pragma unroll
                for (int w = 0; w < THREADS / 32; w++) wbase += w < warp ? S.wsum[w] : 0;
                const int excl = wbase + incl - (part | (num << 20));
                int acc = excl & 0xFFFFF, i = excl >> 20;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    if (k < num) {
                        S.ostart[i] = acc;
                        S.llen[i] = (uint16_t)f_lit[k];
                        S.mlen[i] = f_ml[k];
                        S.lpos[i] = (uint16_t)f_lp[k];
                        S.off[i] = (uint16_t)f_off[k];
                        const int ms = op + acc + f_lit[k];             // absolute match start
                        if (f_ml[k] > 0 && (f_off[k] == 0 || f_off[k] > ms)) S.scal[2] = 1;
                        acc += f_lit[k] + f_ml[k];
                        i++;
                    }
                }
                if (tid == THREADS - 1) {                          // the last thread holds the totals
                    S.ostart[i] = acc;
                    S.scal[7] = i;
                }
                __syncthreads();
                const int nseq = S.scal[7], total = S.ostart[nseq];
                walk = nseq <= WALK_MAX;
                if (S.scal[2] || total > osz - op) { bad = true; break; }
                // output in groups of at most DCAP bytes
                int a = 0;
                while (a < nseq) {
                    const int base = S.ostart[a];
                    int lo = a + 1, hi = nseq;                      // largest b with ostart[b] - base <= DCAP
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (S.ostart[mid] - base <= DCAP) lo = mid; else hi = mid - 1;
                    }
                    const int b = lo;
                    if (S.ostart[b] - base <= DCAP) {
                        const int span = S.ostart[b] - base;
                        // Bytes first, first + step, ... of sequence i: literal bytes as values,
                        // match bytes as their sources' places (match byte k's at m0 - d + (k mod d):
                        // below the match start even when the match overlaps itself).
                        auto fill = [&](int i, int first, int step) {
                            const int s0 = S.ostart[i] - base, lit = S.llen[i], ml = S.mlen[i];
                            const uint8_t *lp = win + S.lpos[i];
                            for (int x = first; x < lit; x += step) S.st[s0 + x] = RES | lp[x];
                            const int d = S.off[i];
                            uint32_t *st = S.st + s0 + lit;
                            const uint32_t src = BIAS + (uint32_t)(s0 + lit - d);
                            if (ml <= d) {
                                for (int k = first; k < ml; k += step) st[k] = src + k;
                            } else {
                                const int inc = step < d ? step : step % d;
                                for (int k = first, km = first < d ? first : first % d; k < ml; k += step) {
                                    st[k] = src + km;
                                    km += inc;
                                    if (km >= d) km -= d;
                                }
                            }
                        };
                        for (int i = a + tid; i < b; i += THREADS) {
                            const int len = S.llen[i] + S.mlen[i];
                            if (len <= LONGSEQ) fill(i, 0, 1);
                            else if (len <= VLONG) S.longs[atomicAdd(&S.nlong, 1)] = (uint16_t)i;
                            else S.vlongs[atomicAdd(&S.nvlong, 1)] = (uint16_t)i;
                        }
                        __syncthreads();
                        const int nlong = S.nlong, nvlong = S.nvlong;
                        for (int j = tid / GROUP; j < nlong; j += THREADS / GROUP) fill(S.longs[j], tid % GROUP, GROUP);
                        for (int j = 0; j < nvlong; j++) fill(S.vlongs[j], tid, THREADS);
                        __syncthreads();
                        if (tid == 0) S.nlong = S.nvlong = 0;          // read above, before the barrier
                        uint8_t *o = out + op + base;
                        // sources before the group: the ring, as far as this group's bytes do not
                        // replace it, else the written output
                        const int hist_lo = max(hist_from, op + base + span - HB);
                        for (;;) {                                 // follow the sources, write
                            int open = 0;
                            for (int x = tid; x < span; x += THREADS) {
                                uint32_t v = S.st[x];
                                for (int h = 0; h < HOPS && v - BIAS < (uint32_t)DCAP; h++) v = S.st[v - BIAS];
                                if (v < BIAS) {
                                    const int abs = op + base + (int)v - (int)BIAS;
                                    v = RES | (abs >= hist_lo ? (uint32_t)S.hist[abs & (HB - 1)] : (uint32_t)__ldcg(out + abs));
                                }
                                S.st[x] = v;
                                if (v & RES) {
                                    o[x] = (uint8_t)v;
                                    S.hist[(op + base + x) & (HB - 1)] = (uint8_t)v;
                                } else {
                                    open = 1;
                                }
                            }
                            if (!__syncthreads_or(open)) break;
                        }
                        hist_from = max(hist_from, op + base + span - HB);
                        a = b;
                    } else {
                        // one sequence larger than DCAP: literals, then the match from global memory
                        const int abs0 = op + base, lit = S.llen[a], ml = S.mlen[a], d = S.off[a];
                        for (int x = tid; x < lit; x += THREADS) out[abs0 + x] = win[S.lpos[a] + x];
                        __syncthreads();
                        const int m0 = abs0 + lit;
                        for (int x = tid; x < ml; x += THREADS) out[m0 + x] = __ldcg(out + m0 - d + (d > x ? x : x % d));
                        hist_from = m0 + ml;                        // the ring missed this sequence
                        a = a + 1;
                    }
                    __syncthreads();
                }
                op += total;
                if (term == ENDS) { done = true; break; }
                p = pnext;
                continue;
            }
            // the sequence at p does not fit in a window: decode it alone, header from global.
            // Every thread has to be here before scal is written: it branched on scal[1] and scal[3].
            __syncthreads();
            if (tid == 0) {
                int r = p, f = 0, lit = 0, mo = 0, ml = 0, fin = 0;
                const int tok = __ldg(in + r++);
                lit = tok >> 4;
                if (lit == 15) {
                    int bb = 255;
                    while (bb == 255) {
                        if (r >= isz) { f = 1; break; }
                        bb = __ldg(in + r++);
                        lit += bb;
                    }
                }
                const int lp = r;
                if (!f && (lit > isz - r || lit > osz - op)) f = 1;
                if (!f) {
                    r += lit;
                    if (r == isz) {
                        fin = 1;
                    } else if (isz - r < 2) {
                        f = 1;
                    } else {
                        mo = __ldg(in + r) | (__ldg(in + r + 1) << 8);
                        r += 2;
                        ml = tok & 15;
                        if (ml == 15) {
                            int bb = 255;
                            while (bb == 255) {
                                if (r >= isz) { f = 1; break; }
                                bb = __ldg(in + r++);
                                ml += bb;
                            }
                        }
                        ml += 4;
                        if (!f && (mo == 0 || mo > op + lit || ml > osz - op - lit)) f = 1;
                    }
                }
                S.scal[2] = f; S.scal[3] = lit; S.scal[4] = lp; S.scal[5] = mo; S.scal[6] = ml; S.scal[7] = fin ? -1 : r;
            }
            __syncthreads();
            if (S.scal[2]) { bad = true; break; }
            {
                const int lit = S.scal[3], lp = S.scal[4], mo = S.scal[5], ml = S.scal[6], nr = S.scal[7];
                for (int x = tid; x < lit; x += THREADS) out[op + x] = __ldg(in + lp + x);
                __syncthreads();
                const int m0 = op + lit;
                for (int x = tid; x < ml; x += THREADS) out[m0 + x] = __ldcg(out + m0 - mo + (mo > x ? x : x % mo));
                __syncthreads();
                op += lit + ml;
                hist_from = op;                            // the ring missed this sequence
                if (nr < 0) done = true; else p = nr;
                if (!done) pre = fetch(in, p, isz);
            }
        }
        if (!bad && op != osz) bad = true;
        if (bad && tid == 0) dev_fail(jb.err, DE_LZ4);
    }
}

constexpr int TILE = 1024;

__device__ __forceinline__ void store_item(uint8_t *o, int ts, uint64_t v)
{
    switch (ts) {
    case 8: *reinterpret_cast<uint64_t *>(o) = v; break;
    case 4: *reinterpret_cast<uint32_t *>(o) = (uint32_t)v; break;
    case 2: *reinterpret_cast<uint16_t *>(o) = (uint16_t)v; break;
    default: for (int j = 0; j < ts; j++) o[j] = (uint8_t)(v >> (8 * j)); break;
    }
}

__device__ __forceinline__ uint64_t load_item(const uint8_t *o, int ts)
{
    switch (ts) {
    case 8: return *reinterpret_cast<const uint64_t *>(o);
    case 4: return *reinterpret_cast<const uint32_t *>(o);
    case 2: return *reinterpret_cast<const uint16_t *>(o);
    default: { uint64_t v = 0; for (int j = 0; j < ts; j++) v |= (uint64_t)o[j] << (8 * j); return v; }
    }
}

// An item at any byte offset (a special-value chunk's value sits right after the chunk's
// 32-byte header, and chunks lie back to back at arbitrary offsets).
__device__ __forceinline__ uint64_t load_item_bytes(const uint8_t *o, int ts)
{
    uint64_t v = 0;
    for (int j = 0; j < ts; j++) v |= (uint64_t)__ldg(o + j) << (8 * j);
    return v;
}

// Map item i of block b of chunk c to its logical (row, col); false if it is padding.
__device__ __forceinline__ bool item_pos(const Geom &g, int64_t c, int64_t b, int64_t i, int64_t &row, int64_t &col)
{
    const int64_t ci0 = c / g.cgrid[1], ci1 = c - ci0 * g.cgrid[1];
    const int64_t bi0 = b / g.bgrid[1], bi1 = b - bi0 * g.bgrid[1];
    const int64_t r = i / g.block[1], cc = i - r * g.block[1];
    const int64_t rin = bi0 * g.block[0] + r, cin = bi1 * g.block[1] + cc;
    if (rin >= g.chunk[0] || cin >= g.chunk[1]) return false;
    row = ci0 * g.chunk[0] + rin;
    col = ci1 * g.chunk[1] + cin;
    return row < g.shape[0] && col < g.shape[1];
}

// Partitions with items of 4 or 8 bytes take the fast paths below, edge blocks included:
// where block rows hold whole groups of 4 items, 4 items and a word of each plane at a time,
// else item by item.
__host__ __device__ __forceinline__ bool geom_quads(const Geom &g) { return !(g.block[1] & 3); }

// D2 fast path: shuffled, split blocks of 4- and 8-byte items, in slices of SC_ITEMS items
// (one CTA per slice at a time).  One thread stages the slice's bytes of every byte plane (read
// in place from raw streams or the LZ4 scratch) into shared memory with bulk asynchronous
// copies completing on an mbarrier; then each thread rebuilds items and writes the logical ones
// to the dense row (edge blocks: the items in chunk or array padding are not written; slices of
// padding only are skipped): 4 consecutive items from one 4-byte word per plane, stored as they lie
// in a row where block rows hold whole groups of 4, else as two pairs where they are of an even
// width, else one by one (4000 x 6000 float64 in blocks of 100 x 150: 0.12 ms; 0.15 by one byte
// per plane and item, 0.79 by the general path's bytewise tiles).  Blocks of other kinds go by the
// general path.
constexpr int SC_ITEMS = 4096;
constexpr int GA_ITEMS = 16384;                    // items of a gather slice
constexpr int SC_PLANE = SC_ITEMS + 32;            // a slice of a plane from its 16-byte boundary
constexpr uint32_t SC_WAIT_POLLS = 1u << 22;

__device__ __forceinline__ void bulk_g2s(void *sdst, const void *gsrc, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc::smem_addr(sdst)), "l"(gsrc), "r"(bytes), "r"(tc::smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool sc_wait(uint64_t *bar, uint32_t parity)
{
    for (uint32_t i = 0; i < SC_WAIT_POLLS; i++)
        if (tc::mbar_try_wait(bar, parity)) return true;
    return false;
}

// D2 general path: unshuffle one tile of TILE items of one block through shared memory
// and scatter it to the dense array (other item sizes; plain, special and unsplit blocks).
__device__ __forceinline__ void scatter_tile(const Geom &g, const uint8_t *__restrict__ ch,
                                             const BlockDesc *__restrict__ bd, const StreamDesc *__restrict__ sd,
                                             const uint8_t *__restrict__ scratch, uint8_t *__restrict__ out, int64_t ld,
                                             int64_t t, int64_t i0, uint8_t *planes)
{
    const int ts = g.itemsize;
    const int cnt = (int)min((int64_t)TILE, g.blockn - i0);
    const int64_t c = t / g.nblocks, b = t - c * g.nblocks;
    const BlockDesc d = bd[t];
    const StreamDesc *s = sd + t * 8;
    const uint8_t *blk_scratch = scratch + t * g.blocksize;
    if (d.mode == BM_SHUFFLED) {
        for (int j = 0; j < ts; j++) {
            const int64_t pos = (int64_t)j * g.blockn + i0;
            const int sidx = (int)(pos / d.neblock);
            const int64_t so = pos - (int64_t)sidx * d.neblock;
            const StreamDesc q = s[sidx];
            uint8_t *pl = planes + j * TILE;
            if (q.kind == SK_RUN) {
                for (int x = threadIdx.x; x < cnt; x += blockDim.x) pl[x] = (uint8_t)q.len;
            } else if (q.kind == SK_RAW) {
                const uint8_t *src = ch + q.src + so;
                for (int x = threadIdx.x; x < cnt; x += blockDim.x) pl[x] = __ldg(src + x);
            } else {
                const uint8_t *src = blk_scratch + (int64_t)sidx * d.neblock + so;
                for (int x = threadIdx.x; x < cnt; x += blockDim.x) pl[x] = __ldcg(src + x);
            }
        }
    } else if (d.mode == BM_PLAIN && d.nstreams == 1) {          // (stored as it is, or one stream)
        const StreamDesc q = s[0];
        const uint8_t *src = q.kind == SK_RAW ? ch + q.src + i0 * ts : blk_scratch + i0 * ts;
        for (int x = threadIdx.x; x < cnt * ts; x += blockDim.x)
            planes[x] = q.kind == SK_RUN ? (uint8_t)q.len : __ldcg(src + x);
    } else if (d.mode == BM_PLAIN) {
        for (int x = threadIdx.x; x < cnt * ts; x += blockDim.x) {
            const int64_t pos = i0 * ts + x;
            const int sidx = (int)(pos / d.neblock);
            const int64_t so = pos - (int64_t)sidx * d.neblock;
            const StreamDesc q = s[sidx];
            uint8_t v;
            if (q.kind == SK_RUN) v = (uint8_t)q.len;
            else if (q.kind == SK_RAW) v = __ldg(ch + q.src + so);
            else v = __ldcg(blk_scratch + (int64_t)sidx * d.neblock + so);
            planes[x] = v;
        }
    }
    __syncthreads();
    for (int x = threadIdx.x; x < cnt; x += blockDim.x) {
        int64_t row, col;
        if (!item_pos(g, c, b, i0 + x, row, col)) continue;
        uint8_t *o = out + (row * ld + col) * ts;
        uint64_t v = 0;
        if (d.mode == BM_SHUFFLED) {
            for (int j = 0; j < ts; j++) v |= (uint64_t)planes[j * TILE + x] << (8 * j);
        } else if (d.mode == BM_PLAIN) {
            for (int j = 0; j < ts; j++) v |= (uint64_t)planes[x * ts + j] << (8 * j);
        } else if (d.mode == BM_NAN) {
            v = ts == 8 ? 0x7FF8000000000000ull : 0x7FC00000ull;
        } else {
            v = load_item_bytes(ch + d.value_src, ts);
        }
        store_item(o, ts, v);
    }
    __syncthreads();
}

// One slice (t, sl) of the fast scatter; false when a bounded wait gave up (the CTA must
// leave).  Blocks of other kinds are left out and set `general`.
template <int TS>
__device__ __forceinline__ bool scatter_fast_unit(const Geom &g, const uint8_t *__restrict__ ch, const uint8_t *ch_end,
                                                  const BlockDesc *__restrict__ bd, const StreamDesc *__restrict__ sd,
                                                  const uint8_t *__restrict__ scratch, const uint8_t *scratch_end,
                                                  uint8_t *__restrict__ out, int64_t ld, int *err, int64_t t, int sl, uint8_t (*stage)[SC_PLANE],
                                                  uint64_t *bar, uint32_t &parity, int *abort_all, bool &general)
{
    const int tid = threadIdx.x;
    const int rowlen = (int)g.block[1];
    int64_t c, b;
    divmod(t, g.nblocks, c, b);
    const BlockDesc d = bd[t];
    if (d.mode != BM_SHUFFLED || d.nstreams != TS) { general = true; return true; }
    const BlockSpan sp = block_span(g, c, b);
    const int i0s = sl * SC_ITEMS, cnt = (int)min((int64_t)SC_ITEMS, g.blockn - i0s);
    if (sp.nc == 0 || i0s / rowlen >= sp.nr) return true;             // the slice holds only padding
    // per plane: its slice starts at src, 16-byte word a16 = src - shift; the bulk copy
    // takes the whole words of [a16, a16 + want) before the buffer end lim, threads copy
    // the bytes that the buffer end cuts off (zeros past it)
    auto plane = [&](int j, const uint8_t *&src, const uint8_t *&lim, int &want, int &bulk) {
        const StreamDesc q = sd[t * 8 + j];
        src = nullptr; lim = nullptr;
        if (q.kind == SK_RAW) { src = ch + q.src + i0s; lim = ch_end; }
        else if (q.kind == SK_LZ4) { src = scratch + t * g.blocksize + (int64_t)j * d.neblock + i0s; lim = scratch_end; }
        want = bulk = 0;
        if (src) {
            const uint8_t *a16 = src - (reinterpret_cast<uintptr_t>(src) & 15);
            want = ((int)(src - a16) + cnt + 15) & ~15;
            bulk = (int)min((int64_t)want, (lim - a16) & ~int64_t(15));
        }
        return q;
    };
    if (tid == 0) {
        uint32_t tx = 0;
#pragma unroll
        for (int j = 0; j < TS; j++) {
            const uint8_t *src, *lim;
            int want, bulk;
            plane(j, src, lim, want, bulk);
            tx += (uint32_t)bulk;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // earlier reads of stage precede the copies
        tc::mbar_arrive_expect_tx(bar, tx);
#pragma unroll
        for (int j = 0; j < TS; j++) {
            const uint8_t *src, *lim;
            int want, bulk;
            plane(j, src, lim, want, bulk);
            if (bulk > 0) bulk_g2s(stage[j], src - (reinterpret_cast<uintptr_t>(src) & 15), (uint32_t)bulk, bar);
        }
    }
    int code[TS];                                  // 0..15: the plane's shift in stage; 256 + v: a run of byte v
#pragma unroll
    for (int j = 0; j < TS; j++) {
        const uint8_t *src, *lim;
        int want, bulk;
        const StreamDesc q = plane(j, src, lim, want, bulk);
        code[j] = src ? (int)(reinterpret_cast<uintptr_t>(src) & 15) : 256 + (q.kind == SK_RUN ? (q.len & 255) : 0);
        if (bulk < want) {
            const uint8_t *a16 = src - code[j];
            for (int x = bulk + tid; x < want; x += blockDim.x) stage[j][x] = a16 + x < lim ? __ldg(a16 + x) : (uint8_t)0;
        }
    }
    const bool ok = sc_wait(bar, parity);
    parity ^= 1;
    if (!ok) *abort_all = 1;
    __syncthreads();
    if (*abort_all) {                              // the copies did not complete: report, wait once more, leave
        if (tid == 0) {
            dev_fail(err, DE_WAIT);
            sc_wait(bar, parity ^ 1);
        }
        return false;
    }
    uint8_t *const obase = out + (sp.row0 * ld + sp.col0) * TS;
    const int nr = sp.nr, nc = sp.nc;
    if (!geom_quads(g)) {
        // quads as two pairs, each in one row, or (rows of an odd width) item by item
        const bool pairs = rowlen % 2 == 0;
        const int step = (int)blockDim.x * 4, step_r = step / rowlen, step_c = step - step_r * rowlen;
        int r = (i0s + tid * 4) / rowlen, cc = i0s + tid * 4 - r * rowlen;
        for (int qd = tid; qd * 4 < cnt; qd += blockDim.x, r += step_r, cc += step_c) {
            if (cc >= rowlen) { cc -= rowlen; r++; }
            uint32_t w[TS];
#pragma unroll
            for (int j = 0; j < TS; j++) {
                if (code[j] >= 256) { w[j] = (uint32_t)(code[j] - 256) * 0x01010101u; continue; }
                const uint32_t *pw = reinterpret_cast<const uint32_t *>(stage[j]);
                const int byte = code[j] + qd * 4, wi = byte >> 2;
                w[j] = __funnelshift_r(pw[wi], pw[wi + 1], (byte & 3) * 8);
            }
            uint32_t v[4], h[4];
            transpose4x4(w[0], w[1], w[2], w[3], v[0], v[1], v[2], v[3]);
            if constexpr (TS == 8) transpose4x4(w[4], w[5], w[6], w[7], h[0], h[1], h[2], h[3]);
            int rr = r, c2 = cc;
            if (!pairs) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (u && ++c2 >= rowlen) { c2 = 0; rr++; }
                    if (qd * 4 + u >= cnt || rr >= nr || c2 >= nc) continue;
                    uint8_t *o = obase + ((int64_t)rr * ld + c2) * TS;
                    if constexpr (TS == 8) *reinterpret_cast<uint2 *>(o) = make_uint2(v[u], h[u]);
                    else *reinterpret_cast<uint32_t *>(o) = v[u];
                }
                continue;
            }
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
                if (u) {
                    c2 += 2;
                    if (c2 >= rowlen) { c2 = 0; rr++; }
                    if (qd * 4 + 2 >= cnt) break;
                }
                if (rr >= nr || c2 >= nc) continue;                       // padding items
                uint8_t *o = obase + ((int64_t)rr * ld + c2) * TS;
                const bool both = c2 + 1 < nc;
                if constexpr (TS == 8) {
                    if (both && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
                        *reinterpret_cast<uint4 *>(o) = make_uint4(v[u], h[u], v[u + 1], h[u + 1]);
                    } else {
                        *reinterpret_cast<uint2 *>(o) = make_uint2(v[u], h[u]);
                        if (both) *reinterpret_cast<uint2 *>(o + 8) = make_uint2(v[u + 1], h[u + 1]);
                    }
                } else {
                    if (both && (reinterpret_cast<uintptr_t>(o) & 7) == 0) {
                        *reinterpret_cast<uint2 *>(o) = make_uint2(v[u], v[u + 1]);
                    } else {
                        *reinterpret_cast<uint32_t *>(o) = v[u];
                        if (both) *reinterpret_cast<uint32_t *>(o + 4) = v[u + 1];
                    }
                }
            }
        }
        __syncthreads();                           // stage is read before the next slice's copies
        return true;
    }
    // (row, column) of each thread's quad, advanced by a fixed step per iteration (one
    // division per slice instead of one per quad)
    const int step = (int)blockDim.x * 4;
    const int step_r = step / rowlen, step_c = step - step_r * rowlen;
    int r = (i0s + tid * 4) / rowlen, cc = i0s + tid * 4 - r * rowlen;
    for (int qd = tid; qd < cnt / 4; qd += blockDim.x, r += step_r, cc += step_c) {
        if (cc >= rowlen) { cc -= rowlen; r++; }
        if (r >= nr || cc >= nc) continue;                                // padding items
        uint32_t w[TS];
#pragma unroll
        for (int j = 0; j < TS; j++) {
            if (code[j] >= 256) { w[j] = (uint32_t)(code[j] - 256) * 0x01010101u; continue; }
            const uint32_t *pw = reinterpret_cast<const uint32_t *>(stage[j]);
            const int byte = code[j] + qd * 4, wi = byte >> 2, sh = (byte & 3) * 8;
            w[j] = sh ? __funnelshift_r(pw[wi], pw[wi + 1], sh) : pw[wi];
        }
        uint8_t *o = obase + ((int64_t)r * ld + cc) * TS;
        uint32_t v[4];
        transpose4x4(w[0], w[1], w[2], w[3], v[0], v[1], v[2], v[3]);
        const bool whole = cc + 4 <= nc;
        const bool o16a = (reinterpret_cast<uintptr_t>(o) & 15) == 0;
        if constexpr (TS == 8) {
            uint32_t h[4];
            transpose4x4(w[4], w[5], w[6], w[7], h[0], h[1], h[2], h[3]);
            if (whole && o16a) {
                uint4 *o16 = reinterpret_cast<uint4 *>(o);
                o16[0] = make_uint4(v[0], h[0], v[1], h[1]);
                o16[1] = make_uint4(v[2], h[2], v[3], h[3]);
            } else {
                uint64_t *o8 = reinterpret_cast<uint64_t *>(o);
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (cc + u < nc) o8[u] = ((uint64_t)h[u] << 32) | v[u];
            }
        } else {
            if (whole && o16a) {
                *reinterpret_cast<uint4 *>(o) = make_uint4(v[0], v[1], v[2], v[3]);
            } else {
                uint32_t *o4 = reinterpret_cast<uint32_t *>(o);
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (cc + u < nc) o4[u] = v[u];
            }
        }
    }
    __syncthreads();                               // stage is read before the next slice's copies
    return true;
}

// D2 general path over the blocks that the fast one does not take: those that are not shuffled in
// fast_streams streams, *ngeneral of them as counted by the parse; every block where fast_streams is 0.
__device__ __forceinline__ void scatter_general(const Geom &g, int fast_streams, const int *ngeneral, const uint8_t *__restrict__ ch,
                                                const BlockDesc *__restrict__ bd, const StreamDesc *__restrict__ sd,
                                                const uint8_t *__restrict__ scratch, uint8_t *__restrict__ out, int64_t ld,
                                                uint8_t *planes)
{
    if (fast_streams && !__ldg(ngeneral)) return;
    const int64_t tpb = (g.blockn + TILE - 1) / TILE;
    const int64_t nwork = g.nchunks * g.nblocks * tpb;
    // Up to 32 tiles are looked at together, a lane each, the same in every warp.  The groups are an
    // even division of a CTA's share, for where the fast path took none.
    const int64_t share = (nwork + gridDim.x - 1) / gridDim.x, rounds = (share + 31) / 32;
    const int group = (int)((share + rounds - 1) / rounds);
    const int lane = threadIdx.x & 31;
    for (int64_t w0 = (int64_t)blockIdx.x * group; w0 < nwork; w0 += (int64_t)gridDim.x * group) {
        int64_t t = 0, i0 = 0;
        bool mine = lane < group && w0 + lane < nwork;
        if (mine) {
            divmod(w0 + lane, tpb, t, i0);
            mine = !(bd[t].mode == BM_SHUFFLED && bd[t].nstreams == fast_streams);
        }
        for (unsigned m = __ballot_sync(FULLMASK, mine); m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            scatter_tile(g, ch, bd, sd, scratch, out, ld, __shfl_sync(FULLMASK, t, l), __shfl_sync(FULLMASK, i0, l) * TILE,
                         planes);
        }
    }
}
// (Not inlined into the fast kernel, whose registers it would make spill.  By tiles rather than the fast
// kernel's slices: 200 x 200 float64 stored as they are, in blocks of 100 x 200: 0.070 ms inlined and by
// slices, 0.019 now, 0.027 by two launches.)
__device__ __noinline__ void scatter_general_call(const Geom &g, int fast_streams, const int *ngeneral, const uint8_t *ch,
                                                  const BlockDesc *bd, const StreamDesc *sd, const uint8_t *scratch,
                                                  uint8_t *out, int64_t ld, uint8_t *planes)
{
    scatter_general(g, fast_streams, ngeneral, ch, bd, sd, scratch, out, ld, planes);
}

template <int TS, bool ALL>
__global__ void __launch_bounds__(256, 6) k_scatter_fast(const __grid_constant__ Geom g, const uint8_t *__restrict__ ch,
                                                      const uint8_t *ch_end, const BlockDesc *__restrict__ bd,
                                                      const StreamDesc *__restrict__ sd,
                                                      const uint8_t *__restrict__ scratch, const uint8_t *scratch_end,
                                                      uint8_t *__restrict__ out, int64_t ld, int *err, const int *ngeneral)
{
    __shared__ __align__(128) uint8_t stage[TS][SC_PLANE];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_all;
    const int tid = threadIdx.x;
    if (tid == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
        abort_all = 0;
    }
    __syncthreads();
    const int64_t nbl = g.nchunks * g.nblocks;
    const int64_t nsl = (g.blockn + SC_ITEMS - 1) / SC_ITEMS;
    uint32_t parity = 0;
    bool general = false;
    for (int64_t u = blockIdx.x; u < nbl * nsl; u += gridDim.x) {
        int64_t t, s64;
        divmod(u, nsl, t, s64);
        const int sl = (int)s64;
        if (!scatter_fast_unit<TS>(g, ch, ch_end, bd, sd, scratch, scratch_end, out, ld, err, t, sl,
                                   stage, &bar, parity, &abort_all, general))
            return;
    }
    // the blocks of other kinds (no bulk copy follows: the stage is free)
    if (ALL && __ldg(ngeneral)) scatter_general_call(g, TS, ngeneral, ch, bd, sd, scratch, out, ld, stage[0]);
}

__global__ void __launch_bounds__(256, 8) k_scatter(const __grid_constant__ Geom g, int fast_streams, const uint8_t *__restrict__ ch,
                                                 const BlockDesc *__restrict__ bd, const StreamDesc *__restrict__ sd,
                                                 const uint8_t *__restrict__ scratch, uint8_t *__restrict__ out, int64_t ld,
                                                 const int *ngeneral)
{
    __shared__ __align__(16) uint8_t planes[8 * TILE];
    scatter_general(g, fast_streams, ngeneral, ch, bd, sd, scratch, out, ld, planes);
}

// ============================================================================ encode
// E1 fast path: shuffle on, items of 4 or 8 bytes (zero for the items in chunk or array
// padding).  Block rows of whole groups of 4 items: each thread reads 4 consecutive items of a
// row and writes one 4-byte word into each byte plane of the image.  Other blocks, whose planes
// may start at any byte: one item per thread, a byte into each plane, the bytes of a warp
// next to each other (5000 x 6000 float32 in blocks of 125 x 150: 0.13 ms, 0.29 by the
// general path).  A few large blocks go in slices, which spread over the SMs (three results of
// 1000 x 1001 float64 of a batch, each one block: 1.10 ms by a CTA a block, now 0.03).
template <int TS, bool QUADS>
__device__ __forceinline__ void gather_fast_block(const Geom &g, const uint8_t *__restrict__ in, int64_t ld,
                                                  uint8_t *__restrict__ img, int64_t t, int i0s, int cnt, int tid, int nt)
{
    int64_t c, b;
    divmod(t, g.nblocks, c, b);
    const BlockSpan sp = block_span(g, c, b);
    uint8_t *blk = img + t * g.blocksize;
    if constexpr (!QUADS) {
        const int rowlen = (int)g.block[1], step = nt, step_r = step / rowlen, step_c = step - step_r * rowlen;
        int r = (i0s + tid) / rowlen, cc = i0s + tid - r * rowlen;
        for (int i = i0s + tid; i < i0s + cnt; i += step, r += step_r, cc += step_c) {
            if (cc >= rowlen) { cc -= rowlen; r++; }
            uint64_t x = 0;
            if (r < sp.nr && cc < sp.nc) {
                const uint8_t *src = in + ((sp.row0 + r) * ld + sp.col0 + cc) * TS;
                x = TS == 8 ? __ldg(reinterpret_cast<const uint64_t *>(src)) : __ldg(reinterpret_cast<const uint32_t *>(src));
            }
#pragma unroll
            for (int j = 0; j < TS; j++) blk[(int64_t)j * g.blockn + i] = (uint8_t)(x >> (8 * j));
        }
        return;
    }
    const int qpr = (int)(g.block[1] / 4), q0 = i0s / 4, nq = cnt / 4;
    // (row, quad column) of each thread's quad, advanced by a fixed step per iteration
    const int step_r = nt / qpr, step_q = nt - step_r * qpr;
    int r = (q0 + tid) / qpr, q = q0 + tid - r * qpr;
    for (int qd = q0 + tid; qd < q0 + nq; qd += nt, r += step_r, q += step_q) {
        if (q >= qpr) { q -= qpr; r++; }
        const int i0 = qd * 4, cc = q * 4;
        const uint8_t *src = in + ((sp.row0 + r) * ld + sp.col0 + cc) * TS;
        uint64_t x[4] = {0, 0, 0, 0};                 // padding items are zero, as in Caterva
        if (r < sp.nr && cc + 4 <= sp.nc) {
            if constexpr (TS == 8) {
                const uint64_t *s8 = reinterpret_cast<const uint64_t *>(src);
#pragma unroll
                for (int u = 0; u < 4; u++) x[u] = __ldg(s8 + u);
            } else {
                const uint32_t *s4 = reinterpret_cast<const uint32_t *>(src);
#pragma unroll
                for (int u = 0; u < 4; u++) x[u] = __ldg(s4 + u);
            }
        } else if (r < sp.nr) {
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (cc + u < sp.nc) x[u] = TS == 8 ? __ldg(reinterpret_cast<const uint64_t *>(src) + u)
                                                   : __ldg(reinterpret_cast<const uint32_t *>(src) + u);
        }
        uint32_t o[TS];
        transpose4x4((uint32_t)x[0], (uint32_t)x[1], (uint32_t)x[2], (uint32_t)x[3], o[0], o[1], o[2], o[3]);
        if constexpr (TS == 8)
            transpose4x4((uint32_t)(x[0] >> 32), (uint32_t)(x[1] >> 32), (uint32_t)(x[2] >> 32), (uint32_t)(x[3] >> 32),
                         o[4], o[5], o[6], o[7]);
#pragma unroll
        for (int j = 0; j < TS; j++) *reinterpret_cast<uint32_t *>(blk + (int64_t)j * g.blockn + i0) = o[j];
    }
}

// Items of a gather slice: a block's slices are of one size, about GA_ITEMS each unless `nbl` blocks in
// fewer fill the `slots` of one wave (600 blocks of 100 x 200 float32: 0.030 ms whole, 0.036 in halves).
static int gather_slice(const Geom &g, int64_t nbl, int64_t slots)
{
    const int64_t nsl = std::min(ceil_div(g.blockn, GA_ITEMS), std::max<int64_t>(slots / std::max<int64_t>(nbl, 1), 1));
    return (int)round_up(ceil_div(g.blockn, nsl), 4);
}
// Threads that take a block: a power of two, a warp at least, a CTA at most.  Blocks of few items share
// a CTA, which else would be all latency.
static int gather_threads(const Geom &g)
{
    const int64_t n = geom_quads(g) ? g.blockn / 4 : g.blockn;
    int nt = 32;
    while (nt < 256 && nt < n) nt *= 2;
    return nt;
}
// (A kernel for each of the two kinds of blocks, as both in one cost registers.  250,000 blocks of 8 x 8
// float32: 0.73 ms with a CTA a block and one kernel for both, now 0.10; float64 0.80 and 0.11.)
template <int TS, bool QUADS>
__global__ void __launch_bounds__(256, !QUADS ? 4 : TS == 8 ? 6 : 8) k_gather_fast(Geom g, const uint8_t *__restrict__ in, int64_t ld,
                                                                               uint8_t *__restrict__ img, int slice, int nt)
{
    const int64_t nsl = (g.blockn + slice - 1) / slice, nu = g.nchunks * g.nblocks * nsl;
    const int per = 256 / nt, tid = threadIdx.x & (nt - 1);
    for (int64_t u = (int64_t)blockIdx.x * per + threadIdx.x / nt; u < nu; u += (int64_t)gridDim.x * per) {
        int64_t t = u, sl = 0;
        if (nsl > 1) divmod(u, nsl, t, sl);
        gather_fast_block<TS, QUADS>(g, in, ld, img, t, (int)sl * slice, (int)min((int64_t)slice, g.blockn - sl * slice), tid, nt);
    }
}

// E1 general path: dense -> byte-plane image (shuffled: plane j holds byte j of every
// item; plain: items back to back).  Padding items are zero, as in Caterva.
__device__ __forceinline__ void gather_tile(const Geom &g, const uint8_t *__restrict__ in, int64_t ld, bool shuffle,
                                            uint8_t *__restrict__ img, int64_t t, int64_t i0, uint8_t *planes)
{
    const int ts = g.itemsize;
    const int cnt = (int)min((int64_t)TILE, g.blockn - i0);
    const int64_t c = t / g.nblocks, b = t - c * g.nblocks;
    for (int x = threadIdx.x; x < cnt; x += blockDim.x) {
        int64_t row, col;
        uint64_t v = 0;
        if (item_pos(g, c, b, i0 + x, row, col)) v = load_item(in + (row * ld + col) * ts, ts);
        if (shuffle) {
            for (int j = 0; j < ts; j++) planes[j * TILE + x] = (uint8_t)(v >> (8 * j));
        } else {
            for (int j = 0; j < ts; j++) planes[x * ts + j] = (uint8_t)(v >> (8 * j));
        }
    }
    __syncthreads();
    uint8_t *blk = img + t * g.blocksize;
    if (shuffle) {
        for (int j = 0; j < ts; j++) {
            uint8_t *dst = blk + (int64_t)j * g.blockn + i0;
            for (int x = threadIdx.x; x < cnt; x += blockDim.x) dst[x] = planes[j * TILE + x];
        }
    } else {
        uint8_t *dst = blk + i0 * ts;
        for (int x = threadIdx.x; x < cnt * ts; x += blockDim.x) dst[x] = planes[x];
    }
    __syncthreads();
}

__global__ void __launch_bounds__(256) k_gather(Geom g, const uint8_t *__restrict__ in, int64_t ld,
                                                bool shuffle, uint8_t *__restrict__ img)
{
    __shared__ __align__(16) uint8_t planes[8 * TILE];
    const int64_t tpb = (g.blockn + TILE - 1) / TILE;
    const int64_t nwork = g.nchunks * g.nblocks * tpb;
    for (int64_t w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int64_t t = w / tpb, i0 = (w - t * tpb) * TILE;
        gather_tile(g, in, ld, shuffle, img, t, i0, planes);
    }
}

// ---------------------------------------------------------------- LZ4 encoder (warp)
// Unaligned little-endian reads from a source whose stream base is 4-byte aligned: two
// aligned word loads and a funnel shift.  Callers only read where p + 7 stays inside the
// stream (hash positions are at most n - 12; match candidates lie before them).
__device__ __forceinline__ uint32_t ld4u(const uint8_t *p)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~uintptr_t(3));
    return __funnelshift_r(__ldg(w), __ldg(w + 1), (uint32_t)(a & 3) * 8);
}

// Position offset of the t-th probe of a search, relative to its start: the step is
// 1 for probes 0..64 and grows by one every 64 probes after that.  (Below 2^32 for every
// stream: a search stops at the first probe past the stream, less than 2^31 bytes long.)
__device__ __forceinline__ uint32_t probe_offset(uint32_t t)
{
    if (t == 0) return 0;
    const uint32_t m = 62 + t, q = m >> 6, r = m - (q << 6);
    return 1 + 32 * (q * (q - 1)) + q * (r + 1);
}

// Shared-memory window over one stream for the encoder: positions [lo, hi) sit at
// r[x & (cap - 1)], the first EMIRROR ring bytes mirrored past its end so that reads of up to
// 32 bytes never wrap.  The window follows the parse position; reads outside it (far search
// probes, old match candidates) go to global memory.  Without it the candidate reads of
// low-entropy streams, spread over the last few KiB, mostly miss L1.
// The liblz4-identical encoder's warps (one per CTA) hold 16 KiB of table each; with a 2 KiB
// window eleven of them fit an SM (f32 blocks of 125 x 150, 5000 x 6000 product: 0.98 ms; ten
// with 4 KiB windows 1.26 ms, twelve with 1 KiB 0.91 ms there but 1.02x the time on 64 KiB
// streams, whose candidates then come from global memory).
constexpr int XCTAS = 11, XRING = 2048;
constexpr int ERING = 4096, ESEG = 512, ELOOK = 256, EMIRROR = 32;
constexpr int EPEER = 128 + 64;                    // words of the lanes-by-hash masks of warp_lz4_compress

struct EncSrc {
    const uint8_t *g;   // the stream in global memory
    uint8_t *r;         // cap + EMIRROR bytes, 16-byte aligned
    int cap;            // ring size, a power of two
    int lo, hi, n;
};

__device__ __forceinline__ uint32_t es_byte(const EncSrc &s, int x)
{
    return (x >= s.lo && x < s.hi) ? (uint32_t)s.r[x & (s.cap - 1)] : (uint32_t)__ldg(s.g + x);
}

__device__ __forceinline__ uint32_t es_rd32(const EncSrc &s, int x)
{
    if (x >= s.lo && x + 4 <= s.hi) {
        const int o = x & (s.cap - 1);
        const uint32_t *w = reinterpret_cast<const uint32_t *>(s.r) + (o >> 2);
        return __funnelshift_r(w[0], w[1], (uint32_t)(o & 3) * 8);
    }
    return ld4u(s.g + x);
}

// liblz4's hash of the 4 (byU16 tables) or 5 (byU32 tables) bytes at p.
__device__ __forceinline__ uint32_t es_hash(const EncSrc &s, int p, bool small)
{
    if (small) return (es_rd32(s, p) * 2654435761u) >> (32 - 13);
    const uint64_t v = (uint64_t)es_rd32(s, p) | ((uint64_t)es_byte(s, p + 4) << 32);
    return (uint32_t)(((v << 24) * 889523592379ull) >> (64 - 12));
}

// Extends the window up to position `want` (warp-uniform) in ESEG pieces; a piece's loads are
// all issued before its stores.
__device__ __forceinline__ void es_fill(EncSrc &s, int want)
{
    const int lane = threadIdx.x & 31;
    while (s.hi < s.n && s.hi < want) {
        const int base = s.hi, cnt = min(ESEG, s.n - base);
        uint32_t v[ESEG / 128];
#pragma unroll
        for (int i = 0; i < ESEG / 128; i++) {
            const int x = lane * 4 + i * 128;
            v[i] = 0;
            if (base + x + 8 <= s.n) {
                v[i] = ld4u(s.g + base + x);
            } else {
                for (int k = 0; k < 4; k++)
                    if (base + x + k < s.n) v[i] |= (uint32_t)__ldg(s.g + base + x + k) << (8 * k);
            }
        }
        __syncwarp();                                    // reads of the slots being replaced are done
#pragma unroll
        for (int i = 0; i < ESEG / 128; i++) {
            const int x = lane * 4 + i * 128, o = (base + x) & (s.cap - 1);
            if (x >= cnt) continue;
            *reinterpret_cast<uint32_t *>(s.r + o) = v[i];
            if (o < EMIRROR) *reinterpret_cast<uint32_t *>(s.r + s.cap + o) = v[i];
        }
        s.hi = base + cnt;
        s.lo = max(s.lo, base + ESEG - s.cap);
        __syncwarp();
    }
}

// Shared-memory word through a 32-bit shared-window address.
__device__ __forceinline__ uint32_t lds32(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
// liblz4's hash of the 4 bytes v4 at a position (byU16 tables) or of those and the fifth
// byte b4 (byU32 tables).
template <bool SMALL>
__device__ __forceinline__ uint32_t lz_hash_v(uint32_t v4, uint32_t b4)
{
    if (SMALL) return (v4 * 2654435761u) >> (32 - 13);
    const uint64_t v = (uint64_t)v4 | ((uint64_t)b4 << 32);
    return (uint32_t)(((v << 24) * 889523592379ull) >> (64 - 12));
}

// Warp-cooperative LZ4 block compressor in limited-output mode with capacity `cap`.
// Returns the compressed size, or 0 when it does not fit; *need_out receives the
// smallest capacity for which it would have fit.  All lanes must call it; every
// position, candidate and output offset below is warp-uniform.  SMALL selects liblz4's
// byU16 table (inputs below 64 KiB + 11 bytes: 13-bit hash of 4 bytes) over its byU32
// table (12-bit hash of 5 bytes, 65535-byte distance limit).
//
// liblz4's parse is one serial chain (what a position finds depends on which earlier positions
// were inserted), and its latency bounds the kernel: a launch has far fewer compressible streams
// than the SMs have warp slots.  So 32 consecutive positions, one per lane, are handled at once:
// the bytes, the hash, the table's candidate as of the window's start, whether it matches, how
// far forwards (to 16 bytes) and backwards (to 4), and from that the chain of matches from every
// lane by pointer doubling over the lanes.  This chain is liblz4's as long as no tested lane has
// an inserted lane of the same hash before it in the window (that lane would be its candidate):
// one ballot finds the first step where it has.  The steps before it are written together, the
// step itself is walked exactly (its candidates are the inserted lanes, a bit mask, else the
// table's), and the chain goes on from its end.  Steps with long matches or literal runs and
// long backward extensions are walked too, with warp-wide loops.  Inserted lanes enter the table
// at the window's end.  Searches past their 64th probe, whose step grows, take 32 probes per step
// at the probes' own positions.
// Measured against one scalar step per sequence: sign/exponent planes of gaussian float64 values, a
// stream by itself, 64 KiB 4.57 -> 3.19 ms (3,060 cycles for 32 positions; five-byte hashes, of 256
// KiB, 2,070); k_lz4_encode on the 5000 x 6000 float32 product 4.75 -> 0.98 ms, on the 4056 x 3712
// float64 one 2.30 -> 0.88 ms.  Where every match is long and follows another, a window holds one
// step, and the scalar step was the faster: (i + j) / 50 rounded down as float64, 4000 x 3000 in
// blocks of 500 x 500, 4.8 -> 7.0 ms, counting 5.4 -> 6.9.  A form of the function for such streams,
// chosen after 2 KiB by what they had compressed to, lost more on streams of a few KiB (1.7 -> 4.3
// ms) than it gave there, and leaving out the chain where the first lane has a long match cost the
// other streams 3 to 5%.
template <bool SMALL>
__device__ __forceinline__ int warp_lz4_compress(const uint8_t *__restrict__ src, int n, uint8_t *__restrict__ dst,
                                                 int cap, uint32_t *tab, uint32_t *bm, uint8_t *ring, int rcap,
                                                 int *need_out)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint16_t *tab16 = reinterpret_cast<uint16_t *>(tab);
    for (int i = lane; i < 1024; i += 32) reinterpret_cast<uint4 *>(tab)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int i = lane; i < EPEER; i += 32) bm[i] = 0u;
    EncSrc s;
    s.g = src; s.r = ring; s.cap = rcap; s.lo = 0; s.hi = 0; s.n = n;
    const uint32_t *rw = reinterpret_cast<const uint32_t *>(ring);
    const int wmask = (rcap >> 2) - 1;
    __syncwarp();
    int need = 0, op = 0, anchor = 0;
    const int mfl1 = n - 12 + 1, mlimit = n - 5;
#define TGET(h) (SMALL ? (uint32_t)tab16[h] : tab[h])
#define TPUT(h, v) do { if (SMALL) tab16[h] = (uint16_t)(v); else tab[h] = (uint32_t)(v); } while (0)
    // The sequence that ends with the match of position pr at distance d: L bytes are known to
    // match (`longer`: perhaps more), `back` bytes before pr match too (`more_back`: perhaps
    // more).  Sets anchor to its end; false when the output does not fit.
    auto sequence = [&](int pr, int d, int L, bool longer, int back, bool more_back) -> bool {
        const int lits = pr - anchor, lim = mlimit - pr;
        back = min(back, lits);
        if (L >= lim) { L = lim; longer = false; }
        if (more_back) {
            for (;;) {
                const int k = back + lane + 1;
                const bool ok = k <= lits && pr - d - k >= 0 && es_byte(s, pr - k) == es_byte(s, pr - d - k);
                const unsigned badm = __ballot_sync(FULLMASK, !ok);
                const int ext = badm ? __ffs((int)badm) - 1 : 32;
                back += ext;
                if (ext < 32) break;
            }
        }
        if (longer) {
            for (;;) {
                const int a = pr + L + lane;
                if (pr + L + 64 > s.hi) es_fill(s, pr + L + ELOOK);
                const bool eq = a < mlimit && es_byte(s, a) == es_byte(s, a - d);
                const unsigned ne = __ballot_sync(FULLMASK, !eq);
                const int cnum = ne ? __ffs((int)ne) - 1 : 32;
                L += cnum;
                if (cnum < 32) break;
            }
        }
        const int lit = lits - back, mc = L + back - 4;
        anchor = pr + L;
        if (lit < 15 && mc < 15) {
            need = max(need, op + lit + 9);
            if (need > cap) return false;
            if (lane < lit + 3)
                dst[op + lane] = (uint8_t)(lane == 0 ? (uint32_t)((lit << 4) | mc)
                                                     : lane <= lit ? es_byte(s, pr - lits + lane - 1)
                                                                   : (uint32_t)d >> (8 * (lane - lit - 1)));
            op += lit + 3;
            return true;
        }
        const int eb = (lit >= 15 ? (lit - 15) / 255 + 1 : 0), mb = (mc >= 15 ? (mc - 15) / 255 + 1 : 0);
        const int o = op + 1 + eb;                              // the literals' offset
        need = max(need, max(op + lit + 9 + lit / 255, o + lit + 8 + (mc + 240) / 255));
        if (need > cap) return false;
        if (lane == 0) dst[op] = (uint8_t)((min(lit, 15) << 4) | min(mc, 15));
        for (int x = lane; x < eb; x += 32) dst[op + 1 + x] = (uint8_t)(x < eb - 1 ? 255 : (lit - 15) % 255);
        for (int x = lane; x < lit; x += 32) dst[o + x] = (uint8_t)es_byte(s, pr - lits + x);
        if (lane < 2) dst[o + lit + lane] = (uint8_t)(d >> (8 * lane));
        for (int x = lane; x < mb; x += 32) dst[o + lit + 2 + x] = (uint8_t)(x < mb - 1 ? 255 : (mc - 15) % 255);
        op = o + lit + 2 + mb;
        return true;
    };
    if (n >= 13) {
        es_fill(s, ELOOK);
        if (lane == 0) TPUT(es_hash(s, 0, SMALL), 0);
        __syncwarp();
        // `hot`: ip follows a match (liblz4 inserts ip - 2, then tests ip itself); else a search
        // is under way whose t-th probe is p0 + probe_offset(t), t0 probes done.
        bool hot = false;
        int ip = 0, p0 = 1, t0 = 0;
        const uint32_t head = ld4u(src);                        // the bytes an empty bucket's candidate 0 has
        for (;;) {
            if (hot && ip >= mfl1) break;
            if (!hot && t0 > 33) {
                // ---- probes with a growing step (the step is 1 for the first 66 probes)
                bool end = false;
                int pr = 0, c = 0;
                for (;;) {
                    es_fill(s, (int)min((uint32_t)p0 + probe_offset((uint32_t)t0), (uint32_t)n) + ELOOK);
                    const uint32_t p = (uint32_t)p0 + probe_offset((uint32_t)(t0 + lane)),
                                   pn = (uint32_t)p0 + probe_offset((uint32_t)(t0 + lane + 1));
                    const bool valid = pn <= (uint32_t)mfl1;
                    const uint32_t v = valid ? es_rd32(s, (int)p) : 0u;
                    const uint32_t h = !valid ? 0x80000000u | (uint32_t)lane
                                              : lz_hash_v<SMALL>(v, SMALL ? 0u : es_byte(s, (int)p + 4));
                    const uint32_t ctab = valid ? TGET(h) : 0u;
                    bool m = valid && (SMALL || ctab + 65535u >= p) && (ctab ? es_rd32(s, (int)ctab) : head) == v;
                    const unsigned em = __ballot_sync(FULLMASK, !valid);
                    const int E = em ? __ffs((int)em) - 1 : 32;
                    unsigned mm = __ballot_sync(FULLMASK, m);
                    int W = mm ? __ffs((int)mm) - 1 : 32;
                    // The probes up to the first match enter the table.  Two of them with one hash
                    // (seen when a lane reads back another's position) change what the later
                    // one finds: then the step is taken again with the lanes' candidates among
                    // the probes themselves.
                    const bool put = lane <= min(W, E - 1);
                    __syncwarp();
                    if (put) TPUT(h, p);
                    __syncwarp();
                    const bool clash = put && TGET(h) != (SMALL ? p & 0xffffu : p);
                    uint32_t cand = ctab;
                    if (__any_sync(FULLMASK, clash)) {
                        const unsigned peers = __match_any_sync(FULLMASK, h), lower = peers & lt;
                        const int cl = lower ? 31 - __clz((int)lower) : lane;
                        const uint32_t pl = __shfl_sync(FULLMASK, p, cl), vl = __shfl_sync(FULLMASK, v, cl);
                        if (lower) {
                            cand = pl;
                            m = valid && (SMALL || cand + 65535u >= p) && vl == v;
                        }
                        mm = __ballot_sync(FULLMASK, m);
                        W = mm ? __ffs((int)mm) - 1 : 32;
                        const int lastw = min(W, E - 1);
                        if (put) TPUT(h, ctab);
                        __syncwarp();
                        const unsigned upto = (lastw >= 31) ? FULLMASK : ((2u << lastw) - 1u);
                        if (lane <= lastw && !(peers & ~lt & ~(1u << lane) & upto)) TPUT(h, p);
                        __syncwarp();
                    }
                    if (W < E) {
                        pr = (int)__shfl_sync(FULLMASK, p, W);
                        c = (int)__shfl_sync(FULLMASK, cand, W);
                        break;
                    }
                    if (E < 32) { end = true; break; }
                    t0 += 32;
                }
                if (end) break;
                if (!sequence(pr, pr - c, 4, true, 0, true)) { *need_out = need; return 0; }
                ip = anchor;
                hot = true;
                continue;
            }
            // ---- window of 32 consecutive positions
            const int w0 = hot ? ip - 2 : p0 + t0;
            if (w0 + 64 > s.hi) es_fill(s, w0 + ELOOK);
            const int p = w0 + lane;
            const bool valid = p < mfl1;
            uint32_t prev, v, n0, n1, n2;                       // bytes p-4 .., p .., p+4 .., p+8 .., p+12 ..
            {
                const uint32_t *w = rw + (((p >> 2) - 1) & wmask);
                const uint32_t sh = (uint32_t)(p & 3) * 8;
                prev = __funnelshift_r(w[0], w[1], sh);
                v = __funnelshift_r(w[1], w[2], sh);
                n0 = __funnelshift_r(w[2], w[3], sh);
                n1 = __funnelshift_r(w[3], w[4], sh);
                n2 = __funnelshift_r(w[4], w[5], sh);
            }
            const uint32_t h = lz_hash_v<SMALL>(v, n0 & 0xffu);
            const int c = valid ? (int)TGET(h) : 0;
            // lanes of the same hash: those that share its low 7 bits and those that share the
            // rest, collected in shared memory (__match_any_sync takes about 11 cycles for every
            // distinct value, 350 here; this 80)
            if (valid) {
                atomicOr(bm + (h & 127u), 1u << lane);
                atomicOr(bm + 128 + (h >> 7), 1u << lane);
            }
            __syncwarp();
            // the candidate's bytes: from the window when it (and the 4 bytes before it) are still
            // there, else from global memory; the first 4 positions only as far as the match
            bool hit_t;
            uint32_t info;                                      // match length, backward length, distance
            {
                const bool inring = c - 4 >= s.lo || s.lo == 0;
                const uintptr_t ca = reinterpret_cast<uintptr_t>(src) + (uintptr_t)(max(c, 4) - 4);
                const uint32_t *w = inring ? rw + (((c >> 2) - 1) & wmask)
                                           : reinterpret_cast<const uint32_t *>(ca & ~uintptr_t(3));
                const uint32_t sh = (inring ? (uint32_t)c & 3u : (uint32_t)(ca & 3)) * 8;
                const uint32_t w0_ = w[0], w1_ = w[1], w2_ = w[2], w3_ = w[3], w4_ = w[4], w5_ = w[5];
                const uint32_t cp = __funnelshift_r(w0_, w1_, sh), c0 = __funnelshift_r(w2_, w3_, sh),
                               c1 = __funnelshift_r(w3_, w4_, sh), c2 = __funnelshift_r(w4_, w5_, sh);
                uint32_t cv = __funnelshift_r(w1_, w2_, sh);
                const bool low = !inring && c < 4;
                if (low) cv = __funnelshift_r(cp, cv, 8 * c);
                hit_t = valid && cv == v && (SMALL || c + 65535 >= p);
                const uint32_t x0 = n0 ^ c0, x1 = n1 ^ c1, x2 = n2 ^ c2;
                const uint32_t x = x0 ? x0 : x1 ? x1 : x2;
                int len = (x0 ? 4 : x1 ? 8 : 12) + (x ? (__ffs((int)x) - 1) >> 3 : 4);
                int bk = min(__clz((int)(prev ^ cp)) >> 3, c);
                uint32_t more = (len == 16 ? 1u : 0u) | (bk == 4 ? 2u : 0u);
                if (low) { len = 4; bk = 0; more = 3u; }
                info = (uint32_t)len | (more << 5) | ((uint32_t)bk << 8) | ((uint32_t)(p - c) << 16);
            }
            const unsigned peers = valid ? bm[h & 127u] & bm[128 + (h >> 7)] : 0u;
            __syncwarp();
            if (valid) { bm[h & 127u] = 0u; bm[128 + (h >> 7)] = 0u; }
            const unsigned vmask = __ballot_sync(FULLMASK, valid), H = __ballot_sync(FULLMASK, hit_t);
            // The step from this lane by the table's candidates alone: match at lane rq (32: none
            // left), the next step at lane jq, lit literals and a match of mc + 4 bytes.  `odd`
            // steps are walked below.
            const unsigned hq = H & (FULLMASK << lane), reach = H ? FULLMASK >> __clz((int)H) : 0u;
            const int rq = hq ? __ffs((int)hq) - 1 : 32;
            const uint32_t iq = __shfl_sync(FULLMASK, info, rq & 31);
            const int Lq = (int)(iq & 31u), bq = (int)((iq >> 8) & 7u);
            const int jq = rq < 32 ? rq + Lq : 32;
            auto odd_step = [&](int lits, int lit, int mc) {
                return (iq & 32u) || ((iq & 64u) && lits > bq) || lit >= 15 || mc >= 15 || w0 + jq > mlimit;
            };
            int lit = rq - lane - min(bq, rq - lane), mc = Lq + min(bq, rq - lane) - 4;
            bool odd = odd_step(rq - lane, lit, mc);
            // Along the chain from this lane (at most 8 steps fit in a window): the lanes where a
            // step starts (m), the lanes tested (tq), the bytes written (sq)
            const int sz = rq < 32 ? 3 + lit : 0;
            unsigned m = 1u << lane, tq = (FULLMASK << lane) & (rq < 32 ? FULLMASK >> (31 - rq) : FULLMASK);
            int sq = sz;
            {
                int j = jq;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const unsigned mj = __shfl_sync(FULLMASK, m, j & 31), tj = __shfl_sync(FULLMASK, tq, j & 31);
                    const int js = __shfl_sync(FULLMASK, j | (sq << 8), j & 31);
                    if (j < 32) { m |= mj; tq |= tj; sq += js >> 8; j = js & 255; }
                }
            }
            const unsigned plt = peers & lt;                    // earlier lanes of this lane's hash
            unsigned ins = 0;                                   // inserted lanes
            int q = hot ? 2 : 0;                                // the lane tested next
            bool end = false;
            for (;;) {
                const unsigned vis = __shfl_sync(FULLMASK, m, q), tm = __shfl_sync(FULLMASK, tq, q);
                const int s0 = __shfl_sync(FULLMASK, sq, q);
                const unsigned hv = (hot ? vis : vis & ~(1u << q)) >> 2;
                const int extra = w0 + q - anchor;              // literals before the first step's lane
                int grow = 0;
                if (extra > 0) {
                    const int lits = rq - lane + extra, bk = min(bq, lits), l0 = lit;
                    if (lane == q) {
                        lit = lits - bk;
                        mc = Lq + bk - 4;
                        odd = odd_step(lits, lit, mc);
                    }
                    grow = __shfl_sync(FULLMASK, lit - l0, q);
                }
                const unsigned bit = 1u << lane, steps = vis & reach;
                const unsigned viol = __ballot_sync(FULLMASK, ((steps & bit) && odd) || ((tm & bit) && (plt & (ins | tm | hv))));
                // the steps before the first one to be walked
                unsigned below = FULLMASK;
                if (viol) below = (1u << (31 - __clz((int)(vis & (viol ^ (viol - 1)))))) - 1u;
                const unsigned ems = steps & below;
                ins |= (tm & below) | (hv & (below >> 2));
                if (ems) {
                    const int last = 31 - __clz((int)ems);
                    const int ev = __shfl_sync(FULLMASK, jq | ((sq - sz) << 8), last);
                    const int total = s0 - (ev >> 8) + grow;
                    need = max(need, op + total + 6);           // op + lit + 9 of the last one
                    if (need > cap) { *need_out = need; return 0; }
                    const int off = s0 - sq + (lane == q ? 0 : grow);
                    if (ems & bit) {
                        uint8_t *o = dst + op + off;
                        o[0] = (uint8_t)((lit << 4) | mc);
                        o[1 + lit] = (uint8_t)(iq >> 16);
                        o[2 + lit] = (uint8_t)(iq >> 24);
                    }
                    // literals: one lane each, those before the window's lanes first
                    const unsigned vle = ems & (lt | bit);
                    const int qv = 31 - __clz((int)vle);
                    const int ov = __shfl_sync(FULLMASK, off | (lit << 16), qv & 31);
                    const int x = lane - qv + (qv == q ? extra : 0);
                    if (vle && x < (ov >> 16)) dst[op + (ov & 0xffff) + 1 + x] = (uint8_t)v;
                    if (extra > 0) {
                        const int lq = __shfl_sync(FULLMASK, lit, q);
                        if (lane < min(extra, lq)) dst[op + 1 + lane] = (uint8_t)es_byte(s, anchor + lane);
                    }
                    op += total;
                    hot = true;
                    ip = anchor = w0 + (ev & 255);
                    q = ip - w0;
                    if (q > 31) break;
                }
                // ---- the step at q, walked: a lane past q is probed when all of q .. lane - 1
                // were, which inserted them
                const unsigned from = FULLMASK << q, hb = hot ? 1u << (q - 2) : 0u;
                const unsigned pm = plt & (ins | hb | from);
                const int cl0 = 31 - __clz((int)pm);
                const uint32_t vc = __shfl_sync(FULLMASK, v, cl0 & 31);
                const bool hit = pm ? vc == v : hit_t;
                const unsigned b = __ballot_sync(FULLMASK, hit) & from & vmask;
                if (!b) {
                    ins |= hb | from;
                    end = vmask != FULLMASK;
                    if (hot) p0 = w0 + q + 1;
                    hot = false;
                    t0 = w0 + 32 - p0;
                    break;
                }
                const int r = __ffs((int)b) - 1, pr = w0 + r;
                ins |= hb | (from & (FULLMASK >> (31 - r)));
                const uint32_t inf = __shfl_sync(FULLMASK, info, r);
                const unsigned pmr = __shfl_sync(FULLMASK, pm, r);
                int L, back, d;
                bool longer, more_back;
                if (pmr) {                                      // a match with lane cl of this window
                    const int cl = 31 - __clz((int)pmr);
                    d = r - cl;
                    const uint32_t ob = __shfl_sync(FULLMASK, v, (lane - d) & 31);
                    const unsigned eq = __ballot_sync(FULLMASK, lane >= d && ((v ^ ob) & 0xffu) == 0);
                    L = __ffs((int)~(eq >> r)) - 1;             // r >= 1: the shifted-in bits end the run
                    longer = r + L == 32;
                    back = __clz((int)~(eq << (32 - r)));       // at most cl: lanes below d are not equal
                    more_back = back == cl;
                } else {
                    L = (int)(inf & 31u);
                    back = (int)((inf >> 8) & 7u);
                    d = (int)(inf >> 16);
                    longer = (inf & 32u) != 0;
                    more_back = (inf & 64u) != 0;
                }
                if (!sequence(pr, d, L, longer, back, more_back && pr - anchor > back)) { *need_out = need; return 0; }
                hot = true;
                ip = anchor;
                q = ip - w0;
                if (q > 31) break;
            }
            if (((ins >> lane) & 1u) && !(peers & ins & ~lt & ~(1u << lane))) TPUT(h, p);
            __syncwarp();
            if (end) break;
        }
    }
    {
        const int last = n - anchor;
        need = max(need, op + last + 1 + (last + 255 - 15) / 255);
        if (need > cap) { *need_out = need; return 0; }
        if (last >= 15) {
            const int rem = last - 15, nff = rem / 255;
            if (lane == 0) dst[op] = 15 << 4;
            for (int x = lane; x < nff; x += 32) dst[op + 1 + x] = 255;
            if (lane == 0) dst[op + 1 + nff] = (uint8_t)(rem % 255);
            op += nff + 2;
        } else {
            if (lane == 0) dst[op] = (uint8_t)(last << 4);
            op += 1;
        }
        for (int x = lane; x < last; x += 32) dst[op + x] = (uint8_t)es_byte(s, anchor + x);
        op += last;
    }
#undef TGET
#undef TPUT
    __syncwarp();
    *need_out = need;
    return op;
}

// The k-th stream to be handed out of `total` streams, `per` per block: the last stream of every
// block first, then the one before it.  In little-endian shuffled floats the last byte planes
// (sign, exponent) compress and cost up to a hundred times what an incompressible plane costs; in
// block order the last ones would start when the other streams are done and run on alone.
// A CTA's first stream is that of its own number, the others are handed out as CTAs ask for them: the
// first streams are the long ones, and by order of arrival they go to the SMs that start first, several
// to each (256 compressible streams of 64 KiB among 2,048, parallel encoder 0.88 -> 0.51 ms, decoder
// 0.33 -> 0.25; by block order and arrival 0.79).
__device__ __forceinline__ int64_t stream_at(int64_t k, int64_t total, int per)
{
    int64_t j, b;
    divmod(k, total / per, j, b);
    return b * per + (per - 1 - j);
}

// This thread's share of whether the bytes [b, b + 64 T) of a stream of n bytes all equal `first` (T
// threads): four 16-byte words, the bytes before the stream's first whole word and after its last one
// by themselves.  Bound by the loads' requests: byte by byte the streams of a plane, which lie a block
// apart, took half as long again as those of a block (zeros of 4000 x 3000 float64 in blocks of
// 100 x 200: 0.223 and 0.263 ms in either order by bytes, 0.033 now).
template <int T>
__device__ __forceinline__ bool run_piece(const uint8_t *__restrict__ src, int n, uint8_t first, int b)
{
    const int t = threadIdx.x % T, head = min((int)(-reinterpret_cast<uintptr_t>(src) & 15), n), nv = (n - head) / 16;
    const uint4 *v = reinterpret_cast<const uint4 *>(src + head);
    const uint32_t all = first * 0x01010101u;
    uint4 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int i = b / 16 + k * T + t;
        x[k] = i < nv ? __ldg(v + i) : make_uint4(all, all, all, all);
    }
    uint32_t d = 0;
    if (b == 0 && t < head) d |= __ldg(src + t) ^ first;
    if (b == 0 && head + nv * 16 + t < n) d |= __ldg(src + head + nv * 16 + t) ^ first;
#pragma unroll
    for (int k = 0; k < 4; k++) d |= (x[k].x ^ all) | (x[k].y ^ all) | (x[k].z ^ all) | (x[k].w ^ all);
    return d == 0;
}

// E2: one warp per stream: run check, then LZ4 into the stream's slot (capacity =
// stream length; a stream that does not shrink is stored raw).
// Streams are handed out dynamically (one atomic per stream): compressible streams cost
// far more than incompressible ones, and in shuffled float data they recur at a fixed
// stride, which a static round-robin assignment would pile onto the same warps.
__global__ void __launch_bounds__(32, XCTAS) k_lz4_encode(const uint8_t *__restrict__ img, int64_t nstreams_total,
                                                    int per, int neblock, uint8_t *slots, EncStream *es,
                                                    unsigned long long *next)
{
    extern __shared__ __align__(16) uint32_t sm_tab[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *tab = sm_tab + warp * (4096 + EPEER + (XRING + EMIRROR) / 4);
    uint32_t *bm = tab + 4096;
    uint8_t *ring = reinterpret_cast<uint8_t *>(bm + EPEER);
    for (bool start = true;; start = false) {
        unsigned long long got = blockIdx.x;
        if (lane == 0 && !start) got = gridDim.x + atomicAdd(next, 1ull);
        const int64_t k = (int64_t)__shfl_sync(FULLMASK, got, 0);
        if (k >= nstreams_total) break;
        const int64_t sid = stream_at(k, nstreams_total, per);
        const uint8_t *src = img + sid * neblock;
        const uint8_t first = __ldg(src);
        bool run = true;
        for (int b = 0; b < neblock && run; b += 32 * 64) run = __all_sync(FULLMASK, run_piece<32>(src, neblock, first, b));
        EncStream e;
        e.out = -1;
        if (run) {
            e.kind = SK_RUN; e.csize = first; e.need = 0;
        } else {
            int need = 0;
            const int cs = neblock < 65536 + 12 - 1
                               ? warp_lz4_compress<true>(src, neblock, slots + sid * neblock, neblock, tab, bm, ring, XRING, &need)
                               : warp_lz4_compress<false>(src, neblock, slots + sid * neblock, neblock, tab, bm, ring, XRING, &need);
            if (cs > 0 && cs < neblock) { e.kind = SK_LZ4; e.csize = cs; e.need = need; }
            else { e.kind = SK_RAW; e.csize = neblock; e.need = need; }
        }
        if (lane == 0) es[sid] = e;
        __syncwarp();
    }
}

// ---------------------------------------------------------------- LZ4 encoder, parallel parse
// The second encoder mode.  It writes standard LZ4 blocks (any LZ4 decoder, liblz4 and the
// reference's Blosc2 included, reads them back bit-exactly) but does not retrace liblz4's
// serial search, so its bytes differ from liblz4's.  One CTA of PT threads encodes one
// stream; per window of PW positions:
//  A. every position is hashed (4 bytes, 12 bits); its candidate is the latest position of
//     its bucket among the previous rounds of PT positions (the table keeps the largest
//     position written, so it is the same whatever the order of the writes), and the
//     previous position is a second candidate (runs); the longer match is kept, measured
//     up to PCAP bytes.  Every position enters the table.  A round's candidates are loaded
//     together, 16 bytes each; what is longer is measured by the warp, once for a row of positions
//     at one distance, and candidates inside runs from the lengths of the two runs.
//  B. the greedy parse (from the parse position, take the first position with a match of
//     at least 4 bytes, continue after it) is a chain over match positions: J[q] = the first
//     match position at or after q + L(q).  The chain is located by segment walks (below), the
//     sequences' output sizes are prefix-summed across the CTA, and every thread writes its own
//     sequences.  A chain ends at the window end, after the window's last match, or at a
//     match of PCAP bytes or more, which is extended exactly before it is written.
// The bytes of the next window are loaded before B and stored after it; literal runs of more than
// 16 bytes are copied by a warp.
// What bounds it: the latency of a window's steps (1,024 streams of 64 KiB, seven an SM: 26,000
// cycles a window, 60% of the issue slots; a stream by itself 13,000), and where zero padding makes
// every match long, the measuring of lengths.  A batch of 40 float64 products with extents of 64 to
// 2048: 14.7 -> 13.2 ms; the 16384 x 16384 float32 result of a split product 3.83 -> 3.45 ms.
// Format rules kept: offsets 1..65535, matches start at least 12 bytes before the end and
// end at least 5 bytes before it, so the block ends with >= 5 literals.
constexpr int PW = 1024;
constexpr int PT = 128;                   // threads per stream
constexpr int PCAP = 128;                 // match lengths measured in phase A (PCAP: at least PCAP)
constexpr uint16_t PJ_NONE = 0xFFFF, PJ_OUT = 0xFFFE, PJ_LONG = 0xFFFD;
constexpr int PSTAGE = 1024 + 16;         // staged bytes per probe window (from 4 before it)

struct ParSmem {              // per CTA
    union {
        uint16_t tab16[8192]; // liblz4 search (byU16); probe: four tables of 2048
        uint32_t tab32[4096]; // parallel parse: position + 1 of each bucket (0: empty); liblz4 byU32
    };
    uint8_t ring[ERING + EMIRROR];
    union {
        struct {
            uint16_t cw[PW];  // match distance of each window position
            uint8_t lw[PW];   // match length (0: none, 4..PCAP; PCAP: at least PCAP)
            uint16_t J[PW];   // the match after the one at each position, or why the chain stops
            uint16_t path[PW / 4 + 2];
        } w;
        uint8_t stage[4][PSTAGE];
        uint32_t peer[EPEER]; // liblz4 search: lanes-by-hash masks
    };
    uint32_t bits[32];        // match flags, one word per 32 positions
    int32_t nchain;           // matches on the window's chain
    int32_t red[8];           // block reductions
    long long sid;
};

// First match position at or after window offset rel (PJ_NONE: none left in the window).
__device__ __forceinline__ uint32_t par_next_match(const uint32_t *bits, int rel)
{
    if (rel >= PW) return PJ_OUT;
    int wi = rel >> 5;
    uint32_t m = bits[wi] & (0xFFFFFFFFu << (rel & 31));
    while (!m && ++wi < 32) m = bits[wi];
    return m ? (uint32_t)(wi * 32 + __ffs((int)m) - 1) : PJ_NONE;
}

__device__ __forceinline__ int lz4_seq_bytes(int lit, int ml)
{
    return 1 + (lit >= 15 ? 1 + (lit - 15) / 255 : 0) + lit + 2 + (ml >= 15 ? 1 + (ml - 15) / 255 : 0);
}

// One sequence (literals src[anchor, q), match at q, distance d, length L) at dst + o.
__device__ __forceinline__ void lz4_put_seq(const EncSrc &s, uint8_t *o, int anchor, int q, int d, int L, bool literals)
{
    const int lit = q - anchor, ml = L - 4;
    int k = 1;
    if (lit >= 15) {
        int rem = lit - 15;
        for (; rem >= 255; rem -= 255) o[k++] = 255;
        o[k++] = (uint8_t)rem;
    }
    if (literals)
        for (int x = 0; x < lit; x++) o[k + x] = (uint8_t)es_byte(s, anchor + x);
    k += lit;
    o[0] = (uint8_t)(((lit >= 15 ? 15 : lit) << 4) | (ml >= 15 ? 15 : ml));
    o[k] = (uint8_t)d;
    o[k + 1] = (uint8_t)(d >> 8);
    k += 2;
    if (ml >= 15) {
        int rem = ml - 15;
        for (; rem >= 255; rem -= 255) o[k++] = 255;
        o[k] = (uint8_t)rem;
    }
}

// 4 bytes at stream position x from the window (x must be inside it).
__device__ __forceinline__ uint32_t par_rd32(uint32_t ring_s, int x)
{
    const uint32_t o = (uint32_t)x & (ERING - 1);
    const uint32_t wa = ring_s + (o & ~3u);
    return __funnelshift_r(lds32(wa), lds32(wa + 4), (o & 3) * 8);
}

// es_fill for a whole CTA (every thread calls it with the same `want`).
__device__ __forceinline__ void cta_fill(EncSrc &s, int want)
{
    while (s.hi < s.n && s.hi < want) {
        const int base = s.hi, cnt = min(ESEG, s.n - base);
        __syncthreads();                                 // reads of the slots being replaced are done
        for (int x = threadIdx.x * 4; x < cnt; x += PT * 4) {
            uint32_t v = 0;
            if (base + x + 8 <= s.n) {
                v = ld4u(s.g + base + x);
            } else {
                for (int k = 0; k < 4; k++)
                    if (base + x + k < s.n) v |= (uint32_t)__ldg(s.g + base + x + k) << (8 * k);
            }
            const int o = (base + x) & (ERING - 1);
            *reinterpret_cast<uint32_t *>(s.r + o) = v;
            if (o < EMIRROR) *reinterpret_cast<uint32_t *>(s.r + ERING + o) = v;
        }
        s.hi = base + cnt;
        s.lo = max(s.lo, base + ESEG - ERING);
        __syncthreads();
    }
}

// Block-wide sum / min of one int per thread (uses red[]; ends with every thread holding
// the result and red[] free again).
__device__ __forceinline__ int cta_sum(int v, int32_t *red)
{
    v = (int)__reduce_add_sync(FULLMASK, (unsigned)v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int t = red[0] + red[1] + red[2] + red[3];
    __syncthreads();
    return t;
}

__device__ __forceinline__ int cta_min(int v, int32_t *red)
{
    v = (int)__reduce_min_sync(FULLMASK, (unsigned)v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int t = min(min(red[0], red[1]), min(red[2], red[3]));
    __syncthreads();
    return t;
}

__device__ __forceinline__ int cta_lz4_compress_par(const uint8_t *__restrict__ src, int n,
                                                    uint8_t *__restrict__ dst, int cap, ParSmem &S)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(S.ring);
    for (int i = tid; i < 4096 / 4; i += PT) reinterpret_cast<uint4 *>(S.tab32)[i] = make_uint4(0u, 0u, 0u, 0u);
    EncSrc s;
    s.g = src; s.r = S.ring; s.cap = ERING; s.lo = 0; s.hi = 0; s.n = n;
    __syncthreads();
    int op = 0, anchor = 0, pos = 0;
    const int mfl1 = n - 11, mlimit = n - 5;
    int ahead = -1;                                      // where `next` goes (-1: nowhere)
    uint32_t next[2][2];
    // Lengths past 16 bytes of the lanes that `need` them (position p, distance d, at most lim; every
    // lane calls).  A lane whose neighbour has the same distance has one byte more than that one;
    // for the last of such a row the warp compares 4 bytes a lane, which reaches PCAP.
    auto extend = [&](bool need, int p, int d, int lim) -> int {
        const unsigned nm = __ballot_sync(FULLMASK, need);
        if (!nm) return 0;
        const int dn = __shfl_down_sync(FULLMASK, d, 1);
        const unsigned hm = __ballot_sync(FULLMASK, need && !(lane < 31 && ((nm >> (lane + 1)) & 1u) && dn == d));
        if (__popc(hm) > 6) {                            // every lane by itself
            int l = 16;
            while (need && l < lim) {
                const uint32_t x = par_rd32(ring_s, p + l) ^ (p - d >= s.lo ? par_rd32(ring_s, p - d + l) : ld4u(src + p - d + l));
                l += x ? (__ffs((int)x) - 1) >> 3 : 4;
                if (x) break;
            }
            return min(l, lim);
        }
        const int head = __ffs((int)(hm & (FULLMASK << lane))) - 1;
        int got = 0;
        for (unsigned m = hm; m; m &= m - 1) {
            const int l = __ffs((int)m) - 1;
            const int ph = __shfl_sync(FULLMASK, p, l), dh = __shfl_sync(FULLMASK, d, l), lh = __shfl_sync(FULLMASK, lim, l);
            const int a = ph + 16 + 4 * lane;
            int eq = 0;
            if (a < ph + lh) {
                const uint32_t x = par_rd32(ring_s, a) ^ (ph - dh >= s.lo ? par_rd32(ring_s, a - dh) : ld4u(src + a - dh));
                eq = x ? (__ffs((int)x) - 1) >> 3 : 4;
            }
            const int f = __ffs((int)__ballot_sync(FULLMASK, eq < 4)) - 1;   // (at most 28 lanes compare)
            const int L = min(16 + 4 * f + __shfl_sync(FULLMASK, eq, f), lh);
            if (head == l) got = L + l - lane;
        }
        return min(got, lim);
    };
    for (int w0 = 0; n >= 13 && w0 < mfl1; w0 += PW) {
        const int wend = min(w0 + PW, mfl1), wn = wend - w0;
        if (ahead == s.hi) {                             // the bytes loaded during the last window
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int o = (ahead + k * ESEG + tid * 4) & (ERING - 1);
                const uint32_t v = __funnelshift_r(next[k][0], next[k][1], (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3) * 8);
                *reinterpret_cast<uint32_t *>(s.r + o) = v;
                if (o < EMIRROR) *reinterpret_cast<uint32_t *>(s.r + ERING + o) = v;
            }
            s.hi = ahead + 2 * ESEG;
            s.lo = max(s.lo, s.hi - ERING);
            __syncthreads();
        }
        ahead = -1;
        cta_fill(s, wend + PCAP + 32);
        // ---- A: candidates and lengths.  Positions p .. p + PCAP + 4 lie in the window;
        // a candidate is read from the window when it is still there, else from global memory.
        // Rounds of 2 PT positions (two per thread; a round's positions see the table as it was
        // before the round).  The stream's first PT positions go in rounds of 32 and the next PT
        // in one round of PT, so that short streams keep table candidates for most positions.
        for (int q0 = 0, rsz; q0 < PW; q0 += rsz) {
            rsz = w0 + q0 < PT ? 32 : w0 + q0 < 2 * PT ? PT : 2 * PT;
            int c2[2];
            uint32_t v2[2], h2[2], n2[2][3], cw2[2][5];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int p = w0 + q0 + tid + k * PT;
                const bool valid = tid + k * PT < rsz && p < wend;
                const uint32_t o = (uint32_t)p & (ERING - 1), wa = ring_s + (o & ~3u), sh = (o & 3) * 8;
                const uint32_t a0 = lds32(wa), a1 = lds32(wa + 4), a2 = lds32(wa + 8), a3 = lds32(wa + 12), a4 = lds32(wa + 16);
                v2[k] = __funnelshift_r(a0, a1, sh);
                n2[k][0] = __funnelshift_r(a1, a2, sh);
                n2[k][1] = __funnelshift_r(a2, a3, sh);
                n2[k][2] = __funnelshift_r(a3, a4, sh);
                h2[k] = (v2[k] * 2654435761u) >> (32 - 12);
                c2[k] = valid ? (int)S.tab32[h2[k]] - 1 : -1;
            }
            // 16 bytes at the candidates: all loads of the round are under way together
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int c = max(c2[k], 0);
                const uint32_t *w = c >= s.lo
                                        ? reinterpret_cast<const uint32_t *>(S.ring) + ((c & (ERING - 1)) >> 2)
                                        : reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(src + c) & ~uintptr_t(3));
#pragma unroll
                for (int i = 0; i < 5; i++) cw2[k][i] = w[i];
            }
            __syncthreads();                             // every read of this round precedes its writes
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int p = w0 + q0 + tid + k * PT;
                if (tid + k * PT < rsz && p < wend) atomicMax(&S.tab32[h2[k]], (uint32_t)p + 1u);
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int q = q0 + tid + k * PT, p = w0 + q, cand = c2[k];
                const bool valid = tid + k * PT < rsz && p < wend;
                const uint32_t v = v2[k];
                const int lim = min(mlimit - p, PCAP);
                const uint32_t sh = (cand >= s.lo ? (uint32_t)cand & 3u
                                                  : (uint32_t)(reinterpret_cast<uintptr_t>(src + max(cand, 0)) & 3)) * 8;
                const bool hit = cand >= 0 && p - cand <= 65535 && __funnelshift_r(cw2[k][0], cw2[k][1], sh) == v;
                const uint32_t x0 = n2[k][0] ^ __funnelshift_r(cw2[k][1], cw2[k][2], sh),
                               x1 = n2[k][1] ^ __funnelshift_r(cw2[k][2], cw2[k][3], sh),
                               x2 = n2[k][2] ^ __funnelshift_r(cw2[k][3], cw2[k][4], sh);
                const uint32_t x = x0 ? x0 : x1 ? x1 : x2;
                const int len = (x0 ? 4 : x1 ? 8 : 12) + (x ? (__ffs((int)x) - 1) >> 3 : 4);
                int L = hit ? min(len, lim) : 0, best = cand;
                bool need = hit && len == 16 && lim > 16;
                // a run from p on, R bytes equal
                const bool flat = valid && v == (v & 0xFFu) * 0x01010101u;
                if (__any_sync(FULLMASK, flat)) {
                    const uint32_t y0 = n2[k][0] ^ v, y1 = n2[k][1] ^ v, y2 = n2[k][2] ^ v;
                    const uint32_t y = y0 ? y0 : y1 ? y1 : y2;
                    int R = min((y0 ? 4 : y1 ? 8 : 12) + (y ? (__ffs((int)y) - 1) >> 3 : 4), lim);
                    const bool far = flat && !(y0 | y1 | y2) && lim > 16;
                    const int l = extend(far, p, 1, lim);
                    if (far) R = l;
                    // Candidates inside a run: the positions of a round have the same one, each at another
                    // distance.  The shorter run is the match (two of the same length are compared on).
                    const bool in = far && need;
                    for (unsigned m = __ballot_sync(FULLMASK, in); m;) {
                        const int i = __ffs((int)m) - 1, c = __shfl_sync(FULLMASK, cand, i), a = c + 16 + 4 * lane;
                        const uint32_t b = __shfl_sync(FULLMASK, v, i);
                        const unsigned mates = __ballot_sync(FULLMASK, in && cand == c);
                        int eq = 0;
                        if (lane < (PCAP - 16) / 4) {
                            const uint32_t z = (c >= s.lo ? par_rd32(ring_s, a) : ld4u(src + a)) ^ b;
                            eq = z ? (__ffs((int)z) - 1) >> 3 : 4;
                        }
                        const int f = __ffs((int)__ballot_sync(FULLMASK, eq < 4)) - 1;
                        const int C = 16 + 4 * f + __shfl_sync(FULLMASK, eq, f);
                        if (((mates >> lane) & 1u) && (R >= lim || C != R)) { L = min(C, R); need = false; }
                        m &= ~mates;
                    }
                    const int g = extend(need, p, p - cand, lim);
                    if (need) L = g;
                    // the previous position matches too when the byte before p is the run's
                    if (flat && p > 0 && cand != p - 1 && R > L && S.ring[(p - 1) & (ERING - 1)] == (uint8_t)v) {
                        L = R;
                        best = p - 1;
                    }
                } else {
                    const int g = extend(need, p, p - cand, lim);
                    if (need) L = g;
                }
                if (tid + k * PT < rsz) {
                    S.w.cw[q] = (uint16_t)(p - best);
                    S.w.lw[q] = (uint8_t)L;
                }
                const unsigned bb = __ballot_sync(FULLMASK, L >= 4);
                if (lane == 0 && k * PT + warp * 32 < rsz) S.bits[((q0 + k * PT) >> 5) + warp] = bb;
            }
            __syncthreads();                             // this round's writes precede the next reads
        }
        // the next window's bytes, on their way while this one's sequences are found and written
        if (s.hi + 2 * ESEG + 8 <= n && wend + PW + PCAP + 32 > s.hi) {
            ahead = s.hi;
#pragma unroll
            for (int k = 0; k < 2; k++) {                // (whole words; shifted when they are stored)
                const uint32_t *w = reinterpret_cast<const uint32_t *>(
                    reinterpret_cast<uintptr_t>(src + ahead + k * ESEG + tid * 4) & ~uintptr_t(3));
                next[k][0] = __ldg(w);
                next[k][1] = __ldg(w + 1);
            }
        }
        // ---- B: chains of matches from the parse position
        while (pos < wend) {
            const uint32_t s0 = par_next_match(S.bits, pos - w0);
            if (s0 >= (uint32_t)wn) { pos = wend; break; }   // no match left: literals run on
            // J[q]: the match after the one at q, or why the chain stops there
            const unsigned nz = __ballot_sync(FULLMASK, S.bits[lane] != 0);
#pragma unroll
            for (int k = 0; k < PW / PT; k++) {
                const int q = tid + k * PT, L = S.w.lw[q], e = q + L, sg = min(e >> 5, 31);
                uint32_t r = S.bits[sg] & (FULLMASK << (e & 31));
                const unsigned more = sg < 31 ? nz & (FULLMASK << (sg + 1)) : 0u;
                int s2 = sg;
                if (!r && more) {
                    s2 = __ffs((int)more) - 1;
                    r = S.bits[s2];
                }
                uint32_t v = r ? (uint32_t)(s2 * 32 + __ffs((int)r) - 1) : (uint32_t)PJ_NONE;
                if (e >= wn) v = PJ_OUT;
                if (L >= PCAP) v = PJ_LONG;
                S.w.J[q] = (uint16_t)v;
            }
            __syncthreads();
            // The chain from s0 by segment walks (warp 0): lane t walks J from the first match
            // at or after 32 t, recording the matches it visits; then, in rounds, lane t takes
            // the exit of lane t - 1 as its entry (lane 0: s0), follows its own walk once the
            // chain meets it and publishes its exit, until no exit changes.
            if (warp == 0) {
                const int lo = lane * 32, hi = lo + 32;
                const int nl = (wn + 31) / 32;              // lanes whose segment holds window positions
                const bool act = lane < nl;
                uint32_t mask = 0;
                int ex = PJ_NONE;
                if (act) {
                    int q = (int)par_next_match(S.bits, lo);
                    ex = q;
                    if (q < hi && q < wn) {
                        for (;;) {                          // positions grow: at most 32 steps
                            mask |= 1u << (q - lo);
                            const int v = S.w.J[q];
                            if (v >= hi || v >= wn) { ex = v; break; }
                            q = v;
                        }
                    }
                }
                uint32_t fm = 0;
                int cur = ex;
                for (int round = 0; round < 32; round++) {  // one round settles at least one more lane
                    int entry = __shfl_up_sync(FULLMASK, cur, 1);
                    if (lane == 0) entry = (int)s0;
                    uint32_t m = 0;
                    int e2 = entry;
                    if (act && entry < hi && entry < wn) {
                        int q = entry;
                        for (;;) {
                            const int b = q - lo;
                            if ((mask >> b) & 1u) { m |= mask & (~0u << b); e2 = ex; break; }
                            m |= 1u << b;
                            const int v = S.w.J[q];
                            if (v >= hi || v >= wn) { e2 = v; break; }
                            q = v;
                        }
                    }
                    const bool changed = act && e2 != cur;
                    fm = m;
                    cur = e2;
                    if (!__any_sync(FULLMASK, changed)) break;
                }
                const int chain_end = __shfl_sync(FULLMASK, cur, max(nl, 1) - 1);
                const int c = __popc(fm);
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(FULLMASK, incl, o);
                    if (lane >= o) incl += v;
                }
                int o = incl - c;
                for (uint32_t x = fm; x; x &= x - 1) S.w.path[o++] = (uint16_t)(lo + __ffs((int)x) - 1);
                if (lane == 31) {
                    S.w.path[incl] = (uint16_t)chain_end;   // PJ_NONE, PJ_OUT or PJ_LONG
                    S.nchain = incl;
                }
            }
            __syncthreads();
            const int cnt = S.nchain;
            const uint16_t term = S.w.path[cnt];                // why the chain stopped
            // a capped last match: extend it exactly (CTA-wide) before writing it
            int lastL = S.w.lw[S.w.path[cnt - 1]];
            const int lastq = w0 + S.w.path[cnt - 1], lastd = S.w.cw[S.w.path[cnt - 1]];
            if (term == PJ_LONG) {
                for (;;) {
                    const int a = lastq + lastL;
                    cta_fill(s, a + PT + ELOOK);
                    const bool eq = a + tid < mlimit && es_byte(s, a + tid) == es_byte(s, a - lastd + tid);
                    const unsigned ne = __ballot_sync(FULLMASK, !eq);
                    const int cnum = cta_min(ne ? warp * 32 + __ffs((int)ne) - 1 : PT, S.red);
                    lastL += cnum;
                    if (cnum < PT) break;
                }
            }
            // output sizes, their exclusive scan (two sequences a thread; at most PW / 4), the sequences
            int q2[2], e2[2], L2[2], d2[2], sz2[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int i = 2 * tid + k;
                q2[k] = e2[k] = L2[k] = d2[k] = sz2[k] = 0;
                if (i < cnt) {
                    const int q = S.w.path[i], before = i ? S.w.path[i - 1] : 0;
                    e2[k] = i ? w0 + before + S.w.lw[before] : anchor;
                    q2[k] = w0 + q;
                    L2[k] = i == cnt - 1 ? lastL : S.w.lw[q];
                    d2[k] = S.w.cw[q];
                    sz2[k] = lz4_seq_bytes(q2[k] - e2[k], L2[k] - 4);
                }
            }
            const int both = sz2[0] + sz2[1];
            int incl = both;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULLMASK, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) S.red[warp] = incl;
            __syncthreads();
            int before = 0, total = 0;
#pragma unroll
            for (int k = 0; k < PT / 32; k++) {
                const int t = S.red[k];
                before += k < warp ? t : 0;
                total += t;
            }
            if (op + total + 1 + 6 <= cap) {
                int o = op + before + incl - both;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const int lit = q2[k] - e2[k];
                    if (sz2[k]) lz4_put_seq(s, dst + o, e2[k], q2[k], d2[k], L2[k], lit <= 16);
                    // longer literal runs by the warp
                    const int at = o + 1 + (lit >= 15 ? 1 + (lit - 15) / 255 : 0);
                    for (unsigned m = __ballot_sync(FULLMASK, sz2[k] && lit > 16); m; m &= m - 1) {
                        const int i = __ffs((int)m) - 1;
                        const int to = __shfl_sync(FULLMASK, at, i), from = __shfl_sync(FULLMASK, e2[k], i),
                                  cnt = __shfl_sync(FULLMASK, lit, i);
                        for (int x = lane; x < cnt; x += 32) dst[to + x] = (uint8_t)es_byte(s, from + x);
                    }
                    o += sz2[k];
                }
            }
            __syncthreads();
            if (op + total + 1 + 6 > cap) return 0;
            op += total;
            anchor = lastq + lastL;
            pos = anchor;
            if (term == PJ_NONE) { pos = max(pos, wend); }
        }
    }
    {
        const int last = n - anchor;
        if (op + 1 + last + (last + 240) / 255 > cap) return 0;
        uint8_t *o = dst + op;
        int k = 1;
        if (last >= 15) {
            const int rem = last - 15, nff = rem / 255;
            for (int x = tid; x < nff; x += PT) o[1 + x] = 255;
            if (tid == 0) o[1 + nff] = (uint8_t)(rem % 255);
            k += nff + 1;
        }
        if (tid == 0) o[0] = (uint8_t)((last >= 15 ? 15 : last) << 4);
        for (int x = tid; x < last; x += PT) o[k + x] = (uint8_t)es_byte(s, anchor + x);
        op += k + last;
    }
    __syncthreads();
    return op;
}

// Matches found in four sampled windows of 1024 positions (at 0, 1/4, 1/2 and 3/4 of the
// stream), one window per warp: positions with a 4-byte match against the warp's table of
// recent positions of the window (11-bit hash) or against the previous position.  Each
// window is staged in shared memory first by one round of coalesced word loads.  Returns
// the CTA's total.
__device__ __forceinline__ uint32_t stage_rd32(const uint8_t *stage, int o)
{
    const uint32_t *w = reinterpret_cast<const uint32_t *>(stage) + (o >> 2);
    return __funnelshift_r(w[0], w[1], (uint32_t)(o & 3) * 8);
}

__device__ __forceinline__ int cta_probe(const uint8_t *__restrict__ src, int n, ParSmem &S)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint16_t *tab = S.tab16 + w * 2048;
    uint8_t *stage = S.stage[w];
    for (int i = lane; i < 2048 / 8; i += 32) reinterpret_cast<uint4 *>(tab)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    const int base = (int)(((int64_t)(n - 11) * w / 4) & ~31);
    const int lim = min(n - 11, base + 1024);
    const int b0 = base >= 4 ? base - 4 : 0;                 // word aligned: base is a multiple of 32
    const int cnt = min(PSTAGE, n - b0);
    for (int x = lane * 4; x < cnt; x += 128) {
        uint32_t v = 0;
        if (b0 + x + 8 <= n) {                               // ld4u reads 8 bytes
            v = ld4u(src + b0 + x);
        } else {
            for (int k = 0; k < 4; k++)
                if (b0 + x + k < n) v |= (uint32_t)__ldg(src + b0 + x + k) << (8 * k);
        }
        *reinterpret_cast<uint32_t *>(stage + x) = v;
    }
    __syncwarp();
    int hits = 0;
    for (int r = 0; r < 32; r++) {
        const int p = base + r * 32 + lane;
        const bool valid = p < lim;
        const uint32_t v = valid ? stage_rd32(stage, p - b0) : 0u;
        const uint32_t h = (v * 2654435761u) >> (32 - 11);
        const uint32_t c = valid ? tab[h] : 0xFFFFu;
        __syncwarp();
        if (valid) tab[h] = (uint16_t)p;
        const bool m = valid && ((c < (uint32_t)p && c >= (uint32_t)b0 && stage_rd32(stage, (int)c - b0) == v) ||
                                 (p > b0 && stage_rd32(stage, p - 1 - b0) == v));
        hits += __popc(__ballot_sync(FULLMASK, m));
    }
    return cta_sum(lane == 0 ? hits : 0, S.red);
}

// E2 (parallel mode): one CTA of PT threads per stream, streams handed out dynamically.  A
// probe of four sampled windows routes each stream: almost no matches (incompressible
// byte planes): stored raw; few matches: the liblz4 search (one warp), whose accelerating
// skip makes them cheap; the rest: the parallel parse.
__global__ void __launch_bounds__(PT, 8) k_lz4_encode_par(const uint8_t *__restrict__ img, int64_t nstreams_total,
                                                       int per, int neblock, uint8_t *slots, EncStream *es,
                                                       unsigned long long *next)
{
    extern __shared__ __align__(16) uint8_t sm_par[];
    ParSmem &S = *reinterpret_cast<ParSmem *>(sm_par);
    const int tid = threadIdx.x, warp = tid >> 5;
    for (bool start = true;; start = false) {
        if (tid == 0) S.sid = start ? (long long)blockIdx.x : (long long)(gridDim.x + atomicAdd(next, 1ull));
        __syncthreads();
        const int64_t k = S.sid;
        __syncthreads();
        if (k >= nstreams_total) break;
        const int64_t sid = stream_at(k, nstreams_total, per);
        const uint8_t *src = img + sid * neblock;
        const uint8_t first = __ldg(src);
        bool run = true;
        for (int b = 0; b < neblock && run; b += PT * 64) run = __syncthreads_and(run_piece<PT>(src, neblock, first, b));
        EncStream e;
        e.out = -1;
        if (run) {
            e.kind = SK_RUN; e.csize = first; e.need = 0;
        } else {
            // (LZ4 compresses no block below 13 bytes, and the probe's windows need 11)
            const int hits = neblock < 13 ? 0 : cta_probe(src, neblock, S);
            if (hits < 16) {                     // no matches to speak of: store the stream raw
                e.kind = SK_RAW; e.csize = neblock; e.need = neblock + 1;
            } else if (hits < 256) {
                if (warp == 0) {
                    int need = 0;
                    const int cs = neblock < 65536 + 12 - 1
                                       ? warp_lz4_compress<true>(src, neblock, slots + sid * neblock, neblock, S.tab32, S.peer, S.ring, ERING, &need)
                                       : warp_lz4_compress<false>(src, neblock, slots + sid * neblock, neblock, S.tab32, S.peer, S.ring, ERING, &need);
                    if (cs > 0 && cs < neblock) { e.kind = SK_LZ4; e.csize = cs; e.need = need; }
                    else { e.kind = SK_RAW; e.csize = neblock; e.need = need; }
                }
            } else {
                const int cs = cta_lz4_compress_par(src, neblock, slots + sid * neblock, neblock, S);
                if (cs > 0 && cs < neblock) { e.kind = SK_LZ4; e.csize = cs; e.need = cs; }
                else { e.kind = SK_RAW; e.csize = neblock; e.need = neblock + 1; }
            }
        }
        if (tid == 0) es[sid] = e;
        __syncthreads();
    }
}

// E3: per chunk (one CTA each), the stream layout blosc_c produces: streams in order, each a
// 4-byte csize word and its payload (a run: one byte or none), an LZ4 stream only where its
// output fits the space left (else raw); a chunk that does not fit nbytes + 32 is stored
// memcpyed.  The space left only binds near the end of a chunk, so sizes are prefix-summed
// as if it never binds, and thread 0 replays the stream-by-stream walk from the first stream
// where it could.
constexpr int LAYOUT_T = 256;

// The blosc_c walk for one stream from running size ntb; false: the chunk does not fit.
__device__ __forceinline__ bool layout_step(EncStream &e, int64_t &ntb, int64_t destsize, int neblock)
{
    ntb += 4;
    if (e.kind == SK_RUN) {
        if (ntb > destsize) return false;
        e.out = (int32_t)(ntb - 4);
        if (e.csize != 0) {
            if (ntb + 1 > destsize) return false;
            ntb += 1;
        }
        return true;
    }
    int64_t maxout = neblock;
    if (ntb + maxout > destsize) {
        maxout = destsize - ntb;
        if (maxout <= 0) return false;
    }
    int64_t sz;
    if (e.kind == SK_LZ4 && e.need <= maxout) {
        sz = e.csize;
    } else {
        if (ntb + neblock > destsize) return false;
        e.kind = SK_RAW;
        sz = neblock;
    }
    e.out = (int32_t)(ntb - 4);
    ntb += sz;
    return true;
}

// memcpy_only (compression level 0): c-blosc2 stores every chunk memcpyed.
__device__ __forceinline__ void layout_chunk(const Geom &g, int nstreams, int neblock, EncStream *es, EncChunk *ec,
                                             int memcpy_only, int64_t c, int64_t *wsum, int64_t &s_before, int &s_first)
{
    const int64_t destsize = g.chunk_nbytes + 32, ns = g.nblocks * nstreams;
    if (memcpy_only) {
        if (threadIdx.x == 0) { ec[c].memcpyed = 1; ec[c].cbytes = (int32_t)destsize; }
        return;
    }
    const int64_t ntb0 = 32 + 4 * g.nblocks;
    EncStream *e0 = es + c * ns;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_first = 0x7FFFFFFF;
    __syncthreads();
    int64_t base = ntb0;
    for (int64_t r0 = 0; ntb0 <= destsize && r0 < ns; r0 += LAYOUT_T) {
        const int64_t i = r0 + threadIdx.x;
        EncStream e;
        e.kind = SK_RAW; e.csize = 0; e.need = 0; e.out = -1;
        int64_t sz = 0;
        if (i < ns) {
            e = e0[i];
            sz = e.kind == SK_RUN ? 4 + (e.csize != 0) : e.kind == SK_LZ4 ? 4 + (int64_t)e.csize : 4 + (int64_t)neblock;
        }
        int64_t incl = sz;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(FULLMASK, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int64_t before = base + incl - sz, all = 0;
#pragma unroll
        for (int w = 0; w < LAYOUT_T / 32; w++) {
            before += w < warp ? wsum[w] : 0;
            all += wsum[w];
        }
        // the unconstrained choice holds while the stream (raw, at worst) still fits
        const bool safe = e.kind == SK_RUN ? before + sz <= destsize
                                           : before + 4 + neblock <= destsize && (e.kind != SK_LZ4 || e.need <= neblock);
        if (i < ns && !safe) atomicMin(&s_first, (int)i);
        __syncthreads();
        const int first = s_first;
        if (i < ns && i < first) e0[i].out = (int32_t)before;
        if (i == first) s_before = before;
        base += all;
        __syncthreads();
        if (first != 0x7FFFFFFF) break;
    }
    if (threadIdx.x == 0) {
        bool ok = ntb0 <= destsize;
        int64_t ntb = base;
        if (ok && s_first != 0x7FFFFFFF) {
            ntb = s_before;
            for (int64_t i = s_first; ok && i < ns; i++) ok = layout_step(e0[i], ntb, destsize, neblock);
        }
        ec[c].memcpyed = ok ? 0 : 1;
        ec[c].cbytes = (int32_t)(ok ? ntb : destsize);
    }
}

// Chunk offsets: exclusive scan of the chunk sizes (one CTA, V chunks a thread at a time); off / len
// (optional): the chunk index as the decoder reads it.
template <int V>
__device__ __forceinline__ void chunk_offsets(int64_t nchunks, EncChunk *ec, int64_t *total, int64_t *off, int32_t *len,
                                              int64_t *wsum)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (int)blockDim.x >> 5;
    int64_t base = 0;
    for (int64_t r0 = 0; r0 < nchunks; r0 += (int64_t)blockDim.x * V) {
        // chunk v of this thread: r0 + warp * 32 V + v * 32 + lane, neighbours side by side
        const int64_t i0 = r0 + (int64_t)warp * 32 * V + lane;
        int32_t size[V];
#pragma unroll
        for (int v = 0; v < V; v++) size[v] = i0 + v * 32 < nchunks ? __ldcg(&ec[i0 + v * 32].cbytes) : 0;
        int64_t sum[V], mine = 0;                  // each chunk's offset within its warp's chunks
#pragma unroll
        for (int v = 0; v < V; v++) {
            int64_t incl = size[v];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(FULLMASK, incl, o);
                if (lane >= o) incl += t;
            }
            sum[v] = mine + incl - size[v];
            mine += __shfl_sync(FULLMASK, incl, 31);
        }
        if (lane == 31) wsum[warp] = mine;
        __syncthreads();
        int64_t before = base, all = 0;
        for (int w = 0; w < warps; w++) {
            before += w < warp ? wsum[w] : 0;
            all += wsum[w];
        }
#pragma unroll
        for (int v = 0; v < V; v++) {
            const int64_t i = i0 + v * 32;
            if (i < nchunks) {
                ec[i].offset = before + sum[v];
                if (off) { off[i] = before + sum[v]; len[i] = size[v]; }
            }
        }
        base += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = base;
}

// One CTA per chunk; the last one to finish (tot[2] counts them) adds the chunks' offsets: no
// launch of its own, and no upload of the index by the host.  More chunks than LAYOUT_OWN have a launch
// for the offsets: the counts come one after the other (about 4 ns each), and a thread of that launch
// takes 8 chunks at a time (250,000 chunks of 8 x 8 float64: layout and offsets 1.05 ms with a launch of a
// chunk a thread, 1.44 with the count, now 0.72).
constexpr int64_t LAYOUT_OWN = 1024;
__global__ void __launch_bounds__(LAYOUT_T) k_layout(Geom g, int nstreams, int neblock, EncStream *es, EncChunk *ec,
                                                    int memcpy_only, int64_t *tot, int64_t *off, int32_t *len, bool own)
{
    __shared__ int64_t wsum[LAYOUT_T / 32];
    __shared__ int64_t s_before;
    __shared__ int s_first;
    layout_chunk(g, nstreams, neblock, es, ec, memcpy_only, blockIdx.x, wsum, s_before, s_first);
    if (!own) return;
    if (threadIdx.x == 0) {                        // (thread 0 wrote the chunk's size)
        __threadfence();
        s_first = atomicAdd(reinterpret_cast<unsigned long long *>(tot + 2), 1ull) + 1 == gridDim.x;
    }
    __syncthreads();
    if (!s_first) return;
    __threadfence();
    chunk_offsets<1>(g.nchunks, ec, tot, off, len, wsum);
}
__global__ void __launch_bounds__(1024) k_chunk_offsets(int64_t nchunks, EncChunk *ec, int64_t *tot, int64_t *off, int32_t *len)
{
    __shared__ int64_t wsum[32];
    chunk_offsets<8>(nchunks, ec, tot, off, len, wsum);
}

// Copies len bytes with nt threads (tid: this one's number): 16-byte aligned stores to dst, each fed by five
// aligned 32-bit loads of src funnel-shifted into place.  Source words are only read
// inside [lo, hi); pieces whose words would leave it are copied bytewise.
__device__ __forceinline__ void group_copy(uint8_t *__restrict__ dst, const uint8_t *__restrict__ src, int len,
                                           const uint8_t *lo, const uint8_t *hi, int tid, int nt)
{
    int head = (int)((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15);
    if (head > len) head = len;
    for (int x = tid; x < head; x += nt) dst[x] = __ldg(src + x);
    const int nvec = (len - head) >> 4;
    for (int v = tid; v < nvec; v += nt) {
        const int s = head + (v << 4);
        const uint8_t *sp = src + s;
        const uint8_t *sa = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(sp) & ~uintptr_t(3));
        uint4 o;
        if (sa >= lo && sa + 20 <= hi) {
            const uint32_t *w = reinterpret_cast<const uint32_t *>(sa);
            const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(sp) & 3) * 8;
            const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3), w4 = __ldg(w + 4);
            o.x = __funnelshift_r(w0, w1, sh);
            o.y = __funnelshift_r(w1, w2, sh);
            o.z = __funnelshift_r(w2, w3, sh);
            o.w = __funnelshift_r(w3, w4, sh);
        } else {
            uint32_t b[4];
            for (int k = 0; k < 4; k++)
                b[k] = (uint32_t)__ldg(sp + 4 * k) | ((uint32_t)__ldg(sp + 4 * k + 1) << 8) |
                       ((uint32_t)__ldg(sp + 4 * k + 2) << 16) | ((uint32_t)__ldg(sp + 4 * k + 3) << 24);
            o = make_uint4(b[0], b[1], b[2], b[3]);
        }
        *reinterpret_cast<uint4 *>(dst + s) = o;
    }
    for (int x = head + (nvec << 4) + tid; x < len; x += nt) dst[x] = __ldg(src + x);
}

// E5: write headers, bstarts, csize words and payloads.  One CTA per stream: where there are few
// blocks the copies of their streams are under way together, where there are many the last ones
// are shorter (300 x 200 float64 9 us, by one CTA per block 15; 8192 x 8192 0.19 ms, 0.26).  Streams
// below EMIT_WARP bytes, where there are more of them than CTAs at once, take a warp each: a CTA spends
// most of its time on the loads before the copy (4000 x 4000 float64 in blocks of 8 x 8, 2 million
// streams: 3.6 ms by a CTA a stream, 0.57 by a CTA a block, 0.74 by warps; of 32 x 32 0.34, 0.36 and
// 0.08; of 90 x 90 0.068, 0.072 and 0.058; of 128 x 128 0.052 by CTAs, 0.064 by warps).
constexpr int EMIT_WARP = 8192;
static int emit_threads(int64_t streams, int neblock, int sms) { return neblock < EMIT_WARP && streams > (int64_t)sms * 8 ? 32 : 256; }
static unsigned emit_grid(int64_t streams, int nt, int sms)
{
    return (unsigned)std::max<int64_t>(std::min<int64_t>(ceil_div(streams, 256 / nt), (int64_t)sms * 8), 1);
}
__device__ __forceinline__ void emit_block(const Geom &g, int nstreams, int neblock, bool shuffle, int splitflag,
                                           const uint8_t *__restrict__ img, const uint8_t *__restrict__ slots,
                                           int64_t img_bytes, const EncStream *__restrict__ es,
                                           const EncChunk *__restrict__ ec, uint8_t *__restrict__ outbuf, int64_t t, int j,
                                           int tid, int nt)
{
    const int ts = g.itemsize;
    do {
        int64_t c, b;
        divmod(t, g.nblocks, c, b);
        const EncStream e = es[t * nstreams + j];      // (loaded beside the chunk's entry; unused when memcpyed)
        const EncChunk cc = ec[c];
        uint8_t *chunk = outbuf + cc.offset;
        if (b == 0 && j == 0 && tid < 32) {
            const int flags = 0x05 | (1 << 5) | (splitflag ? 0 : 0x10) | (cc.memcpyed ? 0x02 : 0);
            uint8_t hb = 0;
            const int x = tid;
            if (x == 0) hb = 5;
            else if (x == 1) hb = 1;
            else if (x == 2) hb = (uint8_t)flags;
            else if (x == 3) hb = (uint8_t)ts;
            else if (x >= 4 && x < 8) hb = (uint8_t)(g.chunk_nbytes >> (8 * (x - 4)));
            else if (x >= 8 && x < 12) hb = (uint8_t)(g.blocksize >> (8 * (x - 8)));
            else if (x >= 12 && x < 16) hb = (uint8_t)((uint32_t)cc.cbytes >> (8 * (x - 12)));
            else if (x == 21) hb = shuffle ? 1 : 0;
            else if (x == 22) hb = 1;   // compcode LZ4
            chunk[x] = hb;
        }
        const uint8_t *blk_img = img + t * g.blocksize;
        if (cc.memcpyed) {
            uint8_t *dst = chunk + 32 + b * g.blocksize;
            for (int64_t x = (int64_t)j * neblock + tid; x < (int64_t)(j + 1) * neblock; x += nt) {
                uint8_t v;
                if (shuffle) { const int64_t i = x / ts, k = x - i * ts; v = blk_img[k * g.blockn + i]; }
                else v = blk_img[x];
                dst[x] = v;
            }
            continue;
        }
        if (j == 0 && tid < 4) chunk[32 + 4 * b + tid] = (uint8_t)((uint32_t)e.out >> (8 * tid));
        uint8_t *w = chunk + e.out;
        int32_t word;
        const uint8_t *payload = nullptr;
        int plen = 0;
        if (e.kind == SK_RUN) { word = -e.csize; }
        else if (e.kind == SK_LZ4) { word = e.csize; payload = slots + (t * nstreams + j) * (int64_t)neblock; plen = e.csize; }
        else { word = neblock; payload = blk_img + (int64_t)j * neblock; plen = neblock; }
        if (tid < 4) w[tid] = (uint8_t)((uint32_t)word >> (8 * tid));
        if (e.kind == SK_RUN && e.csize != 0 && tid == 4) w[4] = 1;
        if (plen > 0) {
            const uint8_t *base = e.kind == SK_LZ4 ? slots : img;
            group_copy(w + 4, payload, plen, base, base + img_bytes, tid, nt);
        }
    } while (false);
}

template <int NT>
__global__ void __launch_bounds__(256) k_emit(Geom g, int nstreams, int neblock, bool shuffle, int splitflag,
                                              const uint8_t *__restrict__ img, const uint8_t *__restrict__ slots,
                                              int64_t img_bytes,
                                              const EncStream *__restrict__ es, const EncChunk *__restrict__ ec,
                                              uint8_t *__restrict__ outbuf)
{
    constexpr int per = 256 / NT;
    for (int64_t u = (int64_t)blockIdx.x * per + threadIdx.x / NT; u < g.nchunks * g.nblocks * nstreams; u += (int64_t)gridDim.x * per) {
        int64_t t, j;
        divmod(u, nstreams, t, j);
        emit_block(g, nstreams, neblock, shuffle, splitflag, img, slots, img_bytes, es, ec, outbuf, t, (int)j, threadIdx.x % NT, NT);
    }
}

// ============================================================================ host launchers
static int sm_count()
{
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

int decode_container(const Geom &g, const uint8_t *d_chunks, int64_t chunks_bytes, const int64_t *d_off, const int32_t *d_len,
                     void *out, int64_t ld, cudaStream_t st)
{
    DecodeWork w;
    int r = decode_launch(g, d_chunks, chunks_bytes, d_off, d_len, out, ld, st, &w);
    if (r) return r;
    return decode_finish(&w, st);
}

int decode_finish_queue(DecodeQueue *q, DecodeWork *const *w, int n, cudaStream_t st)
{
    int h[64];
    const int slots = q->slots;
    if (slots < 0 || (slots + 1) * 16 > 64) return -101;
    cudaMemcpyAsync(h, q->counters.p, 64 * (size_t)(slots + 1), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return -101;
    int r = 0;
    for (int k = 0; k < n; k++) {
        const int64_t at = w[k]->ext_counters ? w[k]->ext_counters - q->counters.as<int>() : 0;
        if (at < 16 || at > 16 * slots) return -101;
        w[k]->nzero = h[at + 4];
        if (!r) r = h[at + 1];
    }
    return r;
}

int decode_finish(DecodeWork *w, cudaStream_t st)
{
    int h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int *cnt = w->ext_counters ? w->ext_counters : w->counters.as<int>();
    cudaMemcpyAsync(h, cnt, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return -101;
    w->nzero = h[4];
    return h[1];
}

// Grid of the fast scatter: the CTAs resident at once (one wave), at most one per slice, or per tile
// where it also takes the general path.
template <int TS>
static int64_t scatter_fast_grid(const Geom &g, int64_t nbl, bool all)
{
    static int per_sm = 0;
    if (!per_sm) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_scatter_fast<TS, true>, 256, 0) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = 4;
        }
        per_sm = n;
    }
    const int64_t units = nbl * ceil_div(g.blockn, all ? TILE : SC_ITEMS);
    return std::max<int64_t>(std::min<int64_t>(units, (int64_t)sm_count() * per_sm), 1);
}

int64_t decode_max_jobs(const Geom &g) { return g.nchunks * g.nblocks * 8; }

int decode_queue_init(DecodeQueue *q, int64_t max_jobs, int slots, cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const size_t bytes = 64 * (size_t)(1 + slots);
    if (!q->jobs.allocate(sizeof(Lz4Job) * (size_t)std::max<int64_t>(max_jobs, 1), dev) || !q->counters.allocate(bytes, dev))
        return -100;
    q->cap = max_jobs;
    q->slots = slots;
    q->used = 0;
    cudaMemsetAsync(q->counters.p, 0, bytes, st);
    return 0;
}

int decode_parse(const DecodeArgs &a, DecodeQueue *q, DecodeWork *w, cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const Geom &g = a.g;
    const int64_t nbl = g.nchunks * g.nblocks;
    if (!w->bd.allocate(sizeof(BlockDesc) * nbl, dev) || !w->sd.allocate(sizeof(StreamDesc) * nbl * 8, dev) ||
        !w->scratch.allocate((size_t)(nbl * g.blocksize), dev))
        return -100;
    if (!w->ext_counters && q->used < q->slots) {
        w->ext_counters = q->counters.as<int>() + 16 * ++q->used;      // zeroed with the queue's counters
    } else {
        if (!w->ext_counters && !w->counters.allocate(64, dev)) return -100;
        cudaMemsetAsync(w->ext_counters ? (void *)w->ext_counters : w->counters.p, 0, 64, st);
    }
    int *cnt = w->ext_counters ? w->ext_counters : w->counters.as<int>();
    if (!w->zf.allocate((size_t)std::max<int64_t>(nbl, 1), dev)) return -100;
    IAB_TIMED("k_parse", st, k_parse<<<parse_grid(nbl, sm_count()), PARSE_T, 0, st>>>(
        g, a.chunks, a.off, a.len, w->bd.as<BlockDesc>(), w->sd.as<StreamDesc>(), q->jobs.as<Lz4Job>(),
        q->counters.as<int>(), q->cap, cnt + 1, cnt + 2, w->scratch.as<uint8_t>(), w->zf.as<uint8_t>(), cnt + 4));
    return 0;
}

int decode_lz4(DecodeQueue *q, cudaStream_t st)
{
    static bool attr = false;
    const int smem = (int)sizeof(dcta::Smem);
    if (!attr) {
        cudaFuncSetAttribute(k_lz4_decode_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        attr = true;
    }
    int *qc = q->counters.as<int>();
    IAB_TIMED("k_lz4_decode_cta", st, k_lz4_decode_cta<<<sm_count() * 6, dcta::THREADS, smem, st>>>(
        q->jobs.as<Lz4Job>(), qc, q->cap, reinterpret_cast<unsigned *>(qc + 8)));
    return 0;
}

// The decoded streams to the dense array.  Small containers by one launch, the blocks the fast
// path does not take included; from SC_SPLIT bytes on those have a launch of their own, which costs
// 5 us where it finds nothing, but writes them with the registers and CTAs that they need (4000 x 4000
// float32, 61 MiB: 66 us by one launch, 70 by two; stored as it is 0.29 and 0.21 ms, 0.41 by two launches
// with a list of the blocks between them).  Items of 1 and 2 bytes go by the general path.
constexpr int64_t SC_SPLIT = int64_t(64) << 20;
template <int TS>
static void scatter_launch(const Geom &g, bool all, const uint8_t *chunks, const uint8_t *cend, const BlockDesc *bd,
                           const StreamDesc *sd, const uint8_t *scratch, const uint8_t *send, void *out, int64_t ld, int *err,
                           const int *ngeneral, cudaStream_t st)
{
    const unsigned grid = (unsigned)scatter_fast_grid<TS>(g, g.nchunks * g.nblocks, all);
    if (all)
        IAB_TIMED("k_scatter_fast", st, k_scatter_fast<TS, true><<<grid, 256, 0, st>>>(
            g, chunks, cend, bd, sd, scratch, send, (uint8_t *)out, ld, err, ngeneral));
    else
        IAB_TIMED("k_scatter_fast", st, k_scatter_fast<TS, false><<<grid, 256, 0, st>>>(
            g, chunks, cend, bd, sd, scratch, send, (uint8_t *)out, ld, err, ngeneral));
}
static void scatter_launch(const Geom &g, const uint8_t *chunks, int64_t chunks_bytes, const BlockDesc *bd, const StreamDesc *sd,
                           const uint8_t *scratch, void *out, int64_t ld, int *err, const int *ngeneral, cudaStream_t st)
{
    const int64_t nbl = g.nchunks * g.nblocks;
    const uint8_t *cend = chunks + chunks_bytes, *send = scratch + nbl * g.blocksize;
    const bool fast = g.itemsize == 8 || g.itemsize == 4, all = fast && nbl * g.blocksize < SC_SPLIT;
    if (g.itemsize == 8) scatter_launch<8>(g, all, chunks, cend, bd, sd, scratch, send, out, ld, err, ngeneral, st);
    else if (g.itemsize == 4) scatter_launch<4>(g, all, chunks, cend, bd, sd, scratch, send, out, ld, err, ngeneral, st);
    if (!all) {
        const int64_t blocks = std::min<int64_t>(nbl * ceil_div(g.blockn, TILE), (int64_t)sm_count() * 8);
        IAB_TIMED("k_scatter", st, k_scatter<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, st>>>(
            g, fast ? g.itemsize : 0, chunks, bd, sd, scratch, (uint8_t *)out, ld, ngeneral));
    }
}

int decode_scatter(const DecodeArgs &a, DecodeWork *w, cudaStream_t st)
{
    int *cnt = w->ext_counters ? w->ext_counters : w->counters.as<int>();
    scatter_launch(a.g, a.chunks, a.chunks_bytes, w->bd.as<BlockDesc>(), w->sd.as<StreamDesc>(), w->scratch.as<uint8_t>(),
                   a.out, a.ld, cnt + 1, cnt + 2, st);
    return 0;
}

int decode_launch(const Geom &g, const uint8_t *d_chunks, int64_t chunks_bytes, const int64_t *d_off, const int32_t *d_len, void *out,
                  int64_t ld, cudaStream_t st, DecodeWork *w)
{
    const DecodeArgs a{g, d_chunks, chunks_bytes, d_off, d_len, out, ld};
    int r = decode_queue_init(&w->queue, decode_max_jobs(g), 1, st);
    if (!r) r = decode_parse(a, &w->queue, w, st);
    if (!r) r = decode_lz4(&w->queue, st);
    if (!r) r = decode_scatter(a, w, st);
    return r;
}

// c-blosc2's split rule for LZ4 (always / never / automatic: LZ4 + shuffle, typesize <= 16
// and at least 32 items per block); a split block has one stream per item byte.
static bool encode_split(const Geom &g, bool shuffle, int splitmode)
{
    if (splitmode == 1) return true;
    if (splitmode == 2) return false;
    return shuffle && g.itemsize <= 16 && (g.blocksize / g.itemsize) >= 32;
}

int encode_nstreams(const Geom &g, bool shuffle, int splitmode)
{
    return encode_split(g, shuffle, splitmode) ? g.itemsize : 1;
}

int encode_gather(const Geom &g, const void *in, int64_t ld, bool shuffle, int splitmode, EncodeWork *w, cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const int ts = g.itemsize;
    const int64_t nbl = g.nchunks * g.nblocks;
    const int64_t img_bytes = nbl * g.blocksize;
    const int nstreams = encode_nstreams(g, shuffle, splitmode);
    const bool ext = w->ext_img != nullptr;
    const bool ready = w->img_ready && !ext && w->img.n >= (size_t)img_bytes;
    if ((!ext && ((!ready && !w->img.allocate(img_bytes, dev)) || !w->slots.allocate(img_bytes, dev) ||
                  !w->es.allocate(sizeof(EncStream) * nbl * nstreams, dev))) ||
        (!w->ext_chunks && !w->ec.allocate(sizeof(EncChunk) * g.nchunks, dev)) || !w->tot.allocate(64, dev))
        return -100;
    w->nchunks = g.nchunks;
    uint8_t *img = ext ? w->ext_img : w->img.as<uint8_t>();
    cudaMemsetAsync(w->tot.p, 0, 64, st);
    if (ready) return 0;                   // the product wrote the image
    const int sms = sm_count();
    const int64_t tpb = (g.blockn + TILE - 1) / TILE;
    const int64_t blocks = std::min<int64_t>(nbl * tpb, (int64_t)sms * 8);
    const bool fast = shuffle && (ts == 4 || ts == 8);
    if (fast) {
        const int nt = gather_threads(g), slice = gather_slice(g, nbl, (int64_t)sms * 8);
        const int64_t fb = std::min<int64_t>(ceil_div(nbl * ceil_div(g.blockn, slice), 256 / nt), (int64_t)sms * 8);
        auto launch = [&](auto kernel) {
            IAB_TIMED("k_gather_fast", st, kernel<<<(unsigned)std::max<int64_t>(fb, 1), 256, 0, st>>>(g, (const uint8_t *)in, ld, img, slice, nt));
        };
        if (ts == 8) launch(geom_quads(g) ? k_gather_fast<8, true> : k_gather_fast<8, false>);
        else launch(geom_quads(g) ? k_gather_fast<4, true> : k_gather_fast<4, false>);
    } else {
        IAB_TIMED("k_gather", st, k_gather<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, st>>>(
            g, (const uint8_t *)in, ld, shuffle, img));
    }
    return 0;
}

void encode_streams(const uint8_t *img, int64_t ns, int per, int neblock, uint8_t *slots, EncStream *es,
                    unsigned long long *cursor, bool exact_lz4, cudaStream_t st)
{
    const int sms = sm_count();
    if (exact_lz4) {
        static bool attr = false;
        // per warp: 16 KiB hash table, lane masks, the source window; 1 warp per CTA, XCTAS per SM
        const int wpb = 1, smem = wpb * (4096 * 4 + EPEER * 4 + XRING + EMIRROR);
        if (!attr) {
            cudaFuncSetAttribute(k_lz4_encode, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            attr = true;
        }
        const int64_t blocks = std::min<int64_t>((ns + wpb - 1) / wpb, (int64_t)sms * XCTAS);
        IAB_TIMED("k_lz4_encode", st, k_lz4_encode<<<(unsigned)std::max<int64_t>(blocks, 1), wpb * 32, smem, st>>>(
            img, ns, per, neblock, slots, es, cursor));
    } else {
        static bool attr = false;
        const int smem = (int)sizeof(ParSmem);                 // one stream per CTA of PT threads, 8 CTAs per SM
        if (!attr) {
            cudaFuncSetAttribute(k_lz4_encode_par, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            attr = true;
        }
        const int64_t blocks = std::min<int64_t>(ns, (int64_t)sms * 8);
        IAB_TIMED("k_lz4_encode_par", st, k_lz4_encode_par<<<(unsigned)std::max<int64_t>(blocks, 1), PT, smem, st>>>(
            img, ns, per, neblock, slots, es, cursor));
    }
}

int encode_emit(const Geom &g, bool shuffle, int splitmode, DevBuf *d_out, EncodeWork *w, cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const int64_t nbl = g.nchunks * g.nblocks;
    const int64_t img_bytes = nbl * g.blocksize;
    const int nstreams = encode_nstreams(g, shuffle, splitmode);
    const int neblock = (int)(g.blocksize / nstreams);
    if (!d_out->allocate((size_t)(g.nchunks * (g.chunk_nbytes + 32)), dev)) return -100;
    const bool ext = w->ext_img != nullptr;
    const uint8_t *img = ext ? w->ext_img : w->img.as<uint8_t>();
    const uint8_t *slots = ext ? w->ext_slots : w->slots.as<uint8_t>();
    EncStream *es = ext ? w->ext_es : w->es.as<EncStream>();
    EncChunk *ec = w->ext_chunks ? w->ext_chunks : w->ec.as<EncChunk>();
    if (!w->d_off.allocate(sizeof(int64_t) * (size_t)std::max<int64_t>(g.nchunks, 1), dev) ||
        !w->d_len.allocate(sizeof(int32_t) * (size_t)std::max<int64_t>(g.nchunks, 1), dev))
        return -100;
    const bool own = g.nchunks <= LAYOUT_OWN;
    IAB_TIMED("k_layout", st, k_layout<<<(unsigned)std::max<int64_t>(g.nchunks, 1), LAYOUT_T, 0, st>>>(
        g, nstreams, neblock, es, ec, w->memcpy_only ? 1 : 0, w->tot.as<int64_t>(), w->d_off.as<int64_t>(),
        w->d_len.as<int32_t>(), own));
    if (!own)
        IAB_TIMED("k_chunk_offsets", st, k_chunk_offsets<<<1, 1024, 0, st>>>(g.nchunks, ec, w->tot.as<int64_t>(),
                                                                            w->d_off.as<int64_t>(), w->d_len.as<int32_t>()));
    const int nt = emit_threads(nbl * nstreams, neblock, sm_count());
    auto *emit = nt == 32 ? k_emit<32> : k_emit<256>;
    IAB_TIMED("k_emit", st, emit<<<emit_grid(nbl * nstreams, nt, sm_count()), 256, 0, st>>>(
        g, nstreams, neblock, shuffle, encode_split(g, shuffle, splitmode) ? 1 : 0, img, slots, img_bytes, es, ec,
        d_out->as<uint8_t>()));
    return 0;
}

int encode_launch(const Geom &g, const void *in, int64_t ld, bool shuffle, int splitmode, DevBuf *d_out, EncodeWork *w,
                  cudaStream_t st)
{
    w->ext_img = nullptr;
    w->ext_slots = nullptr;
    w->ext_es = nullptr;
    const int r = encode_gather(g, in, ld, shuffle, splitmode, w, st);
    if (r) return r;
    const int nstreams = encode_nstreams(g, shuffle, splitmode);
    if (!w->memcpy_only)
        encode_streams(w->img.as<uint8_t>(), g.nchunks * g.nblocks * nstreams, nstreams, (int)(g.blocksize / nstreams),
                       w->slots.as<uint8_t>(), w->es.as<EncStream>(),
                       reinterpret_cast<unsigned long long *>(w->tot.as<int64_t>() + 1), w->exact_lz4, st);
    return encode_emit(g, shuffle, splitmode, d_out, w, st);
}

int encode_finish(EncodeWork *w, std::vector<int64_t> *h_off, std::vector<int32_t> *h_len, cudaStream_t st)
{
    const int64_t n = w->nchunks;
    std::vector<EncChunk> hc((size_t)n);
    const EncChunk *ec = w->ext_chunks ? w->ext_chunks : w->ec.as<EncChunk>();
    cudaMemcpyAsync(hc.data(), ec, sizeof(EncChunk) * n, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return -101;
    h_off->resize((size_t)n);
    h_len->resize((size_t)n);
    for (int64_t c = 0; c < n; c++) { (*h_off)[c] = hc[c].offset; (*h_len)[c] = hc[c].cbytes; }
    return 0;
}

bool encode_image_ok(const Geom &g, bool shuffle, bool memcpy_only)
{
    return g.ndim == 2 && g.itemsize == 8 && shuffle && !memcpy_only && g.nchunks > 0 && !(g.block[1] & 3) &&
           !(g.chunk[1] & 3) && g.blocksize > 0;
}

int encode_image_prepare(const Geom &g, EncodeWork *w)
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (!w->img.allocate((size_t)(g.nchunks * g.nblocks * g.blocksize), dev)) return -100;
    w->img_ready = true;
    return 0;
}

int encode_image_finish(const Geom &g, bool shuffle, int splitmode, DevBuf *d_out, std::vector<int64_t> *h_off,
                        std::vector<int32_t> *h_len, cudaStream_t st, EncodeWork *w)
{
    if (!w->img_ready) return -1;
    w->memcpy_only = false;
    return encode_container(g, nullptr, 0, shuffle, splitmode, d_out, h_off, h_len, st, w);
}

int encode_container(const Geom &g, const void *in, int64_t ld, bool shuffle, int splitmode, DevBuf *d_out,
                     std::vector<int64_t> *h_off, std::vector<int32_t> *h_len, cudaStream_t st, EncodeWork *w)
{
    const int r = encode_launch(g, in, ld, shuffle, splitmode, d_out, w, st);
    if (r) return r;
    return encode_finish(w, h_off, h_len, st);
}

// ============================================================================ decode-fused GEMV
// y = A x straight from A's chunks, after the parse and the LZ4 launch: the dense A is never
// written.  A unit is one slice of whole rows of one block (SC_ITEMS / block[1] rows): its items
// are rebuilt as the scatter rebuilds them (word-level from the staged byte planes for shuffled
// split blocks, item by item from the stream descriptors otherwise), multiplied by x over the
// block's columns, and each row's sum is stored in part[jb * M + row] (jb: the block's column in
// the global block grid); k_gemv_rows then sums part over jb in order.  Every sum runs in a fixed
// order, so the result does not vary from run to run.

// Item i of a block from its stream descriptors (any block mode).
__device__ __forceinline__ uint64_t item_bits(const Geom &g, const uint8_t *__restrict__ ch, const BlockDesc &d,
                                              const StreamDesc *__restrict__ s, const uint8_t *__restrict__ blk_scratch,
                                              int64_t i)
{
    const int ts = g.itemsize;
    if (d.mode == BM_NAN) return ts == 8 ? 0x7FF8000000000000ull : 0x7FC00000ull;
    if (d.mode == BM_VALUE) return load_item_bytes(ch + d.value_src, ts);
    uint64_t v = 0;
    for (int j = 0; j < ts; j++) {
        const int64_t pos = d.mode == BM_SHUFFLED ? (int64_t)j * g.blockn + i : i * ts + j;
        const int sidx = (int)(pos / d.neblock);
        const int64_t so = pos - (int64_t)sidx * d.neblock;
        const StreamDesc q = s[sidx];
        uint8_t b;
        if (q.kind == SK_RUN) b = (uint8_t)q.len;
        else if (q.kind == SK_RAW) b = __ldg(ch + q.src + so);
        else b = __ldcg(blk_scratch + (int64_t)sidx * d.neblock + so);
        v |= (uint64_t)b << (8 * j);
    }
    return v;
}

template <typename T> __device__ __forceinline__ T bits_as(uint64_t v);
template <> __device__ __forceinline__ float bits_as<float>(uint64_t v) { return __uint_as_float((uint32_t)v); }
template <> __device__ __forceinline__ double bits_as<double>(uint64_t v) { return __longlong_as_double((long long)v); }

// One unit of the fused GEMV: one slice of whole rows of one block (block-uniform values).
struct GvUnit {
    int64_t t, jb;
    BlockSpan sp;
    BlockDesc d;
    int r0, nrow, i0s, cnt;
    bool active, fast;         // active: the slice holds logical items; fast: word-level path
};

__device__ __forceinline__ GvUnit gv_unit(const Geom &g, const BlockDesc *__restrict__ bd, int64_t u, int64_t nsl,
                                          int rps, int ts)
{
    GvUnit w;
    int64_t s64, c, b, cq, cr, bq, br;
    divmod(u, nsl, w.t, s64);
    divmod(w.t, g.nblocks, c, b);
    w.sp = block_span(g, c, b);
    w.r0 = (int)s64 * rps;
    w.active = w.sp.nc > 0 && w.r0 < w.sp.nr;
    w.nrow = w.active ? min(rps, w.sp.nr - w.r0) : 0;
    w.i0s = w.r0 * (int)g.block[1];
    w.cnt = w.nrow * (int)g.block[1];
    w.d = bd[w.t];
    w.fast = w.d.mode == BM_SHUFFLED && w.d.nstreams == ts;
    divmod(c, g.cgrid[1], cq, cr);
    divmod(b, g.bgrid[1], bq, br);
    w.jb = cr * g.bgrid[1] + br;
    return w;
}

// Plane j of a fast unit: its slice starts at src (nullptr for a run), 16-byte word a16 =
// src - shift; the bulk copy takes the whole words of [a16, a16 + want) before the buffer end
// lim, threads copy the bytes that the buffer end cuts off (zeros past it).
__device__ __forceinline__ StreamDesc gv_plane(const Geom &g, const uint8_t *ch, const uint8_t *ch_end,
                                               const StreamDesc *__restrict__ sd, const uint8_t *scratch,
                                               const uint8_t *scratch_end, const GvUnit &w, int j,
                                               const uint8_t *&src, const uint8_t *&lim, int &want, int &bulk)
{
    const StreamDesc q = sd[w.t * 8 + j];
    src = nullptr; lim = nullptr;
    if (q.kind == SK_RAW) { src = ch + q.src + w.i0s; lim = ch_end; }
    else if (q.kind == SK_LZ4) { src = scratch + w.t * g.blocksize + (int64_t)j * w.d.neblock + w.i0s; lim = scratch_end; }
    want = bulk = 0;
    if (src) {
        const uint8_t *a16 = src - (reinterpret_cast<uintptr_t>(src) & 15);
        want = ((int)(src - a16) + w.cnt + 15) & ~15;
        bulk = (int)min((int64_t)want, (lim - a16) & ~int64_t(15));
    }
    return q;
}

template <int TS, typename T>
__global__ void __launch_bounds__(256, 4) k_scatter_gemv(Geom g, const uint8_t *__restrict__ ch, const uint8_t *ch_end,
                                                      const BlockDesc *__restrict__ bd,
                                                      const StreamDesc *__restrict__ sd,
                                                      const uint8_t *__restrict__ scratch, const uint8_t *scratch_end,
                                                      const T *__restrict__ x, T *__restrict__ part, int64_t M,
                                                      int *err)
{
    __shared__ __align__(128) uint8_t stage[TS][SC_PLANE];
    __shared__ T qsum[SC_ITEMS / 4];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_all;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
        abort_all = 0;
    }
    __syncthreads();
    const int qpr = (int)(g.block[1] / 4);
    const int rps = (int)(SC_ITEMS / g.block[1]);            // whole rows per slice (>= 1: checked by the host)
    const int64_t nsl = (g.block[0] + rps - 1) / rps;
    const int64_t total = g.nchunks * g.nblocks * nsl;
    uint32_t parity = 0;
    for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {          // block-uniform loop
        const GvUnit w = gv_unit(g, bd, u, nsl, rps, TS);
        if (!w.active) continue;                              // padding only
        const T *__restrict__ xb = x + w.sp.col0;
        if (w.fast) {
            if (tid == 0) {
                uint32_t tx = 0;
#pragma unroll
                for (int j = 0; j < TS; j++) {
                    const uint8_t *src, *lim;
                    int want, bulk;
                    gv_plane(g, ch, ch_end, sd, scratch, scratch_end, w, j, src, lim, want, bulk);
                    tx += (uint32_t)bulk;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // earlier reads of stage precede the copies
                tc::mbar_arrive_expect_tx(&bar, tx);
#pragma unroll
                for (int j = 0; j < TS; j++) {
                    const uint8_t *src, *lim;
                    int want, bulk;
                    gv_plane(g, ch, ch_end, sd, scratch, scratch_end, w, j, src, lim, want, bulk);
                    if (bulk > 0) bulk_g2s(stage[j], src - (reinterpret_cast<uintptr_t>(src) & 15), (uint32_t)bulk, &bar);
                }
            }
            int code[TS];
#pragma unroll
            for (int j = 0; j < TS; j++) {
                const uint8_t *src, *lim;
                int want, bulk;
                const StreamDesc q = gv_plane(g, ch, ch_end, sd, scratch, scratch_end, w, j, src, lim, want, bulk);
                code[j] = src ? (int)(reinterpret_cast<uintptr_t>(src) & 15) : 256 + (q.kind == SK_RUN ? (q.len & 255) : 0);
                if (bulk < want) {
                    const uint8_t *a16 = src - code[j];
                    for (int xx = bulk + tid; xx < want; xx += blockDim.x)
                        stage[j][xx] = a16 + xx < lim ? __ldg(a16 + xx) : (uint8_t)0;
                }
            }
            const bool ok = sc_wait(&bar, parity);
            parity ^= 1;
            if (!ok) abort_all = 1;
            __syncthreads();
            if (abort_all) {                                  // the copies did not complete: report, wait once more, leave
                if (tid == 0) {
                    dev_fail(err, DE_WAIT);
                    sc_wait(&bar, parity ^ 1);
                }
                return;
            }
            const int step_r = (int)blockDim.x / qpr, step_q = (int)blockDim.x - step_r * qpr;
            int q = tid - (tid / qpr) * qpr;
            for (int qd = tid; qd < w.cnt / 4; qd += blockDim.x, q += step_q) {
                if (q >= qpr) q -= qpr;
                const int cc = q * 4;
                T sum = 0;
                if (cc < w.sp.nc) {
                    uint32_t wd[TS];
#pragma unroll
                    for (int j = 0; j < TS; j++) {
                        if (code[j] >= 256) { wd[j] = (uint32_t)(code[j] - 256) * 0x01010101u; continue; }
                        const uint32_t *pw = reinterpret_cast<const uint32_t *>(stage[j]);
                        const int byte = code[j] + qd * 4, wi = byte >> 2, sh = (byte & 3) * 8;
                        wd[j] = sh ? __funnelshift_r(pw[wi], pw[wi + 1], sh) : pw[wi];
                    }
                    uint32_t v[4];
                    transpose4x4(wd[0], wd[1], wd[2], wd[3], v[0], v[1], v[2], v[3]);
                    uint64_t item[4];
                    if constexpr (TS == 8) {
                        uint32_t h[4];
                        transpose4x4(wd[4], wd[5], wd[6], wd[7], h[0], h[1], h[2], h[3]);
#pragma unroll
                        for (int k = 0; k < 4; k++) item[k] = ((uint64_t)h[k] << 32) | v[k];
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; k++) item[k] = v[k];
                    }
                    const T *xq = xb + cc;
                    if (cc + 4 <= w.sp.nc && (reinterpret_cast<uintptr_t>(xq) & 15) == 0) {
                        T xv[4];
                        if constexpr (TS == 8) {
                            const double2 x0 = __ldg(reinterpret_cast<const double2 *>(xq));
                            const double2 x1 = __ldg(reinterpret_cast<const double2 *>(xq) + 1);
                            xv[0] = x0.x; xv[1] = x0.y; xv[2] = x1.x; xv[3] = x1.y;
                        } else {
                            const float4 x0 = __ldg(reinterpret_cast<const float4 *>(xq));
                            xv[0] = x0.x; xv[1] = x0.y; xv[2] = x0.z; xv[3] = x0.w;
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++) sum = fma(bits_as<T>(item[k]), xv[k], sum);
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (cc + k < w.sp.nc) sum = fma(bits_as<T>(item[k]), xq[k], sum);
                    }
                }
                qsum[qd] = sum;
            }
        } else {
            const StreamDesc *s = sd + w.t * 8;
            const uint8_t *bs = scratch + w.t * g.blocksize;
            for (int qd = tid; qd < w.cnt / 4; qd += blockDim.x) {
                const int cc = (qd % qpr) * 4;
                T sum = 0;
                for (int k = 0; k < 4; k++)
                    if (cc + k < w.sp.nc)
                        sum = fma(bits_as<T>(item_bits(g, ch, w.d, s, bs, w.i0s + qd * 4 + k)), xb[cc + k], sum);
                qsum[qd] = sum;
            }
        }
        __syncthreads();
        // row sums: warp w takes rows w, w + 8, ...; lanes stride the row's quads, then a shuffle tree
        for (int rr = warp; rr < w.nrow; rr += blockDim.x / 32) {
            T acc = 0;
            for (int q = lane; q < qpr; q += 32) acc += qsum[rr * qpr + q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(FULLMASK, acc, o);
            if (lane == 0) part[w.jb * M + w.sp.row0 + w.r0 + rr] = acc;
        }
        __syncthreads();                                  // stage and qsum are read before the next slice
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_gemv_rows(const T *__restrict__ part, int64_t JB, int64_t M, T *__restrict__ y)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (int64_t)gridDim.x * blockDim.x) {
        T acc = 0;
        for (int64_t jb = 0; jb < JB; jb++) acc += part[jb * M + i];
        y[i] = acc;
    }
}

bool decode_gemv_fits(const Geom &g)
{
    return g.ndim == 2 && (g.itemsize == 4 || g.itemsize == 8) && !(g.block[1] & 3) && g.block[1] <= SC_ITEMS &&
           g.block[1] > 0;
}

int64_t decode_gemv_part_items(const Geom &g) { return g.cgrid[1] * g.bgrid[1] * g.shape[0]; }

int decode_gemv(const DecodeArgs &a, DecodeWork *w, const void *x, void *part, void *y, cudaStream_t st)
{
    const Geom &g = a.g;
    if (!decode_gemv_fits(g)) return -102;
    const int64_t M = g.shape[0], JB = g.cgrid[1] * g.bgrid[1], nbl = g.nchunks * g.nblocks;
    cudaMemsetAsync(part, 0, (size_t)(JB * M * g.itemsize), st);
    int *cnt = w->ext_counters ? w->ext_counters : w->counters.as<int>();
    const uint8_t *scratch = w->scratch.as<uint8_t>();
    const uint8_t *cend = a.chunks + a.chunks_bytes, *send = scratch + nbl * g.blocksize;
    const int rps = (int)(SC_ITEMS / g.block[1]);
    const int64_t units = nbl * ((g.block[0] + rps - 1) / rps);
    static int per_sm[2] = {0, 0};
    const int slot = g.itemsize == 8;
    if (!per_sm[slot]) {
        int m = 0;
        const cudaError_t e = slot ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_scatter_gemv<8, double>, 256, 0)
                                   : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_scatter_gemv<4, float>, 256, 0);
        if (e != cudaSuccess || m < 1) { cudaGetLastError(); m = 4; }
        per_sm[slot] = m;
    }
    const int64_t grid = std::max<int64_t>(std::min<int64_t>(units, (int64_t)sm_count() * per_sm[slot]), 1);
    const unsigned rb = (unsigned)std::max<int64_t>(std::min<int64_t>((M + 255) / 256, (int64_t)sm_count() * 8), 1);
    if (slot) {
        IAB_TIMED("k_scatter_gemv", st, k_scatter_gemv<8, double><<<(unsigned)grid, 256, 0, st>>>(
            g, a.chunks, cend, w->bd.as<BlockDesc>(), w->sd.as<StreamDesc>(), scratch, send, (const double *)x,
            (double *)part, M, cnt + 1));
        IAB_TIMED("k_gemv_rows", st, k_gemv_rows<double><<<rb, 256, 0, st>>>((const double *)part, JB, M, (double *)y));
    } else {
        IAB_TIMED("k_scatter_gemv", st, k_scatter_gemv<4, float><<<(unsigned)grid, 256, 0, st>>>(
            g, a.chunks, cend, w->bd.as<BlockDesc>(), w->sd.as<StreamDesc>(), scratch, send, (const float *)x,
            (float *)part, M, cnt + 1));
        IAB_TIMED("k_gemv_rows", st, k_gemv_rows<float><<<rb, 256, 0, st>>>((const float *)part, JB, M, (float *)y));
    }
    return 0;
}

// ============================================================================ grouped codec
// Largest k with start[k] <= u (containers with no units share their start with the next).
__device__ __forceinline__ int group_find(const int64_t *__restrict__ start, int n, int64_t u)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(start + mid) <= u) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__global__ void k_group_reset(const CodecItem *__restrict__ items, int n)
{
    const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (x < (int64_t)n * 16) items[x >> 4].cnt[x & 15] = 0;
}

__global__ void __launch_bounds__(PARSE_T) k_parse_g(const CodecItem *__restrict__ items, const int64_t *__restrict__ bstart,
                                                     int n, int64_t nbl, Lz4Job *jobs, int *njobs, int64_t jcap)
{
    for (int64_t u0 = (int64_t)blockIdx.x * (PARSE_T / 8); u0 < nbl; u0 += (int64_t)gridDim.x * (PARSE_T / 8)) {
        const int64_t u = u0 + threadIdx.x / 8;
        const bool valid = u < nbl;
        const int k = group_find(bstart, n, valid ? u : nbl - 1);
        const CodecItem &it = items[k];
        const int64_t t = u - bstart[k];
        ParsedStream ps;
        parse_block(it.g, it.ch, it.off, it.len, it.bd, it.sd, it.cnt + 1, nullptr, nullptr, t, valid, ps);
        queue_streams(ps, it.scratch + t * it.g.blocksize, it.cnt + 1, jobs, njobs, jcap);
    }
}

template <int TS>
__global__ void __launch_bounds__(256, 4) k_scatter_fast_g(const CodecItem *__restrict__ items,
                                                        const int64_t *__restrict__ sstart, int n, int64_t nsf)
{
    __shared__ __align__(128) uint8_t stage[TS][SC_PLANE];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_all;
    const int tid = threadIdx.x;
    if (tid == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
        abort_all = 0;
    }
    __syncthreads();
    uint32_t parity = 0;
    bool general = false;
    for (int64_t u = blockIdx.x; u < nsf; u += gridDim.x) {
        const int k = group_find(sstart, n, u);
        const CodecItem &it = items[k];
        const int64_t nsl = (it.g.blockn + SC_ITEMS - 1) / SC_ITEMS;
        const int64_t lu = u - sstart[k], t = lu / nsl;
        const int sl = (int)(lu - t * nsl);
        const int64_t nbk = it.g.nchunks * it.g.nblocks;
        if (!scatter_fast_unit<TS>(it.g, it.ch, it.ch + it.ch_bytes, it.bd, it.sd, it.scratch,
                                   it.scratch + nbk * it.g.blocksize, it.dense, it.ld, it.cnt + 1, t, sl, stage, &bar, parity, &abort_all,
                                   general))
            return;
    }
    for (int64_t u = blockIdx.x; general && u < nsf; u += gridDim.x) {      // as in k_scatter_fast
        const int k = group_find(sstart, n, u);
        const CodecItem &it = items[k];
        int64_t t, sl;
        divmod(u - sstart[k], (it.g.blockn + SC_ITEMS - 1) / SC_ITEMS, t, sl);
        if (it.bd[t].mode == BM_SHUFFLED && it.bd[t].nstreams == TS) continue;
        const int64_t end = min(it.g.blockn, (sl + 1) * SC_ITEMS);
        for (int64_t i0 = sl * SC_ITEMS; i0 < end; i0 += TILE)
            scatter_tile(it.g, it.ch, it.bd, it.sd, it.scratch, it.dense, it.ld, t, i0, stage[0]);
    }
}

// (The group's blocks are of one size: `nsl` slices of `slice` items a block, `nt` threads a slice.)
template <int TS>
__global__ void __launch_bounds__(256) k_gather_fast_g(const CodecItem *__restrict__ items,
                                                       const int64_t *__restrict__ bstart, int n, int64_t nu, int nsl,
                                                       int slice, int nt)
{
    const int per = 256 / nt, tid = threadIdx.x & (nt - 1);
    for (int64_t u = (int64_t)blockIdx.x * per + threadIdx.x / nt; u < nu; u += (int64_t)gridDim.x * per) {
        int64_t gb, sl;
        divmod(u, nsl, gb, sl);
        const int k = group_find(bstart, n, gb);
        const CodecItem &it = items[k];
        const int i0 = (int)sl * slice, cnt = (int)min((int64_t)slice, it.g.blockn - i0);
        if (geom_quads(it.g)) gather_fast_block<TS, true>(it.g, it.dense, it.ld, it.img, gb - bstart[k], i0, cnt, tid, nt);
        else gather_fast_block<TS, false>(it.g, it.dense, it.ld, it.img, gb - bstart[k], i0, cnt, tid, nt);
    }
}

__global__ void __launch_bounds__(LAYOUT_T) k_layout_g(const CodecItem *__restrict__ items,
                                                      const int64_t *__restrict__ cstart, int n, int nstreams,
                                                      int neblock, int memcpy_only)
{
    __shared__ int64_t wsum[LAYOUT_T / 32];
    __shared__ int64_t s_before;
    __shared__ int s_first;
    const int64_t u = blockIdx.x;
    const int k = group_find(cstart, n, u);
    const CodecItem &it = items[k];
    layout_chunk(it.g, nstreams, neblock, it.es, it.ec, memcpy_only, u - cstart[k], wsum, s_before, s_first);
}

__global__ void __launch_bounds__(1024) k_chunk_offsets_g(CodecItem *items)
{
    __shared__ int64_t wsum[32];
    CodecItem &it = items[blockIdx.x];
    chunk_offsets<1>(it.g.nchunks, it.ec, &it.out_bytes, nullptr, nullptr, wsum);
}

template <int NT>
__global__ void __launch_bounds__(256) k_emit_g(const CodecItem *__restrict__ items, const int64_t *__restrict__ bstart,
                                                int n, int64_t nbl, int nstreams, int neblock, bool shuffle, int splitflag)
{
    constexpr int per = 256 / NT;
    for (int64_t u = (int64_t)blockIdx.x * per + threadIdx.x / NT; u < nbl * nstreams; u += (int64_t)gridDim.x * per) {
        int64_t t, j;
        divmod(u, nstreams, t, j);
        const int k = group_find(bstart, n, t);
        const CodecItem &it = items[k];
        const int64_t img_bytes = it.g.nchunks * it.g.nblocks * it.g.blocksize;
        emit_block(it.g, nstreams, neblock, shuffle, splitflag, it.img, it.slots, img_bytes, it.es, it.ec, it.outbuf,
                   t - bstart[k], (int)j, threadIdx.x % NT, NT);
    }
}

// Start tables (blocks, fast-scatter slices, chunks; n + 1 entries each) and the item table
// on the device.  Synchronises `st` (setup only, before any capture).
static int group_upload(CodecGroup *grp, cudaStream_t st)
{
    const int n = grp->n;
    int dev = 0;
    cudaGetDevice(&dev);
    std::vector<int64_t> s(3 * (size_t)(n + 1), 0);
    for (int k = 0; k < n; k++) {
        const Geom &g = grp->h[(size_t)k].g;
        const int64_t nbl = g.nchunks * g.nblocks;
        s[(size_t)k + 1] = s[(size_t)k] + nbl;
        s[(size_t)(n + 1) + k + 1] = s[(size_t)(n + 1) + k] + nbl * ((g.blockn + SC_ITEMS - 1) / SC_ITEMS);
        s[(size_t)(2 * (n + 1)) + k + 1] = s[(size_t)(2 * (n + 1)) + k] + g.nchunks;
    }
    grp->nbl = s[(size_t)n];
    grp->nsf = s[(size_t)(2 * n + 1)];
    grp->nch = s[(size_t)(3 * n + 2)];
    if (grp->nbl > INT32_MAX) return -102;
    if (!grp->items.allocate(sizeof(CodecItem) * (size_t)n, dev) || !grp->starts.allocate(sizeof(int64_t) * s.size(), dev))
        return -100;
    cudaMemcpyAsync(grp->items.p, grp->h.data(), sizeof(CodecItem) * (size_t)n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(grp->starts.p, s.data(), sizeof(int64_t) * s.size(), cudaMemcpyHostToDevice, st);
    return cudaStreamSynchronize(st) == cudaSuccess ? 0 : -101;
}

int decode_group_setup(const std::vector<DecodeArgs> &a, const std::vector<int *> &cnt, CodecGroup *grp, cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const int n = (int)a.size();
    if (n <= 0 || cnt.size() != a.size()) return -102;
    grp->n = n;
    grp->ts = a[0].g.itemsize;
    if (grp->ts != 4 && grp->ts != 8) return -102;
    int64_t nbl = 0, img = 0, jobs = 0;
    for (const DecodeArgs &x : a) {
        if (x.g.itemsize != grp->ts) return 1;
        nbl += x.g.nchunks * x.g.nblocks;
        img += x.g.nchunks * x.g.nblocks * x.g.blocksize;
        jobs += decode_max_jobs(x.g);
    }
    if (!grp->bd.allocate(sizeof(BlockDesc) * (size_t)std::max<int64_t>(nbl, 1), dev) ||
        !grp->sd.allocate(sizeof(StreamDesc) * 8 * (size_t)std::max<int64_t>(nbl, 1), dev) ||
        !grp->scratch.allocate((size_t)std::max<int64_t>(img, 16), dev))
        return -100;
    int r = decode_queue_init(&grp->q, jobs, 0, st);
    if (r) return r;
    grp->h.assign((size_t)n, CodecItem{});
    int64_t bo = 0, io = 0;
    for (int k = 0; k < n; k++) {
        const DecodeArgs &x = a[(size_t)k];
        CodecItem &it = grp->h[(size_t)k];
        it.g = x.g;
        it.ch = x.chunks; it.ch_bytes = x.chunks_bytes; it.off = x.off; it.len = x.len;
        it.bd = grp->bd.as<BlockDesc>() + bo;
        it.sd = grp->sd.as<StreamDesc>() + bo * 8;
        it.scratch = grp->scratch.as<uint8_t>() + io;
        it.dense = static_cast<uint8_t *>(x.out);
        it.ld = x.ld;
        it.cnt = cnt[(size_t)k];
        bo += x.g.nchunks * x.g.nblocks;
        io += x.g.nchunks * x.g.nblocks * x.g.blocksize;
    }
    return group_upload(grp, st);
}

int decode_group_launch(CodecGroup *grp, cudaStream_t st)
{
    const int n = grp->n, sms = sm_count();
    const CodecItem *items = grp->items.as<CodecItem>();
    const int64_t *bstart = grp->starts.as<int64_t>(), *sstart = bstart + (n + 1);
    cudaMemsetAsync(grp->q.counters.p, 0, 64, st);
    IAB_TIMED("k_group_reset", st, k_group_reset<<<(unsigned)((n * 16 + 255) / 256), 256, 0, st>>>(items, n));
    if (grp->nbl == 0) return 0;
    IAB_TIMED("k_parse", st, k_parse_g<<<parse_grid(grp->nbl, sms), PARSE_T, 0, st>>>(items, bstart, n, grp->nbl, grp->q.jobs.as<Lz4Job>(),
                                                                     grp->q.counters.as<int>(), grp->q.cap));
    int r = decode_lz4(&grp->q, st);
    if (r) return r;
    static int per_sm[2] = {0, 0};
    const int slot = grp->ts == 8;
    if (!per_sm[slot]) {
        int m = 0;
        const cudaError_t e = slot ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_scatter_fast_g<8>, 256, 0)
                                   : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_scatter_fast_g<4>, 256, 0);
        if (e != cudaSuccess || m < 1) { cudaGetLastError(); m = 4; }
        per_sm[slot] = m;
    }
    const int64_t grid = std::max<int64_t>(std::min<int64_t>(grp->nsf, (int64_t)sms * per_sm[slot]), 1);
    if (slot)
        IAB_TIMED("k_scatter_fast", st, k_scatter_fast_g<8><<<(unsigned)grid, 256, 0, st>>>(
            items, sstart, n, grp->nsf));
    else
        IAB_TIMED("k_scatter_fast", st, k_scatter_fast_g<4><<<(unsigned)grid, 256, 0, st>>>(
            items, sstart, n, grp->nsf));
    return 0;
}

int encode_group_setup(const std::vector<Geom> &g, const std::vector<const void *> &dense, const std::vector<int64_t> &ld,
                       const std::vector<EncChunk *> &ec, std::vector<DevBuf> *out, CodecGroup *grp, cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const int n = (int)g.size();
    if (n <= 0 || dense.size() != g.size() || ld.size() != g.size() || ec.size() != g.size() || out->size() != g.size())
        return -102;
    grp->n = n;
    grp->ts = g[0].itemsize;
    if (grp->ts != 4 && grp->ts != 8) return -102;
    grp->shuffle = true;
    grp->nstreams = encode_nstreams(g[0], true, 3 /* automatic split */);
    grp->split = encode_split(g[0], true, 3);
    grp->neblock = (int)(g[0].blocksize / grp->nstreams);
    int64_t img = 0, ns = 0;
    for (const Geom &x : g) {
        const int nsx = encode_nstreams(x, true, 3);
        if (x.itemsize != grp->ts || nsx != grp->nstreams || x.blocksize / nsx != grp->neblock ||
            encode_split(x, true, 3) != grp->split)
            return 1;
        img += x.nchunks * x.nblocks * x.blocksize;
        ns += x.nchunks * x.nblocks * nsx;
    }
    if (!grp->img.allocate((size_t)std::max<int64_t>(img, 16), dev) || !grp->slots.allocate((size_t)std::max<int64_t>(img, 16), dev) ||
        !grp->es.allocate(sizeof(EncStream) * (size_t)std::max<int64_t>(ns, 1), dev) || !grp->counters.allocate(128, dev))
        return -100;
    grp->h.assign((size_t)n, CodecItem{});
    int64_t io = 0, so = 0;
    for (int k = 0; k < n; k++) {
        const Geom &x = g[(size_t)k];
        if (!(*out)[(size_t)k].allocate((size_t)std::max<int64_t>(x.nchunks * (x.chunk_nbytes + 32), 16), dev)) return -100;
        CodecItem &it = grp->h[(size_t)k];
        it.g = x;
        it.dense = const_cast<uint8_t *>(static_cast<const uint8_t *>(dense[(size_t)k]));
        it.ld = ld[(size_t)k];
        it.img = grp->img.as<uint8_t>() + io;
        it.slots = grp->slots.as<uint8_t>() + io;
        it.es = grp->es.as<EncStream>() + so;
        it.ec = ec[(size_t)k];
        it.outbuf = (*out)[(size_t)k].as<uint8_t>();
        io += x.nchunks * x.nblocks * x.blocksize;
        so += x.nchunks * x.nblocks * grp->nstreams;
    }
    return group_upload(grp, st);
}

int encode_group_launch(CodecGroup *grp, bool exact_lz4, bool memcpy_only, cudaStream_t st)
{
    const int n = grp->n, sms = sm_count(), ts = grp->ts;
    CodecItem *items = grp->items.as<CodecItem>();
    const int64_t *bstart = grp->starts.as<int64_t>(), *cstart = bstart + 2 * (n + 1);
    if (grp->nbl == 0) return 0;
    cudaMemsetAsync(grp->counters.p, 0, 128, st);
    if (!grp->img_ready) {
        const int slice = gather_slice(grp->h[0].g, grp->nbl, (int64_t)sms * 8);
        const int64_t nsl = ceil_div(grp->h[0].g.blockn, slice), nu = grp->nbl * nsl;
        int nt = 32;                              // as many as the group's widest need (rows of whole quads or not)
        for (const CodecItem &it : grp->h) nt = std::max(nt, gather_threads(it.g));
        const unsigned gb = (unsigned)std::min<int64_t>(ceil_div(nu, 256 / nt), (int64_t)sms * 8);
        if (ts == 8)
            IAB_TIMED("k_gather_fast", st, k_gather_fast_g<8><<<gb, 256, 0, st>>>(items, bstart, n, nu, (int)nsl, slice, nt));
        else
            IAB_TIMED("k_gather_fast", st, k_gather_fast_g<4><<<gb, 256, 0, st>>>(items, bstart, n, nu, (int)nsl, slice, nt));
    }
    if (!memcpy_only)
        encode_streams(grp->img.as<uint8_t>(), grp->nbl * grp->nstreams, grp->nstreams, grp->neblock, grp->slots.as<uint8_t>(),
                       grp->es.as<EncStream>(), reinterpret_cast<unsigned long long *>(grp->counters.as<uint8_t>() + 64),
                       exact_lz4, st);
    IAB_TIMED("k_layout", st, k_layout_g<<<(unsigned)std::max<int64_t>(grp->nch, 1), LAYOUT_T, 0, st>>>(
        items, cstart, n, grp->nstreams, grp->neblock, memcpy_only ? 1 : 0));
    IAB_TIMED("k_chunk_offsets", st, k_chunk_offsets_g<<<(unsigned)n, 1024, 0, st>>>(items));
    const int nt = emit_threads(grp->nbl * grp->nstreams, grp->neblock, sms);
    auto *emit = nt == 32 ? k_emit_g<32> : k_emit_g<256>;
    IAB_TIMED("k_emit", st, emit<<<emit_grid(grp->nbl * grp->nstreams, nt, sms), 256, 0, st>>>(
        items, bstart, n, grp->nbl, grp->nstreams, grp->neblock, grp->shuffle, grp->split ? 1 : 0));
    return 0;
}

// ============================================================================ decode without allocation
// For callers that cannot call cudaMalloc: engines whose device memory belongs to their own
// arena or memory-budget manager and that hand the library only buffers they already hold,
// and latency-bound loops that must not pay the device synchronisation of cudaMalloc and
// cudaFree.  decode_noalloc runs the same kernels as decode_launch, but its work buffers (chunk
// index, block and stream descriptors, LZ4 jobs, the decoded-stream image and the
// status counters) live in one file-scope device array instead of pool allocations.
// The array is part of the library's device image: every GPU on which the library's
// kernels are loaded holds it until the process exits, and every call shares it, so
// calls whose kernels overlap on the GPU (two streams, two host threads) race on it.
constexpr int64_t NA_MAX_BLOCKS = NOALLOC_MAX_BLOCKS;
constexpr size_t na_align(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t NA_COUNTERS = 0;
constexpr size_t NA_OFF = 256;
constexpr size_t NA_LEN = na_align(NA_OFF + sizeof(int64_t) * NA_MAX_BLOCKS);
constexpr size_t NA_BD = na_align(NA_LEN + sizeof(int32_t) * NA_MAX_BLOCKS);
constexpr size_t NA_SD = na_align(NA_BD + sizeof(BlockDesc) * NA_MAX_BLOCKS);
constexpr size_t NA_JOBS = na_align(NA_SD + sizeof(StreamDesc) * 8 * NA_MAX_BLOCKS);
constexpr size_t NA_IMG = na_align(NA_JOBS + sizeof(Lz4Job) * 8 * NA_MAX_BLOCKS);
constexpr size_t NA_TOTAL = NA_IMG + (size_t)NOALLOC_MAX_BYTES;

static __device__ __align__(256) uint8_t g_noalloc_scratch[NA_TOTAL];

// Chunk index of back-to-back chunks: one thread walks the headers (cbytes at byte 12).
// A header that does not fit the buffer yields length 0, which the parse kernel reports
// as a header error.
__global__ void k_chunk_walk(const uint8_t *__restrict__ ch, int64_t bytes, int64_t n, int64_t *off, int32_t *len)
{
    if (blockIdx.x || threadIdx.x) return;
    int64_t pos = 0;
    for (int64_t c = 0; c < n; c++) {
        int32_t cb = 0;
        if (pos + 32 <= bytes) {
            cb = ld_s32(ch + pos + 12);
            if (cb < 32 || (int64_t)cb > bytes - pos) cb = 0;
        }
        off[c] = pos;
        len[c] = cb;
        pos = cb ? pos + cb : bytes;
    }
}

// Device address of g_noalloc_scratch on the current device.  The first call on a device
// looks the address up (the symbol's host name is only a stand-in, not a device address)
// and sets the decoder's shared-memory attribute; later calls reuse the cached address.
static uint8_t *noalloc_scratch()
{
    constexpr int MAXDEV = 64;
    static std::mutex mu;
    static uint8_t *ptr[MAXDEV] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAXDEV) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!ptr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) { cudaGetLastError(); return nullptr; }
        if (cudaFuncSetAttribute(k_lz4_decode_cta, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(dcta::Smem)) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        ptr[dev] = static_cast<uint8_t *>(p);
    }
    return ptr[dev];
}

int decode_noalloc(const Geom &g, const uint8_t *d_chunks, int64_t chunks_bytes, void *out, int64_t ld, cudaStream_t st)
{
    if (!noalloc_fits(g)) return -102;
    const int64_t nbl = g.nchunks * g.nblocks;
    if (nbl == 0) return 0;
    uint8_t *base = noalloc_scratch();
    if (!base) return -101;
    int *counters = reinterpret_cast<int *>(base + NA_COUNTERS);
    int64_t *off = reinterpret_cast<int64_t *>(base + NA_OFF);
    int32_t *len = reinterpret_cast<int32_t *>(base + NA_LEN);
    BlockDesc *bd = reinterpret_cast<BlockDesc *>(base + NA_BD);
    StreamDesc *sd = reinterpret_cast<StreamDesc *>(base + NA_SD);
    Lz4Job *jobs = reinterpret_cast<Lz4Job *>(base + NA_JOBS);
    uint8_t *img = base + NA_IMG;
    int *njobs = counters, *err = counters + 9, *ngeneral = counters + 10;
    // the job count, the status word and the job cursor must start at zero; descriptors,
    // the chunk index and the image are fully rewritten before they are read
    if (cudaMemsetAsync(counters, 0, 64, st) != cudaSuccess) return -101;
    const int sms = sm_count();
    IAB_TIMED("k_chunk_walk", st, k_chunk_walk<<<1, 32, 0, st>>>(d_chunks, chunks_bytes, g.nchunks, off, len));
    IAB_TIMED("k_parse", st, k_parse<<<parse_grid(nbl, sms), PARSE_T, 0, st>>>(g, d_chunks, off, len, bd, sd, jobs, njobs,
                                                                              8 * NA_MAX_BLOCKS, err, ngeneral, img, nullptr, nullptr));
    {
        IAB_TIMED("k_lz4_decode_cta", st, k_lz4_decode_cta<<<sms * 6, dcta::THREADS, (int)sizeof(dcta::Smem), st>>>(
            jobs, njobs, 8 * NA_MAX_BLOCKS, reinterpret_cast<unsigned *>(counters + 8)));
    }
    scatter_launch(g, d_chunks, chunks_bytes, bd, sd, img, out, ld, err, ngeneral, st);
    // a launch that failed (a bad configuration, or an error left by earlier work) never
    // wrote the status word: report it instead of the zero it still holds
    if (cudaPeekAtLastError() != cudaSuccess) return -101;
    int h_err = 0;
    if (cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return -101;
    if (cudaStreamSynchronize(st) != cudaSuccess) return -101;
    return h_err;
}

}  // namespace iab
