// Time loops with the wavefield resident on chip.
//
// A step kernel reads and writes every field of every cell from memory once
// per time step (40 bytes and more per cell and shot), and a small survey's
// step is a few microseconds of launch and latency.  Here one cooperative
// launch runs a whole run of consecutive steps of a few shots: the grid of
// each shot is cut into gz x gx tiles, one CTA per SM owns one tile for all
// steps, and each of its computing threads owns a block of RB rows x 4
// columns of it.  A thread keeps its block's fields (and forward the
// materials) in registers; shared memory holds the copies that neighbouring
// blocks difference.  Per step a CTA
//   * computes the ring of cells around its tile that its neighbours also
//     compute (the velocity ring forward, the stress ring backward), so one
//     halo exchange per step is enough: the outermost 2R rows and columns of
//     three stress planes forward, of the two velocity products backward;
//   * writes those strips to a global exchange buffer (two alternate by step
//     parity) in 16-byte words of three values and the step's tag;
//   * reads its up to eight neighbours' words until their tags match and puts
//     the values into its halo (a few words per thread: a warp or two of their
//     own took 4000 to 9000 cycles a step for a tile of 81 x 52 cells, and the
//     warps of the border alone a fifth longer than all of them).
// The tag travels with the data (one 16-byte access is a single transaction),
// so there is neither a flag nor a fence: a release of a flag word waits until
// everything the SM has written is in L2, the difference sets included, which
// measured 4000 (100 x 100 survey) to 11000 cycles a step (500 x 1000).
// What is left of the memory traffic is the imaging's difference sets (20
// bytes per imaged cell, written forward, read backward).
//
// Measured, forward / adjoint per step of all shots, against one launch per
// step: 500 x 1000 cells and 4 shots 50.8 / 59.2 -> 20.9 / 37.0 us; whole
// gradients of 100 x 100 cells, 4 shots, 500 steps 7.1 -> 2.5 ms, and of 200 x
// 400 cells, 10 shots, 1000 steps 48.4 -> 29.5 ms.
//
// The arithmetic is that of fwd_step / adj_step / exact_adj_step, operation
// for operation: the results are the step kernels' bits, whatever the tiling.
// (After an overflow the same samples are finite; where the damping is zero an
// infinity stays one here and becomes NaN there.)
//
// Every wait is bounded by p.limit_ns of the global timer: a CTA that gives
// up sets the workspace error word to 3 and stops, and so does every CTA that
// finds the word set when it starts or while it waits.  A CTA that stops
// leaves NaN in its states, its remaining samples and its gradient
// accumulators, so that no caller mistakes the results for good ones.
#pragma once

#include "persist_kernels.cuh"

namespace pyfwi {

// Threads of a CTA, a block each: 12 warps leave 168 registers a thread.
constexpr int RES_THREADS = 384;
constexpr int RES_HALO = RES_THREADS; // halo groups of a tile, at most: a thread fetches a group's words or fewer
constexpr int RES_MAX_CTAS = 148;     // CTAs of a launch: the SMs of a B200
constexpr int RES_MAX_STRIPS = 65536; // strip groups of all CTAs (a word's index takes 18 bits)
constexpr int RES_PAD = 8;            // floats before the first plane: edge groups read past a row's start
// Every shared plane has the same row stride and size, known when compiling:
// a thread addresses its neighbours in all of them by one register and
// immediate offsets.
constexpr int RES_W = 60, RES_ROWS = 92, RES_PLANE = RES_W * RES_ROWS;
constexpr int RES_NAN = 0x7fc00000;    // what a loop that gave up leaves
constexpr int RES_MAX_SLOTS = 1000;   // 4-cell groups with receivers of a CTA (10 bits)
constexpr size_t RES_XCH_BYTES = 2ull * RES_MAX_STRIPS * 64;  // exchange buffer of a workspace
constexpr int RES_MAX_SAMPLES = 1024; // source samples that travel as launch parameters
constexpr int RES_KEEP_STEPS = 2048;  // steps of a launch that keeps some states

// Tiles of a resident launch.  Rows are dealt out in blocks of rb; the last
// block may reach past the grid, where nothing moves.
struct ResTiles {
    int gz, gx, nslots;  // tiles per shot down and across; shots of the launch (gz * gx * nslots CTAs)
    int rb;              // rows of a thread's block
    int nbz, ncg;        // block rows and 4-column groups of the grid
    int bz, nq;          // block rows and groups of the largest tile
};

template <int R>
struct ResShape {
    static constexpr int HG = R <= 2 ? 1 : 2;  // halo groups (2R columns rounded up to 4)
    static constexpr int HX = 4 * HG;
    static constexpr int NQ = (RES_W - 2 * HX) / 4;  // most groups across a tile
    static constexpr int TH = RES_ROWS - 4 * R;      // most rows
    static constexpr int RING = 2 * R * (NQ + 2) + 2 * TH;  // most items of its ring
    static constexpr int OW = 4 * NQ, OPLANE = OW * TH;     // planes of the tile alone
    // every region of shared memory starts on a float4
    static_assert(RES_W % 4 == 0 && RES_ROWS % 4 == 0 && RING % 4 == 0 && RES_PLANE % 4 == 0 && OPLANE % 4 == 0 &&
                      RES_PAD % 4 == 0,
                  "aligned regions");
};

// A rectangle of H x W items split into a frame (bz rows, bx columns thick)
// and the inside; a rectangle with no inside is all frame.
__host__ __device__ inline int frame_count(int H, int W, int bz, int bx)
{
    return H <= 2 * bz || W <= 2 * bx ? H * W : H * W - (H - 2 * bz) * (W - 2 * bx);
}

__device__ __forceinline__ void frame_item(int e, int H, int W, int bz, int bx, int &r, int &q)
{
    if (H <= 2 * bz || W <= 2 * bx) {
        r = e / W;
        q = e - r * W;
        return;
    }
    const int band = bz * W;
    if (e < 2 * band) {
        r = e / W;
        q = e - r * W;
        if (e >= band) r += H - 2 * bz;
        return;
    }
    e -= 2 * band;
    r = bz + e / (2 * bx);
    q = e % (2 * bx);
    if (q >= bx) q += W - 2 * bx;
}

__device__ __forceinline__ void inner_item(int e, int W, int bz, int bx, int &r, int &q)
{
    const int w = W - 2 * bx;
    r = bz + e / w;
    q = bx + e % w;
}

__device__ __forceinline__ int frame_index(int r, int q, int H, int W, int bz, int bx)
{
    if (H <= 2 * bz || W <= 2 * bx) return r * W + q;
    if (r < bz) return r * W + q;
    if (r >= H - bz) return (r - H + 2 * bz) * W + q;
    return 2 * bz * W + (r - bz) * 2 * bx + (q < bx ? q : q - W + 2 * bx);
}

constexpr unsigned ITEM_DAMP = 1u << 30;  // an item with damping on one of its cells
__device__ __forceinline__ unsigned pack_item(int r, int q) { return (unsigned)r << 12 | (unsigned)q; }
__device__ __forceinline__ int item_row(unsigned e) { return (int)((e >> 12) & 0xFFFu); }
__device__ __forceinline__ int item_col(unsigned e) { return (int)(e & 0xFFFu); }

struct FwdResArgs {
    StepArgs a;        // constant fields; in / out: the states at t0 and t1
    ResTiles tl;
    uint4 *xch;        // exchange buffer: [parity][CTA][frame][4] words
    unsigned tag0;     // tag of the strips of state s: tag0 + s - t0 (new to the buffer in every launch)
    long long state;   // floats per state
    int t0, t1;
    int dt_scale, nt_ext, record;
    float *q;          // difference sets (store 1) or states (2) of slot 0 (a.q_stride apart): S_{t+1}'s at
                       // q + (t - q_t0) * state; 3: the exact adjoint's sets of step t
    int q_t0, store;
    int some;          // store 2: only the states of the steps in `keep`, one after another from q on
    int *err;
    unsigned long long limit_ns;
    unsigned keep[RES_KEEP_STEPS / 32];  // bit t - t0: step t's state
    int k0, nk;        // samples k0 .. k0 + nk - 1 are in wav, the others are zero
    float4 wav[RES_MAX_SAMPLES];
};

struct AdjResArgs {
    AdjArgs a;         // constant fields; in / out: the adjoint states before step t_hi - 1 and after step t_lo
    ResTiles tl;
    uint4 *xch;
    unsigned tag0;     // tag of the strips that step t reads: tag0 + t_hi - 1 - t
    long long state;
    int t_hi, t_lo;    // steps t_hi - 1 .. t_lo (t_lo >= 1)
    int nt, nt_ext, dt_scale;
    const float *q;    // the set of S_{t+1} at q + (t - q_t0) * state, slots a.fwd_stride apart
    int q_t0;
    int slots;         // 4-cell groups with receivers whose residuals a CTA stages
    int *err;
    unsigned long long limit_ns;
};

struct RevResArgs {
    StepArgs a;        // constant fields; in: the state of step t_hi
    ResTiles tl;
    uint4 *xch;
    unsigned tag0;     // tag of the strips that step t reads: tag0 + t_hi - 1 - t
    long long state;
    int t_hi, t_lo;    // the states of steps t_hi - 1 .. t_lo
    float *q;          // that of step t, slot 0, at q + (t % ring) * state, slots q_stride apart
    long long q_stride;
    int ring;
    int *err;
    unsigned long long limit_ns;
};

// Shared memory in floats.
// Forward: materials of the blocks that lie in shared memory: with three rows
// in registers the fields alone fill them.
template <int RB>
constexpr int FWD_SHARED_MATS = RB < 3 ? 0 : 3;
template <int R, int RB>
constexpr int FWD_RES_FLOATS = RES_PAD + 5 * RES_PLANE + 6 * ResShape<R>::RING + 2 * RES_ROWS + 2 * RES_W + 8 +
                               4 * RES_MAX_SAMPLES + 4 * RES_THREADS + 4 * FWD_SHARED_MATS<RB> * RB * RES_THREADS;
// Adjoint: a thread's places for difference sets on their way, four floats
// each: three rows share six places, asked for in turns.  Blocks of more than
// one row keep one of the three gradient accumulators in shared memory: with
// all of them in registers the loop spills.
template <int RB>
constexpr int RES_SETS = RB < 3 ? 0 : 6;
template <int R, int RB>
constexpr int RES_OWN = RB < 3 ? 4 * RB * RES_THREADS : ResShape<R>::OPLANE;  // a plane of the blocks alone
template <int R, int RB>
constexpr int ADJ_RES_FLOATS = RES_PAD + 5 * RES_PLANE + (RB < 2 ? 2 : 3) * RES_OWN<R, RB> + 22 * ResShape<R>::RING + 2 * RES_ROWS +
                               3 * RES_W + 4 * RES_SETS<RB> * RES_THREADS;
template <int R, int RB>
constexpr int REV_RES_FLOATS = RES_PAD + 5 * RES_PLANE + 21 * ResShape<R>::RING + RES_ROWS + RES_W +
                               4 * FWD_SHARED_MATS<RB> * RB * RES_THREADS;
template <int R, int RB>
constexpr int EXA_RES_FLOATS = RES_PAD + 5 * RES_PLANE + 2 * RES_OWN<R, RB> + 14 * ResShape<R>::RING + RES_ROWS + RES_W +
                               4 * RES_THREADS;
constexpr int RES_SLOT_FLOATS = 44;  // and per slot of staged residuals (adjoint)

// 16-byte words that are written and read as one transaction.
__device__ __forceinline__ void st_word(uint4 *p, float a, float b, float c, unsigned tag)
{
    const unsigned long long lo = (unsigned long long)__float_as_uint(b) << 32 | __float_as_uint(a),
                             hi = (unsigned long long)tag << 32 | __float_as_uint(c);
    asm volatile("{\n.reg .b128 w;\nmov.b128 w, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], w;\n}\n" ::"l"(p), "l"(lo),
                 "l"(hi)
                 : "memory");
}

__device__ __forceinline__ uint4 ld_word(const uint4 *p)
{
    unsigned long long lo, hi;
    asm volatile("{\n.reg .b128 w;\nld.relaxed.gpu.global.b128 w, [%2];\nmov.b128 {%0, %1}, w;\n}\n"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}

// Where a halo group of tile (tz, tx) comes from: the strip group of the CTA
// that owns it, or ~0u outside the grid (where the halo stays zero).
template <int R>
__device__ __forceinline__ unsigned halo_source(const Grid &g, const ResTiles &tl, int frame, int slot, int tz, int tx,
                                                int i0, int th, int q0, int nq, int gi, int gq)
{
    if (gi < 0 || gi >= g.tnz || gq < 0 || gq >= tl.ncg) return ~0u;
    const int z = gi < i0 ? tz - 1 : gi >= i0 + th ? tz + 1 : tz, x = gq < q0 ? tx - 1 : gq >= q0 + nq ? tx + 1 : tx;
    const int oi = tl.rb * (tl.nbz * z / tl.gz), oh = tl.rb * (tl.nbz * (z + 1) / tl.gz) - oi;
    const int oq = tl.ncg * x / tl.gx, ow = tl.ncg * (x + 1) / tl.gx - oq;
    return (unsigned)(((slot * tl.gz + z) * tl.gx + x) * frame + frame_index(gi - oi, gq - oq, oh, ow, 2 * R, ResShape<R>::HG));
}

// A thread's halo words (W in all: a group has W): where each lies in the
// exchange buffer (18 bits) and where its values go (14 bits); ~0u: none.
template <int R, int W>
__device__ __forceinline__ void halo_words(unsigned *word, const Grid &g, const ResTiles &tl, int frame, int slot, int tz, int tx,
                                           int i0, int th, int q0, int nq)
{
    constexpr int HG = ResShape<R>::HG;
    const int n = W * ((th + 4 * R) * (nq + 2 * HG) - th * nq);
#pragma unroll 1
    for (int u = threadIdx.x; u < W * RES_THREADS; u += RES_THREADS) {
        word[u] = ~0u;
        if (u >= n) continue;
        int r, q;
        frame_item(u / W, th + 4 * R, nq + 2 * HG, 2 * R, HG, r, q);
        const unsigned src = halo_source<R>(g, tl, frame, slot, tz, tx, i0, th, q0, nq, i0 - 2 * R + r, q0 - HG + q);
        if (src != ~0u) word[u] = (4 * src + u % W) << 14 | (unsigned)(r * RES_W + 4 * q);
    }
}

// Each of the words read until its tag is `tag`, then handed to put(offset,
// word of the group, value).  False when the wait gave up (error word set,
// here or by another CTA).
template <int W, class Put>
__device__ __forceinline__ bool fetch_halo(const uint4 *buf, unsigned tag, const unsigned *words, int *err,
                                           unsigned long long limit_ns, Put put)
{
    unsigned long long t0 = 0;
    unsigned open = 0, word[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
        word[k] = words[k * RES_THREADS + threadIdx.x];
        if (word[k] != ~0u) open |= 1u << k;
    }
    for (unsigned n = 1; open; ++n) {
        uint4 v[W];
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (open >> k & 1) v[k] = ld_word(buf + (word[k] >> 14));
#pragma unroll
        for (int k = 0; k < W; ++k)
            if ((open >> k & 1) && v[k].w == tag) {
                const unsigned u = word[k];
                open &= ~(1u << k);
                put((int)(u & 0x3FFFu), (int)(u >> 14 & 3u), v[k]);
            }
        if (open && (n & 63u) == 0) {
            if (ld_relaxed_gpu(err) != 0) return false;
            if (!t0) {
                t0 = global_ns();
            } else if (global_ns() - t0 > limit_ns) {
                atomicCAS(err, 0, 3);
                return false;
            }
        }
    }
    return true;
}

// This thread's halo group: where it lies in the exchange buffer (its strip
// group, 16 bits) and where its values go (14 bits); ~0u: none.
template <int R>
__device__ __forceinline__ unsigned halo_group(const Grid &g, const ResTiles &tl, int frame, int slot, int tz, int tx, int i0,
                                               int th, int q0, int nq)
{
    constexpr int HG = ResShape<R>::HG;
    if ((int)threadIdx.x >= (th + 4 * R) * (nq + 2 * HG) - th * nq) return ~0u;
    int r, q;
    frame_item(threadIdx.x, th + 4 * R, nq + 2 * HG, 2 * R, HG, r, q);
    const unsigned src = halo_source<R>(g, tl, frame, slot, tz, tx, i0, th, q0, nq, i0 - 2 * R + r, q0 - HG + q);
    return src == ~0u ? src : src << 14 | (unsigned)(r * RES_W + 4 * q);
}

// The W words of a halo group, each read until its tag is `tag`, then handed to
// put(offset, words); as fetch_halo.  A thread that takes a whole group needs one
// address and stores four values at a time, where words dealt out evenly are
// fewer per thread.  Measured, us per step: backward (three words, the two
// velocity products) 240 x 440 cells, 1 shot 2.96 with dealt words, 2.65 with
// groups; forward (four, three stresses) 2.39 and 2.50.
template <int W, class Put>
__device__ __forceinline__ bool fetch_group(const uint4 *buf, unsigned tag, unsigned group, int *err,
                                           unsigned long long limit_ns, Put put)
{
    if (group == ~0u) return true;
    buf += 4 * (group >> 14);
    unsigned long long t0 = 0;
    unsigned open = (1u << W) - 1;
    uint4 v[W];
    for (unsigned n = 1; open; ++n) {
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (open >> k & 1) v[k] = ld_word(buf + k);
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (v[k].w == tag) open &= ~(1u << k);
        if (open && (n & 63u) == 0) {
            if (ld_relaxed_gpu(err) != 0) return false;
            if (!t0) {
                t0 = global_ns();
            } else if (global_ns() - t0 > limit_ns) {
                atomicCAS(err, 0, 3);
                return false;
            }
        }
    }
    put((int)(group & 0x3FFFu), v);
    return true;
}

// A row of 4 own columns `c` with its neighbours in shared memory, in row12's
// places (v[4 + k] is column k of the group at `row`): what forward (backward)
// differences of the four read.
template <int R, bool FWD>
__device__ __forceinline__ void xrow(float (&v)[12], const float4 &c, const float *row)
{
    v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
    if constexpr (R == 2) {
        v[0] = v[1] = v[10] = v[11] = 0.f;
        if (FWD) {
            const float2 r = *reinterpret_cast<const float2 *>(row + 4);
            v[2] = 0.f;
            v[3] = row[-1];
            v[8] = r.x; v[9] = r.y;
        } else {
            const float2 l = *reinterpret_cast<const float2 *>(row - 2);
            v[2] = l.x; v[3] = l.y;
            v[8] = row[4];
            v[9] = 0.f;
        }
    } else {
        const float4 l = ld4s(row - 4), r = ld4s(row + 4);
        v[0] = l.x; v[1] = l.y; v[2] = l.z; v[3] = l.w;
        v[8] = r.x; v[9] = r.y; v[10] = r.z; v[11] = r.w;
    }
}

// Rows of a window around the RB own rows of a plane that backward (FWD:
// forward) z differences read: own(r) for row r of the block, the rows above
// and below from shared memory (row 0 of the block at p, rows W apart).
template <int R, int RB, bool FWD>
struct ZWindow {
    static constexpr int UP = FWD ? R - 1 : R, N = RB + 2 * R - 1;
    float4 w[N];
    template <class Own>
    __device__ __forceinline__ ZWindow(Own own, const float *p)
    {
#pragma unroll
        for (int m = 0; m < N; ++m) {
            const int row = m - UP;
            if (row >= 0 && row < RB)
                w[m] = own(row);
            else
                w[m] = ld4s(p + row * RES_W);
        }
    }
    // The difference at row r, column k, in the operation order of zbwd / zfwd.
    __device__ __forceinline__ float at(int r, int k, const float *c) const
    {
        const int o = r + UP;
        float s = FWD ? c[0] * (f4(w[o + 1], k) - f4(w[o], k)) : c[0] * (f4(w[o], k) - f4(w[o - 1], k));
#pragma unroll
        for (int q = 1; q < R; ++q)
            s = FWD ? fmaf(c[q], f4(w[o + q + 1], k) - f4(w[o - q], k), s) : fmaf(c[q], f4(w[o + q], k) - f4(w[o - q - 1], k), s);
        return s;
    }
};

// The same window moving down row by row: the 2R rows that the difference at
// the current row reads.
template <int R, bool FWD>
struct ZSlide {
    static constexpr int UP = FWD ? R - 1 : R, DN = FWD ? R : R - 1;
    float4 w[2 * R];
    template <class Row>
    __device__ __forceinline__ ZSlide(Row row)
    {
#pragma unroll
        for (int m = 1; m < 2 * R; ++m) w[m] = row(m - 1 - UP);
    }
    __device__ __forceinline__ void next(const float4 &v)
    {
#pragma unroll
        for (int m = 1; m < 2 * R; ++m) w[m - 1] = w[m];
        w[2 * R - 1] = v;
    }
    __device__ __forceinline__ const float4 &centre() const { return w[UP]; }
    __device__ __forceinline__ float at(int k, const float *c) const
    {
        float s = FWD ? c[0] * (f4(w[UP + 1], k) - f4(w[UP], k)) : c[0] * (f4(w[UP], k) - f4(w[UP - 1], k));
#pragma unroll
        for (int q = 1; q < R; ++q)
            s = FWD ? fmaf(c[q], f4(w[UP + q + 1], k) - f4(w[UP - q], k), s)
                    : fmaf(c[q], f4(w[UP + q], k) - f4(w[UP - q - 1], k), s);
        return s;
    }
};

// Difference values are written once and read once: streaming accesses.
__device__ __forceinline__ void qst4s(float *q, float4 v) { __stcs(reinterpret_cast<float4 *>(q), v); }
// Keeps the compiler from loading early what comes after, where that would cost registers.
__device__ __forceinline__ void in_order() { asm volatile("" ::: "memory"); }

// Difference values are read once: past L1.
__device__ __forceinline__ float4 qld4s(const float *q)
{
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(q));
    return v;
}

// Groups of asynchronous copies.
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ void qprefetch4(const float *q) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(q)); }
__device__ __forceinline__ float4 mk4(const float (&v)[4]) { return make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ float4 times4(const float4 &u, const float4 &v)
{
    return make_float4(__fmul_rn(u.x, v.x), __fmul_rn(u.y, v.y), __fmul_rn(u.z, v.z), __fmul_rn(u.w, v.w));
}

// Receivers k0 .. k0 + n - 1 of line l on rows [r0, r1), columns [c0, c1).
__device__ __forceinline__ void line_range(const Lines &L, int l, int r0, int r1, int c0, int c1, int &k0, int &n)
{
    int lo, hi;  // first and one past the last receiver
    if (L.drow[l] == 0) {
        const int d = L.dcol[l];
        lo = c0 > L.col0[l] ? (c0 - L.col0[l] + d - 1) / d : 0;
        hi = c1 > L.col0[l] ? (c1 - 1 - L.col0[l]) / d + 1 : 0;
        if (L.row0[l] < r0 || L.row0[l] >= r1) hi = lo;
    } else {
        const int d = L.drow[l];
        lo = r0 > L.row0[l] ? (r0 - L.row0[l] + d - 1) / d : 0;
        hi = r1 > L.row0[l] ? (r1 - 1 - L.row0[l]) / d + 1 : 0;
        if (L.col0[l] < c0 || L.col0[l] >= c1) hi = lo;
    }
    if (hi > L.count[l]) hi = L.count[l];
    k0 = lo;
    n = hi > lo ? hi - lo : 0;
}

// The tile of this CTA.
struct ResTile {
    int slot, tz, tx, i0, th, q0, nq, j0;
    int nblk, nin;  // blocks; the first nin reach neither the halo nor the strips
};

template <int R, int RB>
__device__ __forceinline__ ResTile res_tile(const ResTiles &tl)
{
    constexpr int HG = ResShape<R>::HG, BZ = (2 * R + RB - 1) / RB;  // block rows that hold the strips
    ResTile t;
    const int per = tl.gz * tl.gx, tile = blockIdx.x % per;
    t.slot = blockIdx.x / per;
    t.tz = tile / tl.gx;
    t.tx = tile - t.tz * tl.gx;
    const int b0 = tl.nbz * t.tz / tl.gz, b1 = tl.nbz * (t.tz + 1) / tl.gz;
    t.i0 = RB * b0;
    t.th = RB * (b1 - b0);
    t.q0 = tl.ncg * t.tx / tl.gx;
    t.nq = tl.ncg * (t.tx + 1) / tl.gx - t.q0;
    t.j0 = 4 * t.q0;
    t.nblk = (b1 - b0) * t.nq;
    t.nin = t.nblk - frame_count(b1 - b0, t.nq, BZ, HG);
    return t;
}

// Block row and group of block e: the inside first, then the frame.
template <int R, int RB>
__device__ __forceinline__ void res_block(const ResTile &t, int e, int &bz, int &q)
{
    constexpr int BZ = (2 * R + RB - 1) / RB, HG = ResShape<R>::HG;
    if (e < t.nin)
        inner_item(e, t.nq, BZ, HG, bz, q);
    else
        frame_item(e - t.nin, t.th / RB, t.nq, BZ, HG, bz, q);
}

// ---------------------------------------------------------------------------
// forward steps t0 .. t1 - 1 (fwd_step's arithmetic)
// ---------------------------------------------------------------------------
// QD: 1 stores the difference sets of the states, 2 the states, 3 the exact
// adjoint's sets (stress differences of S_t with step t's source, velocity
// differences of S_{t+1}; zero outside the update domain), 0 neither.
template <int R, int RB, int QD>
__global__ void __launch_bounds__(RES_THREADS, 1) fwd_resident(const __grid_constant__ FwdResArgs p)
{
    constexpr int NT = RES_THREADS, HX = ResShape<R>::HX, HG = ResShape<R>::HG;
    extern __shared__ float4 smem4[];
    __shared__ int s_stop, s_line[3][4];
    const StepArgs &a = p.a;
    const Grid &g = a.g;
    const long long P = g.plane;
    const int tid = threadIdx.x;
    const ResTile T = res_tile<R, RB>(p.tl);
    const int i0 = T.i0, j0 = T.j0, th = T.th, nq = T.nq;
    constexpr int W = RES_W, PL = RES_PLANE, RING = ResShape<R>::RING;
    float *const sm = reinterpret_cast<float *>(smem4) + RES_PAD;
    // Cell (r, c) of the tile lies at (r + 2R) * W + HX + c of every plane.
    float *const s_txx = sm, *const s_tzz = sm + PL, *const s_txz = sm + 2 * PL, *const s_vx = sm + 3 * PL, *const s_vz = sm + 4 * PL;
    float *const s_rb = sm + 5 * PL;                              // buoyancy of the ring's items
    float *const s_dx = s_rb + 4 * RING, *const s_dz = s_dx + W;  // damping of columns j0 - HX .., rows i0 - 2R ..
    float *const s_org = s_dz + RES_ROWS;                         // the source cell's stresses before the add
    float4 *const s_wav = reinterpret_cast<float4 *>(s_org + 4);
    unsigned *const t_ring = reinterpret_cast<unsigned *>(s_wav + RES_MAX_SAMPLES);
    unsigned *const t_word = t_ring + RING;                       // the threads' halo words
    float *const s_mat = reinterpret_cast<float *>(t_word + 4 * NT);  // [lam, mu, b][row][thread][4], RB 3
    constexpr int SM = FWD_SHARED_MATS<RB>;
    const int frame = frame_count(RB * p.tl.bz, p.tl.nq, 2 * R, HG);  // strip groups of the largest tile
    const int nring = (th + 2 * R) * (nq + 2) - th * nq;
    const int shot = a.shot0 + T.slot;
    const float dt = a.k.dt;
    const float *in = a.in + T.slot * a.in_stride;
    const int xpar = 4 * gridDim.x * frame;  // words per parity
    uint4 *const strip = p.xch + 4 * blockIdx.x * frame;

    // the tile with its halo, the ring's table and buoyancy, the damping
    if (tid == 0) s_stop = ld_relaxed_gpu(p.err) != 0;
    for (int e = tid; e < (th + 4 * R) * (nq + 2 * HG); e += NT) {
        const int r = e / (nq + 2 * HG), q = e - r * (nq + 2 * HG), o = r * W + 4 * q;
        const int gi = i0 - 2 * R + r, gj = j0 - HX + 4 * q;
        cp4(s_txx + o, in + TXX * P, g, gi, gj);
        cp4(s_tzz + o, in + TZZ * P, g, gi, gj);
        cp4(s_txz + o, in + TXZ * P, g, gi, gj);
        cp4(s_vx + o, in + VX * P, g, gi, gj);
        cp4(s_vz + o, in + VZ * P, g, gi, gj);
    }
    for (int e = tid; e < p.nk; e += NT) s_wav[e] = p.wav[e];
    // Outside the update domain nothing moves: zero materials there leave every
    // field as it is (x + dt * (0 * y) = x; no source sits there).
    auto masked = [&](const float *plane, int gi, int gj) {
        float4 v = ld4(plane, g, gi, gj);
        if (!in_domain(g, R, gi, gj)) v.x = 0.f;
        if (!in_domain(g, R, gi, gj + 1)) v.y = 0.f;
        if (!in_domain(g, R, gi, gj + 2)) v.z = 0.f;
        if (!in_domain(g, R, gi, gj + 3)) v.w = 0.f;
        return v;
    };
    auto row_damp = [&](int gi) { return gi + ZO >= 0 && gi + ZO < g.rows ? __ldg(a.dampz + gi + ZO) : 0.f; };
    auto damped = [&](int gi, int gj) {
        const float4 x = damp4(a.dampx, g, gj);
        return row_damp(gi) != 0.f || x.x != 0.f || x.y != 0.f || x.z != 0.f || x.w != 0.f;
    };
    for (int e = tid; e < nring; e += NT) {
        int r, q;
        frame_item(e, th + 2 * R, nq + 2, R, 1, r, q);
        t_ring[e] = pack_item(r, q) | (damped(i0 - R + r, j0 - 4 + 4 * q) ? ITEM_DAMP : 0u);
        st4s(s_rb + 4 * e, masked(a.mat + 2 * P, i0 - R + r, j0 - 4 + 4 * q));
    }
    for (int e = tid; e < 4 * nq + 2 * HX; e += NT) {
        const int c = j0 - HX + e + XO;
        s_dx[e] = c >= 0 && c < g.pitch ? __ldg(a.dampx + c) : 0.f;
    }
    for (int e = tid; e < th + 4 * R; e += NT) s_dz[e] = row_damp(i0 - 2 * R + e);
    if (tid < a.lines.n) {
        // receivers of the tile, per line: how many, the first one's place and the stride in the
        // planes, its trace column
        const Lines &L = a.lines;
        int k0, n;
        line_range(L, tid, i0, min(i0 + th, g.tnz), j0, min(j0 + 4 * nq, g.tnx), k0, n);
        const int r = L.row0[tid] + k0 * L.drow[tid] - i0, c = L.col0[tid] + k0 * L.dcol[tid] - j0;
        s_line[tid][0] = n;
        s_line[tid][1] = (r + 2 * R) * W + c + HX;
        s_line[tid][2] = L.drow[tid] * W + L.dcol[tid];
        s_line[tid][3] = shot * a.nr + L.slot0[tid] + k0;
    }
    cp_wait_all();
    __syncthreads();

    halo_words<R, 4>(t_word, g, p.tl, frame, T.slot, T.tz, T.tx, i0, th, T.q0, nq);
    auto put = [&](int o, int c, const uint4 &w) {
        s_txx[o + c] = __uint_as_float(w.x);
        s_tzz[o + c] = __uint_as_float(w.y);
        s_txz[o + c] = __uint_as_float(w.z);
    };

    // this thread's block
    const bool mine = tid < T.nblk, inside = tid < T.nin;
    int bz = 0, bq = 0;
    if (mine) res_block<R, RB>(T, tid, bz, bq);
    const int br = bz * RB;                                // its first row in the tile
    const int ot = (br + 2 * R) * W + HX + 4 * bq;         // and its place in the planes
    const int gi0 = i0 + br, gj0 = j0 + 4 * bq;
    const int co = (gi0 + ZO) * g.pitch + gj0 + XO;        // its first cell in a plane
    float4 vx[RB], vz[RB], sxx[RB], szz[RB], sxz[RB];
    float4 b[RB], lam[RB], mu[RB];
    constexpr bool SETS = QD == 1 || QD == 3;
    bool damp = false;
    unsigned img = 0;                                      // rows with imaged cells
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        vx[r] = vz[r] = sxx[r] = szz[r] = sxz[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        b[r] = lam[r] = mu[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!mine) continue;
        const int gi = gi0 + r;
        vx[r] = ld4s(s_vx + ot + r * W);
        vz[r] = ld4s(s_vz + ot + r * W);
        sxx[r] = ld4s(s_txx + ot + r * W);
        szz[r] = ld4s(s_tzz + ot + r * W);
        sxz[r] = ld4s(s_txz + ot + r * W);
        b[r] = masked(a.mat + 2 * P, gi, gj0);
        lam[r] = masked(a.mat, gi, gj0);
        mu[r] = masked(a.mat + P, gi, gj0);
        if (SM > 0) st4s(s_mat + 4 * (r * NT + tid), lam[r]);
        if (SM > 1) st4s(s_mat + 4 * ((RB + r) * NT + tid), mu[r]);
        if (SM > 2) st4s(s_mat + 4 * ((2 * RB + r) * NT + tid), b[r]);
        damp = damp || damped(gi, gj0);
        if (SETS && gi >= a.qlo && gi <= a.qhi_z && gj0 + 3 >= a.qlo && gj0 <= a.qhi_x) img |= 1u << r;
    }

    // The strip group of row r of the tile in this thread's column, -1: none.
    auto strip_group = [&](int r) {
        return r < 2 * R || r >= th - 2 * R || bq < HG || bq >= nq - HG ? frame_index(r, bq, th, nq, 2 * R, HG) : -1;
    };

    // the source cell: in the tile, or in its halo
    const int si = __ldg(a.srcz + shot), sj = __ldg(a.srcx + shot);
    const int s_r = si - i0 + 2 * R, s_c = sj - j0 + HX, so = s_r * W + s_c;
    const bool src_t = s_r >= 0 && s_r < th + 4 * R && s_c >= 0 && s_c < 4 * nq + 2 * HX;
    const bool src_own = si >= i0 && si < i0 + th && sj >= j0 && sj < j0 + 4 * nq;
    const bool my_src = mine && si >= gi0 && si < gi0 + RB && sj >= gj0 && sj < gj0 + 4;

    // This thread's receiver (a tile has fewer than there are threads): its place in the planes and its
    // trace column.
    int rec_o = -1;
    bool rec_vzx = false;
    float *rec_tr = a.traces;
    for (int l = 0, e = tid; p.record && l < a.lines.n; e -= s_line[l++][0])
        if (e >= 0 && e < s_line[l][0]) {
            rec_o = s_line[l][1] + e * s_line[l][2];
            rec_vzx = a.lines.vzx[l];
            rec_tr += s_line[l][3] + e;
        }
    const int rec_row = a.ns * a.nr;
    // Its traces of row `row`: the velocities (as soon as they are there), the stresses (before the next source).
    auto record_v = [&](int row) {
        float *tr = rec_tr + (long long)row * rec_row;
        tr[0] = s_vx[rec_o];
        tr[a.trace_plane] = rec_vzx ? s_vx[rec_o] : s_vz[rec_o];
    };
    auto record_t = [&](int row) {
        float *tr = rec_tr + (long long)row * rec_row;
        tr[2 * a.trace_plane] = s_txx[rec_o];
        tr[3 * a.trace_plane] = s_tzz[rec_o];
        tr[4 * a.trace_plane] = s_txz[rec_o];
    };

    auto lam_of = [&](int r) { return SM > 0 ? ld4s(s_mat + 4 * (r * NT + tid)) : lam[r]; };
    auto mu_of = [&](int r) { return SM > 1 ? ld4s(s_mat + 4 * ((RB + r) * NT + tid)) : mu[r]; };
    auto b_of = [&](int r) { return SM > 2 ? ld4s(s_mat + 4 * ((2 * RB + r) * NT + tid)) : b[r]; };
    // Four values of a set: (QD 3) zero on columns outside the update domain.
    auto within = [&](float (&s)[4]) {
        if (QD == 3)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (gj0 + k < a.qlo || gj0 + k > a.qhi_x) s[k] = 0.f;
        return mk4(s);
    };
    // New velocities of the block; qi: the difference set of the input state (null: none).
    auto velocity = [&](float *qi) {
        {
            const ZWindow<R, RB, false> z([&](int r) { return sxz[r]; }, s_txz + ot);  // Dz- txz
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                float x[12], s[4], n[4];
                const float4 br4 = b_of(r);
                xrow<R, false>(x, sxx[r], s_txx + ot + r * W);  // Dx- txx
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s[k] = xbwd<R>(x, k, a.k.cx) + z.at(r, k, a.k.cz);
                    n[k] = f4(vx[r], k) + dt * (f4(br4, k) * s[k]);
                }
                if (SETS && qi && (img >> r & 1)) qst4s(qi + Q_TXS * P + co + r * g.pitch, within(s));
                vx[r] = mk4(n);
            }
        }
        {
            const ZWindow<R, RB, true> z([&](int r) { return szz[r]; }, s_tzz + ot);  // Dz+ tzz
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                float x[12], s[4], n[4];
                const float4 br4 = b_of(r);
                xrow<R, true>(x, sxz[r], s_txz + ot + r * W);  // Dx+ txz
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s[k] = z.at(r, k, a.k.cz) + xfwd<R>(x, k, a.k.cx);
                    n[k] = f4(vz[r], k) + dt * (f4(br4, k) * s[k]);
                }
                if (SETS && qi && (img >> r & 1)) qst4s(qi + Q_TZS * P + co + r * g.pitch, within(s));
                vz[r] = mk4(n);
            }
        }
        if (damp) {
            const float4 dx = ld4s(s_dx + HX + 4 * bq);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const float dr = s_dz[br + r + 2 * R];
                float nx[4], nz[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float d = f4(dx, k) + dr;
                    nx[k] = f4(vx[r], k) + dt * (-d * f4(vx[r], k));
                    nz[k] = f4(vz[r], k) + dt * (-d * f4(vz[r], k));
                }
                vx[r] = mk4(nx);
                vz[r] = mk4(nz);
            }
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            st4s(s_vx + ot + r * W, vx[r]);
            st4s(s_vz + ot + r * W, vz[r]);
        }
    };

    // New velocities of ring item e.
    auto ring = [&](int e) {
        const unsigned item = t_ring[e];
        const int r = item_row(item), q = item_col(item), c = (r + R) * W + HX - 4 + 4 * q;
        const float4 ovx = ld4s(s_vx + c), ovz = ld4s(s_vz + c), bb = ld4s(s_rb + 4 * e), cxz = ld4s(s_txz + c);
        float x[12], nx[4], nz[4];
        const ZWindow<R, 1, false> zx([&](int) { return cxz; }, s_txz + c);
        xrow<R, false>(x, ld4s(s_txx + c), s_txx + c);
#pragma unroll
        for (int k = 0; k < 4; ++k) nx[k] = f4(ovx, k) + dt * (f4(bb, k) * (xbwd<R>(x, k, a.k.cx) + zx.at(0, k, a.k.cz)));
        const ZWindow<R, 1, true> zz([&](int) { return ld4s(s_tzz + c); }, s_tzz + c);
        xrow<R, true>(x, cxz, s_txz + c);
#pragma unroll
        for (int k = 0; k < 4; ++k) nz[k] = f4(ovz, k) + dt * (f4(bb, k) * (zz.at(0, k, a.k.cz) + xfwd<R>(x, k, a.k.cx)));
        if (item & ITEM_DAMP) {
            const float4 dx = ld4s(s_dx + HX - 4 + 4 * q);
            const float dr = s_dz[r + R];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float d = f4(dx, k) + dr;
                nx[k] = nx[k] + dt * (-d * nx[k]);
                nz[k] = nz[k] + dt * (-d * nz[k]);
            }
        }
        st4s(s_vx + c, mk4(nx));
        st4s(s_vz + c, mk4(nz));
    };

    // New stresses of the block; its strips to xo, the velocity differences to qo.
    auto stress = [&](uint4 *xo, unsigned tag, float *qo) {
        float4 hx[RB];  // Dx- vz
        {               // normal stresses: Dx+ vx, Dz- vz (and, imaged, Dz+ vz)
            const ZWindow<R, RB, false> zz([&](int r) { return vz[r]; }, s_vz + ot);
            const ZWindow<R, RB, true> zi([&](int r) { return vz[r]; }, s_vz + ot);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                float x[12], ex[4], ez[4], h[4], oxx[4], ozz[4];
                xrow<R, true>(x, vx[r], s_vx + ot + r * W);
#pragma unroll
                for (int k = 0; k < 4; ++k) ex[k] = xfwd<R>(x, k, a.k.cx);
                xrow<R, false>(x, vz[r], s_vz + ot + r * W);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    h[k] = xbwd<R>(x, k, a.k.cx);
                    ez[k] = zz.at(r, k, a.k.cz);
                }
                hx[r] = mk4(h);
                if (QD == 3 && (img >> r & 1)) {
                    qst4s(qo + Q_DXP_VX * P + co + r * g.pitch, within(ex));
                    qst4s(qo + Q_DZM_VZ * P + co + r * g.pitch, within(ez));
                }
                if (QD == 1 && (img >> r & 1)) {
                    float *q = qo + co + r * g.pitch, s[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) s[k] = zi.at(r, k, a.k.cz) + h[k];
                    qst4s(q + Q_DXP_VX * P, mk4(ex));
                    qst4s(q + Q_DZM_VZ * P, mk4(ez));
                    qst4s(q + Q_VZS * P, mk4(s));
                }
                const float4 l4 = lam_of(r), m4 = mu_of(r);
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // normal_pair_fwd, the damping apart
                    const float l = f4(l4, k), m = f4(m4, k), l2m = l + 2.f * m;
                    oxx[k] = __fmaf_rn(dt, __fmaf_rn(l2m, ex[k], __fmul_rn(l, ez[k])), f4(sxx[r], k));
                    ozz[k] = __fmaf_rn(dt, __fmaf_rn(l, ex[k], __fmul_rn(l2m, ez[k])), f4(szz[r], k));
                }
                sxx[r] = mk4(oxx);
                szz[r] = mk4(ozz);
            }
        }
        const ZWindow<R, RB, true> zx([&](int r) { return vx[r]; }, s_vx + ot);  // Dz+ vx
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            float oxz[4];
            const float4 m4 = mu_of(r);
#pragma unroll
            for (int k = 0; k < 4; ++k) oxz[k] = f4(sxz[r], k) + dt * (f4(m4, k) * (f4(hx[r], k) + zx.at(r, k, a.k.cz)));
            if (QD == 3 && (img >> r & 1)) {
                float s[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) s[k] = f4(hx[r], k) + zx.at(r, k, a.k.cz);
                qst4s(qo + Q_VZS * P + co + r * g.pitch, within(s));
            }
            if (damp) {
                const float4 dx = ld4s(s_dx + HX + 4 * bq);
                const float dr = s_dz[br + r + 2 * R];
                float oxx[4], ozz[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float d = f4(dx, k) + dr;
                    oxx[k] = __fmaf_rn(dt, __fmul_rn(-d, f4(sxx[r], k)), f4(sxx[r], k));
                    ozz[k] = __fmaf_rn(dt, __fmul_rn(-d, f4(szz[r], k)), f4(szz[r], k));
                    oxz[k] = oxz[k] + dt * (-d * oxz[k]);
                }
                sxx[r] = mk4(oxx);
                szz[r] = mk4(ozz);
            }
            sxz[r] = mk4(oxz);
            if (!inside) {
                const int s = strip_group(br + r);
                if (s >= 0) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) st_word(xo + 4 * s + k, f4(sxx[r], k), f4(szz[r], k), oxz[k], tag);
                }
            }
            st4s(s_txx + ot + r * W, sxx[r]);
            st4s(s_tzz + ot + r * W, szz[r]);
            st4s(s_txz + ot + r * W, sxz[r]);
        }
    };

    int k = p.t0 / p.dt_scale, sub = p.t0 - k * p.dt_scale;  // sample index and position inside it
    if (rec_o >= 0 && sub == 0 && k < p.nt_ext) record_v(k);
    __syncthreads();
    // ring items go to the threads without a block first, then to those inside
    const int rank = tid >= T.nblk ? tid - T.nblk : tid + NT - T.nblk;
    bool stop = s_stop;
    int nkept = 0;
    for (int t = p.t0; t < p.t1 && !stop; ++t) {
        if (rec_o >= 0 && sub == 0 && k < p.nt_ext) record_t(k);
        // this step's source sample, where it reaches the tile (uniform over the CTA)
        float4 src = make_float4(0.f, 0.f, 0.f, 0.f);
        if (src_t && sub == 0 && k >= p.k0 && k - p.k0 < p.nk) src = s_wav[k - p.k0];
        const bool add = src.x != 0.f || src.y != 0.f || src.z != 0.f || src.w != 0.f;
        float *qi = nullptr, *qo = nullptr;
        if constexpr (QD) {
            qo = p.q + (long long)(t - p.q_t0) * p.state + T.slot * a.q_stride;
            if (QD == 1 && t > p.q_t0) qi = qo - p.state;
            if (QD == 3) qi = qo;
        }
        if (add) {
            __syncthreads();
            if (tid == 0) {
                if (src_own) {
                    s_org[0] = s_txx[so];
                    s_org[1] = s_tzz[so];
                    s_txx[so] += src.z;
                    s_tzz[so] += src.w;
                }
                s_vx[so] += src.x;  // outside the ring: not read
                s_vz[so] += src.y;
            }
            __syncthreads();
            if (my_src) {  // the block's own copies
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    vx[r] = ld4s(s_vx + ot + r * W);
                    vz[r] = ld4s(s_vz + ot + r * W);
                    sxx[r] = ld4s(s_txx + ot + r * W);
                    szz[r] = ld4s(s_tzz + ot + r * W);
                }
            }
        }
        // velocities: the blocks inside, then, with the halo, the others
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            if (pass == 1) {
                if (t > p.t0) {  // the neighbours' strips of S_t
                    if (!fetch_halo<4>(p.xch + (t & 1) * xpar, p.tag0 + (unsigned)(t - p.t0), t_word, p.err, p.limit_ns, put))
                        s_stop = 1;
                    __syncthreads();
                    stop = s_stop;
                    if (stop) break;
                }
                if (add && !src_own) {
                    if (t == p.t0) __syncthreads();
                    if (tid == 0) {
                        s_org[0] = s_txx[so];
                        s_org[1] = s_tzz[so];
                        s_txx[so] += src.z;
                        s_tzz[so] += src.w;
                    }
                    __syncthreads();
                }
            }
            if (mine && inside == (pass == 0)) velocity(qi);
        }
        if (stop) break;
        for (int e = rank; e < nring; e += NT) ring(e);
        if constexpr (QD == 1) {
            // the stress differences near the source cell again, without this
            // step's source (see fwd_step)
            if (qi && add) {
                __syncthreads();
                if (tid < 4 * R) {
                    const int gi = tid < 2 * R ? si : si - R + (tid - 2 * R), gj = tid < 2 * R ? sj - R + 1 + tid : sj;
                    if (gi >= i0 && gi < i0 + th && gi < g.tnz && gj >= j0 && gj < j0 + 4 * nq && gj < g.tnx) {
                        const long long sc = so;
                        const float oxx = s_org[0], ozz = s_org[1];
                        auto lxx = [&](long long m) { return m == sc ? oxx : s_txx[m]; };
                        auto lzz = [&](long long m) { return m == sc ? ozz : s_tzz[m]; };
                        auto lxz = [&](long long m) { return s_txz[m]; };
                        const long long c = (gi - i0 + 2 * R) * W + gj - j0 + HX;
                        const long long o = cell_off(g, gi, gj);
                        qi[Q_TXS * P + o] = lbwd<R>(lxx, c, 1, a.k.cx) + lbwd<R>(lxz, c, W, a.k.cz);
                        qi[Q_TZS * P + o] = lfwd<R>(lzz, c, W, a.k.cz) + lfwd<R>(lxz, c, 1, a.k.cx);
                    }
                }
            }
        }
        __syncthreads();
        if (mine) stress(strip + ((t + 1) & 1) * xpar, p.tag0 + (unsigned)(t + 1 - p.t0), qo);
        if constexpr (QD == 2) {
            const bool keep = !p.some || (p.keep[(t - p.t0) >> 5] >> ((t - p.t0) & 31) & 1u);
            if (p.some) qo = p.q + (long long)nkept * p.state + T.slot * a.q_stride;
            nkept += keep;
            if (mine && keep)
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    if (gi0 + r >= g.tnz) break;
                    float *o = qo + co + r * g.pitch;
                    qst4s(o + VX * P, vx[r]);
                    qst4s(o + VZ * P, vz[r]);
                    qst4s(o + TXX * P, sxx[r]);
                    qst4s(o + TZZ * P, szz[r]);
                    qst4s(o + TXZ * P, sxz[r]);
                }
        }
        if (rec_o >= 0 && t + 1 < p.t1 && sub + 1 == p.dt_scale && k + 1 < p.nt_ext) record_v(k + 1);
        if (++sub == p.dt_scale) {
            sub = 0;
            ++k;
        }
        __syncthreads();
    }
    if (stop && rec_o >= 0)
        for (; k < p.nt_ext; ++k)
            for (int f = 0; f < 5; ++f)
                rec_tr[f * a.trace_plane + (long long)k * a.ns * a.nr] = __int_as_float(RES_NAN);
    if (!mine) return;
    const float nan = __int_as_float(RES_NAN);
    float *out = a.out + T.slot * a.out_stride;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        if (gi0 + r >= g.tnz) break;
        if (stop) vx[r] = vz[r] = sxx[r] = szz[r] = sxz[r] = make_float4(nan, nan, nan, nan);
        float *o = out + co + r * g.pitch;
        *reinterpret_cast<float4 *>(o + VX * P) = vx[r];
        *reinterpret_cast<float4 *>(o + VZ * P) = vz[r];
        *reinterpret_cast<float4 *>(o + TXX * P) = sxx[r];
        *reinterpret_cast<float4 *>(o + TZZ * P) = szz[r];
        *reinterpret_cast<float4 *>(o + TXZ * P) = sxz[r];
    }
}

// ---------------------------------------------------------------------------
// adjoint steps t_hi - 1 .. t_lo with imaging (adj_step's arithmetic)
// ---------------------------------------------------------------------------
// Each thread keeps its block's velocities and stresses in registers, and its
// gradient accumulators (one of the three only with one row per block).  Shared
// memory holds what neighbouring blocks difference (b * Av on the tile and its
// 2R halo; the sums of adj_sums and mu * Atxz on the tile and its ring), the
// block's lam and mu, and the ring's stresses and materials.
// What bounds it is latency: the exchange with the neighbours, two barriers and
// the chains between them.  A register spilled costs more than any arithmetic,
// since next to this much shared memory there is hardly an L1: 100 bytes of
// spills a thread cost a third of a 500 x 1000 survey's step.
template <int R, int RB>
__global__ void __launch_bounds__(RES_THREADS, 1) adj_resident(const __grid_constant__ AdjResArgs p)
{
    constexpr int NT = RES_THREADS, HX = ResShape<R>::HX, HG = ResShape<R>::HG;
    extern __shared__ float4 smem4[];
    __shared__ int s_stop, s_nslot, s_line[4][6], s_t[4];
    const AdjArgs &a = p.a;
    const Grid &g = a.g;
    const long long P = g.plane;
    const int tid = threadIdx.x;
    const ResTile T = res_tile<R, RB>(p.tl);
    // With three rows what the loop needs of the tile is read from shared memory, and a thread's places are
    // worked out again from its block's number in each phase: kept in registers, they would spill the fields.
    if (tid == 0) {
        s_t[0] = T.i0;
        s_t[1] = T.j0;
        s_t[2] = T.th;
        s_t[3] = T.nq;
    }
    const int i0 = T.i0, j0 = T.j0, th = T.th, nq = T.nq;
    constexpr int W = RES_W, PL = RES_PLANE, RING = ResShape<R>::RING;
    float *const sm = reinterpret_cast<float *>(smem4) + RES_PAD;
    // Cell (r, c) of the tile lies at (r + 2R) * W + HX + c of the first five planes, at r * OW + c of the others.
    float *const s_pvx = sm, *const s_pvz = sm + PL, *const s_px = sm + 2 * PL, *const s_pz = sm + 3 * PL, *const s_pxz = sm + 4 * PL;
    constexpr int OWN = RES_OWN<R, RB>;
    float *const s_lam = sm + 5 * PL, *const s_mu = s_lam + OWN;  // row r of a block at om + r * OM
    float *const s_rho = s_mu + OWN;                              // RB > 1: grho
    float *const s_set = s_rho + (RB < 2 ? 0 : OWN);              // [place][thread][4]: difference sets on their way
    float *const s_ring = s_set + 4 * RES_SETS<RB> * NT;          // [ring item][5][4]: its stresses, lam, mu
    float *const s_dx = s_ring + 20 * RING, *const s_mx = s_dx + W, *const s_dz = s_mx + W;  // damping; -dt on the domain's columns
    unsigned *const t_ring = reinterpret_cast<unsigned *>(s_dz + RES_ROWS);
    int *const t_rslot = reinterpret_cast<int *>(t_ring + RING);  // slots of the ring's items
    float *const s_res = reinterpret_cast<float *>(t_rslot + RING);  // [2][5][slots][4] staged residuals
    int *const t_dst = reinterpret_cast<int *>(s_res + 40 * p.slots);  // [4 slots] where a receiver's residual goes
    const int nring = (th + 2 * R) * (nq + 2) - th * nq;
    const float dt = a.k.dt;
    const float *in = a.in + T.slot * a.in_stride;
    const int frame = frame_count(RB * p.tl.bz, p.tl.nq, 2 * R, HG);
    const int xpar = 4 * gridDim.x * frame;
    const int shot = a.shot0 + T.slot;
    const int glo = a.npml + R, ghi_z = g.tnz - R - a.npml, ghi_x = g.tnx - R - a.npml;

    // receivers of the tile and its ring, per line: how many, the first one's
    // index, trace column and staged entry; [3]: all of them
    if (tid < 32) {
        int k0 = 0, n = 0;
        const Lines &L = a.lines;
        if (tid < L.n) line_range(L, tid, i0 - R, i0 + th + R, j0 - 4, j0 + 4 * nq + 4, k0, n);
        const int n0 = __shfl_sync(0xffffffffu, n, 0), n1 = __shfl_sync(0xffffffffu, n, 1), n2 = __shfl_sync(0xffffffffu, n, 2);
        if (tid < L.n) {
            s_line[tid][0] = n;
            s_line[tid][1] = k0;
            s_line[tid][2] = shot * a.nr + L.slot0[tid] + k0;
            s_line[tid][3] = tid == 0 ? 0 : tid == 1 ? n0 : n0 + n1;
        }
        if (tid == 0) {
            s_line[3][0] = n0 + n1 + n2;
            s_nslot = 0;
            s_stop = ld_relaxed_gpu(p.err) != 0;
        }
    }
    for (int e = tid; e < 40 * p.slots; e += NT) s_res[e] = 0.f;
    __syncthreads();
    const int nrec = s_line[3][0];
    // A slot of staged residuals for each line with receivers on the four cells from (gi, gj): 10 bits
    // a line, slot + 1.
    auto slots_of = [&](int gi, int gj) {
        int w = 0;
        for (int l = 0; nrec && l < a.lines.n; ++l) {
            int slot = 0;
            for (int c = 0; c < 4; ++c) {
                const int ks = line_slot(a.lines, l, gi, gj + c);
                if (ks < 0) continue;
                if (!slot) slot = atomicAdd(&s_nslot, 1) + 1;
                t_dst[s_line[l][3] + ks - s_line[l][1]] = 4 * (slot - 1) + c;
            }
            w |= slot << 10 * l;
        }
        return w;
    };
    for (int e = tid; e < (th + 4 * R) * (nq + 2 * HG); e += NT) {
        const int r = e / (nq + 2 * HG), q = e - r * (nq + 2 * HG), o = r * W + 4 * q;
        const int gi = i0 - 2 * R + r, gj = j0 - HX + 4 * q;
        const float4 b = ld4(a.mat + 2 * P, g, gi, gj);
        st4s(s_pvx + o, times4(ld4(in + VX * P, g, gi, gj), b));
        st4s(s_pvz + o, times4(ld4(in + VZ * P, g, gi, gj), b));
    }
    for (int e = tid; e < nring; e += NT) {
        int r, q;
        frame_item(e, th + 2 * R, nq + 2, R, 1, r, q);
        t_ring[e] = pack_item(r, q);
        const int gi = i0 - R + r, gj = j0 - 4 + 4 * q;
        t_rslot[e] = slots_of(gi, gj);
        float *s = s_ring + 20 * e;
        st4s(s, ld4(in + TXX * P, g, gi, gj));
        st4s(s + 4, ld4(in + TZZ * P, g, gi, gj));
        st4s(s + 8, ld4(in + TXZ * P, g, gi, gj));
        st4s(s + 12, ld4(a.mat, g, gi, gj));
        st4s(s + 16, ld4(a.mat + P, g, gi, gj));
    }
    for (int e = tid; e < 4 * nq + 2 * HX; e += NT) {
        const int c = j0 - HX + e + XO;
        s_dx[e] = c >= 0 && c < g.pitch ? __ldg(a.dampx + c) : 0.f;
        s_mx[e] = in_domain(g, R, R, j0 - HX + e) ? -dt : 0.f;
    }
    for (int e = tid; e < th + 4 * R; e += NT) {
        const int i = i0 - 2 * R + e + ZO;
        s_dz[e] = i >= 0 && i < g.rows ? __ldg(a.dampz + i) : 0.f;
    }

    // this thread's block
    const bool mine = tid < T.nblk, inside = tid < T.nin;
    int bz = 0, bq = 0;
    if (mine) res_block<R, RB>(T, tid, bz, bq);
    const int br = bz * RB;
    const int ot = (br + 2 * R) * W + HX + 4 * bq;
    constexpr int OM = RB < 3 ? 4 * NT : ResShape<R>::OW;
    const int om = RB < 3 ? 4 * tid : br * OM + 4 * bq;
    const int gi0 = i0 + br, gj0 = j0 + 4 * bq;
    const int co = (gi0 + ZO) * g.pitch + gj0 + XO;
    const unsigned own = (unsigned)bz << 8 | (unsigned)bq;
    struct Own {
        int br, bq, ot, gi0, gj0;
    };
    auto place = [&]() {
        unsigned w = own;
        if (RB == 3) asm volatile("" : "+r"(w));  // anew each time
        Own o;
        o.br = RB * (int)(w >> 8);
        o.bq = (int)(w & 255u);
        o.ot = (o.br + 2 * R) * W + HX + 4 * o.bq;
        o.gi0 = (RB == 3 ? s_t[0] : i0) + o.br;
        o.gj0 = (RB == 3 ? s_t[1] : j0) + 4 * o.bq;
        return o;
    };
    auto om_of = [&](const Own &o) { return RB < 3 ? 4 * tid : o.br * OM + 4 * o.bq; };
    auto co_of = [&](const Own &o) { return (o.gi0 + ZO) * g.pitch + o.gj0 + XO; };
    float4 vx[RB], vz[RB], ax[RB], az[RB], axz[RB];
    float4 gmu[RB], glam[RB], grho;  // its gradient accumulators
    int rs[RB];         // its slots of staged residuals
    unsigned img = 0;   // rows with imaged cells
    float *const G = a.gacc + T.slot * a.gacc_stride;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        vx[r] = vz[r] = ax[r] = az[r] = axz[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        gmu[r] = glam[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (RB < 2) grho = gmu[r];
        rs[r] = 0;
        if (!mine) continue;
        const int gi = gi0 + r;
        vx[r] = ld4(in + VX * P, g, gi, gj0);
        vz[r] = ld4(in + VZ * P, g, gi, gj0);
        ax[r] = ld4(in + TXX * P, g, gi, gj0);
        az[r] = ld4(in + TZZ * P, g, gi, gj0);
        axz[r] = ld4(in + TXZ * P, g, gi, gj0);
        st4s(s_lam + om + r * OM, ld4(a.mat, g, gi, gj0));
        st4s(s_mu + om + r * OM, ld4(a.mat + P, g, gi, gj0));
        if (gi < g.tnz) {
            gmu[r] = *reinterpret_cast<const float4 *>(G + co + r * g.pitch);
            glam[r] = *reinterpret_cast<const float4 *>(G + P + co + r * g.pitch);
            const float4 gr = *reinterpret_cast<const float4 *>(G + 2 * P + co + r * g.pitch);
            if (RB < 2)
                grho = gr;
            else
                st4s(s_rho + om + r * OM, gr);
        }
        rs[r] = slots_of(gi, gj0);
        if (gi >= glo && gi <= ghi_z && gj0 + 3 >= glo && gj0 <= ghi_x) img |= 1u << r;
    }
    __syncthreads();

    const bool res_v = nrec && (a.res[VX] || a.res[VZ]), res_s = nrec && (a.res[TXX] || a.res[TZZ] || a.res[TXZ]);
    // This thread's receiver (the tile and its ring have fewer than there are threads): where its residuals
    // go and its trace column.
    int rec_d = -1, rec_c = 0;
    for (int l = 0, e = tid; l < a.lines.n; e -= s_line[l++][0])
        if (e >= 0 && e < s_line[l][0]) {
            rec_d = t_dst[s_line[l][3] + e];
            rec_c = s_line[l][2] + e;
        }
    // Its residuals of row `row`, step t, into buffer t & 1.
    auto stage = [&](int row, int t) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(s_res + (t & 1) * 20 * p.slots + rec_d);
        const long long o = (long long)row * a.ns * a.nr + rec_c;
#pragma unroll
        for (int f = 0; f < 5; ++f)
            if (a.res[f])
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d + f * 16 * p.slots), "l"(a.res[f] + o) : "memory");
    };
    // Adds the staged residuals of field f, step t, of the slots in w to a group, one receiver line after
    // another (the cells of a slot without a receiver hold zero).
    auto inject = [&](float4 &v, int t, int f, int w) {
        const float *d = s_res + ((t & 1) * 5 + f) * 4 * p.slots;
        for (; w; w = (int)((unsigned)w >> 10)) {
            const int s = w & 1023;
            if (!s) continue;
            const float4 x = ld4s(d + 4 * (s - 1));
            v.x += x.x;
            v.y += x.y;
            v.z += x.z;
            v.w += x.w;
        }
    };
    const int t_first = p.t_hi - 1;
    const unsigned halo = halo_group<R>(g, p.tl, frame, T.slot, T.tz, T.tx, i0, th, T.q0, nq);
    // word w of a group holds values 3 w .. of its 4 vx and 4 vz products
    auto put = [&](int o, const uint4 (&w)[3]) {
        auto f = [](unsigned u) { return __uint_as_float(u); };
        st4s(s_pvx + o, make_float4(f(w[0].x), f(w[0].y), f(w[0].z), f(w[1].x)));
        st4s(s_pvz + o, make_float4(f(w[1].y), f(w[1].z), f(w[2].x), f(w[2].y)));
    };
    // A step injects where its t mod dt_scale is 0 (step 0 never runs); kept by counting down: that of t, and
    // the residual row of the next injecting step below t.
    int sub_t = t_first % p.dt_scale;
    int row = inj_row_dev((t_first - 1) / p.dt_scale * p.dt_scale, p.nt, p.nt_ext, p.dt_scale);

    // What the adjoint velocities difference, from new stresses.
    auto sums = [&](const float4 &l, const float4 &m, const float4 &x, const float4 &z, const float4 &xz, int o) {
        float4 sx, sz;
        adj_sums(l.x, m.x, x.x, z.x, sx.x, sz.x);
        adj_sums(l.y, m.y, x.y, z.y, sx.y, sz.y);
        adj_sums(l.z, m.z, x.z, z.z, sx.z, sz.z);
        adj_sums(l.w, m.w, x.w, z.w, sx.w, sz.w);
        st4s(s_px + o, sx);
        st4s(s_pz + o, sz);
        st4s(s_pxz + o, times4(m, xz));
    };
    // -dt on the cells of a row that are updated, else zero (x + 0 * y = x).
    auto step4 = [&](int gi, int c) { return gi >= R && gi <= g.tnz - R ? ld4s(s_mx + c) : make_float4(0.f, 0.f, 0.f, 0.f); };
    // New stresses of four cells from their differences Dx+ (b vx), Dz- (b vz), Dz+ (b vx) + Dx- (b vz).
    auto update = [&](float4 &x, float4 &z, float4 &xz, const float4 &dx, float dz, const float4 &md, const float (&ex)[4],
                      const float (&ez)[4], const float (&exz)[4]) {
        float ox[4], oz[4], oxz[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            ox[k] = f4(x, k) + f4(md, k) * (f4(dx, k) * f4(x, k) + ex[k]);
            oz[k] = f4(z, k) + f4(md, k) * (dz * f4(z, k) + ez[k]);
            oxz[k] = f4(xz, k) + f4(md, k) * ((f4(dx, k) + dz) * f4(xz, k) + exz[k]);
        }
        x = mk4(ox);
        z = mk4(oz);
        xz = mk4(oxz);
    };

    // The strip group of row r of the tile in this thread's column, -1: none.
    auto strip_group = [&](int r, int q) {
        const int h = RB == 3 ? s_t[2] : th, w = RB == 3 ? s_t[3] : nq;
        return r < 2 * R || r >= h - 2 * R || q < HG || q >= w - HG ? frame_index(r, q, h, w, 2 * R, HG) : -1;
    };

    // Difference sets of step t.  One or two rows read a row's into registers, ahead of their use, and ask for
    // those of the step after it into L2.
    auto sets_of = [&](int t) { return p.q + (long long)(t - p.q_t0) * p.state + T.slot * a.fwd_stride + co_of(place()); };
    float4 qv[5];
    auto load_set = [&](int t, int r) {
        if (!(img >> r & 1)) return;
        const float *q = sets_of(t) + r * g.pitch;
#pragma unroll
        for (int f = 0; f < 5; ++f) qv[f] = qld4s(q + f * P);
        if (t > p.t_lo)
#pragma unroll
            for (int f = 0; f < 5; ++f) qprefetch4(q + f * P - p.state);
    };
    // With three rows asynchronous copies, by each thread for itself: the little L1 that this much shared memory
    // leaves holds up plain loads, and their registers spill.  500 x 1000 cells, 4 shots: 44.2 us per step
    // with loads, 37.6 with copies.
    auto set_at = [&](int place) { return ld4s(s_set + 4 * (place * NT + tid)); };
    auto ask = [&](const float *q, int f, int r, int place) {
        if (img >> r & 1)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                             (unsigned)__cvta_generic_to_shared(s_set + 4 * (place * NT + tid))),
                         "l"(q + f * P + r * g.pitch)
                         : "memory");
    };
    // What the new stresses of row r add to the gradient (in the step kernels' contractions).
    auto image_stress = [&](int r, int gj0, const float4 &q0, const float4 &q1, const float4 &q2) {
        if (img >> r & 1) {
            float m0[4], m1[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                m0[k] = f4(gmu[r], k);
                m1[k] = f4(glam[r], k);
                if (gj0 + k >= glo && gj0 + k <= ghi_x) {
                    const float atx = f4(ax[r], k), atz = f4(az[r], k), atxz = f4(axz[r], k);
                    image_stress_terms(dt, atx, atz, atxz, f4(q0, k), f4(q1, k), f4(q2, k), m0[k], m1[k]);
                }
            }
            gmu[r] = mk4(m0);
            glam[r] = mk4(m1);
        }
    };
    // And its new velocities.
    auto image_velocity = [&](int r, int gj0, int om, const float4 &b, const float4 &q3, const float4 &q4) {
        if (img >> r & 1) {
            const float4 gr4 = RB < 2 ? grho : ld4s(s_rho + om + r * OM);
            float m2[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                m2[k] = f4(gr4, k);
                if (gj0 + k >= glo && gj0 + k <= ghi_x) {
                    const float bk = f4(b, k), avx = f4(vx[r], k), avz = f4(vz[r], k);
                    image_velocity_terms(dt, bk, avx, avz, f4(q3, k), f4(q4, k), m2[k]);
                }
            }
            if (RB < 2)
                grho = mk4(m2);
            else
                st4s(s_rho + om + r * OM, mk4(m2));
        }
    };
    // New stresses of the block.
    auto stress = [&]() {
        const Own o = place();
        const int om = om_of(o);
        const float4 dx = ld4s(s_dx + HX + 4 * o.bq);
        {
            auto row = [&](int r) { return ld4s(s_pvx + o.ot + r * W); };
            ZSlide<R, true> zx(row);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const float4 md = step4(o.gi0 + r, HX + 4 * o.bq);
                const float dz = s_dz[o.br + r + 2 * R];
                float x[12], ox[4], oxz[4];
                zx.next(row(r + R));
                xrow<R, true>(x, zx.centre(), s_pvx + o.ot + r * W);
#pragma unroll
                for (int k = 0; k < 4; ++k) ox[k] = f4(ax[r], k) + f4(md, k) * (f4(dx, k) * f4(ax[r], k) + xfwd<R>(x, k, a.k.cx));
                xrow<R, false>(x, ld4s(s_pvz + o.ot + r * W), s_pvz + o.ot + r * W);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    oxz[k] = f4(axz[r], k) + f4(md, k) * ((f4(dx, k) + dz) * f4(axz[r], k) +
                                                         (zx.at(k, a.k.cz) + xbwd<R>(x, k, a.k.cx)));
                ax[r] = mk4(ox);
                axz[r] = mk4(oxz);
            }
        }
        auto row = [&](int r) { return ld4s(s_pvz + o.ot + r * W); };
        ZSlide<R, false> zz(row);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const float4 md = step4(o.gi0 + r, HX + 4 * o.bq);
            const float dz = s_dz[o.br + r + 2 * R];
            zz.next(row(r + R - 1));
            float oz[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) oz[k] = f4(az[r], k) + f4(md, k) * (dz * f4(az[r], k) + zz.at(k, a.k.cz));
            az[r] = mk4(oz);
            sums(ld4s(s_lam + om + r * OM), ld4s(s_mu + om + r * OM), ax[r], az[r], axz[r], o.ot + r * W);
        }
    };
    // New stresses of ring item e, first, where it is due, what the residual of step t adds to them.
    auto ring = [&](int e, int t, bool due) {
        const int r = item_row(t_ring[e]), q = item_col(t_ring[e]), c = (r + R) * W + HX - 4 + 4 * q;
        float x[12], ex[4], ez[4], exz[4];
        {
            const ZWindow<R, 1, true> zx([&](int) { return ld4s(s_pvx + c); }, s_pvx + c);
            xrow<R, true>(x, zx.w[R - 1], s_pvx + c);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                ex[k] = xfwd<R>(x, k, a.k.cx);
                exz[k] = zx.at(0, k, a.k.cz);
            }
        }
        in_order();
        {
            const ZWindow<R, 1, false> zz([&](int) { return ld4s(s_pvz + c); }, s_pvz + c);
            xrow<R, false>(x, zz.w[R], s_pvz + c);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                ez[k] = zz.at(0, k, a.k.cz);
                exz[k] += xbwd<R>(x, k, a.k.cx);
            }
        }
        in_order();
        float *s = s_ring + 20 * e;
        float4 x4 = ld4s(s), z4 = ld4s(s + 4), xz4 = ld4s(s + 8);
        const int w = t_rslot[e];
        if (due && w) {
            if (a.res[TXX]) inject(x4, t, TXX, w);
            if (a.res[TZZ]) inject(z4, t, TZZ, w);
            if (a.res[TXZ]) inject(xz4, t, TXZ, w);
        }
        update(x4, z4, xz4, ld4s(s_dx + HX - 4 + 4 * q), s_dz[r + R], step4(s_t[0] - R + r, HX - 4 + 4 * q), ex, ez, exz);
        st4s(s, x4);
        st4s(s + 4, z4);
        st4s(s + 8, xz4);
        sums(ld4s(s + 12), ld4s(s + 16), x4, z4, xz4, c);
    };

    // The first copies for step t: two rows' for the stresses; the others are asked into L2.
    auto ask_first = [&](int t) {
        const float *q = sets_of(t);
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int f = 0; f < 5; ++f)
                if (r < 2 && f < 3)
                    ask(q, f, r, 3 * r + f);
                else if (img >> r & 1)
                    qprefetch4(q + f * P + r * g.pitch);
        cp_commit();
    };
    if (RB == 3) ask_first(t_first);

    // ring items go to the threads without a block first, then to those inside
    const int rank = tid >= T.nblk ? tid - T.nblk : tid + NT - T.nblk;
    bool stop = s_stop;
    for (int t = t_first; t >= p.t_lo && !stop; --t) {
        // the residual that this step's input lacks in its stresses (the first state of a launch has it)
        const bool due = res_s && t < t_first && sub_t == 0;
        if (due) {
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                if (!rs[r]) continue;
                if (a.res[TXX]) inject(ax[r], t, TXX, rs[r]);
                if (a.res[TZZ]) inject(az[r], t, TZZ, rs[r]);
                if (a.res[TXZ]) inject(axz[r], t, TXZ, rs[r]);
            }
        }
        sub_t = sub_t ? sub_t - 1 : p.dt_scale - 1;  // of t - 1
        const bool epi = nrec && t > 1 && sub_t == 0;
        if (epi) {  // what this step adds at its end, on its way meanwhile
            if (rec_d >= 0) stage(row, t - 1);
            row = row ? row - 1 : p.nt_ext - 1;
        }
        cp_commit();
        // stresses: the blocks inside, then, with the halo, the others
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            if (pass == 1 && t < t_first) {  // the neighbours' products of this step's input
                if (!fetch_group<3>(p.xch + (t & 1) * xpar, p.tag0 + (unsigned)(t_first - t), halo, p.err, p.limit_ns, put))
                    s_stop = 1;
                __syncthreads();
                stop = s_stop;
                if (stop) break;
            }
            if (mine && inside == (pass == 0)) {
                if (RB == 3) cp_wait<1>();
                stress();
                if (RB == 3) {
                    const int gj = place().gj0;
                    image_stress(0, gj, set_at(0), set_at(1), set_at(2));
                    image_stress(1, gj, set_at(3), set_at(4), set_at(5));
                    const float *q = sets_of(t);
                    for (int f = 0; f < 3; ++f) ask(q, f, 2, f);
                    for (int f = 3; f < 5; ++f) ask(q, f, 0, f);
                    cp_commit();
                }
            }
        }
        if (stop) break;
        for (int e = rank; e < nring; e += NT) ring(e, t, due);
        if (RB < 3) load_set(t, 0);
        // the staged residuals are there
        if (RB == 3 && mine)
            cp_wait<1>();
        else
            cp_wait<0>();
        __syncthreads();
        if (mine) {
            const Own o = place();
            const float *gb = a.mat + 2 * P + co_of(o);
            uint4 *const xo = p.xch + 4 * blockIdx.x * frame + ((t - 1) & 1) * xpar;  // what step t - 1 reads
            const unsigned tag = p.tag0 + (unsigned)(t_first - t + 1);
            const float4 dx4 = ld4s(s_dx + HX + 4 * o.bq);
            {
                auto row = [&](int r) { return ld4s(s_pxz + o.ot + r * W); };
                ZSlide<R, false> zxz(row);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const float4 m4 = step4(o.gi0 + r, HX + 4 * o.bq);
                    const float dz = s_dz[o.br + r + 2 * R];
                    zxz.next(row(r + R - 1));
                    float x[12], nx[4];
                    xrow<R, false>(x, ld4s(s_px + o.ot + r * W), s_px + o.ot + r * W);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        nx[k] = f4(vx[r], k) + f4(m4, k) * ((2.f * f4(dx4, k) + dz) * f4(vx[r], k) +
                                                          (xbwd<R>(x, k, a.k.cx) + zxz.at(k, a.k.cz)));
                    vx[r] = mk4(nx);
                }
            }
            if (RB == 3) {
                cp_wait<0>();
                image_stress(RB - 1, o.gj0, set_at(0), set_at(1), set_at(2));
                const float *q = sets_of(t);
                ask(q, 3, 1, 0);
                ask(q, 4, 1, 1);
                ask(q, 3, 2, 2);
                ask(q, 4, 2, 5);
                cp_commit();
            }
            auto row = [&](int r) { return ld4s(s_pz + o.ot + r * W); };
            ZSlide<R, true> zz(row);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const float4 m4 = step4(o.gi0 + r, HX + 4 * o.bq);
                const float dz = s_dz[o.br + r + 2 * R];
                const float4 b = __ldg(reinterpret_cast<const float4 *>(gb + r * g.pitch));
                zz.next(row(r + R));
                float x[12], nz[4];
                xrow<R, true>(x, ld4s(s_pxz + o.ot + r * W), s_pxz + o.ot + r * W);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    nz[k] = f4(vz[r], k) + f4(m4, k) * ((f4(dx4, k) + 2.f * dz) * f4(vz[r], k) +
                                                      (zz.at(k, a.k.cz) + xfwd<R>(x, k, a.k.cx)));
                vz[r] = mk4(nz);
                if (RB < 3) {
                    image_stress(r, o.gj0, qv[0], qv[1], qv[2]);
                    image_velocity(r, o.gj0, om_of(o), b, qv[3], qv[4]);
                    if (r + 1 < RB) load_set(t, r + 1);
                }
                float4 px = vx[r], pzz = vz[r];
                if (epi && res_v && rs[r]) {  // with what step t - 1 finds in its input
                    if (a.res[VX]) inject(px, t - 1, VX, rs[r]);
                    if (a.res[VZ]) inject(pzz, t - 1, VZ, rs[r]);
                }
                if (RB < 3) {
                    vx[r] = px;
                    vz[r] = pzz;
                }
                px = times4(px, b);
                pzz = times4(pzz, b);
                st4s(s_pvx + o.ot + r * W, px);
                st4s(s_pvz + o.ot + r * W, pzz);
                if (!inside) {
                    const int s = strip_group(o.br + r, o.bq);
                    if (s >= 0) {
                        st_word(xo + 4 * s, px.x, px.y, px.z, tag);
                        st_word(xo + 4 * s + 1, px.w, pzz.x, pzz.y, tag);
                        st_word(xo + 4 * s + 2, pzz.z, pzz.w, 0.f, tag);
                    }
                }
            }
        }
        __syncthreads();
        if (RB == 3 && mine) {  // with the strips on their way
            cp_wait<0>();
            {
                const Own o = place();
                const float *gb = a.mat + 2 * P + co_of(o);
#pragma unroll
                for (int r = 0; r < RB; ++r)
                    image_velocity(r, o.gj0, om_of(o), __ldg(reinterpret_cast<const float4 *>(gb + r * g.pitch)),
                                   set_at(r == 0 ? 3 : r == 1 ? 0 : 2), set_at(r == 0 ? 4 : r == 1 ? 1 : 5));
            }
            if (epi && res_v) {
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    if (!rs[r]) continue;
                    if (a.res[VX]) inject(vx[r], t - 1, VX, rs[r]);
                    if (a.res[VZ]) inject(vz[r], t - 1, VZ, rs[r]);
                }
            }
            if (t > p.t_lo) ask_first(t - 1);
        }
    }
    if (!mine) return;
    // the state that step t_lo - 1 finds, its residual included
    const bool last = res_s && p.t_lo > 1 && sub_t == 0;
    const float nan = __int_as_float(RES_NAN);
    float *out = a.out + T.slot * a.out_stride;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        if (gi0 + r >= g.tnz) break;
        if (last && rs[r]) {
            if (a.res[TXX]) inject(ax[r], p.t_lo - 1, TXX, rs[r]);
            if (a.res[TZZ]) inject(az[r], p.t_lo - 1, TZZ, rs[r]);
            if (a.res[TXZ]) inject(axz[r], p.t_lo - 1, TXZ, rs[r]);
        }
        if (stop) {
            vx[r] = vz[r] = ax[r] = az[r] = axz[r] = make_float4(nan, nan, nan, nan);
            gmu[r] = glam[r] = vx[r];
            if (RB < 2)
                grho = vx[r];
            else
                st4s(s_rho + om + r * OM, vx[r]);
        }
        float *o = out + co + r * g.pitch;
        *reinterpret_cast<float4 *>(o + VX * P) = vx[r];
        *reinterpret_cast<float4 *>(o + VZ * P) = vz[r];
        *reinterpret_cast<float4 *>(o + TXX * P) = ax[r];
        *reinterpret_cast<float4 *>(o + TZZ * P) = az[r];
        *reinterpret_cast<float4 *>(o + TXZ * P) = axz[r];
        *reinterpret_cast<float4 *>(G + co + r * g.pitch) = gmu[r];
        *reinterpret_cast<float4 *>(G + P + co + r * g.pitch) = glam[r];
        *reinterpret_cast<float4 *>(G + 2 * P + co + r * g.pitch) = RB < 2 ? grho : ld4s(s_rho + om + r * OM);
    }
}

// ---------------------------------------------------------------------------
// exact adjoint steps t_hi - 1 .. t_lo (exact_adj_step's formulas)
// ---------------------------------------------------------------------------
// The transpose runs as the forward loop does, velocities from differences of
// three stress planes (P1 .. P3), then stresses from differences of two
// velocity planes (Q1, Q2), so it exchanges and recomputes what that does: the
// P planes' outermost 2R rows and columns, the Q planes of the ring.  The
// residuals are staged as in adj_resident, and added to the new state at the
// end of a step (to the ring's velocities at the start of the next one).  The
// materials are zero outside the update domain, which is all that keeps P and Q
// zero there.  Latency bounds it, as the other loops: for 101 x 203 cells and 4
// shots a step took 15.6 us in exact_adj_step and 3.5 in the injection after it,
// and takes 4.0 us here.
template <int R, int RB>
__global__ void __launch_bounds__(RES_THREADS, 1) exact_resident(const __grid_constant__ AdjResArgs p)
{
    constexpr int NT = RES_THREADS, HX = ResShape<R>::HX, HG = ResShape<R>::HG;
    extern __shared__ float4 smem4[];
    __shared__ int s_stop, s_nslot, s_line[4][6];
    const AdjArgs &a = p.a;
    const Grid &g = a.g;
    const long long P = g.plane;
    const int tid = threadIdx.x;
    const ResTile T = res_tile<R, RB>(p.tl);
    const int i0 = T.i0, j0 = T.j0, th = T.th, nq = T.nq;
    constexpr int W = RES_W, PL = RES_PLANE, RING = ResShape<R>::RING, OWN = RES_OWN<R, RB>;
    float *const sm = reinterpret_cast<float *>(smem4) + RES_PAD;
    // Cell (r, c) of the tile lies at (r + 2R) * W + HX + c of every plane.
    float *const s_p1 = sm, *const s_p2 = sm + PL, *const s_p3 = sm + 2 * PL, *const s_q1 = sm + 3 * PL, *const s_q2 = sm + 4 * PL;
    float *const s_lam = sm + 5 * PL, *const s_mu = s_lam + OWN;  // [row][thread][4] of the blocks
    float *const s_ring = s_mu + OWN;                             // [ring item][3][4]: its velocities, buoyancy
    float *const s_dx = s_ring + 12 * RING, *const s_dz = s_dx + W;  // damping
    unsigned *const t_ring = reinterpret_cast<unsigned *>(s_dz + RES_ROWS);
    int *const t_rslot = reinterpret_cast<int *>(t_ring + RING);
    unsigned *const t_word = reinterpret_cast<unsigned *>(t_rslot + RING);
    float *const s_res = reinterpret_cast<float *>(t_word + 4 * RES_THREADS);  // [2][5][slots][4] staged residuals
    int *const t_dst = reinterpret_cast<int *>(s_res + 40 * p.slots);
    const int nring = (th + 2 * R) * (nq + 2) - th * nq;
    const float dt = a.k.dt;
    const float *in = a.in + T.slot * a.in_stride;
    const int frame = frame_count(RB * p.tl.bz, p.tl.nq, 2 * R, HG);
    const int xpar = 4 * gridDim.x * frame;
    uint4 *const strip = p.xch + 4 * blockIdx.x * frame;
    const int shot = a.shot0 + T.slot;

    // receivers of the tile and its ring, as in adj_resident
    if (tid < 32) {
        int k0 = 0, n = 0;
        const Lines &L = a.lines;
        if (tid < L.n) line_range(L, tid, i0 - R, i0 + th + R, j0 - 4, j0 + 4 * nq + 4, k0, n);
        const int n0 = __shfl_sync(0xffffffffu, n, 0), n1 = __shfl_sync(0xffffffffu, n, 1), n2 = __shfl_sync(0xffffffffu, n, 2);
        if (tid < L.n) {
            s_line[tid][0] = n;
            s_line[tid][1] = k0;
            s_line[tid][2] = shot * a.nr + L.slot0[tid] + k0;
            s_line[tid][3] = tid == 0 ? 0 : tid == 1 ? n0 : n0 + n1;
        }
        if (tid == 0) {
            s_line[3][0] = n0 + n1 + n2;
            s_nslot = 0;
            s_stop = ld_relaxed_gpu(p.err) != 0;
        }
    }
    for (int e = tid; e < 40 * p.slots; e += NT) s_res[e] = 0.f;
    for (int e = tid; e < 4 * nq + 2 * HX; e += NT) {
        const int c = j0 - HX + e + XO;
        s_dx[e] = c >= 0 && c < g.pitch ? __ldg(a.dampx + c) : 0.f;
    }
    for (int e = tid; e < th + 4 * R; e += NT) {
        const int i = i0 - 2 * R + e + ZO;
        s_dz[e] = i >= 0 && i < g.rows ? __ldg(a.dampz + i) : 0.f;
    }
    __syncthreads();
    const int nrec = s_line[3][0];
    auto slots_of = [&](int gi, int gj) {
        int w = 0;
        for (int l = 0; nrec && l < a.lines.n; ++l) {
            int slot = 0;
            for (int c = 0; c < 4; ++c) {
                const int ks = line_slot(a.lines, l, gi, gj + c);
                if (ks < 0) continue;
                if (!slot) slot = atomicAdd(&s_nslot, 1) + 1;
                t_dst[s_line[l][3] + ks - s_line[l][1]] = 4 * (slot - 1) + c;
            }
            w |= slot << 10 * l;
        }
        return w;
    };
    auto masked = [&](const float *plane, int gi, int gj) {
        float4 v = ld4(plane, g, gi, gj);
        if (!in_domain(g, R, gi, gj)) v.x = 0.f;
        if (!in_domain(g, R, gi, gj + 1)) v.y = 0.f;
        if (!in_domain(g, R, gi, gj + 2)) v.z = 0.f;
        if (!in_domain(g, R, gi, gj + 3)) v.w = 0.f;
        return v;
    };
    // 1 - dt d of four cells: column place c of s_dx, row place r of s_dz
    auto damp4_of = [&](int r, int c) {
        const float4 dx = ld4s(s_dx + c);
        const float dz = s_dz[r];
        return make_float4(exact_damp(dt, dx.x, dz), exact_damp(dt, dx.y, dz), exact_damp(dt, dx.z, dz), exact_damp(dt, dx.w, dz));
    };
    // P1 .. P3 of four cells
    auto products = [&](const float4 &l, const float4 &m, const float4 &d, const float4 &xx, const float4 &zz, const float4 &xz,
                        float4 &p1, float4 &p2, float4 &p3) {
        float v1[4], v2[4], v3[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            exact_products(dt, f4(l, k), f4(m, k), __fmul_rn(f4(d, k), f4(xx, k)), __fmul_rn(f4(d, k), f4(zz, k)),
                           __fmul_rn(f4(d, k), f4(xz, k)), v1[k], v2[k], v3[k]);
        }
        p1 = mk4(v1);
        p2 = mk4(v2);
        p3 = mk4(v3);
    };
    for (int e = tid; e < (th + 4 * R) * (nq + 2 * HG); e += NT) {
        const int r = e / (nq + 2 * HG), q = e - r * (nq + 2 * HG), o = r * W + 4 * q;
        const int gi = i0 - 2 * R + r, gj = j0 - HX + 4 * q;
        float4 p1, p2, p3;
        products(masked(a.mat, gi, gj), masked(a.mat + P, gi, gj), damp4_of(r, 4 * q), ld4(in + TXX * P, g, gi, gj),
                 ld4(in + TZZ * P, g, gi, gj), ld4(in + TXZ * P, g, gi, gj), p1, p2, p3);
        st4s(s_p1 + o, p1);
        st4s(s_p2 + o, p2);
        st4s(s_p3 + o, p3);
    }
    for (int e = tid; e < nring; e += NT) {
        int r, q;
        frame_item(e, th + 2 * R, nq + 2, R, 1, r, q);
        t_ring[e] = pack_item(r, q);
        const int gi = i0 - R + r, gj = j0 - 4 + 4 * q;
        t_rslot[e] = slots_of(gi, gj);
        float *s = s_ring + 12 * e;
        st4s(s, ld4(in + VX * P, g, gi, gj));
        st4s(s + 4, ld4(in + VZ * P, g, gi, gj));
        st4s(s + 8, masked(a.mat + 2 * P, gi, gj));
    }

    // this thread's block
    const bool mine = tid < T.nblk, inside = tid < T.nin;
    int bz = 0, bq = 0;
    if (mine) res_block<R, RB>(T, tid, bz, bq);
    const int br = bz * RB;
    const int ot = (br + 2 * R) * W + HX + 4 * bq;
    const int gi0 = i0 + br, gj0 = j0 + 4 * bq;
    const int co = (gi0 + ZO) * g.pitch + gj0 + XO;
    float4 vx[RB], vz[RB], xx[RB], zz[RB], xz[RB], b[RB];
    float4 glam[RB], gmu[RB], gb[RB];  // its gradient accumulators
    int rs[RB];
    unsigned img = 0;                  // rows of the update domain
    float *const G = a.gacc + T.slot * a.gacc_stride;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        vx[r] = vz[r] = xx[r] = zz[r] = xz[r] = b[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        glam[r] = gmu[r] = gb[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        rs[r] = 0;
        if (!mine) continue;
        const int gi = gi0 + r;
        vx[r] = ld4(in + VX * P, g, gi, gj0);
        vz[r] = ld4(in + VZ * P, g, gi, gj0);
        xx[r] = ld4(in + TXX * P, g, gi, gj0);
        zz[r] = ld4(in + TZZ * P, g, gi, gj0);
        xz[r] = ld4(in + TXZ * P, g, gi, gj0);
        b[r] = masked(a.mat + 2 * P, gi, gj0);
        st4s(s_lam + 4 * (r * NT + tid), masked(a.mat, gi, gj0));
        st4s(s_mu + 4 * (r * NT + tid), masked(a.mat + P, gi, gj0));
        if (gi < g.tnz) {
            glam[r] = *reinterpret_cast<const float4 *>(G + co + r * g.pitch);
            gmu[r] = *reinterpret_cast<const float4 *>(G + P + co + r * g.pitch);
            gb[r] = *reinterpret_cast<const float4 *>(G + 2 * P + co + r * g.pitch);
        }
        rs[r] = slots_of(gi, gj0);
        if (gi >= R && gi <= g.tnz - R && gj0 + 3 >= R && gj0 <= g.tnx - R) img |= 1u << r;
    }
    __syncthreads();

    int rec_d = -1, rec_c = 0;
    for (int l = 0, e = tid; l < a.lines.n; e -= s_line[l++][0])
        if (e >= 0 && e < s_line[l][0]) {
            rec_d = t_dst[s_line[l][3] + e];
            rec_c = s_line[l][2] + e;
        }
    auto stage = [&](int row, int t) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(s_res + (t & 1) * 20 * p.slots + rec_d);
        const long long o = (long long)row * a.ns * a.nr + rec_c;
#pragma unroll
        for (int f = 0; f < 5; ++f)
            if (a.res[f])
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d + f * 16 * p.slots), "l"(a.res[f] + o) : "memory");
    };
    // Adds the staged residuals of step t to field f of a group: line after line, and the residual of a line's vz
    // trace to the field it was recorded from.
    auto add4 = [&](float4 &v, int t, int f, int slot) {
        if (!a.res[f]) return;
        const float4 x = ld4s(s_res + (((t & 1) * 5 + f) * p.slots + slot) * 4);
        v.x += x.x;
        v.y += x.y;
        v.z += x.z;
        v.w += x.w;
    };
    auto inject = [&](float4 &v, int t, int f, int w) {
        for (int l = 0; w; w = (int)((unsigned)w >> 10), ++l) {
            const int s = w & 1023;
            if (!s) continue;
            if (f != VZ || !a.lines.vzx[l]) add4(v, t, f, s - 1);
            if (f == VX && a.lines.vzx[l]) add4(v, t, VZ, s - 1);
        }
    };
    const int t_first = p.t_hi - 1;
    halo_words<R, 4>(t_word, g, p.tl, frame, T.slot, T.tz, T.tx, i0, th, T.q0, nq);
    auto put = [&](int o, int c, const uint4 &w) {
        s_p1[o + c] = __uint_as_float(w.x);
        s_p2[o + c] = __uint_as_float(w.y);
        s_p3[o + c] = __uint_as_float(w.z);
    };
    const float *const q0 = p.q + T.slot * a.fwd_stride + co;
    auto set_of = [&](int t, int f, int r) { return q0 + (long long)(t - p.q_t0) * p.state + f * P + r * g.pitch; };

    // New velocities of the block, and Q1, Q2.
    auto velocity = [&](int t) {
        float4 qx[RB], qz[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            qx[r] = qz[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!(img >> r & 1)) continue;
            qx[r] = qld4s(set_of(t, Q_TXS, r));
            qz[r] = qld4s(set_of(t, Q_TZS, r));
        }
        {
            auto row = [&](int r) { return ld4s(s_p2 + ot + r * W); };
            ZSlide<R, false> z(row);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                z.next(row(r + R - 1));
                float x[12], n[4];
                xrow<R, false>(x, ld4s(s_p1 + ot + r * W), s_p1 + ot + r * W);
#pragma unroll
                for (int k = 0; k < 4; ++k) n[k] = f4(vx[r], k) - xbwd<R>(x, k, a.k.cx) - z.at(k, a.k.cz);
                vx[r] = mk4(n);
            }
        }
        auto row = [&](int r) { return ld4s(s_p3 + ot + r * W); };
        ZSlide<R, true> z(row);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            z.next(row(r + R));
            float x[12], n[4], m[4], w[4], u[4], gg[4];
            const float4 d = damp4_of(br + r + 2 * R, HX + 4 * bq);
            xrow<R, true>(x, ld4s(s_p2 + ot + r * W), s_p2 + ot + r * W);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                n[k] = __fmul_rn(f4(d, k), f4(vz[r], k) - z.at(k, a.k.cz) - xfwd<R>(x, k, a.k.cx));
                m[k] = __fmul_rn(f4(d, k), f4(vx[r], k));
                u[k] = exact_q(dt, f4(b[r], k), m[k]);
                w[k] = exact_q(dt, f4(b[r], k), n[k]);
                gg[k] = f4(gb[r], k);
                exact_velocity_terms(dt, m[k], n[k], f4(qx[r], k), f4(qz[r], k), gg[k]);
            }
            vx[r] = mk4(m);
            vz[r] = mk4(n);
            gb[r] = mk4(gg);
            st4s(s_q1 + ot + r * W, mk4(u));
            st4s(s_q2 + ot + r * W, mk4(w));
        }
    };
    // The same for ring item e, first, where it is due, what the residual of step t + 1 added to its velocities.
    auto ring = [&](int e, int t, bool due) {
        const int r = item_row(t_ring[e]), q = item_col(t_ring[e]), c = (r + R) * W + HX - 4 + 4 * q;
        float *s = s_ring + 12 * e;
        float4 ovx = ld4s(s), ovz = ld4s(s + 4);
        const float4 bb = ld4s(s + 8), d = damp4_of(r + R, HX - 4 + 4 * q);
        const int w = t_rslot[e];
        if (due && w) {
            inject(ovx, t + 1, VX, w);
            inject(ovz, t + 1, VZ, w);
        }
        float x[12], nx[4], nz[4], u[4], v[4];
        const ZWindow<R, 1, false> z2([&](int) { return ld4s(s_p2 + c); }, s_p2 + c);
        xrow<R, false>(x, ld4s(s_p1 + c), s_p1 + c);
#pragma unroll
        for (int k = 0; k < 4; ++k) nx[k] = __fmul_rn(f4(d, k), f4(ovx, k) - xbwd<R>(x, k, a.k.cx) - z2.at(0, k, a.k.cz));
        const ZWindow<R, 1, true> z3([&](int) { return ld4s(s_p3 + c); }, s_p3 + c);
        xrow<R, true>(x, ld4s(s_p2 + c), s_p2 + c);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            nz[k] = __fmul_rn(f4(d, k), f4(ovz, k) - z3.at(0, k, a.k.cz) - xfwd<R>(x, k, a.k.cx));
            u[k] = exact_q(dt, f4(bb, k), nx[k]);
            v[k] = exact_q(dt, f4(bb, k), nz[k]);
        }
        st4s(s, mk4(nx));
        st4s(s + 4, mk4(nz));
        st4s(s_q1 + c, mk4(u));
        st4s(s_q2 + c, mk4(v));
    };
    auto strip_group = [&](int r) {
        return r < 2 * R || r >= th - 2 * R || bq < HG || bq >= nq - HG ? frame_index(r, bq, th, nq, 2 * R, HG) : -1;
    };
    // New stresses of the block with the residual of step t, their products, and the strips to xo.
    auto stress = [&](int t, bool epi, uint4 *xo, unsigned tag) {
        float4 q0v[RB], q1v[RB], q2v[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            q0v[r] = q1v[r] = q2v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!(img >> r & 1)) continue;
            q0v[r] = qld4s(set_of(t, Q_DXP_VX, r));
            q1v[r] = qld4s(set_of(t, Q_DZM_VZ, r));
            q2v[r] = qld4s(set_of(t, Q_VZS, r));
        }
        {
            auto row = [&](int r) { return ld4s(s_q2 + ot + r * W); };
            ZSlide<R, false> z(row);  // Dz- Q2
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                z.next(row(r + R - 1));
                const float4 d = damp4_of(br + r + 2 * R, HX + 4 * bq);
                float x[12], oz[4], oxz[4], gl[4], gm[4], ax[4];
                xrow<R, false>(x, z.centre(), s_q2 + ot + r * W);  // Dx- Q2
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    ax[k] = __fmul_rn(f4(d, k), f4(xx[r], k));
                    const float az = __fmul_rn(f4(d, k), f4(zz[r], k)), axz = __fmul_rn(f4(d, k), f4(xz[r], k));
                    gl[k] = f4(glam[r], k);
                    gm[k] = f4(gmu[r], k);
                    exact_stress_terms(dt, ax[k], az, axz, f4(q0v[r], k), f4(q1v[r], k), f4(q2v[r], k), gl[k], gm[k]);
                    oz[k] = __fsub_rn(az, z.at(k, a.k.cz));
                    oxz[k] = xbwd<R>(x, k, a.k.cx);  // taken off after Dz+ Q1
                }
                xx[r] = mk4(ax);
                zz[r] = mk4(oz);
                glam[r] = mk4(gl);
                gmu[r] = mk4(gm);
                xz[r] = times4(d, xz[r]);
                q2v[r] = mk4(oxz);
            }
        }
        auto row = [&](int r) { return ld4s(s_q1 + ot + r * W); };
        ZSlide<R, true> z(row);  // Dz+ Q1
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            z.next(row(r + R));
            float x[12], ox[4], oxz[4];
            xrow<R, true>(x, z.centre(), s_q1 + ot + r * W);  // Dx+ Q1
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                ox[k] = __fsub_rn(f4(xx[r], k), xfwd<R>(x, k, a.k.cx));
                oxz[k] = __fsub_rn(__fsub_rn(f4(xz[r], k), z.at(k, a.k.cz)), f4(q2v[r], k));
            }
            xx[r] = mk4(ox);
            xz[r] = mk4(oxz);
            if (epi && rs[r]) {
                inject(vx[r], t, VX, rs[r]);
                inject(vz[r], t, VZ, rs[r]);
                inject(xx[r], t, TXX, rs[r]);
                inject(zz[r], t, TZZ, rs[r]);
                inject(xz[r], t, TXZ, rs[r]);
            }
            float4 p1, p2, p3;
            products(ld4s(s_lam + 4 * (r * NT + tid)), ld4s(s_mu + 4 * (r * NT + tid)), damp4_of(br + r + 2 * R, HX + 4 * bq),
                     xx[r], zz[r], xz[r], p1, p2, p3);
            st4s(s_p1 + ot + r * W, p1);
            st4s(s_p2 + ot + r * W, p2);
            st4s(s_p3 + ot + r * W, p3);
            if (!inside) {
                const int s = strip_group(br + r);
                if (s >= 0) {
                    st_word(xo + 4 * s, p1.x, p2.x, p3.x, tag);
                    st_word(xo + 4 * s + 1, p1.y, p2.y, p3.y, tag);
                    st_word(xo + 4 * s + 2, p1.z, p2.z, p3.z, tag);
                    st_word(xo + 4 * s + 3, p1.w, p2.w, p3.w, tag);
                }
            }
        }
    };

    const int rank = tid >= T.nblk ? tid - T.nblk : tid + NT - T.nblk;
    bool stop = s_stop, due = false;
    for (int t = t_first; t >= p.t_lo && !stop; --t) {
        const bool epi = nrec && t % p.dt_scale == 0 && t / p.dt_scale < p.nt_ext;
        if (epi && rec_d >= 0) stage(t / p.dt_scale, t);
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            if (pass == 1 && t < t_first) {
                if (!fetch_halo<4>(p.xch + (t & 1) * xpar, p.tag0 + (unsigned)(t_first - t), t_word, p.err, p.limit_ns, put))
                    s_stop = 1;
                __syncthreads();
                stop = s_stop;
                if (stop) break;
            }
            if (mine && inside == (pass == 0)) velocity(t);
        }
        if (stop) break;
        for (int e = rank; e < nring; e += NT) ring(e, t, due);
        cp_wait<0>();
        __syncthreads();
        if (mine) stress(t, epi, strip + ((t - 1) & 1) * xpar, p.tag0 + (unsigned)(t_first - t + 1));
        due = epi;
        __syncthreads();
    }
    if (!mine) return;
    const float nan = __int_as_float(RES_NAN);
    float *out = a.out + T.slot * a.out_stride;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        if (gi0 + r >= g.tnz) break;
        if (stop) {
            vx[r] = vz[r] = xx[r] = zz[r] = xz[r] = make_float4(nan, nan, nan, nan);
            glam[r] = gmu[r] = gb[r] = vx[r];
        }
        // nothing is kept beyond the grid's last column
        auto kept = [&](const float4 &v) {
            return make_float4(v.x, gj0 + 1 < g.tnx ? v.y : 0.f, gj0 + 2 < g.tnx ? v.z : 0.f, gj0 + 3 < g.tnx ? v.w : 0.f);
        };
        float *o = out + co + r * g.pitch;
        *reinterpret_cast<float4 *>(o + VX * P) = kept(vx[r]);
        *reinterpret_cast<float4 *>(o + VZ * P) = kept(vz[r]);
        *reinterpret_cast<float4 *>(o + TXX * P) = kept(xx[r]);
        *reinterpret_cast<float4 *>(o + TZZ * P) = kept(zz[r]);
        *reinterpret_cast<float4 *>(o + TXZ * P) = kept(xz[r]);
        *reinterpret_cast<float4 *>(G + co + r * g.pitch) = glam[r];
        *reinterpret_cast<float4 *>(G + P + co + r * g.pitch) = gmu[r];
        *reinterpret_cast<float4 *>(G + 2 * P + co + r * g.pitch) = gb[r];
    }
}

// ---------------------------------------------------------------------------
// reverse-time steps (rev_step's arithmetic)
// ---------------------------------------------------------------------------
// The state of step t from that of step t + 1: stresses first, then velocities,
// so it exchanges velocities and recomputes the ring's stresses, as
// adj_resident does with its products.  Every state goes to memory, 20 bytes a
// cell.  190 x 290 cells, 5 shots: 5.1 us a step in runs of nine, 8.2 in rev_step.
template <int R, int RB>
__global__ void __launch_bounds__(RES_THREADS, 1) rev_resident(const __grid_constant__ RevResArgs p)
{
    constexpr int NT = RES_THREADS, HX = ResShape<R>::HX, HG = ResShape<R>::HG;
    extern __shared__ float4 smem4[];
    __shared__ int s_stop;
    const StepArgs &a = p.a;
    const Grid &g = a.g;
    const long long P = g.plane;
    const int tid = threadIdx.x;
    const ResTile T = res_tile<R, RB>(p.tl);
    const int i0 = T.i0, j0 = T.j0, th = T.th, nq = T.nq;
    constexpr int W = RES_W, PL = RES_PLANE, RING = ResShape<R>::RING, SM = FWD_SHARED_MATS<RB>;
    float *const sm = reinterpret_cast<float *>(smem4) + RES_PAD;
    // Cell (r, c) of the tile lies at (r + 2R) * W + HX + c of every plane.
    float *const s_vx = sm, *const s_vz = sm + PL, *const s_txx = sm + 2 * PL, *const s_tzz = sm + 3 * PL, *const s_txz = sm + 4 * PL;
    float *const s_ring = sm + 5 * PL;                               // [ring item][5][4]: its stresses, lam, mu
    float *const s_dx = s_ring + 20 * RING, *const s_dz = s_dx + W;  // damping
    unsigned *const t_ring = reinterpret_cast<unsigned *>(s_dz + RES_ROWS);
    float *const s_mat = reinterpret_cast<float *>(t_ring + RING);   // [lam, mu, b][row][thread][4], RB 3
    const int nring = (th + 2 * R) * (nq + 2) - th * nq;
    const float dt = a.k.dt;
    const float *in = a.in + T.slot * a.in_stride;
    const int frame = frame_count(RB * p.tl.bz, p.tl.nq, 2 * R, HG);
    const int xpar = 4 * gridDim.x * frame;
    uint4 *const strip = p.xch + 4 * blockIdx.x * frame;

    if (tid == 0) s_stop = ld_relaxed_gpu(p.err) != 0;
    for (int e = tid; e < (th + 4 * R) * (nq + 2 * HG); e += NT) {
        const int r = e / (nq + 2 * HG), q = e - r * (nq + 2 * HG), o = r * W + 4 * q;
        const int gi = i0 - 2 * R + r, gj = j0 - HX + 4 * q;
        st4s(s_vx + o, ld4(in + VX * P, g, gi, gj));
        st4s(s_vz + o, ld4(in + VZ * P, g, gi, gj));
    }
    // Zero materials outside the update domain, where every field is zero, keep it so.
    auto masked = [&](const float *plane, int gi, int gj) {
        float4 v = ld4(plane, g, gi, gj);
        if (!in_domain(g, R, gi, gj)) v.x = 0.f;
        if (!in_domain(g, R, gi, gj + 1)) v.y = 0.f;
        if (!in_domain(g, R, gi, gj + 2)) v.z = 0.f;
        if (!in_domain(g, R, gi, gj + 3)) v.w = 0.f;
        return v;
    };
    for (int e = tid; e < nring; e += NT) {
        int r, q;
        frame_item(e, th + 2 * R, nq + 2, R, 1, r, q);
        t_ring[e] = pack_item(r, q);
        const int gi = i0 - R + r, gj = j0 - 4 + 4 * q;
        float *s = s_ring + 20 * e;
        st4s(s, ld4(in + TXX * P, g, gi, gj));
        st4s(s + 4, ld4(in + TZZ * P, g, gi, gj));
        st4s(s + 8, ld4(in + TXZ * P, g, gi, gj));
        st4s(s + 12, masked(a.mat, gi, gj));
        st4s(s + 16, masked(a.mat + P, gi, gj));
    }
    for (int e = tid; e < 4 * nq + 2 * HX; e += NT) {
        const int c = j0 - HX + e + XO;
        s_dx[e] = c >= 0 && c < g.pitch ? __ldg(a.dampx + c) : 0.f;
    }
    for (int e = tid; e < th + 4 * R; e += NT) {
        const int i = i0 - 2 * R + e + ZO;
        s_dz[e] = i >= 0 && i < g.rows ? __ldg(a.dampz + i) : 0.f;
    }

    const bool mine = tid < T.nblk, inside = tid < T.nin;
    int bz = 0, bq = 0;
    if (mine) res_block<R, RB>(T, tid, bz, bq);
    const int br = bz * RB;
    const int ot = (br + 2 * R) * W + HX + 4 * bq;
    const int gi0 = i0 + br, gj0 = j0 + 4 * bq;
    const int co = (gi0 + ZO) * g.pitch + gj0 + XO;
    float4 vx[RB], vz[RB], sxx[RB], szz[RB], sxz[RB], b[RB], lam[RB], mu[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        vx[r] = vz[r] = sxx[r] = szz[r] = sxz[r] = b[r] = lam[r] = mu[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!mine) continue;
        const int gi = gi0 + r;
        vx[r] = ld4(in + VX * P, g, gi, gj0);
        vz[r] = ld4(in + VZ * P, g, gi, gj0);
        sxx[r] = ld4(in + TXX * P, g, gi, gj0);
        szz[r] = ld4(in + TZZ * P, g, gi, gj0);
        sxz[r] = ld4(in + TXZ * P, g, gi, gj0);
        lam[r] = masked(a.mat, gi, gj0);
        mu[r] = masked(a.mat + P, gi, gj0);
        b[r] = masked(a.mat + 2 * P, gi, gj0);
        if (SM) {
            st4s(s_mat + 4 * (r * NT + tid), lam[r]);
            st4s(s_mat + 4 * ((RB + r) * NT + tid), mu[r]);
            st4s(s_mat + 4 * ((2 * RB + r) * NT + tid), b[r]);
        }
    }
    auto lam_of = [&](int r) { return SM ? ld4s(s_mat + 4 * (r * NT + tid)) : lam[r]; };
    auto mu_of = [&](int r) { return SM ? ld4s(s_mat + 4 * ((RB + r) * NT + tid)) : mu[r]; };
    auto b_of = [&](int r) { return SM ? ld4s(s_mat + 4 * ((2 * RB + r) * NT + tid)) : b[r]; };
    const unsigned halo = halo_group<R>(g, p.tl, frame, T.slot, T.tz, T.tx, i0, th, T.q0, nq);
    auto put = [&](int o, const uint4 (&w)[3]) {
        auto f = [](unsigned u) { return __uint_as_float(u); };
        st4s(s_vx + o, make_float4(f(w[0].x), f(w[0].y), f(w[0].z), f(w[1].x)));
        st4s(s_vz + o, make_float4(f(w[1].y), f(w[1].z), f(w[2].x), f(w[2].y)));
    };
    __syncthreads();

    // New stresses of four cells.
    auto update = [&](float4 &xx, float4 &zz, float4 &xz, const float4 &l, const float4 &m, const float4 &dx, float dz,
                      const float (&ex)[4], const float (&ez)[4], const float (&exz)[4]) {
        float oxx[4], ozz[4], oxz[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float d = f4(dx, k) + dz;
            float txx = f4(xx, k), tzz = f4(zz, k), txz = f4(xz, k);
            txz = txz - dt * (d * txz);
            txz = txz - dt * (f4(m, k) * exz[k]);
            normal_pair_rev(f4(l, k), f4(m, k), ex[k], ez[k], d, dt, txx, tzz);
            oxx[k] = txx;
            ozz[k] = tzz;
            oxz[k] = txz;
        }
        xx = mk4(oxx);
        zz = mk4(ozz);
        xz = mk4(oxz);
    };
    auto stress = [&]() {
        const float4 dx = ld4s(s_dx + HX + 4 * bq);
        auto row_x = [&](int r) { return ld4s(s_vx + ot + r * W); };
        auto row_z = [&](int r) { return ld4s(s_vz + ot + r * W); };
        ZSlide<R, true> zx(row_x);
        ZSlide<R, false> zz(row_z);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            zx.next(row_x(r + R));
            zz.next(row_z(r + R - 1));
            float x[12], ex[4], ez[4], exz[4];
            xrow<R, true>(x, zx.centre(), s_vx + ot + r * W);
#pragma unroll
            for (int k = 0; k < 4; ++k) ex[k] = xfwd<R>(x, k, a.k.cx);
            xrow<R, false>(x, zz.centre(), s_vz + ot + r * W);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                exz[k] = xbwd<R>(x, k, a.k.cx) + zx.at(k, a.k.cz);
                ez[k] = zz.at(k, a.k.cz);
            }
            update(sxx[r], szz[r], sxz[r], lam_of(r), mu_of(r), dx, s_dz[br + r + 2 * R], ex, ez, exz);
            st4s(s_txx + ot + r * W, sxx[r]);
            st4s(s_tzz + ot + r * W, szz[r]);
            st4s(s_txz + ot + r * W, sxz[r]);
        }
    };
    auto ring = [&](int e) {
        const int r = item_row(t_ring[e]), q = item_col(t_ring[e]), c = (r + R) * W + HX - 4 + 4 * q;
        float *s = s_ring + 20 * e;
        float x[12], ex[4], ez[4], exz[4];
        {
            const ZWindow<R, 1, true> zx([&](int) { return ld4s(s_vx + c); }, s_vx + c);
            xrow<R, true>(x, zx.w[R - 1], s_vx + c);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                ex[k] = xfwd<R>(x, k, a.k.cx);
                exz[k] = zx.at(0, k, a.k.cz);
            }
        }
        const ZWindow<R, 1, false> zz([&](int) { return ld4s(s_vz + c); }, s_vz + c);
        xrow<R, false>(x, zz.w[R], s_vz + c);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            ez[k] = zz.at(0, k, a.k.cz);
            exz[k] = xbwd<R>(x, k, a.k.cx) + exz[k];
        }
        float4 xx = ld4s(s), zz4 = ld4s(s + 4), xz = ld4s(s + 8);
        update(xx, zz4, xz, ld4s(s + 12), ld4s(s + 16), ld4s(s_dx + HX - 4 + 4 * q), s_dz[r + R], ex, ez, exz);
        st4s(s, xx);
        st4s(s + 4, zz4);
        st4s(s + 8, xz);
        st4s(s_txx + c, xx);
        st4s(s_tzz + c, zz4);
        st4s(s_txz + c, xz);
    };

    const int rank = tid >= T.nblk ? tid - T.nblk : tid + NT - T.nblk;
    const int t_first = p.t_hi - 1;
    bool stop = s_stop;
    for (int t = t_first; t >= p.t_lo && !stop; --t) {
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            if (pass == 1 && t < t_first) {
                if (!fetch_group<3>(p.xch + (t & 1) * xpar, p.tag0 + (unsigned)(t_first - t), halo, p.err, p.limit_ns, put)) s_stop = 1;
                __syncthreads();
                stop = s_stop;
                if (stop) break;
            }
            if (mine && inside == (pass == 0)) stress();
        }
        if (stop) break;
        for (int e = rank; e < nring; e += NT) ring(e);
        __syncthreads();
        if (mine) {
            uint4 *const xo = strip + ((t - 1) & 1) * xpar;
            const unsigned tag = p.tag0 + (unsigned)(t_first - t + 1);
            float *const o0 = p.q + (long long)(t % p.ring) * p.state + T.slot * p.q_stride + co;
            const float4 dx = ld4s(s_dx + HX + 4 * bq);
            {
                auto row = [&](int r) { return ld4s(s_txz + ot + r * W); };
                ZSlide<R, false> z(row);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    z.next(row(r + R - 1));
                    const float4 bb = b_of(r);
                    const float dz = s_dz[br + r + 2 * R];
                    float x[12], n[4];
                    xrow<R, false>(x, sxx[r], s_txx + ot + r * W);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float d = f4(dx, k) + dz;
                        float v = f4(vx[r], k);
                        v = v - dt * (d * v);
                        n[k] = v - dt * (f4(bb, k) * (xbwd<R>(x, k, a.k.cx) + z.at(k, a.k.cz)));
                    }
                    vx[r] = mk4(n);
                }
            }
            auto row = [&](int r) { return ld4s(s_tzz + ot + r * W); };
            ZSlide<R, true> z(row);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                z.next(row(r + R));
                const float4 bb = b_of(r);
                const float dz = s_dz[br + r + 2 * R];
                float x[12], n[4];
                xrow<R, true>(x, sxz[r], s_txz + ot + r * W);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float d = f4(dx, k) + dz;
                    float v = f4(vz[r], k);
                    v = v - dt * (d * v);
                    n[k] = v - dt * (f4(bb, k) * (z.at(k, a.k.cz) + xfwd<R>(x, k, a.k.cx)));
                }
                vz[r] = mk4(n);
                st4s(s_vx + ot + r * W, vx[r]);
                st4s(s_vz + ot + r * W, vz[r]);
                if (!inside) {
                    const int rr = br + r;
                    if (rr < 2 * R || rr >= th - 2 * R || bq < HG || bq >= nq - HG) {
                        uint4 *const s = xo + 4 * frame_index(rr, bq, th, nq, 2 * R, HG);
                        st_word(s, vx[r].x, vx[r].y, vx[r].z, tag);
                        st_word(s + 1, vx[r].w, vz[r].x, vz[r].y, tag);
                        st_word(s + 2, vz[r].z, vz[r].w, 0.f, tag);
                    }
                }
                if (gi0 + r < g.tnz) {
                    float *o = o0 + r * g.pitch;
                    qst4s(o + VX * P, vx[r]);
                    qst4s(o + VZ * P, vz[r]);
                    qst4s(o + TXX * P, sxx[r]);
                    qst4s(o + TZZ * P, szz[r]);
                    qst4s(o + TXZ * P, sxz[r]);
                }
            }
        }
        __syncthreads();
    }
    if (!stop || !mine) return;
    const float nan = __int_as_float(RES_NAN);
    for (int t = t_first; t >= p.t_lo; --t)
        for (int r = 0; r < RB && gi0 + r < g.tnz; ++r)
            for (int f = 0; f < 5; ++f)
                qst4s(p.q + (long long)(t % p.ring) * p.state + T.slot * p.q_stride + co + r * g.pitch + f * P,
                      make_float4(nan, nan, nan, nan));
}

}  // namespace pyfwi
