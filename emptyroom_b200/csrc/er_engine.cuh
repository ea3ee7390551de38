// er_engine.cuh -- the probe-framework Lennard-Jones pair-sum engine (sm_100a).
//
// What it computes is the sum of src/computegridsheet.h:54-92 (and the same
// sum in src/doHenry.h:70-98): at every point p, over every kept atom image
// a + T n, 4 eps s^6 (s^6 - 1) with s = sig^2 / r^2 when r^2 < rc^2.
// How it computes it is its own:
//
//  * Positions live in the framework's positioning frame R (an upper-
//    triangular rotation of the cell matrix T, equal to T bit for bit when T
//    is already upper triangular, as the reference's cells are). Distances are
//    frame-independent; the exact cutoff decision below still uses T.
//  * A CTA owns up to 8 warp tasks of <= 32*P points (a lattice sub-brick of
//    the grid, or a chunk of one spatial bin of Widom insertions). The CTA box
//    is the FP64 bounding box of its points; all FP32 coordinates are relative
//    to the box centre, so FP32 never holds magnitudes above rc + box.
//  * Candidate atom images come from the framework's cell list: one contiguous
//    image range per (y, z) row of cells, with the x range of each row pruned
//    by the cutoff circle. Passing candidates are compacted in order (ballots
//    and prefix sums, so the order is deterministic) into shared memory.
//  * Atoms far from a fine grid's brick and inside the cutoff of all of it are
//    summed at fewer nodes and interpolated to its points (far_field).
//  * Each warp splits the CTA candidates against its own box into an inner
//    list (inside the cutoff for every point of the warp: no test needed) and
//    a shell list (cutoff tested per pair). Lists are u16 byte offsets.
//  * Lattice points of one lane differ only along the grid's first axis, which
//    R maps to Cartesian x; so per atom the lane forms dy^2 + dz^2 once and per
//    point only dx and r^2 = dx^2 + (dy^2 + dz^2). Point pairs run as packed
//    FP32x2 instructions (add/mul/fma .f32x2): per two pair terms 5 packed ops
//    and 2 MUFU.RCP, E += u^3 (C12 u^3 - C6), u = 1 / r^2.
//  * Shell pairs whose FP32 r^2 lies within a proven error window of rc^2 are
//    re-decided in FP64 with the reference's own expression order, so the set
//    of summed pairs equals the FP64 reference's set exactly.
//  * Accumulation: FP32 over chunks of 8 to 64 atoms, chunk sums added into FP64
//    per-point totals (ER_PREC_COMP, ER_PREC_NEAR64), or FP32 over the whole
//    list (ER_PREC_FP32). ER_PREC_NEAR64 (the default) evaluates the pairs of
//    atoms within kNearR of a warp's points in FP64: those large terms carry
//    the FP32 error where they cancel to a small |E|.
#pragma once
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "er_internal.h"
#include "er_philox.h"

namespace er {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
// points per thread (P) and the CTA brick are set by the point policy (Tile)
constexpr int kWJ = 4, kWK = 8;            // lanes of a warp sub-brick along j, k
constexpr int kPMax = 8;                   // largest P any policy uses
constexpr int kAxisMax = 2 * (kPMax + kWJ + kWK);  // lattice lines of the largest brick, all axes
constexpr int kMaxCand = 1024;             // CTA candidate capacity per flush
constexpr int kRowChunk = kThreads;        // cell rows examined per producer pass
constexpr int kAccChunk = 64;              // atoms per FP32 partial sum (shell lists,
                                           // and every list of ER_PREC_COMP)
constexpr float kEnergyCap = 1.0e30f;      // overflow cap (ER_ENERGY_CAP)

// PREC_COUNT writes the number of in-cutoff pair terms per point instead of
// the energy (same traversal; used to count the algorithmic work of a job).
// PREC_NEAR64 is PREC_COMP with the pairs of atoms within kNearR of a warp's
// box evaluated in FP64 (they carry most of |E| where terms cancel).
// PREC_FP64 evaluates every pair term in FP64 (same pair set).
enum { PREC_COMP = 0, PREC_FP32 = 1, PREC_COUNT = 2, PREC_NEAR64 = 3, PREC_FP64 = 4 };

template <int PREC>
struct PrecTraits {
    static constexpr bool comp = PREC == PREC_COMP || PREC == PREC_NEAR64;
    static constexpr bool near64 = PREC == PREC_NEAR64;
    static constexpr bool fp64 = PREC == PREC_FP64;
    static constexpr bool far = near64;  // the brick's far field is interpolated
    // Atoms per FP32 partial sum of an inner list. Once NEAR64 has taken the
    // near terms to FP64, the rounding of the FP32 partial sums (its error
    // grows with the chunk length times the partial's magnitude) is what is
    // left: 16-atom partials keep every E < -10 K point of the 256-framework
    // batch within 1e-5 of FP64, 64-atom ones leave 82 of 1.4e8 above it;
    // 32-atom ones were 0.8 % faster but raised the sampled p99 error from
    // 5.1e-7 to 6.6e-7.
    static constexpr int inner_chunk = PREC == PREC_NEAR64 ? 16 : 64;
};

// The same for two policies whose other choices would raise the error a little.
// Where a brick has a far field, for its nodes and for what is left of the inner
// lists: with 16 the mean error on E < -10 K points was within 3 % of the one
// without a far field, either way; with 8 it is 4-10 % below it (five cells at
// 0.1-0.155 A), for 2 % more time. And for Widom warps of 128 points, whose boxes
// have fewer atoms within kNearR than those of 256: with 8 the mean error of 2e5
// and 32768 insertions is 2-4 % below the one with 16.
constexpr int kShortChunk = 8;
template <class Pol, int PREC>
struct InnerChunk {
    static constexpr int value =
        PREC == PREC_NEAR64 && Pol::kShort ? kShortChunk : PrecTraits<PREC>::inner_chunk;
};
constexpr int kNearCap = 256;     // near-list capacity per warp (overflow stays FP32)
constexpr int kRec = 3;           // borderline shell atoms recorded per thread and flush
                                  // (10-bit list positions packed in one register)
constexpr float kNearR = 5.0f;    // near radius (A) from the warp box

// One candidate atom image in shared memory (32 bytes, so a list entry can be
// the byte offset of its record). x, C12 and -C6 are stored twice so that a
// 128-bit load yields them as packed FP32x2 operands; the position is the
// first 16 bytes (one vector load in the per-warp split).
struct __align__(32) Cand {
    float ax, ax_, ay, az;       // x (twice), y, z relative to the CTA centre
    float c12, c12_, nc6, nc6_;  // C12 (twice), -C6 (twice)
};

// 74.8 KB: at most (228 KB / 3) - 1 KB, so that three CTAs share an SM.
struct __align__(32) EngineSmem {
    Cand cand[kMaxCand];                   // CTA candidates
    int cid[kMaxCand];                     // their image indices (FP64 paths)
    unsigned short wl[kWarps][kMaxCand];   // per-warp inner (front) / shell (back) lists of
                                           // byte offsets into cand
    unsigned short wn[kWarps][kNearCap];   // per-warp near lists (PREC_NEAR64): atoms inside
                                           // the cutoff for every point (front) and atoms
                                           // crossing it (back)
    double tot[kPMax][kThreads];           // FP64 per-point sums, [p][thread]
    union {
        int row_beg[kRowChunk];
        double red[kWarps][6];             // warp boxes of the CTA box, before the producer
    };
    int row_off[kRowChunk];
    int wcnt[2][kWarps];                   // warp counts of block_prefix, two in turn
    double box[6];                         // CTA box (FP64 lo, hi; generic points)
    double org[3];                         // its centre, the origin of FP32 coordinates
    float cbox[6];                         // CTA box (local FP32 lo, hi)
    float fbox[6];                         // box of the whole brick (far field)
    float wbox[kWarps][6];                 // warp boxes (local FP32 lo, hi)
    double axis[kAxisMax];                 // fractional coordinates of a brick's lattice lines
};

// Atoms a warp holds in FP64 (near_lists, fp64_lists): position relative to the
// CTA centre and FP64 (C12, C6).
struct __align__(16) NearAtom {
    double x, y, z, c12, c6, pad;
};
constexpr int kNearStage = 32;  // one per lane
// Shared memory of a block: PREC_FP64 has a stage per warp behind EngineSmem
// (its two CTAs per SM have the room), PREC_NEAR64 uses a consumed list.
__host__ __device__ constexpr size_t engine_smem_bytes(int prec) {
    return sizeof(EngineSmem) +
           (prec == PREC_FP64 ? kWarps * kNearStage * sizeof(NearAtom) : (size_t)0);
}

// The block's EngineSmem, by the shared array itself: a reference handed to an
// out-of-line function arrives as a generic pointer, and the pair loops then
// run on generic loads (half again as long in a 32^3 grid).
__device__ __forceinline__ EngineSmem& engine_smem() {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    return *reinterpret_cast<EngineSmem*>(smem_raw);
}
// This warp's stage of PREC_FP64.
__device__ __forceinline__ NearAtom* fp64_stage() {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    return reinterpret_cast<NearAtom*>(smem_raw + sizeof(EngineSmem)) +
           (threadIdx.x >> 5) * kNearStage;
}

// ----------------------------------------------------------- packed FP32x2
typedef unsigned long long f2_t;

__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
    f2_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b) {
    f2_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
    f2_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
    f2_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
    f2_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// 1.0f when a < b, else 0.0f
__device__ __forceinline__ float set_lt(float a, float b) {
    float d;
    asm("set.lt.f32.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Sum of the warps' counts below this warp's; *total gets the sum of all. One
// barrier per call: consecutive calls use `buf` 0 and 1 in turn, so a warp
// writes a buffer again only after the barrier of the call between, which
// every warp reaches after its reads.
__device__ __forceinline__ int block_prefix(EngineSmem& s, int buf, int count, int* total) {
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) s.wcnt[buf][w] = count;
    __syncthreads();
    int below = 0, all = 0;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) {
        const int c = s.wcnt[buf][k];
        below += k < w ? c : 0;
        all += c;
    }
    *total = all;
    return below;
}

__device__ __forceinline__ void frac_to_cart(const double* t, double xf, double yf, double zf,
                                             double& x, double& y, double& z) {
    // src/computegridsheet.h:25-27, strict IEEE order (no contraction)
    x = __dadd_rn(__dadd_rn(__dmul_rn(t[0], xf), __dmul_rn(t[1], yf)), __dmul_rn(t[2], zf));
    y = __dadd_rn(__dadd_rn(__dmul_rn(t[3], xf), __dmul_rn(t[4], yf)), __dmul_rn(t[5], zf));
    z = __dadd_rn(__dadd_rn(__dmul_rn(t[6], xf), __dmul_rn(t[7], yf)), __dmul_rn(t[8], zf));
}

// The reference's FP64 in-cutoff decision for point f and image gid:
// src/computegridsheet.h:61-79 evaluated in IEEE double without contraction,
// in the caller's cell matrix T.
static __device__ __noinline__ bool exact_in_cutoff(const FwDev& fw, const double* f, int gid,
                                                    double r2min) {
    const uint32_t id = fw.img_id[gid];
    const int atom = (int)(id / (uint32_t)fw.imgs_per_atom);
    const int m = (int)(id - (uint32_t)atom * (uint32_t)fw.imgs_per_atom);
    const int n2 = 2 * fw.rep[2] + 1, n1 = 2 * fw.rep[1] + 1;
    const int kk = m % n2 - fw.rep[2];
    const int jj = (m / n2) % n1 - fw.rep[1];
    const int ii = m / (n2 * n1) - fw.rep[0];
    const double4 a = fw.atom_frac[atom];
    double x, y, z, xw, yw, zw;
    frac_to_cart(fw.t, f[0], f[1], f[2], x, y, z);
    frac_to_cart(fw.t, __dadd_rn(a.x, (double)ii), __dadd_rn(a.y, (double)jj),
                 __dadd_rn(a.z, (double)kk), xw, yw, zw);
    const double dx = __dsub_rn(x, xw), dy = __dsub_rn(y, yw), dz = __dsub_rn(z, zw);
    double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    r2 = (r2 > r2min) ? r2 : r2min;
    return r2 < fw.rc2;
}

// One atom image for FP64 pair terms: position relative to the CTA centre and
// FP64 (C12, C6).
struct Atom64 {
    double x, y, z, c12, c6;
};
__device__ __forceinline__ Atom64 atom64(const FwDev& fw, int gid, double o0, double o1,
                                         double o2) {
    const double4 a = fw.img_xyz[gid];
    const double2 lj = fw.img_lj64[gid];
    return Atom64{a.x - o0, a.y - o1, a.z - o2, lj.x, lj.y};
}
// 1/x in FP64 for the near pairs of PREC_NEAR64: one Newton step
// y = y0 (1 + e), e = 1 - x y0, from the hardware seed y0 =
// rcp.approx.ftz.f64(x), whose relative error e0 is below 2^-16 (asserted by
// the tests; er_probe_rcp64_seed measures 9.9e-7, about 2^-20), leaves a
// relative error of order e0^2 < 2^-32 plus two FP64 roundings. A near term then carries at
// most ~6 x 2^-32 of its own size, far below the 1e-5 relative bound on the
// energy even where near terms cancel a thousandfold (a third-order step,
// e0^3, gave the same errors on 71,378 sampled E < -10 K points of the
// 256-framework batch and took 0.8 % longer; a seed from the FP32
// reciprocal, converted, took 4.7 % longer). x is a squared distance,
// clamped to >= min_r^2 > 0 by the caller, so the seed is finite and normal.
__device__ __forceinline__ double rcp64_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, e, y);
}
// acc + the FP64 pair term of a near pair (PREC_NEAR64): r^2 = dx^2 + yzc from
// dx and yzc = dy^2 + dz^2 + min_r^2, formed once per atom and lane, with the
// reference's clamp r^2 >= min_r^2 (src/computegridsheet.h:77) folded into
// yzc: both keep r^2 >= min_r^2, and min_r^2 (1e-24 or 1e-32 A^2) lies below
// the FP64 resolution of r^2 unless r^2 < ~1e-8 A^2, a point within 1e-4 A of
// an atom, whose energy (> 1e40 K) is capped either way. (The clamp as a
// separate FP64 max cost 3 % of the 256-framework batch.) Reciprocal by
// rcp64_nr, the term added by one FMA.
__device__ __forceinline__ double near_acc64(double acc, double dx, double yzc, double c12,
                                             double c6) {
    const double u = rcp64_nr(fma(dx, dx, yzc));
    const double u3 = u * u * u;
    return fma(u3, fma(c12, u3, -c6), acc);
}

// FP32 r^2 of the generic form (each point has its own x, y, z) and of the
// lattice form (ss = dy^2 + dz^2 shared by a lane's points). Both are fixed
// instruction sequences, so a later re-evaluation reproduces the same bits.
__device__ __forceinline__ float r2_generic(float px, float py, float pz, float ax, float ay,
                                            float az) {
    const float dx = __fsub_rn(px, ax);
    const float dy = __fsub_rn(py, ay);
    const float dz = __fsub_rn(pz, az);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}
__device__ __forceinline__ float ss_lattice(float py, float pz, float ay, float az) {
    const float dy = __fsub_rn(py, ay);
    const float dz = __fsub_rn(pz, az);
    return __fmaf_rn(dz, dz, __fmul_rn(dy, dy));
}
__device__ __forceinline__ float r2_lattice(float px, float ax, float ss) {
    const float dx = __fsub_rn(px, ax);
    return __fmaf_rn(dx, dx, ss);
}
// E_pair = u3 * t with u = 1/r^2, u3 = u^3, t = C12 u3 - C6.
__device__ __forceinline__ float pair_term(float r2, float c12, float nc6) {
    const float u = rcp_approx(r2);
    const float u3 = __fmul_rn(__fmul_rn(u, u), u);
    return __fmul_rn(u3, __fmaf_rn(c12, u3, nc6));
}

// ---------------------------------------------------------------------------
// Point sources. A policy maps (warp, lane, p) to an FP64 fractional point
// and stores its energy. kLattice: a lane's P points differ only in the
// first fractional coordinate.

// Lattice points of one (2P) x 8 x 16 brick of a grid job: warp w owns the
// P x 4 x 8 sub-brick at ((w & 1) P, ((w >> 1) & 1) 4, (w >> 2) 8); lane l the
// (j, k) = (l / 8, l % 8) column of it and its P points along i.
//
// The brick's fractional coordinates i / (N - 1) (FP64 divisions) are formed
// once per lattice line, one thread each, in `axis` (shared memory); points
// are products of the table. The boxes need no reduction over the points: a
// Cartesian coordinate is a chain of rounded products and sums, each monotone
// in every fractional coordinate, so its extremes over a product set of
// lattice lines are its values at corners of the set, bit for bit. With every
// point forming its own divisions twice and FP64 shuffles for the boxes, this
// took 11,000 of the 84,000 clocks of a CTA (129^3 grid of a 424-atom cell).
//
// SPLIT > 1 spreads one brick over SPLIT CTAs, for grids of few bricks: CTA
// `item % SPLIT` takes kWarps / SPLIT of the sub-bricks, SPLIT warps to each
// with P / SPLIT of its points a lane. Box, origin, candidates and lists stay
// those of the brick and the sub-brick, so every energy keeps its bits.
template <int SPLIT>
struct BrickPart {  // which of its brick's SPLIT CTAs this is
    int part;
    __device__ explicit BrickPart(int item) : part(item % SPLIT) {}
};
template <>
struct BrickPart<1> {
    static constexpr int part = 0;
    __device__ explicit BrickPart(int) {}
};

template <int P_, int SPLIT = 1>
struct GridPolicy : BrickPart<SPLIT> {
    static constexpr int kP = P_ / SPLIT, kBoxP = kP;
    static constexpr bool kLattice = true;
    static constexpr int kBI = 2 * P_, kBJ = 2 * kWJ, kBK = 2 * kWK;
    static_assert(P_ % SPLIT == 0 && kWarps % SPLIT == 0, "whole points and sub-bricks per warp");
    const GridTask* T;
    int i0, j0, k0;
    __device__ GridPolicy(const GridTask* task, int item) : BrickPart<SPLIT>(item), T(task) {
        const int brick = item / SPLIT;
        const int nbk = task->nb[2], nbj = task->nb[1];
        const int bk = brick % nbk;
        const int bj = (brick / nbk) % nbj;
        const int bi = brick / (nbk * nbj);
        i0 = bi * kBI; j0 = bj * kBJ; k0 = bk * kBK;
    }
    // the sub-brick of warp w
    __device__ __forceinline__ int sub(int w) const {
        return this->part * (kWarps / SPLIT) + w / SPLIT;
    }
    __device__ __forceinline__ void index(int w, int lane, int p, int& i, int& j, int& k) const {
        const int b = sub(w);
        i = i0 + (b & 1) * P_ + w % SPLIT * kP + p;
        j = j0 + ((b >> 1) & 1) * kWJ + lane / kWK;
        k = k0 + (b >> 2) * kWK + lane % kWK;
    }
    // One thread per lattice line; the caller synchronises. Lines past the
    // grid repeat its last one (such points are never stored).
    __device__ __forceinline__ void fill_axes(int tid) const {
        if (tid >= kBI + kBJ + kBK) return;
        double* axis = engine_smem().axis;
        int i, n;
        if (tid < kBI) { i = i0 + tid; n = T->nx; }
        else if (tid < kBI + kBJ) { i = j0 + tid - kBI; n = T->ny; }
        else { i = k0 + tid - kBI - kBJ; n = T->nz; }
        // axes 1.0 * i / (N - 1), src/writegrid.cu:122-127
        axis[tid] = __ddiv_rn((double)min(i, n - 1), (double)(n - 1));
    }
    // Out-of-range points are clamped onto the lattice (same j, k when only i
    // overshoots, so a lane's points keep sharing y and z) and never stored.
    __device__ __forceinline__ bool point(int w, int lane, int p, double* f) const {
        int i, j, k;
        index(w, lane, p, i, j, k);
        const double* axis = engine_smem().axis;
        f[0] = axis[i - i0];
        f[1] = axis[kBI + j - j0];
        f[2] = axis[kBI + kBJ + k - k0];
        return i < T->nx && j < T->ny && k < T->nz;
    }
    // the point's Cartesian position in the positioning frame r
    __device__ __forceinline__ bool cart(const double* r, int w, int lane, int p, double& x,
                                         double& y, double& z) const {
        double f[3];
        const bool ok = point(w, lane, p, f);
        frac_to_cart(r, f[0], f[1], f[2], x, y, z);
        return ok;
    }
    // FP64 Cartesian box of the lattice points [bi, bi + ni) x [bj, bj + nj) x
    // [bk, bk + nk) of the brick that lie on the grid; false when there are none.
    __device__ __forceinline__ bool box(const double* r, int bi, int ni, int bj, int nj, int bk,
                                        int nk, double* lo, double* hi) const {
        const int ei = min(bi + ni, T->nx - i0) - 1, ej = min(bj + nj, T->ny - j0) - 1;
        const int ek = min(bk + nk, T->nz - k0) - 1;
        if (ei < bi || ej < bj || ek < bk) return false;
        const double* axis = engine_smem().axis;
        const double a[3] = {axis[bi], axis[kBI + bj], axis[kBI + kBJ + bk]};
        const double b[3] = {axis[ei], axis[kBI + ej], axis[kBI + kBJ + ek]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double* t = r + 3 * d;
            double l[3], h[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const double u = __dmul_rn(t[e], a[e]), v = __dmul_rn(t[e], b[e]);
                l[e] = fmin(u, v);
                h[e] = fmax(u, v);
            }
            lo[d] = __dadd_rn(__dadd_rn(l[0], l[1]), l[2]);
            hi[d] = __dadd_rn(__dadd_rn(h[0], h[1]), h[2]);
        }
        return true;
    }
    __device__ __forceinline__ bool cta_box(const double* r, double* lo, double* hi) const {
        return box(r, 0, kBI, 0, kBJ, 0, kBK, lo, hi);
    }
    // Far field of this brick: the distance (squared) from which on atoms are
    // interpolated, 0 for none. Bricks with less than half their points on the
    // grid do without: the nodes would cost more than the points.
    static constexpr bool kFar = P_ == 8 && SPLIT == 1;
    static constexpr bool kShort = kFar;
    __device__ __forceinline__ float far_from2() const {
        const int ni = min(kBI, T->nx - i0), nj = min(kBJ, T->ny - j0), nk = min(kBK, T->nz - k0);
        return 2 * ni * nj * nk >= kBI * kBJ * kBK ? T->far2 : 0.f;
    }
    // Cartesian position at lattice coordinates (a, b, c) of the brick, on the
    // grid or past its end
    __device__ __forceinline__ void lattice_at(const double* r, double a, double b, double c,
                                               double& x, double& y, double& z) const {
        frac_to_cart(r, (i0 + a) / (T->nx - 1), (j0 + b) / (T->ny - 1), (k0 + c) / (T->nz - 1), x,
                     y, z);
    }
    __device__ __forceinline__ bool warp_box(const double* r, int w, double* lo,
                                             double* hi) const {
        const int b = sub(w);
        return box(r, (b & 1) * P_, P_, ((b >> 1) & 1) * kWJ, kWJ, (b >> 2) * kWK, kWK, lo, hi);
    }
    // where point p goes, for points on the grid
    __device__ __forceinline__ size_t offset(int w, int lane, int p) const {
        int i, j, k;
        index(w, lane, p, i, j, k);
        return (size_t)k + (size_t)j * T->nz + (size_t)i * T->ny * T->nz;
    }
    __device__ __forceinline__ float* target(int w, int lane, int p) const {
        return T->out + offset(w, lane, p);
    }
    __device__ __forceinline__ double* target64(int w, int lane, int p) const {
        return T->out64 + offset(w, lane, p);
    }
};

// Widom insertion points: CTA c owns sorted positions [256 P c, 256 P (c + 1))
// of `order` (points stored in that order); warp w the 32 P positions from
// 256 P c + 32 P w, lane l position p * 32 + l of them. SPLIT > 1 as for grid
// bricks: SPLIT CTAs share those positions, SPLIT warps a warp's 32 P of them.
template <int P_, int SPLIT = 1>
struct PointPolicy : BrickPart<SPLIT> {
    static constexpr int kP = P_ / SPLIT;
    static constexpr int kBoxP = P_;  // points per lane of the box passes
    static constexpr bool kFar = false;
    static constexpr bool kShort = P_ == 4;  // (shared by its split forms)
    static constexpr bool kLattice = false;
    static_assert(P_ % SPLIT == 0 && kWarps % SPLIT == 0, "whole points and warps");
    const PointTask* T;
    int base, nv;
    __device__ PointPolicy(const PointTask* task, int item)
        : BrickPart<SPLIT>(item), T(task), base(item / SPLIT * (kWarps * 32 * P_)),
          nv(*task->n_valid) {}
    // the position of point p of lane `lane`, warp w
    __device__ __forceinline__ int raw_pos(int w, int lane, int p) const {
        return base + (this->part * (kWarps / SPLIT) + w / SPLIT) * (32 * P_) +
               (w % SPLIT * kP + p) * 32 + lane;
    }
    __device__ __forceinline__ int pos_of(int w, int lane, int p, bool& ok) const {
        const int pos = raw_pos(w, lane, p);
        ok = pos < nv;
        return ok ? pos : min(base, nv - 1);  // a finite stand-in, never stored
    }
    // Cartesian position of a sorted position that is in range
    __device__ __forceinline__ void at(int pos, double& x, double& y, double& z) const {
        x = T->pts[3 * (size_t)pos];
        y = T->pts[3 * (size_t)pos + 1];
        z = T->pts[3 * (size_t)pos + 2];
    }
    // point q (of kBoxP) that warp w brings to the CTA box, and to the box of
    // the 32 P positions it works on
    __device__ __forceinline__ bool cta_point(int w, int lane, int q, double& x, double& y,
                                              double& z) const {
        const int pos = base + w * (32 * P_) + q * 32 + lane;
        if (pos < nv) at(pos, x, y, z);
        return pos < nv;
    }
    __device__ __forceinline__ bool warp_point(int w, int lane, int q, double& x, double& y,
                                               double& z) const {
        const int pos =
            base + (this->part * (kWarps / SPLIT) + w / SPLIT) * (32 * P_) + q * 32 + lane;
        if (pos < nv) at(pos, x, y, z);
        return pos < nv;
    }
    // Cartesian position (frame r), stored at its bin-order position by the
    // placement pass
    __device__ __forceinline__ bool cart(const double*, int w, int lane, int p, double& x,
                                         double& y, double& z) const {
        bool ok;
        at(pos_of(w, lane, p, ok), x, y, z);
        return ok;
    }
    // fractional position, regenerated from the insertion's Philox counter
    // (only the exact cutoff decisions need it)
    __device__ __forceinline__ bool point(int w, int lane, int p, double* f) const {
        bool ok;
        const int pos = pos_of(w, lane, p, ok);
        insertion_point(T->seed, (uint64_t)T->order[pos], f);
        return ok;
    }
    // where the energy of point p, which is in range, goes
    __device__ __forceinline__ float* target(int w, int lane, int p) const {
        return T->energies + T->order[raw_pos(w, lane, p)];
    }
};

// ---------------------------------------------------------------------------
// Half-width (in ulps of fl32(rc^2)) of the window around rc^2 inside which
// an FP32 r^2 may sit on the other side of rc^2 from the exact FP64 r^2.
// Coordinates relative to the CTA centre are bounded by M = rc + margin +
// box diagonal; each displacement component then carries at most 1.5 ulp(M)
// of rounding (two roundings into FP32, one subtraction), which moves r^2 by
// at most 2 sqrt(3) rc * 1.5 ulp(M) near the cutoff; the FMUL/FFMA chain adds
// at most 1.5 ulp(rc^2). The window is twice that bound plus two ulps.
__device__ __forceinline__ int borderline_ulps(double rc, float rc2f, double box_diag) {
    const double M = rc + 1e-3 + box_diag;
    int e;
    frexp(M, &e);
    const double ulpM = ldexp(1.0, e - 24);
    frexp((double)rc2f, &e);
    const double ulpR = ldexp(1.0, e - 24);
    const double err = 2.0 * 1.7320508075688772 * rc * 1.5 * ulpM + 1.5 * ulpR + 1e-9;
    return 2 * ((int)ceil(err / ulpR) + 2);
}

// Per-thread state of one CTA pass. The FP64 per-point sums live in shared
// memory (EngineSmem::tot), the warp box and the CTA centre too.
template <class Pol, int PREC>
struct Lane {
    static constexpr int P = Pol::kP;
    static constexpr int NY = Pol::kLattice ? 1 : P;  // distinct y, z per lane
    float px[P], py[NY], pz[NY];
    unsigned vmask;
    bool warp_live;
    int bul;
};

__device__ __forceinline__ double& tot_at(EngineSmem& s, int p) {
    return s.tot[p][threadIdx.x];
}

template <int N>
struct Int {
    static constexpr int value = N;
};

// Folds FP32 chunk sums into FP64 registers.
template <int M>
__device__ __forceinline__ void fold_regs(double* acc64, f2_t* acc2) {
#pragma unroll
    for (int m = 0; m < M; ++m) {
        float a0, a1;
        f2_unpack(acc2[m], a0, a1);
        acc64[2 * m] += (double)a0;
        acc64[2 * m + 1] += (double)a1;
        acc2[m] = 0ull;
    }
}

// Folds FP32 chunk sums into the FP64 totals.
template <int M>
__device__ __forceinline__ void fold_packed(EngineSmem& s, f2_t* acc2) {
#pragma unroll
    for (int m = 0; m < M; ++m) {
        float a0, a1;
        f2_unpack(acc2[m], a0, a1);
        tot_at(s, 2 * m) += (double)a0;
        tot_at(s, 2 * m + 1) += (double)a1;
        acc2[m] = 0ull;
    }
}

// Lattice inner list: every pair inside the cutoff, packed over point pairs.
template <class Pol, int PREC>
__device__ __forceinline__ void lattice_inner(EngineSmem& s, const unsigned short* wl,
                                              int n_in, Lane<Pol, PREC>& L) {
    constexpr int M = Pol::kP / 2;
    constexpr bool kComp = PrecTraits<PREC>::comp;
    constexpr int kChunk = InnerChunk<Pol, PREC>::value;
    f2_t px2[M], acc2[M];
    double acc64[2 * M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        px2[m] = f2_pack(L.px[2 * m], L.px[2 * m + 1]);
        acc2[m] = 0ull;
        acc64[2 * m] = acc64[2 * m + 1] = 0.0;
    }
    const f2_t one2 = f2_pack(1.0f, 1.0f);
    const float py = L.py[0], pz = L.pz[0];
    const char* cbase = reinterpret_cast<const char*>(s.cand);
    const unsigned* wl32 = reinterpret_cast<const unsigned*>(wl);
    auto atom = [&](const ulonglong2 v0, const ulonglong2 v1) {  // x x | y z, C12 | -C6
        if (PREC == PREC_COUNT) {
#pragma unroll
            for (int m = 0; m < M; ++m) acc2[m] = f2_add(acc2[m], one2);
            return;
        }
        float ay, az;
        f2_unpack(v0.y, ay, az);
        const float ss = ss_lattice(py, pz, ay, az);
        const f2_t ss2 = f2_pack(ss, ss);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const f2_t dx = f2_sub(px2[m], v0.x);
            const f2_t r2 = f2_fma(dx, dx, ss2);
            float r0, r1;
            f2_unpack(r2, r0, r1);
            const f2_t u = f2_pack(rcp_approx(r0), rcp_approx(r1));
            const f2_t u3 = f2_mul(f2_mul(u, u), u);
            acc2[m] = f2_fma(u3, f2_fma(v1.x, u3, v1.y), acc2[m]);
        }
    };
    auto atoms = [&](auto n_, const unsigned* off) {
        constexpr int N = decltype(n_)::value;
        ulonglong2 v0[N], v1[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            v0[k] = *reinterpret_cast<const ulonglong2*>(cbase + off[k]);
            v1[k] = *reinterpret_cast<const ulonglong2*>(cbase + off[k] + 16);
        }
#pragma unroll
        for (int k = 0; k < N; ++k) atom(v0[k], v1[k]);
    };
    int q = 0;
    while (q < n_in) {
        const int qe = kComp ? min(q + kChunk, n_in) : n_in;
        // eight atoms per iteration (one 128-bit load of their list entries):
        // more independent chains between the MUFU results (256-framework
        // batch: 350 -> 342 ms against two atoms per iteration)
        for (; q + 7 < qe; q += 8) {  // q is a multiple of 8 here (chunk starts are)
            const uint4 e = *reinterpret_cast<const uint4*>(wl32 + (q >> 1));
            const unsigned o0[4] = {e.x & 0xffffu, e.x >> 16, e.y & 0xffffu, e.y >> 16};
            const unsigned o1[4] = {e.z & 0xffffu, e.z >> 16, e.w & 0xffffu, e.w >> 16};
            atoms(Int<4>{}, o0);
            atoms(Int<4>{}, o1);
        }
        for (; q + 3 < qe; q += 4) {
            const uint2 e = *reinterpret_cast<const uint2*>(wl32 + (q >> 1));
            const unsigned o[4] = {e.x & 0xffffu, e.x >> 16, e.y & 0xffffu, e.y >> 16};
            atoms(Int<4>{}, o);
        }
        for (; q < qe; ++q) {
            const unsigned o[1] = {wl[q]};
            atoms(Int<1>{}, o);
        }
        fold_regs<M>(acc64, acc2);
    }
#pragma unroll
    for (int p = 0; p < 2 * M; ++p) tot_at(s, p) += acc64[p];
}

// Lattice shell list: cutoff tested per pair (mask 1.0 / 0.0), and the
// smallest |r^2 - fl32(rc^2)| per point pair kept for the borderline test.
template <class Pol, int PREC>
__device__ __forceinline__ int lattice_shell(EngineSmem& s, const unsigned short* wl, int n_sh,
                                             float rc2f, float win, Lane<Pol, PREC>& L,
                                             unsigned& rec) {
    constexpr int M = Pol::kP / 2;
    constexpr bool kComp = PrecTraits<PREC>::comp;
    f2_t px2[M], acc2[M];
    int nrec = 0;
    rec = 0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        px2[m] = f2_pack(L.px[2 * m], L.px[2 * m + 1]);
        acc2[m] = 0ull;
    }
    const f2_t rc2 = f2_pack(rc2f, rc2f);
    const float py = L.py[0], pz = L.pz[0];
    const char* cbase = reinterpret_cast<const char*>(s.cand);
    // the shell list runs backwards from the end of wl
    const unsigned* wl32 = reinterpret_cast<const unsigned*>(wl);
    // the pair terms of one atom; returns its smallest |r^2 - fl32(rc^2)|
    auto atom = [&](const ulonglong2 v0, const ulonglong2 v1) {  // x x | y z, C12 | -C6
        float ay, az;
        f2_unpack(v0.y, ay, az);
        const float ss = ss_lattice(py, pz, ay, az);
        const f2_t ss2 = f2_pack(ss, ss);
        float mn = INFINITY;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const f2_t dx = f2_sub(px2[m], v0.x);
            const f2_t r2 = f2_fma(dx, dx, ss2);
            float r0, r1, d0, d1;
            f2_unpack(r2, r0, r1);
            const f2_t in = f2_pack(set_lt(r0, rc2f), set_lt(r1, rc2f));
            f2_unpack(f2_sub(r2, rc2), d0, d1);
            mn = fminf(mn, fminf(fabsf(d0), fabsf(d1)));
            if (PREC == PREC_COUNT) {
                acc2[m] = f2_add(acc2[m], in);
            } else {
                const f2_t u = f2_pack(rcp_approx(r0), rcp_approx(r1));
                const f2_t u3 = f2_mul(f2_mul(u, u), u);
                acc2[m] = f2_fma(f2_mul(u3, in), f2_fma(v1.x, u3, v1.y), acc2[m]);
            }
        }
        return mn;
    };
    // N atoms (positions q .. q + N - 1 of the list): one branch for them all
    auto atoms = [&](auto n_, const unsigned* off, int q) {
        constexpr int N = decltype(n_)::value;
        ulonglong2 v0[N], v1[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            v0[k] = *reinterpret_cast<const ulonglong2*>(cbase + off[k]);
            v1[k] = *reinterpret_cast<const ulonglong2*>(cbase + off[k] + 16);
        }
        float mn[N], all = INFINITY;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            mn[k] = atom(v0[k], v1[k]);
            all = fminf(all, mn[k]);
        }
        if (all <= win) {  // rare: a pair of these atoms sits near the cutoff
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (mn[k] <= win) {
                    rec = (rec << 10) | (unsigned)(q + k);
                    ++nrec;
                }
        }
    };
    int q = 0;
    while (q < n_sh) {
        const int qe = kComp ? min(q + kAccChunk, n_sh) : n_sh;
        for (; q + 3 < qe; q += 4) {
            // entries q .. q + 3 sit at wl[K - 1 - q] .. wl[K - 4 - q]: one aligned
            // 64-bit load (q is a multiple of 4 here: chunks are)
            const uint2 four = *reinterpret_cast<const uint2*>(wl32 + ((kMaxCand - 4 - q) >> 1));
            const unsigned off[4] = {four.y >> 16, four.y & 0xffffu, four.x >> 16,
                                     four.x & 0xffffu};
            atoms(Int<4>{}, off, q);
        }
        for (; q < qe; ++q) {
            const unsigned off[1] = {wl[kMaxCand - 1 - q]};
            atoms(Int<1>{}, off, q);
        }
        if (kComp) fold_packed<M>(s, acc2);
    }
    if (!kComp) fold_packed<M>(s, acc2);
    return nrec;
}

// Generic (per-point x, y, z) inner and shell lists, packed over point pairs
// (2m, 2m + 1): per two pair terms 9 packed FP32x2 instructions and 2
// MUFU.RCP; r^2 = fma(dz, dz, fma(dy, dy, dx * dx)) as in r2_generic, so the
// borderline re-check reproduces it bit for bit.
template <class Pol, int PREC>
__device__ __forceinline__ int generic_packed_lists(EngineSmem& s, const unsigned short* wl,
                                                    int n_in, int n_sh, float rc2f, float win,
                                                    Lane<Pol, PREC>& L, unsigned& rec) {
    constexpr int M = Pol::kP / 2;
    constexpr bool kComp = PrecTraits<PREC>::comp;
    f2_t px2[M], py2[M], pz2[M], acc2[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        px2[m] = f2_pack(L.px[2 * m], L.px[2 * m + 1]);
        py2[m] = f2_pack(L.py[2 * m], L.py[2 * m + 1]);
        pz2[m] = f2_pack(L.pz[2 * m], L.pz[2 * m + 1]);
        acc2[m] = 0ull;
    }
    const f2_t one2 = f2_pack(1.0f, 1.0f);
    const f2_t rc2 = f2_pack(rc2f, rc2f);
    const char* cbase = reinterpret_cast<const char*>(s.cand);
    int nrec = 0;
    rec = 0;
    auto inner_atom = [&](const ulonglong2 v0, const ulonglong2 v1) {  // x x | y z, C12 | -C6
        if (PREC == PREC_COUNT) {
#pragma unroll
            for (int m = 0; m < M; ++m) acc2[m] = f2_add(acc2[m], one2);
            return;
        }
        float ay, az;
        f2_unpack(v0.y, ay, az);
        const f2_t ay2 = f2_pack(ay, ay), az2 = f2_pack(az, az);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const f2_t dx = f2_sub(px2[m], v0.x);
            const f2_t dy = f2_sub(py2[m], ay2);
            const f2_t dz = f2_sub(pz2[m], az2);
            const f2_t r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
            float r0, r1;
            f2_unpack(r2, r0, r1);
            const f2_t u = f2_pack(rcp_approx(r0), rcp_approx(r1));
            const f2_t u3 = f2_mul(f2_mul(u, u), u);
            acc2[m] = f2_fma(u3, f2_fma(v1.x, u3, v1.y), acc2[m]);
        }
    };
    // returns the atom's smallest |r^2 - fl32(rc^2)|
    auto shell_atom = [&](const ulonglong2 v0, const ulonglong2 v1) {
        float ay, az;
        f2_unpack(v0.y, ay, az);
        const f2_t ay2 = f2_pack(ay, ay), az2 = f2_pack(az, az);
        float mn = INFINITY;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const f2_t dx = f2_sub(px2[m], v0.x);
            const f2_t dy = f2_sub(py2[m], ay2);
            const f2_t dz = f2_sub(pz2[m], az2);
            const f2_t r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
            float r0, r1, d0, d1;
            f2_unpack(r2, r0, r1);
            const f2_t in = f2_pack(set_lt(r0, rc2f), set_lt(r1, rc2f));
            f2_unpack(f2_sub(r2, rc2), d0, d1);
            mn = fminf(mn, fminf(fabsf(d0), fabsf(d1)));
            if (PREC == PREC_COUNT) {
                acc2[m] = f2_add(acc2[m], in);
            } else {
                const f2_t u = f2_pack(rcp_approx(r0), rcp_approx(r1));
                const f2_t u3 = f2_mul(f2_mul(u, u), u);
                acc2[m] = f2_fma(f2_mul(u3, in), f2_fma(v1.x, u3, v1.y), acc2[m]);
            }
        }
        return mn;
    };
    auto load = [&](unsigned off, ulonglong2& v0, ulonglong2& v1) {
        v0 = *reinterpret_cast<const ulonglong2*>(cbase + off);
        v1 = *reinterpret_cast<const ulonglong2*>(cbase + off + 16);
    };
    auto inner = [&](auto n_, const unsigned short* l) {
        constexpr int N = decltype(n_)::value;
        ulonglong2 v0[N], v1[N];
#pragma unroll
        for (int k = 0; k < N; ++k) load(l[k], v0[k], v1[k]);
#pragma unroll
        for (int k = 0; k < N; ++k) inner_atom(v0[k], v1[k]);
    };
    // N atoms (positions q .. q + N - 1 of the list): one branch for them all
    auto shell = [&](auto n_, int q) {
        constexpr int N = decltype(n_)::value;
        ulonglong2 v0[N], v1[N];
#pragma unroll
        for (int k = 0; k < N; ++k) load(wl[kMaxCand - 1 - q - k], v0[k], v1[k]);
        float mn[N], all = INFINITY;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            mn[k] = shell_atom(v0[k], v1[k]);
            all = fminf(all, mn[k]);
        }
        if (all <= win) {  // rare: a pair of these atoms sits near the cutoff
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (mn[k] <= win) {
                    rec = (rec << 10) | (unsigned)(q + k);
                    ++nrec;
                }
        }
    };
    int q = 0;
    // the FP32 chunk sums of the inner list fold into FP64 registers, added to
    // the shared totals once (the Widom kernel has the registers for it)
    double acc64[2 * M];
#pragma unroll
    for (int m = 0; m < 2 * M; ++m) acc64[m] = 0.0;
    // atoms whose records are loaded together: as many as the registers hold
    constexpr int kIn = M > 2 ? 4 : 8, kSh = M > 2 ? 2 : 4;
    while (q < n_in) {
        const int qe = kComp ? min(q + InnerChunk<Pol, PREC>::value, n_in) : n_in;
        for (; q + kIn <= qe; q += kIn) inner(Int<kIn>{}, wl + q);
        for (; q + 2 <= qe; q += 2) inner(Int<2>{}, wl + q);
        if (q < qe) inner(Int<1>{}, wl + q++);
        if (kComp) fold_regs<M>(acc64, acc2);
    }
    if (kComp) {
#pragma unroll
        for (int p = 0; p < 2 * M; ++p) tot_at(s, p) += acc64[p];
    }
    q = 0;
    while (q < n_sh) {
        const int qe = kComp ? min(q + kAccChunk, n_sh) : n_sh;
        for (; q + kSh <= qe; q += kSh) shell(Int<kSh>{}, q);
        for (; q < qe; ++q) shell(Int<1>{}, q);
        if (kComp) fold_packed<M>(s, acc2);
    }
    if (!kComp) fold_packed<M>(s, acc2);
    return nrec;
}

// Inner and shell lists of a lane's one point (split bricks), several atoms at a
// time. Per point the same operations in the same order as the packed forms
// above, so the energies are theirs bit for bit.
template <class Pol, int PREC>
__device__ __forceinline__ int single_lists(EngineSmem& s, const unsigned short* wl, int n_in,
                                            int n_sh, float rc2f, float win,
                                            Lane<Pol, PREC>& L, unsigned& rec) {
    constexpr bool kComp = PrecTraits<PREC>::comp;
    // one point's state leaves the registers for many records, and two warps per
    // scheduler need them (32^3 grid, records loaded together: 4 34.9 us, 8 32.4, 16
    // 30.8)
    constexpr int kSh = 16;
    constexpr int kIn = InnerChunk<Pol, PREC>::value < 16 ? InnerChunk<Pol, PREC>::value : 16;
    const float px = L.px[0], py = L.py[0], pz = L.pz[0];
    const char* cbase = reinterpret_cast<const char*>(s.cand);
    float acc = 0.f;
    auto r2_of = [&](const float4 v) {  // x x y z
        return Pol::kLattice ? r2_lattice(px, v.x, ss_lattice(py, pz, v.z, v.w))
                             : r2_generic(px, py, pz, v.x, v.z, v.w);
    };
    auto load = [&](unsigned off, float4& v0, float4& v1) {
        v0 = *reinterpret_cast<const float4*>(cbase + off);
        v1 = *reinterpret_cast<const float4*>(cbase + off + 16);
    };
    auto inner = [&](auto n_, const unsigned short* l) {
        constexpr int N = decltype(n_)::value;
        float4 v0[N], v1[N];
#pragma unroll
        for (int k = 0; k < N; ++k) load(l[k], v0[k], v1[k]);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (PREC == PREC_COUNT) {
                acc += 1.0f;
            } else {
                const float u = rcp_approx(r2_of(v0[k]));
                const float u3 = __fmul_rn(__fmul_rn(u, u), u);
                acc = __fmaf_rn(u3, __fmaf_rn(v1[k].x, u3, v1[k].z), acc);
            }
        }
    };
    double acc64 = 0.0;
    int q = 0;
    while (q < n_in) {
        const int qe = kComp ? min(q + InnerChunk<Pol, PREC>::value, n_in) : n_in;
        for (; q + kIn <= qe; q += kIn) inner(Int<kIn>{}, wl + q);
        for (; q + 2 <= qe; q += 2) inner(Int<2>{}, wl + q);
        if (q < qe) inner(Int<1>{}, wl + q++);
        if (kComp || Pol::kLattice) {
            acc64 += (double)acc;
            acc = 0.f;
        }
    }
    if (kComp || Pol::kLattice) tot_at(s, 0) += acc64;
    int nrec = 0;
    rec = 0;
    auto shell = [&](auto n_, int q) {
        constexpr int N = decltype(n_)::value;
        float4 v0[N], v1[N];
#pragma unroll
        for (int k = 0; k < N; ++k) load(wl[kMaxCand - 1 - q - k], v0[k], v1[k]);
        float d[N], all = INFINITY;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float r2 = r2_of(v0[k]);
            const float in = set_lt(r2, rc2f);
            d[k] = fabsf(__fsub_rn(r2, rc2f));
            all = fminf(all, d[k]);
            if (PREC == PREC_COUNT) {
                acc += in;
            } else {
                const float u = rcp_approx(r2);
                const float u3 = __fmul_rn(__fmul_rn(u, u), u);
                acc = __fmaf_rn(__fmul_rn(u3, in), __fmaf_rn(v1[k].x, u3, v1[k].z), acc);
            }
        }
        if (all <= win) {  // rare: a pair of these atoms sits near the cutoff
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (d[k] <= win) {
                    rec = (rec << 10) | (unsigned)(q + k);
                    ++nrec;
                }
        }
    };
    q = 0;
    while (q < n_sh) {
        const int qe = kComp ? min(q + kAccChunk, n_sh) : n_sh;
        for (; q + kSh <= qe; q += kSh) shell(Int<kSh>{}, q);
        for (; q + 4 <= qe; q += 4) shell(Int<4>{}, q);
        for (; q < qe; ++q) shell(Int<1>{}, q);
        if (kComp) {
            tot_at(s, 0) += (double)acc;
            acc = 0.f;
        }
    }
    if (!kComp) tot_at(s, 0) += (double)acc;
    return nrec;
}

// Exact re-decision of the borderline shell pairs: a pair whose FP32 r^2 is
// within `win` of fl32(rc^2) is decided by exact_in_cutoff, and its term
// added or removed where the FP32 decision differed. The shell loops record
// the list positions of the atoms with such a pair (the last kRec of them,
// 10 bits each, in `rec`); past kRec records the whole shell list is
// re-examined. Kept out of line: it runs for a few
// lanes of some warps.
template <class Pol, int PREC>
static __device__ __noinline__ void recheck_borderline(const Pol& pol, const FwDev& fw,
                                                       const CutoffConsts& cc, int n_sh,
                                                       float win, int nrec, unsigned rec,
                                                       const Lane<Pol, PREC>& L) {
    EngineSmem& s = engine_smem();
    const unsigned short* wl = s.wl[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float rc2f = cc.rc2f;
    const bool all = nrec > kRec;
    const int nq = all ? n_sh : nrec;
    // ascending list positions either way (the latest record sits in the low
    // bits), so the corrections of a point add up in one order whichever
    // points share its thread: an energy depends only on its warp's and CTA's
    // point sets, not on where in the warp the point sits
    for (int r = 0; r < nq; ++r) {
        const int q = all ? r : (int)((rec >> (10 * (nq - 1 - r))) & 1023u);
        const unsigned off = wl[kMaxCand - 1 - q];
        const Cand& cd = s.cand[off >> 5];
        const float ss = Pol::kLattice ? ss_lattice(L.py[0], L.pz[0], cd.ay, cd.az) : 0.f;
#pragma unroll 1
        for (int p = 0; p < Pol::kP; ++p) {
            if (!(L.vmask & (1u << p))) continue;
            const float r2 =
                Pol::kLattice ? r2_lattice(L.px[p], cd.ax, ss)
                              : r2_generic(L.px[p], L.py[Pol::kLattice ? 0 : p],
                                           L.pz[Pol::kLattice ? 0 : p], cd.ax, cd.ay, cd.az);
            const float dd = __fsub_rn(r2, rc2f);
            if (fabsf(dd) <= win) {
                double f[3];
                pol.point(w, lane, p, f);
                const bool ex = exact_in_cutoff(fw, f, s.cid[off >> 5], cc.r2min);
                if (ex != (dd < 0.f)) {
                    const float e = PREC == PREC_COUNT ? 1.0f : pair_term(r2, cd.c12, cd.nc6);
                    tot_at(s, p) += ex ? (double)e : -(double)e;
                }
            }
        }
    }
}

// Near lists of PREC_NEAR64 in FP64: exact positions (FP64 images and points
// relative to the CTA centre) and FP64 (C12, C6), n_ni atoms inside the cutoff
// for every point of the warp and n_ns crossing it. A warp's lanes fetch the
// data of 32 atoms at once into the warp's (by now consumed) inner / shell
// list, so the fetch latency -- list entry, image index, image, each a
// dependent load -- is paid once per 32 atoms instead of once per atom, and
// every lane reads the atoms back by broadcast. Out of line: its FP64 state
// stays out of the FP32 loops' registers.
static_assert(kNearStage * sizeof(NearAtom) <= kMaxCand * sizeof(unsigned short),
              "the staged atoms fit a warp's list");

template <class Pol, int PREC>
static __device__ __noinline__ void near_lists(const Pol& pol, const FwDev& fw,
                                               const CutoffConsts& cc, int n_ni, int n_ns,
                                               const Lane<Pol, PREC>& L) {
    constexpr int P = Pol::kP;
    // lattice lanes take all P points in one pass (dy^2 + dz^2 once per atom);
    // generic points, with their own y and z each, take passes of 4
    constexpr int kNearP = Pol::kLattice ? P : (P < 4 ? P : 4);
    EngineSmem& s = engine_smem();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned short* wn = s.wn[w];
    NearAtom* st = reinterpret_cast<NearAtom*>(s.wl[w]);
    const double o0 = s.org[0], o1 = s.org[1], o2 = s.org[2];
    // list entry q counts from the front (inside) or from the back (crossing)
    auto stage = [&](int q0, int n, bool back) {
        __syncwarp();  // the warp is done with the list, or with the atoms staged before
        const int q = q0 + lane;
        if (q < n) {
            const int gid = s.cid[wn[back ? kNearCap - 1 - q : q] >> 5];
            const Atom64 a = atom64(fw, gid, o0, o1, o2);
            NearAtom& d = st[lane];
            *reinterpret_cast<double2*>(&d.x) = make_double2(a.x, a.y);
            *reinterpret_cast<double2*>(&d.z) = make_double2(a.z, a.c12);
            d.c6 = a.c6;
        }
        __syncwarp();
    };
    auto staged = [&](int k) {
        const double2 u = *reinterpret_cast<const double2*>(&st[k].x);
        const double2 v = *reinterpret_cast<const double2*>(&st[k].z);
        return Atom64{u.x, u.y, v.x, v.y, st[k].c6};
    };
#pragma unroll 1
    for (int p0 = 0; p0 < P; p0 += kNearP) {
        double qx[kNearP], qy[Pol::kLattice ? 1 : kNearP], qz[Pol::kLattice ? 1 : kNearP];
        double nacc[kNearP];
#pragma unroll
        for (int p = 0; p < kNearP; ++p) {
            double x, y, z;
            pol.cart(fw.r, w, lane, p0 + p, x, y, z);
            qx[p] = x - o0;
            if (!Pol::kLattice || p == 0) {
                qy[Pol::kLattice ? 0 : p] = y - o1;
                qz[Pol::kLattice ? 0 : p] = z - o2;
            }
            nacc[p] = 0.0;
        }
        // atoms inside the cutoff for every point of the warp: no test
        for (int q0 = 0; q0 < n_ni; q0 += kNearStage) {
            stage(q0, n_ni, false);
            const int m = min(kNearStage, n_ni - q0);
            for (int k = 0; k < m; ++k) {
                const Atom64 a = staged(k);
                if (Pol::kLattice) {
                    const double dy = qy[0] - a.y, dz = qz[0] - a.z;
                    const double yzc = fma(dz, dz, fma(dy, dy, cc.r2min));
#pragma unroll
                    for (int p = 0; p < kNearP; ++p)
                        nacc[p] = near_acc64(nacc[p], qx[p] - a.x, yzc, a.c12, a.c6);
                } else {
#pragma unroll
                    for (int p = 0; p < kNearP; ++p) {
                        const double dy = qy[Pol::kLattice ? 0 : p] - a.y;
                        const double dz = qz[Pol::kLattice ? 0 : p] - a.z;
                        nacc[p] = near_acc64(nacc[p], qx[p] - a.x,
                                             fma(dz, dz, fma(dy, dy, cc.r2min)), a.c12, a.c6);
                    }
                }
            }
        }
        // atoms crossing the cutoff inside the warp box (boxes wider than
        // rc - kNearR: coarse grids, sparse Widom bins): the cutoff decided per
        // pair on the FP64 r^2. It differs from the reference's FP64 r^2 (cell
        // frame, its own rounding) by far less than 1e-12 rc^2, so outside that
        // window both decide alike and inside it exact_in_cutoff decides.
        const double rc2lo = fw.rc2 * (1.0 - 1e-12), rc2hi = fw.rc2 * (1.0 + 1e-12);
        for (int q0 = 0; q0 < n_ns; q0 += kNearStage) {
            stage(q0, n_ns, true);
            const int m = min(kNearStage, n_ns - q0);
            for (int k = 0; k < m; ++k) {
                const Atom64 a = staged(k);
#pragma unroll
                for (int p = 0; p < kNearP; ++p) {
                    const double dy = qy[Pol::kLattice ? 0 : p] - a.y;
                    const double dz = qz[Pol::kLattice ? 0 : p] - a.z;
                    const double dx = qx[p] - a.x;
                    const double r2 = fmax(fma(dx, dx, fma(dz, dz, dy * dy)), cc.r2min);
                    bool inside = r2 < rc2lo;
                    if (!inside && r2 < rc2hi && (L.vmask & (1u << (p0 + p)))) {
                        double f[3];
                        pol.point(w, lane, p0 + p, f);
                        inside = exact_in_cutoff(fw, f, s.cid[wn[kNearCap - 1 - q0 - k] >> 5],
                                                 cc.r2min);
                    }
                    const double u = rcp64_nr(r2);
                    const double u3 = u * u * u;
                    if (inside) nacc[p] = fma(u3, fma(a.c12, u3, -a.c6), nacc[p]);
                }
            }
        }
#pragma unroll
        for (int p = 0; p < kNearP; ++p) tot_at(s, p0 + p) += nacc[p];
    }
}

// Inner and shell lists of PREC_FP64: every pair term in FP64 (the reference
// mode of the precision sweeps, and a caller's choice), shell pairs decided on
// their FP32 r^2 and by exact_in_cutoff inside the error window. Atoms are
// fetched 32 at a time as in near_lists and serve all of a lane's points; with
// every point fetching every atom the 65 x 63 x 61 grid of a 424-atom cell took
// 280 us, now 167 (bound by FP64 arithmetic, 22 operations a pair).
template <class Pol, int PREC>
__device__ __forceinline__ void fp64_lists(EngineSmem& s, const Pol& pol, const FwDev& fw,
                                           const CutoffConsts& cc, const unsigned short* wl,
                                           int n_in, int n_sh, float win,
                                           const Lane<Pol, PREC>& L) {
    constexpr int P = Pol::kP;
    static_assert(Pol::kLattice, "grids only");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    NearAtom* st = fp64_stage();
    double qx[P], qy, qz, acc[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        pol.cart(fw.r, w, lane, p, qx[p], qy, qz);
        qx[p] -= s.org[0];
        acc[p] = 0.0;
    }
    qy -= s.org[1];
    qz -= s.org[2];
    // list entries q0 .. of a list of n: `step` = 1 from its front, -1 from its back
    auto stage = [&](const unsigned short* list, int step, int q0, int n) {
        __syncwarp();
        if (q0 + lane < n) {
            const Atom64 a = atom64(fw, s.cid[list[step * (q0 + lane)] >> 5], s.org[0], s.org[1],
                                    s.org[2]);
            NearAtom& d = st[lane];
            *reinterpret_cast<double2*>(&d.x) = make_double2(a.x, a.y);
            *reinterpret_cast<double2*>(&d.z) = make_double2(a.z, a.c12);
            d.c6 = a.c6;
        }
        __syncwarp();
    };
    // the correctly rounded reciprocal: a seed refined twice took 31 us less
    // and left errors up to 9 % larger (against 64-bit sums, eight grids)
    auto term = [&](const NearAtom& a, double dy, double dz, int p) {
        const double dx = qx[p] - a.x;
        const double u = __drcp_rn(fmax(fma(dz, dz, fma(dy, dy, dx * dx)), cc.r2min));
        const double u3 = u * u * u;
        return u3 * fma(a.c12, u3, -a.c6);
    };
    for (int q0 = 0; q0 < n_in; q0 += kNearStage) {
        stage(wl, 1, q0, n_in);
        const int m = min(kNearStage, n_in - q0);
        for (int k = 0; k < m; ++k) {
            const NearAtom a = st[k];
            const double dy = qy - a.y, dz = qz - a.z;
#pragma unroll
            for (int p = 0; p < P; ++p) acc[p] += term(a, dy, dz, p);
        }
    }
    const unsigned short* back = wl + kMaxCand - 1;
    for (int q0 = 0; q0 < n_sh; q0 += kNearStage) {
        stage(back, -1, q0, n_sh);
        const int m = min(kNearStage, n_sh - q0);
        for (int k = 0; k < m; ++k) {
            const NearAtom a = st[k];
            const unsigned off = back[-(q0 + k)];
            const Cand& cd = s.cand[off >> 5];
            const float ss = ss_lattice(L.py[0], L.pz[0], cd.ay, cd.az);
            const double dy = qy - a.y, dz = qz - a.z;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const float dd = __fsub_rn(r2_lattice(L.px[p], cd.ax, ss), cc.rc2f);
                bool inside = dd < 0.f;
                if (fabsf(dd) <= win) {
                    double f[3];
                    pol.point(w, lane, p, f);
                    inside = exact_in_cutoff(fw, f, s.cid[off >> 5], cc.r2min);
                }
                const double e = term(a, dy, dz, p);
                if (inside) acc[p] += e;
            }
        }
    }
#pragma unroll
    for (int p = 0; p < P; ++p) tot_at(s, p) += acc[p];
}

// ---------------------------------------------------------------------------
// Far field. Atoms that lie inside the cutoff for every point of a brick and
// at least Rf away from it add a smooth function of the position: it is summed
// at 8 x 8 x 8 nodes (8 Chebyshev nodes for each 16 points along the first and
// third axis, every lattice line along the second) instead of 2048 points, and
// interpolated to the points in FP64. Rf (far_distance2) keeps the error of the
// interpolation, which falls as (x + sqrt(x^2 + 1))^-8 with x = Rf over the
// half-width 7.5 spacings and grows as sigma^12, below the rounding of the FP32
// pair terms (1e-6 to 2e-5 K root mean square at epsilon 94 K, against 2e-5 to
// 5e-3); those are the same here as for the points. At 0.12 A
// about 60 % of a cell's pairs are far and cost a quarter: a 256^3 grid of 4096
// atoms 8.70 -> 6.57 ms, 8 triclinic frameworks (54 M points) 16.76 -> 14.2 ms.
constexpr int kFarN = 8;   // nodes per 16 lattice points
constexpr int kFarL = 16;

struct FarTable {
    double node[kFarN];         // node positions in lattice coordinates, 0 .. 15
    double w[kFarL][kFarN];     // Lagrange weights of the 16 lattice points
};
constexpr FarTable make_far_table() {
    // cos((2 m + 1) pi / 16)
    const double c[4] = {0.98078528040323044913, 0.83146961230254523708, 0.55557023301960222474,
                         0.19509032201612826785};
    FarTable t{};
    for (int m = 0; m < kFarN; ++m) {
        const double x = m < 4 ? -c[m] : c[kFarN - 1 - m];
        t.node[m] = 7.5 + 7.5 * x;
    }
    for (int i = 0; i < kFarL; ++i)
        for (int m = 0; m < kFarN; ++m) {
            double w = 1.0;
            for (int q = 0; q < kFarN; ++q)
                if (q != m) w *= (i - t.node[q]) / (t.node[m] - t.node[q]);
            t.w[i][m] = w;
        }
    return t;
}
static __constant__ FarTable kFarTable = make_far_table();

// Scratch of the far field in the warp lists, which the flush builds after it.
struct FarSmem {
    union {
        double part[kWarps][kFarN][32];            // a column group's partial sums per warp
        double line[kFarN][2 * kWJ][kFarL];        // nodes along i, points along j and k
    };
    double node[2][kFarN][32];                     // per column group: nodes along i, (j, k) column
};
static_assert(sizeof(FarSmem) <= sizeof(EngineSmem::wl) + sizeof(EngineSmem::wn),
              "the far field fits the warp lists");

// Adds the far field of the n_far atoms at the end of the candidate list to
// the points' totals. All warps of the block, which meet at its barriers.
template <class Pol, int PREC>
__device__ __forceinline__ void far_field(EngineSmem& s, const Pol& pol, const FwDev& fw,
                                          int n_far) {
    constexpr int M = kFarN / 2;
    constexpr int kChunk = kShortChunk;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    FarSmem& f = *reinterpret_cast<FarSmem*>(&s.wl[0][0]);
    // this warp's share of the atoms
    const int a0 = n_far * w / kWarps, a1 = n_far * (w + 1) / kWarps;
    const Cand* far = s.cand + (kMaxCand - n_far);
#pragma unroll 1
    for (int g = 0; g < 2; ++g) {  // lattice lines 4 g .. 4 g + 3 along j
        f2_t px2[M], acc2[M];
        double acc64[kFarN];
        float py = 0.f, pz = 0.f;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            float px[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double x, y, z;
                pol.lattice_at(fw.r, kFarTable.node[2 * m + h], g * kWJ + lane / kWK,
                               kFarTable.node[lane % kWK], x, y, z);
                px[h] = (float)(x - s.org[0]);
                py = (float)(y - s.org[1]);
                pz = (float)(z - s.org[2]);
            }
            px2[m] = f2_pack(px[0], px[1]);
            acc2[m] = 0ull;
            acc64[2 * m] = acc64[2 * m + 1] = 0.0;
        }
        auto atom = [&](const ulonglong2 v0, const ulonglong2 v1) {  // x x | y z, C12 | -C6
            float ay, az;
            f2_unpack(v0.y, ay, az);
            const float ss = ss_lattice(py, pz, ay, az);
            const f2_t ss2 = f2_pack(ss, ss);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const f2_t dx = f2_sub(px2[m], v0.x);
                const f2_t r2 = f2_fma(dx, dx, ss2);
                float r0, r1;
                f2_unpack(r2, r0, r1);
                const f2_t u = f2_pack(rcp_approx(r0), rcp_approx(r1));
                const f2_t u3 = f2_mul(f2_mul(u, u), u);
                acc2[m] = f2_fma(u3, f2_fma(v1.x, u3, v1.y), acc2[m]);
            }
        };
        for (int a = a0; a < a1;) {
            const int e = min(a + kChunk, a1);
            for (; a + 3 < e; a += 4) {
                ulonglong2 v0[4], v1[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    v0[k] = *reinterpret_cast<const ulonglong2*>(&far[a + k].ax);
                    v1[k] = *reinterpret_cast<const ulonglong2*>(&far[a + k].c12);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) atom(v0[k], v1[k]);
            }
            for (; a < e; ++a)
                atom(*reinterpret_cast<const ulonglong2*>(&far[a].ax),
                     *reinterpret_cast<const ulonglong2*>(&far[a].c12));
            fold_regs<M>(acc64, acc2);
        }
#pragma unroll
        for (int m = 0; m < kFarN; ++m) f.part[w][m][lane] = acc64[m];
        __syncthreads();
        double sum = 0.0;  // thread (m, column) = (w, lane), in warp order
#pragma unroll
        for (int k = 0; k < kWarps; ++k) sum += f.part[k][w][lane];
        f.node[g][w][lane] = sum;
        __syncthreads();
    }
    // along k: from 8 nodes to 16 points (256 threads: 4 of the 8 x 8 x 16 each)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = u * kThreads + tid, k = e % kFarL, j = e / kFarL % (2 * kWJ);
        const int m = e / (kFarL * 2 * kWJ);
        const double* nd = &f.node[j / kWJ][m][j % kWJ * kWK];
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < kFarN; ++q) v = fma(kFarTable.w[k][q], nd[q], v);
        f.line[m][j][k] = v;
    }
    __syncthreads();
    // along i: this lane's points
    const int j = ((w >> 1) & 1) * kWJ + lane / kWK, k = (w >> 2) * kWK + lane % kWK;
    double v[kFarN];
#pragma unroll
    for (int m = 0; m < kFarN; ++m) v[m] = f.line[m][j][k];
#pragma unroll
    for (int p = 0; p < Pol::kP; ++p) {
        double e = 0.0;
#pragma unroll
        for (int m = 0; m < kFarN; ++m) e = fma(kFarTable.w[(w & 1) * Pol::kP + p][m], v[m], e);
        tot_at(s, p) += e;
    }
    __syncthreads();  // the warps' lists take the scratch's place
}

template <class Pol, int PREC>
__device__ __forceinline__ void warp_flush(EngineSmem& s, const Pol& pol, const FwDev& fw,
                                                const CutoffConsts& cc, int n_cand,
                                                Lane<Pol, PREC>& L) {
    constexpr int P = Pol::kP;
    constexpr bool kNear = PrecTraits<PREC>::near64;
    constexpr bool kF64 = PrecTraits<PREC>::fp64;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (!L.warp_live) return;
    unsigned short* wl = s.wl[w];
    unsigned short* wn = s.wn[w];
    // --- split candidates into inner / shell (/ near) lists for this warp's box
    int n_in = 0, n_sh = 0, n_ni = 0, n_ns = 0;
    const unsigned lt = (1u << lane) - 1u;
    const float rnear2 = kNearR * kNearR;
    const float wl0x = s.wbox[w][0], wl0y = s.wbox[w][1], wl0z = s.wbox[w][2];
    const float wh0x = s.wbox[w][3], wh0y = s.wbox[w][4], wh0z = s.wbox[w][5];
    // groups of 32 per turn: two in split bricks, whose few warps wait for the
    // ballots of one group with the boxes of the other (32^3 grid 36.9 -> 34.9 us);
    // elsewhere other warps fill the wait and the second group only takes registers
    constexpr int kGroups = P == 1 ? 2 : 1;
    for (int base = 0; base < n_cand; base += 32 * kGroups) {
        bool in[kGroups], sh[kGroups], nr[kGroups];
#pragma unroll
        for (int h = 0; h < kGroups; ++h) {
            const int c = base + 32 * h + lane;
            in[h] = sh[h] = nr[h] = false;
            if (c < n_cand) {
                const float4 a = *reinterpret_cast<const float4*>(&s.cand[c].ax);
                const float ax = a.x, ay = a.z, az = a.w;
                const float ex = fmaxf(0.f, fmaxf(wl0x - ax, ax - wh0x));
                const float ey = fmaxf(0.f, fmaxf(wl0y - ay, ay - wh0y));
                const float ez = fmaxf(0.f, fmaxf(wl0z - az, az - wh0z));
                const float dmin2 = ex * ex + ey * ey + ez * ez;
                const float fx = fmaxf(fabsf(ax - wl0x), fabsf(ax - wh0x));
                const float fy = fmaxf(fabsf(ay - wl0y), fabsf(ay - wh0y));
                const float fz = fmaxf(fabsf(az - wl0z), fabsf(az - wh0z));
                const float dmax2 = fx * fx + fy * fy + fz * fz;
                in[h] = dmax2 < cc.rin2;
                sh[h] = !in[h] && dmin2 < cc.rout2;
                nr[h] = kNear && dmin2 < rnear2;
            }
        }
#pragma unroll
        for (int h = 0; h < kGroups; ++h) {
            const unsigned short off =
                (unsigned short)((base + 32 * h + lane) * (int)sizeof(Cand));
            if (kNear) {
                // near atoms inside the cutoff for every point of the warp go to the
                // front of wn, near atoms crossing it (large warp boxes) to the back;
                // past kNearCap entries they stay on the FP32 lists
                const bool ni = nr[h] && in[h], ns = nr[h] && sh[h];
                const unsigned bni = __ballot_sync(0xffffffffu, ni);
                const unsigned bns = __ballot_sync(0xffffffffu, ns);
                const int room = kNearCap - n_ni - n_ns;
                const int ti = min(__popc(bni), room);
                const int ts = min(__popc(bns), room - ti);
                const int ai = __popc(bni & lt), as = __popc(bns & lt);
                if (ni && ai < ti) {
                    wn[n_ni + ai] = off;
                    in[h] = false;
                }
                if (ns && as < ts) {
                    wn[kNearCap - 1 - (n_ns + as)] = off;
                    sh[h] = false;
                }
                n_ni += ti;
                n_ns += ts;
            }
            const unsigned bi = __ballot_sync(0xffffffffu, in[h]);
            const unsigned bs = __ballot_sync(0xffffffffu, sh[h]);
            if (in[h]) wl[n_in + __popc(bi & lt)] = off;
            if (sh[h]) wl[kMaxCand - 1 - (n_sh + __popc(bs & lt))] = off;
            n_in += __popc(bi);
            n_sh += __popc(bs);
        }
    }
    __syncwarp();

    const float rc2f = cc.rc2f;
    float win;
    {
        int e;
        frexpf(rc2f, &e);
        win = ldexpf((float)L.bul, e - 24);
    }

    int nrec = 0;
    unsigned rec = 0;
    if constexpr (kF64) {
        fp64_lists<Pol, PREC>(s, pol, fw, cc, wl, n_in, n_sh, win, L);
        return;
    }

    if constexpr (P == 1) {
        nrec = single_lists<Pol, PREC>(s, wl, n_in, n_sh, rc2f, win, L, rec);
    } else if constexpr (Pol::kLattice) {
        lattice_inner<Pol, PREC>(s, wl, n_in, L);
        nrec = lattice_shell<Pol, PREC>(s, wl, n_sh, rc2f, win, L, rec);
    } else {
        nrec = generic_packed_lists<Pol, PREC>(s, wl, n_in, n_sh, rc2f, win, L, rec);
    }

    // --- exact re-decision of borderline shell pairs (rare); lanes without a
    // flagged point idle through it
    if (nrec > 0) recheck_borderline<Pol, PREC>(pol, fw, cc, n_sh, win, nrec, rec, L);
    if (kNear && n_ni + n_ns > 0) near_lists<Pol, PREC>(pol, fw, cc, n_ni, n_ns, L);
}

template <class Pol, int PREC>
__device__ void process_cta(const Pol& pol, const FwDev& fw, const CutoffConsts& cc) {
    EngineSmem& s = engine_smem();
    constexpr int P = Pol::kP;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    Lane<Pol, PREC> L;

    // 1. the CTA box (FP64 bounding box of the valid points), whose centre is
    // the origin of the FP32 coordinates, and the warp box in them
    double lo0, lo1, lo2, hi0, hi1, hi2;
    L.vmask = 0;
    if constexpr (Pol::kLattice) {
        pol.fill_axes(tid);
        __syncthreads();
        double lo[3], hi[3];
        pol.cta_box(fw.r, lo, hi);  // a brick holds at least one point of the grid
        lo0 = lo[0]; lo1 = lo[1]; lo2 = lo[2];
        hi0 = hi[0]; hi1 = hi[1]; hi2 = hi[2];
    } else {
        double mn0 = INFINITY, mn1 = INFINITY, mn2 = INFINITY;
        double mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY;
#pragma unroll
        for (int q = 0; q < Pol::kBoxP; ++q) {
            double x, y, z;
            // (unsplit, the CTA's points are its own lanes')
            const bool ok = Pol::kBoxP == P ? pol.cart(fw.r, w, lane, q, x, y, z)
                                            : pol.cta_point(w, lane, q, x, y, z);
            if (ok) {
                mn0 = fmin(mn0, x); mn1 = fmin(mn1, y); mn2 = fmin(mn2, z);
                mx0 = fmax(mx0, x); mx1 = fmax(mx1, y); mx2 = fmax(mx2, z);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn0 = fmin(mn0, __shfl_xor_sync(0xffffffffu, mn0, o));
            mn1 = fmin(mn1, __shfl_xor_sync(0xffffffffu, mn1, o));
            mn2 = fmin(mn2, __shfl_xor_sync(0xffffffffu, mn2, o));
            mx0 = fmax(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            mx1 = fmax(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
            mx2 = fmax(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
        }
        if (lane == 0) {
            s.red[w][0] = mn0; s.red[w][1] = mn1; s.red[w][2] = mn2;
            s.red[w][3] = mx0; s.red[w][4] = mx1; s.red[w][5] = mx2;
        }
        __syncthreads();
        if (tid < 6) {
            double v = s.red[0][tid];
            for (int k = 1; k < kWarps; ++k)
                v = (tid < 3) ? fmin(v, s.red[k][tid]) : fmax(v, s.red[k][tid]);
            s.box[tid] = v;
        }
        __syncthreads();
        lo0 = s.box[0]; lo1 = s.box[1]; lo2 = s.box[2];
        hi0 = s.box[3]; hi1 = s.box[4]; hi2 = s.box[5];
        __syncthreads();
        if (!(lo0 <= hi0)) return;  // no valid point in this CTA
    }
    const double o0 = 0.5 * (lo0 + hi0), o1 = 0.5 * (lo1 + hi1), o2 = 0.5 * (lo2 + hi2);
    L.bul = borderline_ulps(
        cc.rc, cc.rc2f,
        sqrt((hi0 - lo0) * (hi0 - lo0) + (hi1 - lo1) * (hi1 - lo1) + (hi2 - lo2) * (hi2 - lo2)));

    // 2. local FP32 coordinates and the warp box (a lattice lane's points
    // share y and z bit for bit: R[1][0] = R[2][0] = 0)
    {
        float wl0x = INFINITY, wl0y = INFINITY, wl0z = INFINITY;
        float wh0x = -INFINITY, wh0y = -INFINITY, wh0z = -INFINITY;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            double x, y, z;
            if (pol.cart(fw.r, w, lane, p, x, y, z)) L.vmask |= 1u << p;
            const float fx = (float)(x - o0), fy = (float)(y - o1), fz = (float)(z - o2);
            L.px[p] = fx;
            if (!Pol::kLattice || p == 0) {
                L.py[Pol::kLattice ? 0 : p] = fy;
                L.pz[Pol::kLattice ? 0 : p] = fz;
            }
            tot_at(s, p) = 0.0;
            // (unsplit, the warp's points are its own lanes')
            if (!Pol::kLattice && Pol::kBoxP == P && (L.vmask & (1u << p))) {
                wl0x = fminf(wl0x, fx); wl0y = fminf(wl0y, fy); wl0z = fminf(wl0z, fz);
                wh0x = fmaxf(wh0x, fx); wh0y = fmaxf(wh0y, fy); wh0z = fmaxf(wh0z, fz);
            }
        }
        if constexpr (Pol::kLattice) {
            // x -> (float)(x - o) is monotone too
            double lo[3], hi[3];
            L.warp_live = pol.warp_box(fw.r, w, lo, hi);
            if (L.warp_live) {
                wl0x = (float)(lo[0] - o0); wl0y = (float)(lo[1] - o1); wl0z = (float)(lo[2] - o2);
                wh0x = (float)(hi[0] - o0); wh0y = (float)(hi[1] - o1); wh0z = (float)(hi[2] - o2);
            }
        } else {
#pragma unroll
            for (int q = 0; q < (Pol::kBoxP == P ? 0 : Pol::kBoxP); ++q) {
                double x, y, z;
                if (pol.warp_point(w, lane, q, x, y, z)) {
                    const float fx = (float)(x - o0), fy = (float)(y - o1), fz = (float)(z - o2);
                    wl0x = fminf(wl0x, fx); wl0y = fminf(wl0y, fy); wl0z = fminf(wl0z, fz);
                    wh0x = fmaxf(wh0x, fx); wh0y = fmaxf(wh0y, fy); wh0z = fmaxf(wh0z, fz);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                wl0x = fminf(wl0x, __shfl_xor_sync(0xffffffffu, wl0x, o));
                wl0y = fminf(wl0y, __shfl_xor_sync(0xffffffffu, wl0y, o));
                wl0z = fminf(wl0z, __shfl_xor_sync(0xffffffffu, wl0z, o));
                wh0x = fmaxf(wh0x, __shfl_xor_sync(0xffffffffu, wh0x, o));
                wh0y = fmaxf(wh0y, __shfl_xor_sync(0xffffffffu, wh0y, o));
                wh0z = fmaxf(wh0z, __shfl_xor_sync(0xffffffffu, wh0z, o));
            }
            L.warp_live = wl0x <= wh0x;
        }
        if (lane == 0) {
            s.wbox[w][0] = wl0x; s.wbox[w][1] = wl0y; s.wbox[w][2] = wl0z;
            s.wbox[w][3] = wh0x; s.wbox[w][4] = wh0y; s.wbox[w][5] = wh0z;
        }
        __syncwarp();
    }

    // 3. producer: rows of cells around the CTA box, streamed into shared memory.
    // What its loops need of the box lies in shared memory: held in registers
    // it would spill around every flush.
    int c0[3], c1[3];
    {
        const double lov[3] = {lo0, lo1, lo2}, hiv[3] = {hi0, hi1, hi2};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            c0[d] = max(0, (int)floor((lov[d] - cc.rcm - fw.cell_lo[d]) * fw.inv_h));
            c1[d] = min(fw.nc[d] - 1, (int)floor((hiv[d] + cc.rcm - fw.cell_lo[d]) * fw.inv_h));
        }
    }
    if (tid == 0) {
        s.org[0] = o0; s.org[1] = o1; s.org[2] = o2;
        s.cbox[0] = (float)(lo0 - o0); s.cbox[1] = (float)(lo1 - o1); s.cbox[2] = (float)(lo2 - o2);
        s.cbox[3] = (float)(hi0 - o0); s.cbox[4] = (float)(hi1 - o1); s.cbox[5] = (float)(hi2 - o2);
    }
    __syncthreads();
    constexpr bool kFar = Pol::kFar && PrecTraits<PREC>::far;
    float far2 = 0.f;  // squared distance of the far field, 0 without one
    if constexpr (kFar) {
        far2 = pol.far_from2();
        if (far2 > 0.f && tid < 3) {
            // extent along Cartesian axis `tid`: each lattice axis adds its own
            double at[3], lo, hi;
            pol.lattice_at(fw.r, 0.0, 0.0, 0.0, at[0], at[1], at[2]);
            lo = hi = tid == 0 ? at[0] : tid == 1 ? at[1] : at[2];
            for (int d = 0; d < 3; ++d) {
                double e[3];
                pol.lattice_at(fw.r, d == 0 ? Pol::kBI - 1.0 : 0.0, d == 1 ? Pol::kBJ - 1.0 : 0.0,
                               d == 2 ? Pol::kBK - 1.0 : 0.0, e[0], e[1], e[2]);
                const double x = (tid == 0 ? e[0] - at[0] : tid == 1 ? e[1] - at[1] : e[2] - at[2]);
                lo += fmin(x, 0.0);
                hi += fmax(x, 0.0);
            }
            s.fbox[tid] = (float)(lo - s.org[tid]);
            s.fbox[3 + tid] = (float)(hi - s.org[tid]);
        }
        __syncthreads();
    }
    const float R2f = (float)(cc.rcm * cc.rcm);
    // rows are pruned in FP32 with 1e-3 A of slack, some hundred times the rounding
    // of these coordinates (|x| < 64 A: 4e-6 A): every image that passes the test
    // below lies in the pruned range
    const float Rrow = (float)cc.rcm + 1e-3f, R2row = Rrow * Rrow;
    // Fills the candidate list, flushes it and goes on until every row is done.
    // One flush site (the pair loops are inlined there), and a chunk of images
    // that no longer fits is taken again after the flush, so that no thread
    // holds an image through the pair loops.
    int nyr = 0, nrows = 0;
    if (c0[0] <= c1[0] && c0[1] <= c1[1] && c0[2] <= c1[2]) {
        nyr = c1[1] - c0[1] + 1;
        nrows = nyr * (c1[2] - c0[2] + 1);
    }
    int rb = 0, cb = 0, tot = 0, nr = 0, buf = 0;
    for (bool more = true; more;) {
        int n_cand = 0, n_far = 0;  // from the front, and from the back
        for (;;) {
            if (cb >= tot) {  // the next chunk of rows
                if (rb >= nrows) {
                    more = false;
                    break;
                }
                const int r = rb + tid;
                int beg = 0, len = 0;
                if (r < nrows) {
                    const int ry = c0[1] + r % nyr, rz = c0[2] + r / nyr;
                    const float y = (float)(fw.cell_lo[1] + ry * fw.h - s.org[1]);
                    const float z = (float)(fw.cell_lo[2] + rz * fw.h - s.org[2]);
                    const float hf = (float)fw.h;
                    const float dy = fmaxf(0.f, fmaxf(y - s.cbox[4], s.cbox[1] - (y + hf)));
                    const float dz = fmaxf(0.f, fmaxf(z - s.cbox[5], s.cbox[2] - (z + hf)));
                    const float d2 = dy * dy + dz * dz;
                    if (d2 < R2row) {
                        const float ex = sqrtf(R2row - d2);
                        const double x0 = s.org[0] - fw.cell_lo[0];
                        const int xa = max(c0[0], (int)floor((x0 + (s.cbox[0] - ex)) * fw.inv_h));
                        const int xb = min(c1[0], (int)floor((x0 + (s.cbox[3] + ex)) * fw.inv_h));
                        if (xa <= xb) {
                            const int rowb = (rz * fw.nc[1] + ry) * fw.nc[0];
                            beg = fw.cell_start[rowb + xa];
                            len = fw.cell_start[rowb + xb + 1] - beg;
                        }
                    }
                }
                int off = len;  // inclusive scan over the warp
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, off, o);
                    if (lane >= o) off += v;
                }
                off += block_prefix(s, buf, __shfl_sync(0xffffffffu, off, 31), &tot) - len;
                buf ^= 1;
                s.row_beg[tid] = beg;
                s.row_off[tid] = off;
                __syncthreads();
                nr = min(kRowChunk, nrows - rb);
                rb += kRowChunk;
                cb = 0;
                continue;
            }
            const int c = cb + tid;
            bool pass = false, far = false;
            int g = 0;
            float ax = 0.f, ay = 0.f, az = 0.f;
            float2 pr = make_float2(0.f, 0.f);
            if (c < tot) {
                int a = 0, b = nr - 1;
                while (a < b) {
                    const int mid = (a + b + 1) >> 1;
                    if (s.row_off[mid] <= c) a = mid; else b = mid - 1;
                }
                g = s.row_beg[a] + (c - s.row_off[a]);
                const double4 ap = fw.img_xyz[g];
                pr = fw.img_par[g];
                ax = (float)(ap.x - s.org[0]);
                ay = (float)(ap.y - s.org[1]);
                az = (float)(ap.z - s.org[2]);
                const float ddx = fmaxf(0.f, fmaxf(s.cbox[0] - ax, ax - s.cbox[3]));
                const float ddy = fmaxf(0.f, fmaxf(s.cbox[1] - ay, ay - s.cbox[4]));
                const float ddz = fmaxf(0.f, fmaxf(s.cbox[2] - az, az - s.cbox[5]));
                pass = (ddx * ddx + ddy * ddy + ddz * ddz) < R2f;
                if (kFar && far2 > 0.f && pass) {
                    const float lx = s.fbox[0] - ax, ly = s.fbox[1] - ay, lz = s.fbox[2] - az;
                    const float hx = ax - s.fbox[3], hy = ay - s.fbox[4], hz = az - s.fbox[5];
                    const float nx = fmaxf(0.f, fmaxf(lx, hx)), ny = fmaxf(0.f, fmaxf(ly, hy));
                    const float nz = fmaxf(0.f, fmaxf(lz, hz));
                    const float mx = fminf(lx, hx), my = fminf(ly, hy), mz = fminf(lz, hz);
                    // max over the box of |x - ax| is -min(lo - ax, ax - hi)
                    far = nx * nx + ny * ny + nz * nz > far2 &&
                          mx * mx + my * my + mz * mz < cc.rin2;
                    pass = !far;
                }
            }
            const unsigned ball = __ballot_sync(0xffffffffu, pass);
            const unsigned fball = kFar ? __ballot_sync(0xffffffffu, far) : 0u;
            const unsigned below = (1u << lane) - 1u;
            int both;  // counts of the two kinds in the halves of a word
            const int at = block_prefix(s, buf, __popc(ball) | (__popc(fball) << 16), &both);
            buf ^= 1;
            const int npass = both & 0xffff, nfar = both >> 16;
            if (n_cand + n_far + npass + nfar > kMaxCand) break;
            if (pass || far) {
                const int pos = pass ? n_cand + (at & 0xffff) + __popc(ball & below)
                                     : kMaxCand - 1 - (n_far + (at >> 16) + __popc(fball & below));
                Cand& dst = s.cand[pos];
                *reinterpret_cast<float4*>(&dst.ax) = make_float4(ax, ax, ay, az);
                *reinterpret_cast<float4*>(&dst.c12) = make_float4(pr.x, pr.x, pr.y, pr.y);
                if (pass) s.cid[pos] = g;
            }
            n_cand += npass;
            n_far += nfar;
            cb += kThreads;
        }
        __syncthreads();
        if constexpr (kFar) {
            if (n_far > 0) far_field<Pol, PREC>(s, pol, fw, n_far);
        }
        if (n_cand > 0) warp_flush<Pol, PREC>(s, pol, fw, cc, n_cand, L);
        if (more) __syncthreads();
    }
    // 4. store
    // lattice points: every address before the first store, which may alias the
    // task the next address is formed from and would make it wait (8 triclinic
    // frameworks 14.23 -> 14.10 ms; the Widom kernel, whose addresses are loads of
    // their own, spills over it and is faster one by one, 1651 against 1677 us per
    // 1e7 insertions)
    if constexpr (PrecTraits<PREC>::fp64) {
#pragma unroll
        for (int p = 0; p < P; ++p)
            if (L.vmask & (1u << p))
                *pol.target64(w, lane, p) = fmin(tot_at(s, p), (double)kEnergyCap);
    } else {
        float* to[P];
        if constexpr (Pol::kLattice) {
#pragma unroll
            for (int p = 0; p < P; ++p) to[p] = pol.target(w, lane, p);
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
            if (L.vmask & (1u << p)) {
                float e = (float)tot_at(s, p);
                if (PREC != PREC_COUNT) e = fminf(e, kEnergyCap);
                if constexpr (Pol::kLattice) {
                    // streaming store: the grid is written once and not read back
                    // here, so its lines are the first the L2 evicts
                    __stcs(to[p], e);
                } else {
                    *pol.target(w, lane, p) = e;
                }
            }
        }
    }
    __syncthreads();
}

}  // namespace er
