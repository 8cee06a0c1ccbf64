// One "axis pass": a batch of power-of-two complex DFTs of length L, each
// computed by one group of L/R threads of a CTA, with the pre- and
// post-processing of the transform kind fused into the load and the store.
//
// Addressing.  Transform b of the batch is split as b0 = b % d0,
// b1 = (b / d0) % d1, b2 = b / (d0*d1); its input starts at
// b0*is0 + b1*is1 + b2*is2 and element n sits at +n*in_n (likewise for the
// output with os*, out_k).  This one form covers rows (in_n = 1), columns of
// a C-order array (in_n = product of trailing dims) and the large-length
// passes of a Stockham FFT over HBM (see plan.cu).
//
// Thread layout.  Row mode: the L/R threads of one transform are adjacent,
// so a warp reads consecutive elements of one row.  Column mode: the cpb
// transforms of the CTA are adjacent in memory (consecutive columns), so the
// thread index runs fastest over the transform.  Either way every global
// access of a warp is a contiguous run.
//
// Within the CTA the DFT is a Stockham autosort FFT: thread j of a transform
// holds elements j + r*(L/R), r < R, in registers; each pass multiplies by
// table twiddles, runs an R-point (or smaller) DFT in registers and exchanges
// through padded shared memory.  The last pass leaves output element
// k = j + r*(L/R) in register r, so the first load and the last store need
// no shared memory at all for the plain complex transform.
//
// Kind roots.  The load and store stages multiply by roots w_M^k of the kind
// tables at k = j + i*(L/R).  Thread j reads only table entry j (one load per
// table) and forms the others as w_M^j * w_M^(i*L/R); for the tables used
// here M is 2L, 4L or 8L, so the second factor is the 128th root of unity
// w_128^(i*128L/(M*R)), a constant-memory operand (w128).  When L/R = 1 the
// only thread is j = 0 and w_M^0 = 1 is not read at all.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "roots128.h"

namespace mb {

// w_128^m, m < 32 (m is a compile-time constant once the caller's loop is unrolled)
__device__ __forceinline__ cpx w128(int m) {
#if MINFFT_SINGLE
  return cmk(roots128::kReF[m], roots128::kImF[m]);
#else
  return cmk(roots128::kReD[m], roots128::kImD[m]);
#endif
}

// Entry j of a kind table: the base of this thread's roots (see above).
template <int TPT>
__device__ __forceinline__ cpx kind_base(const cpx* table, int j) {
  if constexpr (TPT == 1) {
    return cmk(real(1), real(0));
  } else {
    return ldg(table + j);
  }
}

// The roots w^(j + i*(L/R)) of a kind table, i = 0 .. R/2: base times constant
// w_128^(i*kStep), two roundings more than the table's entry unless j = 0.  At 16
// and 32 points radix 16 has such threads for all or half of the roots, radix 8
// for half as many, and a DCT-4 pair of 64 x 64 was less exact so (single 3.1e-7
// for 2.6e-7, double 3.75e-16 for 3.67e-16).  There its kernels read each root
// from the table, in single the other kinds' too, and at 128 points, where
// radix 8 has a pass more (256 x 256: 3.7e-7 for 3.2e-7).  So 64 x 64 rounds to
// 2.5e-7 and 3.4e-16 and 256 x 256 to 2.8e-7.  32768 DCT-4 of 64 points in double,
// bound by L1 traffic, take 20.0 us a pair with table roots, 18.9 without, 28.1
// at radix 16; in single 14.8, 14.6 and 43; with the tables in shared memory
// (nd_pass.cu) reading is the faster way at every length (DCT-2 + DCT-3 of 64 x 64
// in double 11.4 us, 12.4 without).
#ifdef MB_TABLES_GENERIC
constexpr bool kTablesNear = true;
#else
constexpr bool kTablesNear = false;
#endif
template <int L, int R, bool kT4>
constexpr bool kTableRoots = R == 8 && L > R &&
                             (kTablesNear || (kT4 && L == 32) || (sizeof(real) == 4 && (L == 32 || L == 128)));
template <int L, int R, int kStep, bool kT4 = false>
struct KindRoots {
  const cpx* t;
  cpx base;
  __device__ __forceinline__ KindRoots(const cpx* table, int j) : t(table + j), base(czero()) {
    if constexpr (!kTableRoots<L, R, kT4>) base = kind_base<L / R>(table, j);
  }
  __device__ __forceinline__ cpx operator()(int i) const {
    if constexpr (kTableRoots<L, R, kT4>)
      return ldg(t + i * (L / R));
    else
      return cmul(base, w128(i * kStep));
  }
};
template <int L, int R>
using RftRoots = KindRoots<L, R, 64 / R>;  // w_N^k, for 0 < k < L/2 only: i < R/2
template <int L, int R>
using T23Roots = KindRoots<L, R, 16 / R>;  // w_4N^k
template <int L, int R>
using T4Roots = KindRoots<L, R, 32 / R, true>;  // w_2N^k

struct AxisParams {
  const void* in;
  void* out;
  int64_t nbatch;
  int64_t d0, d1;
  int64_t is0, is1, is2;
  int64_t os0, os1, os2;
  int64_t in_n, out_k;
  const cpx* tw;     // w_L^m, m < L (forward roots for the in-CTA passes)
  const cpx* t1;     // kind table 1 (see the load/store stages)
  const cpx* t2;     // kind table 2
  const cpx* st_hi;  // large-length pass roots: w_Lt^(a << st_lobits)
  const cpx* st_lo;  // large-length pass roots: w_Lt^c, c < 2^st_lobits
  int64_t st_ns;     // span of the preceding HBM passes (1: no pre-twiddle)
  int64_t st_div;    // elements per span index (product of trailing dims)
  int st_shift;      // log2(Lt / (st_ns * L))
  int st_lobits;
  int cpb;      // transforms per CTA (per tile in the pipelined kernel)
  int colmode;  // 1: thread index runs fastest over the transform
  int flags;
  int chunk;    // pipelined kernel: bytes per asynchronous copy (16, 8 or 4)
  int64_t ntiles;       // pipelined kernel: number of tiles
  int64_t gpb;          // pipelined kernel, column mode: tiles per d0 block
  int stage_bytes;      // pipelined kernel: bytes of one shared-memory stage
  int lp;               // shared-memory pitch between transforms (tile_pitch)
  int* status;          // set to 1 by a kernel whose bounded device-side wait ran out
  // type-4 steps fused into the first / last pass of a 1-D chain over HBM:
  // real length N of the line, reals between lines of the real input /
  // output, and the fine-table bits of the post-rotation roots (t1, t2)
  int64_t kn, k_in_line, k_out_line;
  int kbits;
  // streamed row pass: stages in flight, bytes copied per row, bytes
  // between rows of a stage
  int nstages, row_bytes, row_pitch;
};

enum : int {
  F_SRC_SMEM = 1 << 9,  // the input pointer is a shared-memory stage (generic loads, no ld.global)
  F_CONJ_IN = 1,      // conjugate the input (inverse DFT = conj . DFT . conj)
  F_CONJ_OUT = 2,     // conjugate the output
  F_DST = 4,          // sine variant of a real symmetric transform
  F_STAGE_ROWS = 8,   // store through shared memory with k running fastest
  F_VEC = 16,         // real rows are aligned for paired (complex) vector access
};

// Shared-memory tile: cpb transforms of L complex values, transform c at
// c*lp, element p at pad16(p) (one spare slot every 16 elements, so strided
// Stockham scatters spread over all banks).  The pitch lp is skewed by the
// host (tile_pitch) so that the threads of one 128-byte wavefront -- several
// short transforms in row mode, several adjacent columns in column mode --
// land in distinct banks.
struct Tile {
  cpx* s;
  int lp;
  __device__ __forceinline__ int idx(int c, int p) const { return c * lp + pad16(p); }
};

// Pitch (in complex elements) between the transforms of a tile.
__host__ __device__ inline int tile_pitch(int L, int R, int cpb, int colmode) {
  const int W = int(128 / sizeof(cpx));  // complex values per wavefront
  const int tpt = L / (L < R ? L : R);
  int target = 0;
  if (colmode)
    target = cpb >= W ? 1 : W / cpb;
  else if (tpt < W)
    target = tpt;
  int lp = padded_len(L);
  if (target > 0)
    while (lp % W != target % W) ++lp;
  return lp;
}

// Per-thread context: which transform, which thread within it, offsets.
struct Ctx {
  int64_t b;
  int64_t b0;
  int64_t oin, oout;
  int c, j;
  bool active;
};

__device__ __forceinline__ void batch_offsets(const AxisParams& p, int64_t b, int64_t& b0, int64_t& oi, int64_t& oo) {
  const int64_t r = udiv(b, p.d0);
  b0 = b - r * p.d0;
  const int64_t b2 = udiv(r, p.d1);
  const int64_t b1 = r - b2 * p.d1;
  oi = b0 * p.is0 + b1 * p.is1 + b2 * p.is2;
  oo = b0 * p.os0 + b1 * p.os1 + b2 * p.os2;
}

// ------------------------------------------------------------ Stockham core
// u[r] *= w^r for r = 1..RP-1 with w = tw[i1]: two table roots (w, w^4) per
// sub-DFT, the other powers formed just before use as products of at most
// four roundings, so only a handful of roots are live at a time.  The radix-8
// kernels (kLoad = 3) take w^2 and w^3 from the table too: they run where the
// array is small and the loads hide, and 32- and 64-point DFTs then round no
// more than radix 16 does (in the same time).  At 128 points radix 8 has three
// passes to radix 16's two, and in single precision (kLoad = 7) takes every
// power from the table (DCT-4 pair of 256 x 256: 3.7e-7 with products, 3.45e-7
// with loads, 3.2e-7 at radix 16).
template <int RP, int kLoad>
__device__ __forceinline__ void apply_root_powers(cpx* u, const cpx* __restrict__ tw, int i1) {
  static_assert(RP <= 16, "radix up to 16");
  const cpx w1 = ldg(tw + i1);
  u[1] = cmul(u[1], w1);
  if constexpr (RP > 2) {
    const cpx w2 = kLoad ? ldg(tw + 2 * i1) : cmul(w1, w1);
    u[2] = cmul(u[2], w2);
    const cpx w3 = kLoad ? ldg(tw + 3 * i1) : cmul(w2, w1);
    u[3] = cmul(u[3], w3);
    if constexpr (RP > 4) {
      const cpx w4 = ldg(tw + 4 * i1);
      u[4] = cmul(u[4], w4);
      u[5] = cmul(u[5], kLoad > 3 ? ldg(tw + 5 * i1) : cmul(w4, w1));
      u[6] = cmul(u[6], kLoad > 3 ? ldg(tw + 6 * i1) : cmul(w4, w2));
      u[7] = cmul(u[7], kLoad > 3 ? ldg(tw + 7 * i1) : cmul(w4, w3));
      if constexpr (RP > 8) {
        const cpx w8 = cmul(w4, w4);
        u[8] = cmul(u[8], w8);
        u[9] = cmul(u[9], cmul(w8, w1));
        u[10] = cmul(u[10], cmul(w8, w2));
        u[11] = cmul(u[11], cmul(w8, w3));
        const cpx w12 = cmul(w8, w4);
        u[12] = cmul(u[12], w12);
        u[13] = cmul(u[13], cmul(w12, w1));
        u[14] = cmul(u[14], cmul(w12, w2));
        u[15] = cmul(u[15], cmul(w12, w3));
      }
    }
  }
}

template <int L, int R, int RP, int NS, bool kScalar = false>
__device__ __forceinline__ void pass_compute(cpx (&v)[R], int j, const cpx* __restrict__ tw) {
  constexpr int S = R / RP;  // sub-DFTs per thread in this pass
#pragma unroll
  for (int s = 0; s < S; ++s) {
    cpx u[RP];
#pragma unroll
    for (int r = 0; r < RP; ++r) u[r] = v[s + r * S];
    if constexpr (NS > 1) {
      const int jp = j + s * (L / R);
      const int q = jp & (NS - 1);
      constexpr int step = L / (NS * RP);
      constexpr int load = R != 8 ? 0 : (sizeof(real) == 4 && L == 128) ? 7 : 3;
      apply_root_powers<RP, load>(u, tw, q * step);
    }
    fft_reg<RP, kScalar>(u);
#pragma unroll
    for (int r = 0; r < RP; ++r) v[s + r * S] = u[r];
  }
}

// Stockham scatter of a pass with span NS: element r of sub-DFT jp goes to
// B + r*NS with B = (jp/NS)*NS*RP + jp%NS.  Either NS = 1 (B is a multiple of
// RP and r < RP) or NS*RP >= 16 (the part of B above jp%NS is a multiple of
// 16 and jp%NS < NS); in both cases pad16(B + r*NS) = pad16(B) + r*NS +
// ((r*NS) >> 4), so each sub-DFT computes one padded base and the offsets of
// its RP elements are compile-time constants.
template <int L, int R, int RP, int NS>
__device__ __forceinline__ void pass_scatter(const cpx (&v)[R], int j, int c, const Tile& t) {
  constexpr int S = R / RP;
  static_assert(NS == 1 || NS * RP >= 16, "padded offsets are linear in r");
  cpx* tb = t.s + c * t.lp;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int jp = j + s * (L / R);
    cpx* q = tb + pad16((jp / NS) * (NS * RP) + (jp & (NS - 1)));
#pragma unroll
    for (int r = 0; r < RP; ++r) q[r * NS + ((r * NS) >> 4)] = v[s + r * S];
  }
}

// Padded position of element j + r*(L/R) relative to that of element j
// (TPT = L/R either divides 16 with j < TPT, or is a multiple of 16).
template <int TPT>
__host__ __device__ constexpr int nat_off(int r) {
  return TPT >= 16 ? r * (TPT + TPT / 16) : r * TPT + ((r * TPT) >> 4);
}

template <int L, int R>
__device__ __forceinline__ void gather_natural(cpx (&v)[R], int j, int c, const Tile& t) {
  constexpr int TPT = L / R;
  const cpx* q = t.s + c * t.lp + (TPT >= 16 ? pad16(j) : j);
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = q[nat_off<TPT>(r)];
}

template <int L, int R>
__device__ __forceinline__ void scatter_natural(const cpx (&v)[R], int j, int c, const Tile& t) {
  constexpr int TPT = L / R;
  cpx* q = t.s + c * t.lp + (TPT >= 16 ? pad16(j) : j);
#pragma unroll
  for (int r = 0; r < R; ++r) q[nat_off<TPT>(r)] = v[r];
}

// All passes from span NS on.  kFresh: nothing has used the tile since the
// CTA's last barrier (the load stage went straight to registers, KeepsTile), so
// the first exchange needs no barrier before its writes: a warp whose loads
// have come goes on to them (round trips: 256^3 f32 258.0 us with the barrier,
// 253.7 without; real DFT 2048 x 2048 f64 70.7 / 69.8).
template <int L, int R, int NS, bool kFresh = false, bool kScalar = false>
__device__ __forceinline__ void run_passes(cpx (&v)[R], int j, int c, const Tile& t, const cpx* __restrict__ tw) {
  constexpr int RP = (L / NS >= R) ? R : (L / NS);
  pass_compute<L, R, RP, NS, kScalar>(v, j, tw);
  if constexpr (NS * RP < L) {
    if constexpr (!kFresh) __syncthreads();
    pass_scatter<L, R, RP, NS>(v, j, c, t);
    __syncthreads();
    gather_natural<L, R>(v, j, c, t);
    run_passes<L, R, NS * RP, false, kScalar>(v, j, c, t, tw);
  }
}

// A streaming (evict-first) load from global memory, or a plain load where
// the kernel reads its input from a shared-memory stage (F_SRC_SMEM): the
// streaming form is a global-only instruction.
template <typename T>
__device__ __forceinline__ T src_ld(const T* q, bool smem) {
  return smem ? *q : __ldcs(q);
}

// A pointer that walks a strided run: step() moves it by one stride.  kUnit
// runs have a compile-time stride, so the compiler folds every position into
// the access's immediate offset; the others add the stride to the pointer
// (two integer instructions per access -- indexing by r * stride cost four,
// 12 of the 52 instructions per point of a 256-point column pass; the asm
// keeps the compiler from turning the additions back into products).
template <typename T, bool kUnit, int kStep>
struct Walk {
  T* q;
  int64_t st;  // stride of one element
  __device__ __forceinline__ Walk(T* base, int64_t stride) : q(base), st(kUnit ? 0 : stride * kStep) {}
  __device__ __forceinline__ void step() {
    if constexpr (kUnit) {
      q += kStep;
    } else {
      q += st;
      asm("" : "+l"(q));
    }
  }
};

// ------------------------------------------------------------- row staging
// In row mode a transform's real row (N = 2L contiguous reals) is moved
// between global memory and the transform's tile slot in shared memory by its
// TPT threads as 16-byte vectors (single elements when either side is not
// 16-byte aligned), so that strided gathers and scatters (stride 4 elements,
// mirrored halves) happen in shared memory while global memory sees whole
// coalesced 16-byte accesses.  Every thread loads all of its share before
// storing any of it.  The type-3 kinds use it for both their load and their
// store (measured: 18% faster in f64, 11% in f32 on 2048-real rows); the
// type-2 and type-4 kinds were measured slower with it and keep direct
// global accesses.
__device__ __forceinline__ real* tile_row(const Tile& t, int c) { return reinterpret_cast<real*>(t.s + c * t.lp); }

template <int L, int R>
__device__ __forceinline__ void row_g2s(real* sr, const real* g, int j, bool smem = false) {
  constexpr int TPT = L / R;
  constexpr int NV = 2 * L * int(sizeof(real)) / 16;  // 16-byte vectors in the row
  static_assert(NV % TPT == 0, "whole vectors per thread");
  if (((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(sr)) & 15) == 0) {
    const uint4* gv = reinterpret_cast<const uint4*>(g) + j;
    uint4* sv = reinterpret_cast<uint4*>(sr) + j;
    uint4 r[NV / TPT];
#pragma unroll
    for (int i = 0; i < NV / TPT; ++i) r[i] = src_ld(gv + i * TPT, smem);
#pragma unroll
    for (int i = 0; i < NV / TPT; ++i) sv[i * TPT] = r[i];
  } else {
    real r[2 * R];
#pragma unroll
    for (int i = 0; i < 2 * R; ++i) r[i] = src_ld(g + j + i * TPT, smem);
#pragma unroll
    for (int i = 0; i < 2 * R; ++i) sr[j + i * TPT] = r[i];
  }
}

template <int L, int R>
__device__ __forceinline__ void row_s2g(real* g, const real* sr, int j) {
  constexpr int TPT = L / R;
  constexpr int NV = 2 * L * int(sizeof(real)) / 16;
  static_assert(NV % TPT == 0, "whole vectors per thread");
  if (((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(sr)) & 15) == 0) {
    uint4* gv = reinterpret_cast<uint4*>(g) + j;
    const uint4* sv = reinterpret_cast<const uint4*>(sr) + j;
    uint4 r[NV / TPT];
#pragma unroll
    for (int i = 0; i < NV / TPT; ++i) r[i] = sv[i * TPT];
#pragma unroll
    for (int i = 0; i < NV / TPT; ++i) __stcs(gv + i * TPT, r[i]);
  } else {
    real r[2 * R];
#pragma unroll
    for (int i = 0; i < 2 * R; ++i) r[i] = sr[j + i * TPT];
#pragma unroll
    for (int i = 0; i < 2 * R; ++i) __stcs(g + j + i * TPT, r[i]);
  }
}

// Column mode: thread j of the transform moves reals n = j + m*TPT (m < 2R)
// of its column (element stride s) into the column's tile slot, all loads
// issued before any store; a warp's load covers cpb adjacent columns of a
// few rows.
template <int L, int R>
__device__ __forceinline__ void col_g2s(real* sr, const real* g, int64_t s, int j, bool smem = false) {
  constexpr int TPT = L / R;
  real r[2 * R];
  Walk<const real, false, TPT> w(g + int64_t(j) * s, s);
#pragma unroll
  for (int m = 0; m < 2 * R; ++m, w.step()) r[m] = src_ld(w.q, smem);
#pragma unroll
  for (int m = 0; m < 2 * R; ++m) sr[j + m * TPT] = r[m];
}

// row mode with unit element strides
__device__ __forceinline__ bool rows_staged_in(const AxisParams& p) { return !p.colmode && p.in_n == 1; }
__device__ __forceinline__ bool rows_staged_out(const AxisParams& p) { return !p.colmode && p.out_k == 1; }

// ------------------------------------------------- root progressions
// The roots of a fused chain pass, W^(g0 + r*D) for a thread's elements r < R:
// W^g0 from the table pair (hi, lo) of W -- hi[e >> lobits] * lo[e & (2^lobits
// - 1)] -- and W^D.  The thread's elements are a whole Lt/R points apart
// whatever the pass (TPT strides of Lt/L), so W^(r*D) does not depend on the
// length: it is the 128th root of unity w_128^(r*K/R), a constant operand,
// with K = 16, 32 or 64 for W of 8 Lt, 4 Lt (or w_16Lt^4) or 2 Lt.  (Formed
// per thread from two more table roots, the steps took 40 of a thread's 700
// instructions and its registers: the first pass of the DCT-4 of 2^24 points
// in f32 went from 44 to 40 us.)  Exponents are 32-bit (the planner keeps
// the tables below 2^32 roots).
template <int R, int K>
struct RootProgression {
  cpx base;
  __device__ __forceinline__ RootProgression(const cpx* __restrict__ hi, const cpx* __restrict__ lo, int lobits,
                                             uint32_t g0)
      : base(cmul(ldg(hi + (g0 >> lobits)), ldg(lo + (g0 & ((1u << lobits) - 1u))))) {}
  __device__ __forceinline__ cpx at(int r) const {
    const int m = r * K / R;  // below 64
    return m < 32 ? cmul(base, w128(m)) : cmul_negi(cmul(base, w128(m - 32)));
  }
};

// The same roots as constant + constant * (W^g0 - 1).  g0 lies within one step, so
// |W^g0 - 1| < 0.2 (0.4 at radix 8), the product's roundings are a fraction of the
// root's, and in single the constant brings along what its own rounding left
// out: the root has one rounding (two in double), where the product form has
// five, counting two tables, and a coarse entry times a fine one, as the
// element-wise steps take, three.  hi and lo hold the roots minus one.
// For the real and type-2/3 lines, which were up to 6% less exact with products
// than with element-wise steps (DCT-2 + DCT-3 of 2^16 in single 3.41e-7 for 3.21e-7,
// 3.15e-7 so; of 2^22 points 49.9 -> 50.1 us in single, 82.2 -> 82.8 in double), and
// the mixed batch, whose type-4 jobs read tables of their own before (jobs of 2^16
// points 2.19e-7 for 2.06e-7, 2.07e-7 so; 20000 jobs of all lengths 979 -> 1011 us).  Type-4 lines
// gain on the element-wise step either way and keep the cheaper products (DCT-4 of
// 2^24 points 171 us, 174 with steps).
template <int R, int K>
struct RootSteps {
  cpx d;  // W^g0 - 1
  __device__ __forceinline__ RootSteps(const cpx* __restrict__ hi, const cpx* __restrict__ lo, int lobits,
                                       uint32_t g0) {
    const cpx a = ldg(hi + (g0 >> lobits)), b = ldg(lo + (g0 & ((1u << lobits) - 1u)));
    d = cadd(cadd(a, b), cmul(a, b));
  }
  __device__ __forceinline__ cpx at(int r) const {
    const int m = r * K / R, n = m & 31;  // m below 64
    const cpx c = w128(n);
#if MINFFT_SINGLE  // with what the constant's rounding left out
    const cpx e = cmk(roots128::kReR[n], roots128::kImR[n]);
    const cpx w = cadd(c, cmk(e.x + c.x * d.x - c.y * d.y, e.y + c.x * d.y + c.y * d.x));
#else  // (not as a fused multiply-add, which would round the larger sum twice)
    const cpx t = cmul(c, d), w = cmk(__dadd_rn(c.x, t.x), __dadd_rn(c.y, t.y));
#endif
    return m < 32 ? w : cmul_negi(w);
  }
};

// ------------------------------------------------------- HBM pre-twiddle
// In a pass of a Stockham FFT over HBM, element n of a sub-DFT with span
// index q is multiplied by w_Lt^g, g = q*n*Lt/(st_ns*L), each root read as
// the product of a coarse and a fine table entry.  Thread j holds
// n = j + r*TPT, so its roots are w^g0 * d^r with w^g0 = w_Lt^(q*j*s) and
// d = w_Lt^(q*TPT*s) (s = 2^st_shift): three table roots per thread (w^g0,
// d, d^4), the other powers of d formed as at most two products, as the
// in-CTA passes form theirs (apply_root_powers).
template <int L, int R>
__device__ __forceinline__ void hbm_pretwiddle(cpx (&v)[R], const AxisParams& p, int64_t b0, int j) {
  constexpr int TPT = L / R;
  // exponents stay below Lt <= 2^31: 32-bit
  const uint32_t q = uint32_t(udiv(b0, p.st_div)) & uint32_t(p.st_ns - 1);
  const uint32_t lomask = (1u << p.st_lobits) - 1u;
  auto root = [&](uint32_t g) { return cmul(ldg(p.st_hi + (g >> p.st_lobits)), ldg(p.st_lo + (g & lomask))); };
  if constexpr (R < 4) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = cmul(v[r], root((q * uint32_t(j + r * TPT)) << p.st_shift));
  } else {
    const uint32_t gd = (q * uint32_t(TPT)) << p.st_shift;
    const cpx base = root((q * uint32_t(j)) << p.st_shift);
    const cpx d1 = root(gd);
    const cpx d2 = cmul(d1, d1);
    const cpx d3 = cmul(d2, d1);
    const cpx d4 = R > 4 ? root(4 * gd) : czero();
    const cpx d8 = cmul(d4, d4);
    const cpx d12 = cmul(d8, d4);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int lo = r & 3, hi = r >> 2;
      cpx w = base;
      if (hi == 1) w = cmul(w, d4);
      if (hi == 2) w = cmul(w, d8);
      if (hi == 3) w = cmul(w, d12);
      if (lo == 1) w = cmul(w, d1);
      if (lo == 2) w = cmul(w, d2);
      if (lo == 3) w = cmul(w, d3);
      v[r] = cmul(v[r], w);
    }
  }
}

// ---------------------------------------------------------------- load ops
// Each load op fills v[r] with complex input element n = j + r*(L/R) of the
// length-L DFT of transform x.b.

// Plain complex input; optional conjugation and large-length pre-twiddle.
struct LoadCplx {
  static constexpr bool kComplexIn = true;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile&, cpx (&v)[R]) {
    constexpr int TPT = L / R;
    const cpx* in = static_cast<const cpx*>(p.in) + x.oin;
    if (!x.active) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = czero();
    } else if (p.in_n == 1) {  // contiguous: compile-time offsets
      const cpx* q = in + x.j;
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = src_ld(q + r * TPT, (p.flags & F_SRC_SMEM) != 0);
    } else {
      Walk<const cpx, false, TPT> w(in + x.j * p.in_n, p.in_n);
#pragma unroll
      for (int r = 0; r < R; ++r, w.step()) v[r] = src_ld(w.q, (p.flags & F_SRC_SMEM) != 0);
    }
    if (p.flags & F_CONJ_IN) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r].y = -v[r].y;
    }
    if (p.st_ns > 1) hbm_pretwiddle<L, R>(v, p, x.b0, x.j);
  }
};

// Real row read as L complex pairs (x[2n], x[2n+1]): the half-length complex
// DFT of the real DFT (reference minfft.c:541-543).
struct LoadR2C {
  static constexpr bool kComplexIn = false;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile&, cpx (&v)[R]) {
    constexpr int TPT = L / R;
    const real* in = static_cast<const real*>(p.in) + x.oin;
    if (!x.active) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = czero();
    } else if (p.flags & F_VEC) {
      const cpx* q = reinterpret_cast<const cpx*>(in) + x.j;
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = src_ld(q + r * TPT, (p.flags & F_SRC_SMEM) != 0);
    } else {
      const real* q = in + 2 * x.j;
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = cmk(q[2 * r * TPT], q[2 * r * TPT + 1]);
    }
  }
};

// Type-2 input permutation (reference minfft.c:707-710, 756-759): the
// length-N sequence u_i = x[2i] (i < N/2), u_i = +-x[2N-1-2i] (i >= N/2)
// read as complex pairs (u_2m, u_2m+1); N = 2L.
struct LoadDCT2 {
  static constexpr bool kComplexIn = false;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  // element m = j + r*TPT lies in the first half (m < L/2) exactly when r < R/2:
  // pair (x[4m], x[4m+2]) there, (x[2N-1-4m], x[2N-3-4m]) (times sg) after
  template <bool kUnit, int L, int R>
  static __device__ __forceinline__ void pairs(const real* in, int64_t s, int j, real sg, cpx (&v)[R]) {
    constexpr int N = 2 * L, TPT = L / R, m0 = (R / 2) * TPT;
    Walk<const real, kUnit, 4 * TPT> a(in + int64_t(4 * j) * s, s), b(in + int64_t(4 * j + 2) * s, s);
#pragma unroll
    for (int r = 0; r < R / 2; ++r, a.step(), b.step()) v[r] = cmk(*a.q, *b.q);
    Walk<const real, kUnit, -4 * TPT> c(in + int64_t(2 * N - 1 - 4 * (j + m0)) * s, s),
        d(in + int64_t(2 * N - 3 - 4 * (j + m0)) * s, s);
#pragma unroll
    for (int r = R / 2; r < R; ++r, c.step(), d.step()) v[r] = cmk(sg * *c.q, sg * *d.q);
  }
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile&, cpx (&v)[R]) {
    const real* in = static_cast<const real*>(p.in) + x.oin;
    const real sg = (p.flags & F_DST) ? real(-1) : real(1);
    if (!x.active) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = czero();
      return;
    }
    if constexpr (L >= 2) {
      if (p.in_n == 1)
        pairs<true, L, R>(in, 1, x.j, sg, v);
      else
        pairs<false, L, R>(in, p.in_n, x.j, sg, v);
    } else {
      v[0] = cmk(in[0], sg * in[p.in_n]);  // L = 1: u = (x0, +-x1)
    }
  }
};

// Type-4 pre-rotation (reference minfft.c:906-910, 953-957):
// t_n = e_n (x[2n] + i x[N-1-2n]) for DCT-4, -e_n (x[2n] - i x[N-1-2n]) for
// DST-4, with e_n = w_2N^n from table t1.
struct LoadT4 {
  static constexpr bool kComplexIn = false;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile&, cpx (&v)[R]) {
    const real* in = static_cast<const real*>(p.in) + x.oin;
    const bool dst = (p.flags & F_DST) != 0;
    constexpr int TPT = L / R;
    if (!x.active) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = czero();
      return;
    }
    const T4Roots<L, R> e(p.t1, x.j);  // w_2N^(j + r*TPT)
    if (p.in_n == 1)
      rotate<true, L, R>(in, 1, x.j, e, dst, v);
    else
      rotate<false, L, R>(in, p.in_n, x.j, e, dst, v);
  }
  template <bool kUnit, int L, int R>
  static __device__ __forceinline__ void rotate(const real* in, int64_t s, int j, const T4Roots<L, R>& e, bool dst,
                                                cpx (&v)[R]) {
    constexpr int N = 2 * L, TPT = L / R;
    const real sg = dst ? real(-1) : real(1);
    Walk<const real, kUnit, 2 * TPT> lo(in + int64_t(2 * j) * s, s);
    Walk<const real, kUnit, -2 * TPT> hi(in + int64_t(N - 1 - 2 * j) * s, s);
#pragma unroll
    for (int r = 0; r < R; ++r, lo.step(), hi.step()) {
      // DST: -(a - ib) = -a + ib
      const real a = sg * *lo.q;
      const real b = *hi.q;
      v[r] = cmul(e(r), cmk(a, b));
    }
  }
};

// Packing step of the inverse real DFT (reference minfft.c:628-656) for the
// spectrum pair (z_k, z_{L-k}); returns t_k and t_{L-k}.  f = w_N^k.
__device__ __forceinline__ void pack_pair(cpx za, cpx zb, cpx f, cpx& ta, cpx& tb) {
  const cpx m = cconj(zb);
  const cpx u = cadd(za, m);
  const cpx d = csub(za, m);
  const cpx vv = cmul(d, cmk(f.y, f.x));  // times i*conj(f)
  ta = cadd(u, vv);
  tb = cconj(csub(u, vv));
}

// Unpacking step of the real DFT (reference minfft.c:556-575) for the pair
// (Z_k, Z_{L-k}) of the half-length DFT; returns X_k and X_{L-k}.
__device__ __forceinline__ void unpack_pair(cpx za, cpx zb, cpx f, cpx& xa, cpx& xb) {
  const cpx m = cconj(zb);
  const real h = real(0.5);
  const cpx u = cscale(cadd(za, m), h);
  const cpx d = csub(za, m);
  const cpx vv = cscale(cmul(d, cmk(f.y, -f.x)), h);  // times f/(2i)
  xa = cadd(u, vv);
  xb = cconj(csub(u, vv));
}

// The same without the factor 1/2: returns 2 X_k and 2 X_{L-k} (for the
// type-2 output, which doubles them; scaling by 1/2 and 2 is exact, so the
// results are the same to the bit with two multiplies fewer per value).
__device__ __forceinline__ void unpack_pair2(cpx za, cpx zb, cpx f, cpx& xa, cpx& xb) {
  const cpx m = cconj(zb);
  const cpx u = cadd(za, m);
  const cpx d = csub(za, m);
  const cpx vv = cmul(d, cmk(f.y, -f.x));  // times f/i
  xa = cadd(u, vv);
  xb = cconj(csub(u, vv));
}

// One value of the packing step (pack_pair) for the spectrum pair (z, zm) of
// points k and L-k: the conjugated inverse-DFT input at k,
// conj(z + conj(zm) + (z - conj(zm)) i conj(f)); f = w_N^k.
__device__ __forceinline__ cpx pack_one(cpx z, cpx zm, cpx f) {
  const real a = z.x + zm.x, b = z.y - zm.y, p = z.x - zm.x, q = z.y + zm.y;
  return cmk(a + (p * f.y - q * f.x), -(b + (p * f.x + q * f.y)));
}
// One value of the unpacking step (unpack_pair2): 2 X_k from Z_k, Z_(L-k),
// z + conj(zm) + (z - conj(zm)) f/i.
__device__ __forceinline__ cpx unpack_one2(cpx z, cpx zm, cpx f) {
  const real a = z.x + zm.x, b = z.y - zm.y, p = z.x - zm.x, q = z.y + zm.y;
  return cmk(a + (p * f.y + q * f.x), b + (q * f.y - p * f.x));
}

// The same pairs' values at L-k (f = w_N^k as above): from the sums of
// pack_one and unpack_one2 with the other signs.
__device__ __forceinline__ cpx pack_mirror(cpx z, cpx zm, cpx f) {
  const real a = z.x + zm.x, b = z.y - zm.y, p = z.x - zm.x, q = z.y + zm.y;
  return cmk(a - (p * f.y - q * f.x), b - (p * f.x + q * f.y));
}
__device__ __forceinline__ cpx unpack_mirror2(cpx z, cpx zm, cpx f) {
  const real a = z.x + zm.x, b = z.y - zm.y, p = z.x - zm.x, q = z.y + zm.y;
  return cmk(a - (p * f.y + q * f.x), (q * f.y - p * f.x) - b);
}

// Visits the spectrum pairs (k, L-k), k = 0 .. L/2, owned by thread j of a
// transform: k = j + i*TPT for i = 0 .. R/2 (only j = 0 reaches k = L/2).
// ends(i, k) handles k = 0 and k = L/2, the self-paired ends; body(i, k) the
// pairs inside.  i is a compile-time constant once unrolled, so only i = 0
// and i = R/2 test for an end; step() runs after each.
template <int L, int R, class Ends, class Body, class Step>
__device__ __forceinline__ void pair_loop(const Ctx& x, const Ends& ends, const Body& body, const Step& step) {
  constexpr int TPT = L / R;
#pragma unroll
  for (int i = 0; i <= R / 2; ++i) {
    const int k = x.j + i * TPT;
    if (i == R / 2) {
      if (x.j == 0) ends(i, k);
    } else if (i == 0) {
      if (x.j == 0)
        ends(i, k);
      else
        body(i, k);
    } else {
      body(i, k);
    }
    step();
  }
}

// w_N^k (N = 2L) at k = j + i*(L/R) from base = w_N^j (kind roots, above);
// used for 0 < k < L/2, i.e. i < R/2 (other i map to w_128^0 and stay
// inside the constant table).
template <int R>
__device__ __forceinline__ cpx rft_root(cpx base, int i) {
  return cmul(base, w128((i < R / 2 ? i : 0) * (64 / R)));
}
// w_4N^k (N = 2L) at k = j + i*(L/R) from base = w_4N^j.
template <int R>
__device__ __forceinline__ cpx t23_root(cpx base, int i) {
  return cmul(base, w128(i * (16 / R)));
}
// w_4N^(L-k) from w_4N^k: w_4N^L = w_8 times the conjugate.
__device__ __forceinline__ cpx t23_mirror(cpx rk) { return cmulc(w128(16), rk); }

// Packs the pair (z_k, z_{L-k}) into the conjugated inverse-DFT inputs t_k,
// t_{L-k} of the tile (k = 0 and k = L/2 are the self-paired ends); f = w_N^k.
__device__ __forceinline__ void pack_into(const Tile& t, int c, int k, int L, cpx z0, cpx z1, cpx f) {
  if (k == 0) {
    t.s[t.idx(c, 0)] = cmk(z0.x + z1.x, -(z0.x - z1.x));
  } else if (2 * k == L) {
    t.s[t.idx(c, k)] = cmk(2 * z0.x, 2 * z0.y);
  } else {
    cpx ta, tb;
    pack_pair(z0, z1, f, ta, tb);
    t.s[t.idx(c, k)] = cconj(ta);
    t.s[t.idx(c, L - k)] = cconj(tb);
  }
}

// Tile addresses of the pairs (k, L-k), k = j + i*TPT, of thread j: element k
// is at lo + nat_off(i), element L-k at hi + nat_off(R-1-i) (thread TPT-j's
// element; for j = 0 that is thread 0's element R-i, see at()).
template <int L, int R>
struct PairSlots {
  static constexpr int TPT = L / R;
  cpx *lo, *hi;
  bool first;  // j = 0
  __device__ __forceinline__ PairSlots(const Tile& t, int c, int j) : first(j == 0) {
    cpx* s = t.s + c * t.lp;
    if constexpr (TPT >= 16) {  // offsets linear in i: thread 0's shift goes into the base
      lo = s + pad16(j);
      hi = s + (j == 0 ? nat_off<TPT>(1) : pad16(TPT - j));
    } else {
      lo = s + j;
      hi = s + (j == 0 ? 0 : TPT - j);
    }
  }
  __device__ __forceinline__ cpx& at(int i) const { return lo[nat_off<TPT>(i)]; }
  // element L-k, 0 < k (thread 0's pairs lie one element further)
  __device__ __forceinline__ cpx& mirror(int i) const {
    return hi[TPT < 16 && first ? nat_off<TPT>((R - i) % R) : nat_off<TPT>(R - 1 - i)];
  }
};

// Inverse real DFT input: spectrum X_k, k = 0..L, packed into L complex
// values, staged in shared memory.  Stored conjugated: the inverse DFT is
// computed as conj(DFT(conj(t))).  t2 = w_N^k, k < L/2.
struct LoadC2R {
  static constexpr bool kComplexIn = true;  // whether the raw input elements are complex
  static constexpr bool kStaged = true;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, cpx (&v)[R]) {
    const cpx* in = static_cast<const cpx*>(p.in) + x.oin;
    const RftRoots<L, R> rft(p.t2, x.j);
    const PairSlots<L, R> at(t, x.c, x.j);
    auto z = [&](int k) { return x.active ? in[k] : czero(); };
    pair_loop<L, R>(
        x,
        [&](int i, int k) {
          const cpx z0 = z(k);
          if (k == 0) {
            const cpx zl = z(L);
            at.at(0) = cmk(z0.x + zl.x, -(z0.x - zl.x));
          } else {
            at.at(i) = cmk(2 * z0.x, 2 * z0.y);
          }
        },
        [&](int i, int k) {
          const cpx za = z(k), zb = z(L - k), f = rft(i);
          at.at(i) = pack_one(za, zb, f);
          at.mirror(i) = pack_mirror(za, zb, f);
        },
        [] {});
    __syncthreads();
    gather_natural<L, R>(v, x.j, x.c, t);
  }
};

// Split column DFT of a 2-D real DFT with Nr = 4Q rows, inverse half.  The
// CTA's four rows j + Q*m (layout as for StoreR2CQ; input block stride is0,
// element stride in_n) receive the last radix-4 stage of the inverse column
// DFTs from row j of the four blocks V_q left by the length-Q inverse DFTs,
//   X_m = sum_q w_4^(-m*q) (w_Nr^(-j*q) V_q),
// and are packed for their inverse real DFTs as LoadC2R does.  One pass over
// the spectrum pairs (k, L-k) covers all four rows: each thread forms both
// columns of the pair for every row and packs them (one root w_N^k for all
// four).  t1 = w_Nr^n, t2 = w_N^k.
struct LoadC2RQ {
  static constexpr bool kComplexIn = true;  // whether the raw input elements are complex
  static constexpr bool kStaged = true;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, cpx (&v)[R]) {
    constexpr int NT = 4 * (L / R);  // threads of the CTA (four transforms)
    const cpx* in = static_cast<const cpx*>(p.in) + (x.oin - int64_t(x.c) * p.is0);  // row j of block 0
    const int64_t jr = umod(udiv(x.b, p.d0), p.d1);  // the CTA's row index j
    const cpx w1 = cconj(ldg(p.t1 + jr)), w2 = cconj(ldg(p.t1 + 2 * jr)), w3 = cconj(ldg(p.t1 + 3 * jr));
    const int64_t bs = p.is0;
    // column col of the four blocks -> the four rows' spectra at col
    auto gather4 = [&](int col, cpx (&X)[4]) {
      const cpx* q = in + col;
      const cpx u0 = q[0], u1 = cmul(q[bs], w1), u2 = cmul(q[2 * bs], w2), u3 = cmul(q[3 * bs], w3);
      const cpx a0 = cadd(u0, u2), a1 = csub(u0, u2), c0 = cadd(u1, u3), c1 = csub(u1, u3);
      const cpx ic1 = cmk(-c1.y, c1.x);  // i * c1
      X[0] = cadd(a0, c0);
      X[1] = cadd(a1, ic1);
      X[2] = csub(a0, c0);
      X[3] = csub(a1, ic1);
    };
#pragma unroll
    for (int it = 0; it < (L / 2 + NT) / NT; ++it) {
      const int k = threadIdx.x + it * NT;  // pair (k, L-k), k = 0 .. L/2
      if (k <= L / 2) {
        cpx Xa[4], Xb[4];
        gather4(k, Xa);
        if (2 * k != L) gather4(k == 0 ? L : L - k, Xb);  // X_L pairs with X_0
        const cpx f = (k > 0 && 2 * k < L) ? ldg(p.t2 + k) : cmk(real(1), real(0));
#pragma unroll
        for (int m = 0; m < 4; ++m) pack_into(t, m, k, L, Xa[m], Xb[m], f);
      }
    }
    __syncthreads();
    gather_natural<L, R>(v, x.j, x.c, t);
  }
};

// Type-3 input (reference minfft.c:807-817, 857-867) followed by the
// inverse-real-DFT packing, staged in shared memory (conjugated as above).
// t1 = w_4N^n (n < N/2), t2 = w_N^k (k < L/2); N = 2L.
struct LoadDCT3 {
  static constexpr bool kComplexIn = false;  // whether the raw input elements are complex
  static constexpr bool kStaged = true;
  // z_n of the type-3 pre-rotation; rd(i) returns input real x_i
  template <class Rd>
  static __device__ __forceinline__ cpx zval_r(const Rd& rd, int n, int L, bool dst, const cpx* e) {
    return zval_w(rd, n, L, dst, [&](int m) { return ldg(e + m); });
  }
  // z_n with the root w_4N^n from a function
  template <class Rd, class Rt>
  static __device__ __forceinline__ cpx zval_w(const Rd& rd, int n, int L, bool dst, const Rt& root) {
    const int N = 2 * L;
    if (n == 0) return cmk(dst ? rd(N - 1) : rd(0), real(0));
    if (n == L) {
      const real r2 = real(1.414213562373095048801688724209698079);
      return cmk(r2 * (dst ? rd(L - 1) : rd(L)), real(0));
    }
    const real a = dst ? rd(N - n - 1) : rd(n);
    const real b = dst ? rd(n - 1) : rd(N - n);
    return cconj(cmul(cmk(a, b), root(n)));
  }
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, cpx (&v)[R]) {
    const real* in = static_cast<const real*>(p.in) + x.oin;
    const bool dst = (p.flags & F_DST) != 0;
    if constexpr (L >= 2) {
      if (rows_staged_in(p) || p.colmode) {
        // the row (or column) through shared memory, its loads all issued
        // up front; every thread reads its pairs before any packed value
        // overwrites the row
        constexpr int TPT = L / R;
        const T23Roots<L, R> t23(p.t1, x.j);
        const RftRoots<L, R> rft(p.t2, x.j);
        real* sr = tile_row(t, x.c);
        if (x.active) {
          if (p.colmode)
            col_g2s<L, R>(sr, in, p.in_n, x.j, (p.flags & F_SRC_SMEM) != 0);
          else
            row_g2s<L, R>(sr, in, x.j, (p.flags & F_SRC_SMEM) != 0);
        }
        __syncthreads();
        // positions of the reals of z_k and z_(L-k): DCT-3 (k, N-k) and
        // (L-k, L+k), DST-3 (N-1-k, k-1) and (L-1+k, L-k-1), walked by i
        constexpr int N = 2 * L, NP = R / 2 + 1;
        const int sa = dst ? -TPT : TPT;
        const real* pa = sr + (dst ? N - 1 - x.j : x.j);
        const real* pb = sr + (dst ? x.j - 1 : N - x.j);
        const real* pc = sr + (dst ? L - 1 + x.j : L - x.j);
        const real* pd = sr + (dst ? L - 1 - x.j : L + x.j);
        const real r2 = real(1.414213562373095048801688724209698079);
        cpx za[NP], zb[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          const cpx rk = t23(i);  // w_4N^k
          if (i == 0 && x.j == 0) {
            za[0] = cmk(*pa, real(0));
            zb[0] = cmk(r2 * *pc, real(0));
          } else if (i < R / 2 || x.j == 0) {
            za[i] = cconj(cmul(cmk(pa[i * sa], pb[-i * sa]), rk));
            if (i < R / 2) zb[i] = cconj(cmul(cmk(pc[-i * sa], pd[i * sa]), t23_mirror(rk)));
          }
        }
        __syncthreads();
        const PairSlots<L, R> at(t, x.c, x.j);
        pair_loop<L, R>(
            x,
            [&](int i, int k) {
              at.at(i) = k == 0 ? cmk(za[0].x + zb[0].x, -(za[0].x - zb[0].x)) : cmk(2 * za[i].x, 2 * za[i].y);
            },
            [&](int i, int) {
              const cpx f = rft(i);
              at.at(i) = pack_one(za[i], zb[i], f);
              at.mirror(i) = pack_mirror(za[i], zb[i], f);
            },
            [] {});
        __syncthreads();
        gather_natural<L, R>(v, x.j, x.c, t);
        return;
      }
    }
    // the pairs (k, L-k) of pair_loop, read straight from global memory
    constexpr int TPT = L / R;
    const T23Roots<L, R> t23(p.t1, x.j);
    const RftRoots<L, R> rft(p.t2, x.j);
    auto rd = [&](int m) { return in[int64_t(m) * p.in_n]; };
#pragma unroll
    for (int i = 0; i <= R / 2; ++i) {
      const int k = x.j + i * TPT;
      if (i == R / 2 && x.j != 0) break;
      const cpx rk = t23(i);  // w_4N^k
      const cpx z0 = x.active ? zval_w(rd, k, L, dst, [&](int) { return rk; }) : czero();
      const cpx z1 = x.active ? zval_w(rd, L - k, L, dst, [&](int) { return t23_mirror(rk); }) : czero();
      pack_into(t, x.c, k, L, z0, z1, i < R / 2 ? rft(i) : czero());
    }
    __syncthreads();
    gather_natural<L, R>(v, x.j, x.c, t);
  }
};

// Type-4 pre-rotation fused into the first pass of a Stockham chain over
// HBM along a 1-D line (reference minfft.c:906-910, 953-957).  Element n of
// sub-DFT b (b1 = its index in the line, b2 = the line) is the line's
// complex point g = b1 + n*in_n: t_g = w_2N^g (x[2g] + i x[N-1-2g]) for
// DCT-4, -w_2N^g (x[2g] - i x[N-1-2g]) for DST-4, x the line's N = kn reals
// at b2 * k_in_line.  w_2N^g is the product of the coarse and fine roots
// (st_hi, st_lo, st_lobits) of 2N: the first pass has no pre-twiddle of its
// own.  The CTA holds mirror pairs of sub-DFTs (MirrorPairs below): point
// g's mirror Lt-1-g (Lt = N/2) is element L-1-n of the partner sub-DFT, and
// x[2g+1] = x[N-1-2(Lt-1-g)].  So each element reads the real pair
// (x[2g], x[2g+1]) as one vector, keeps x[2g] and hands x[2g+1] to its
// mirror element's thread through the tile: every real is read once, in
// whole sectors.
template <template <int, int> class Roots>
struct LoadT4ChainBy {
  static constexpr bool kComplexIn = false;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, cpx (&v)[R]) {
    constexpr int TPT = L / R;
    const int64_t rest = udiv(x.b, p.d0);
    const int64_t b2 = udiv(rest, p.d1), b1 = rest - b2 * p.d1;
    const real* in = static_cast<const real*>(p.in) + b2 * p.k_in_line;
    const bool dst = (p.flags & F_DST) != 0;
    const int h = p.cpb / 2;
    const int pc = x.c < h ? x.c + h : x.c - h;  // the mirror sub-DFT's slot
    real* sb = reinterpret_cast<real*>(t.s);
    const bool vec = (reinterpret_cast<uintptr_t>(in) % sizeof(cpx)) == 0;
    const real sg = dst ? real(-1) : real(1);
    real a[R];
    Walk<const real, false, TPT> w(in + 2 * (b1 * p.is1 + int64_t(x.j) * p.in_n), 2 * p.in_n);
    real* put = sb + pc * 2 * t.lp + (L - 1 - x.j);
    const real* get = sb + x.c * 2 * t.lp + x.j;
#pragma unroll
    for (int r = 0; r < R; ++r, w.step()) {
      real lo, hi;
      if (vec) {
        const cpx q = __ldcs(reinterpret_cast<const cpx*>(w.q));
        lo = q.x;
        hi = q.y;
      } else {
        lo = __ldcs(w.q);
        hi = __ldcs(w.q + 1);
      }
      a[r] = sg * lo;  // DST: -(a - ib) = -a + ib
      put[-r * TPT] = hi;
    }
    __syncthreads();
    // w_2N^g for g = g0 + r*TPT*in_n
    const Roots<R, 32> ew(p.st_hi, p.st_lo, p.st_lobits, uint32_t(b1 * p.is1 + int64_t(x.j) * p.in_n));
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = cmul(ew.at(r), cmk(a[r], get[r * TPT]));
  }
};
using LoadT4Chain = LoadT4ChainBy<RootProgression>;

// ---- type-2, type-3 and real-DFT steps fused into the passes of a 1-D chain
//
// The first and last passes of the half-length chain of a long 1-D line
// (Lt = N/2 points, N = kn reals) also do the line's pre- and
// post-processing, which otherwise are passes over memory of their own.
// Each step combines a point with its mirror, so the CTA holds mirror pairs
// of sub-DFTs (MirrorPairs below), one sub-DFT of a pair in slot c < cpb/2,
// the other in slot c + cpb/2, and hands values over through the tile:
//  * reflected pairs (points m and Lt-1-m; the type-2 permutation and the
//    type-3 de-interleave): element n of sub-DFT i with element L-1-n of
//    sub-DFT M-1-i;
//  * spectrum pairs (points m and Lt-m; the packing and unpacking of the
//    real DFT): element n of sub-DFT i with element L-1-n of sub-DFT M-i;
//    sub-DFTs 0 and M/2 pair with themselves (element n of sub-DFT 0 with
//    L-n) and share a CTA's slots.
// Bound by the same memory traffic as a plain pass: what they save is the
// two passes over memory around the chain (dct2 + dct3 of 2^22 points in
// f64: ten launches in 148 us before, six in 83 us now).

// Slot of the mirror sub-DFT, and the thread whose elements mirror this
// thread's: element j + r*TPT pairs with element jm + (R-1-r)*TPT of that
// slot (jm = TPT-1-j; TPT-j in sub-DFT 0 of spectrum pairs).  In sub-DFT 0
// thread 0 pairs its elements r and R-r among themselves: it puts element r
// where the others put r-1 (`turned`), so that it reads its partners at the
// same places; its element 0 is point 0, which every step treats apart.
struct Mirror {
  int slot, jm;
  bool turned;
};
// Reflected pairs.
template <int TPT>
__device__ __forceinline__ Mirror mirror_reflected(const AxisParams& p, const Ctx& x) {
  const int h = p.cpb / 2;
  return Mirror{x.c < h ? x.c + h : x.c - h, TPT - 1 - x.j, false};
}
// Spectrum pairs; i is the sub-DFT's index in its line.
template <int TPT>
__device__ __forceinline__ Mirror mirror_spectrum(const AxisParams& p, const Ctx& x, int64_t i) {
  const int h = p.cpb / 2;
  if (i == 0) return Mirror{x.c, x.j == 0 ? 0 : TPT - x.j, x.j == 0};
  if (2 * i == p.d0 * p.d1) return Mirror{x.c, TPT - 1 - x.j, false};
  return Mirror{x.c < h ? x.c + h : x.c - h, TPT - 1 - x.j, false};
}
// Tile address of element j of slot c; element j + r*TPT is at nat_off<TPT>(r) from it.
template <int TPT>
__device__ __forceinline__ cpx* slot_at(const Tile& t, int c, int j) {
  return t.s + c * t.lp + (TPT >= 16 ? pad16(j) : j);
}
// The thread's elements into its slot, where their mirrors' threads read
// them: element r's partner is then at slot_at(mi.slot, mi.jm) + nat_off(R-1-r).
template <int L, int R>
__device__ __forceinline__ void scatter_mirror(const cpx (&v)[R], const Ctx& x, const Mirror& mi, const Tile& t) {
  constexpr int TPT = L / R;
  cpx* q = slot_at<TPT>(t, x.c, x.j);
  if (mi.turned) {
#pragma unroll
    for (int r = 0; r < R; ++r) q[nat_off<TPT>((r + R - 1) % R)] = v[r];
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) q[nat_off<TPT>(r)] = v[r];
  }
}

// Four consecutive reals, as 16-byte vectors where `vec`.
struct Real4 {
  real v[4];
};
__device__ __forceinline__ Real4 ld_real4(const real* q, bool vec) {
  Real4 r;
  if (vec) {
#if MINFFT_SINGLE
    const float4 a = __ldcs(reinterpret_cast<const float4*>(q));
    r.v[0] = a.x, r.v[1] = a.y, r.v[2] = a.z, r.v[3] = a.w;
#else
    const double2 a = __ldcs(reinterpret_cast<const double2*>(q)), b = __ldcs(reinterpret_cast<const double2*>(q) + 1);
    r.v[0] = a.x, r.v[1] = a.y, r.v[2] = b.x, r.v[3] = b.y;
#endif
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) r.v[i] = __ldcs(q + i);
  }
  return r;
}
__device__ __forceinline__ void st_real4(real* q, const Real4& r, bool vec) {
  if (vec) {
#if MINFFT_SINGLE
    __stcs(reinterpret_cast<float4*>(q), make_float4(r.v[0], r.v[1], r.v[2], r.v[3]));
#else
    __stcs(reinterpret_cast<double2*>(q), make_double2(r.v[0], r.v[1]));
    __stcs(reinterpret_cast<double2*>(q) + 1, make_double2(r.v[2], r.v[3]));
#endif
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) __stcs(q + i, r.v[i]);
  }
}

// Line and sub-DFT index of a first pass's transform, and the line's input.
struct ChainIn {
  const real* in;
  int64_t i;
};
__device__ __forceinline__ ChainIn chain_in(const AxisParams& p, const Ctx& x) {
  const int64_t rest = udiv(x.b, p.d0);
  const int64_t line = udiv(rest, p.d1);
  return ChainIn{static_cast<const real*>(p.in) + line * p.k_in_line, rest - line * p.d1};
}

// Type-2 permutation (reference minfft.c:707-710, 756-759; LoadDCT2) of
// point g = i + n*in_n: (x[4g], x[4g+2]) for g < Lt/2 (n < L/2), and for its
// mirror Lt-1-g the pair (x[4g+3], x[4g+1]), negated for DST-2: one vector of
// four reals gives both points.
struct LoadDCT2Line {
  static constexpr bool kComplexIn = false;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, cpx (&v)[R]) {
    constexpr int TPT = L / R;
    const ChainIn ci = chain_in(p, x);
    const real sg = (p.flags & F_DST) ? real(-1) : real(1);
    const Mirror mi = mirror_reflected<TPT>(p, x);
    const bool vec = (reinterpret_cast<uintptr_t>(ci.in) & 15) == 0;
    Walk<const real, false, TPT> w(ci.in + 4 * (ci.i + int64_t(x.j) * p.in_n), 4 * p.in_n);
    Real4 q[R / 2];
#pragma unroll
    for (int r = 0; r < R / 2; ++r, w.step()) q[r] = ld_real4(w.q, vec);
    cpx* put = slot_at<TPT>(t, mi.slot, mi.jm);
    const cpx* get = slot_at<TPT>(t, x.c, x.j);
#pragma unroll
    for (int r = 0; r < R / 2; ++r) {
      v[r] = cmk(q[r].v[0], q[r].v[2]);
      put[nat_off<TPT>(R - 1 - r)] = cmk(sg * q[r].v[3], sg * q[r].v[1]);
    }
    __syncthreads();
#pragma unroll
    for (int r = R / 2; r < R; ++r) v[r] = get[nat_off<TPT>(r)];
  }
};

// Packs the tile's spectrum values z (point g of the thread's element r in
// v[r], k0 the value of t_0) into the conjugated inverse-DFT inputs; fw are
// the roots w_N^g.
template <int L, int R>
__device__ __forceinline__ void pack_tile(const Ctx& x, const Tile& t, const Mirror& mi, bool zero, cpx k0,
                                          const RootSteps<R, 64>& fw, cpx (&v)[R]) {
  constexpr int TPT = L / R;
  scatter_mirror<L, R>(v, x, mi, t);
  __syncthreads();
  const cpx* zm = slot_at<TPT>(t, mi.slot, mi.jm);
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = pack_one(v[r], zm[nat_off<TPT>(R - 1 - r)], fw.at(r));
  if (zero) v[0] = k0;
}

// Type-3 pre-rotation (reference minfft.c:807-817, 857-867; LoadDCT3) and
// packing of point g: z_g = conj((x[g] + i x[N-g]) w_4N^g), DST-3 with
// x[N-1-g] and x[g-1].  Roots of 4N (st_hi, st_lo): w_4N^g and w_N^g.
struct LoadDCT3Line {
  static constexpr bool kComplexIn = false;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, cpx (&v)[R]) {
    constexpr int TPT = L / R;
    const ChainIn ci = chain_in(p, x);
    const bool dst = (p.flags & F_DST) != 0;
    const int64_t N = p.kn;
    const Mirror mi = mirror_spectrum<TPT>(p, x, ci.i);
    const bool zero = mi.turned;  // element 0 is point 0: x_0 and x_Lt
    const int64_t g0 = ci.i + int64_t(x.j) * p.in_n;
    const int64_t sa = dst ? -p.in_n : p.in_n;
    Walk<const real, false, TPT> wa(dst ? ci.in + (N - 1 - g0) : ci.in + g0, sa);
    Walk<const real, false, -TPT> wb(dst ? ci.in + (g0 - 1) : ci.in + (N - g0), sa);
#pragma unroll
    for (int r = 0; r < R; ++r, wa.step(), wb.step()) {
      const real* b = wb.q;
      if (r == 0 && zero) b = ci.in + (dst ? N / 2 - 1 : N / 2);
      v[r] = cmk(__ldcs(wa.q), __ldcs(b));
    }
    const real r2 = real(1.414213562373095048801688724209698079);
    const cpx k0 = cmk(v[0].x + r2 * v[0].y, -(v[0].x - r2 * v[0].y));
    {
      const RootSteps<R, 16> ew(p.st_hi, p.st_lo, p.st_lobits, uint32_t(g0));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const cpx e = ew.at(r);
        v[r] = cmk(v[r].x * e.x - v[r].y * e.y, -(v[r].x * e.y) - v[r].y * e.x);
      }
    }
    const RootSteps<R, 64> fw(p.st_hi, p.st_lo, p.st_lobits, uint32_t(4 * g0));
    pack_tile<L, R>(x, t, mi, zero, k0, fw, v);
  }
};

// Packing of the inverse real DFT (reference minfft.c:628-656; LoadC2R) of
// point g: the line's N/2 + 1 complex values at line * k_in_line (complex
// units).  Roots of N (st_hi, st_lo).
struct LoadC2RLine {
  static constexpr bool kComplexIn = true;  // whether the raw input elements are complex
  static constexpr bool kStaged = false;
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, cpx (&v)[R]) {
    constexpr int TPT = L / R;
    const int64_t rest = udiv(x.b, p.d0), line = udiv(rest, p.d1), i = rest - line * p.d1;
    const cpx* in = static_cast<const cpx*>(p.in) + line * p.k_in_line;
    const Mirror mi = mirror_spectrum<TPT>(p, x, i);
    const bool zero = mi.turned;
    const int64_t g0 = i + int64_t(x.j) * p.in_n;
    Walk<const cpx, false, TPT> w(in + g0, p.in_n);
#pragma unroll
    for (int r = 0; r < R; ++r, w.step()) v[r] = __ldcs(w.q);
    cpx k0 = czero();
    if (zero) {
      const cpx zl = in[p.kn / 2];
      k0 = cmk(v[0].x + zl.x, -(v[0].x - zl.x));
    }
    const RootSteps<R, 64> fw(p.st_hi, p.st_lo, p.st_lobits, uint32_t(g0));
    pack_tile<L, R>(x, t, mi, zero, k0, fw, v);
  }
};

// --------------------------------------------------------------- store ops
// Each store op receives output element k = j + r*(L/R) of the length-L DFT
// in v[r].

// Offsets of the CTA's transforms, kept in shared memory so staged stores
// can address any transform of the tile.
struct TileOffsets {
  int64_t* in_off;
  int64_t* out_off;
  int nvalid;  // transforms of the tile that exist (the rest are padding)
};

struct StoreCplx {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets& to,
                                             cpx (&v)[R]) {
    cpx* out = static_cast<cpx*>(p.out);
    const bool cj = (p.flags & F_CONJ_OUT) != 0;
    if (!(p.flags & F_STAGE_ROWS)) {
      if (!x.active) return;
      constexpr int TPT = L / R;
      if (cj) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r].y = -v[r].y;
      }
      if (p.out_k == 1) {
        cpx* q = out + x.oout + x.j;
#pragma unroll
        for (int r = 0; r < R; ++r) q[r * TPT] = v[r];
      } else {
        Walk<cpx, false, TPT> w(out + x.oout + x.j * p.out_k, p.out_k);
#pragma unroll
        for (int r = 0; r < R; ++r, w.step()) *w.q = v[r];
      }
      return;
    }
    // staged: each transform's L outputs written with k running fastest
    __syncthreads();
    scatter_natural<L, R>(v, x.j, x.c, t);
    __syncthreads();
    if ((blockDim.x & (L - 1)) == 0 && p.out_k == 1) {
      // whole transforms per sweep of the CTA: a thread keeps its output k
      const int k = threadIdx.x & (L - 1), step = int(blockDim.x) / L;
      int c = threadIdx.x / L;
      const cpx* q = t.s + t.idx(c, k);
      cpx* o = out + k;
      for (; c < to.nvalid; c += step, q += step * t.lp) {
        cpx w = *q;
        if (cj) w.y = -w.y;
        o[to.out_off[c]] = w;
      }
      return;
    }
    const int total = to.nvalid * L;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const int c = e / L, k = e - c * L;
      cpx o = t.s[t.idx(c, k)];
      if (cj) o.y = -o.y;
      out[to.out_off[c] + int64_t(k) * p.out_k] = o;
    }
  }
};

// Real DFT output (reference minfft.c:547-578): L+1 complex values from the
// half-length DFT, via the pair unpacking; t1 = w_N^k, k < L/2.
struct StoreR2C {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets&,
                                             cpx (&v)[R]) {
    __syncthreads();
    scatter_natural<L, R>(v, x.j, x.c, t);
    __syncthreads();
    if (!x.active) return;
    cpx* out = static_cast<cpx*>(p.out) + x.oout;
    const RftRoots<L, R> rft(p.t1, x.j);
    const PairSlots<L, R> at(t, x.c, x.j);
    pair_loop<L, R>(
        x,
        [&](int i, int k) {
          const cpx za = at.at(i);
          if (k == 0) {
            out[0] = cmk(za.x + za.y, real(0));
            out[L] = cmk(za.x - za.y, real(0));
          } else {
            out[k] = cconj(za);
          }
        },
        [&](int i, int k) {
          const cpx za = at.at(i), zb = at.mirror(i), f = rft(i);
          out[k] = cscale(unpack_one2(za, zb, f), real(0.5));
          out[L - k] = cscale(unpack_mirror2(za, zb, f), real(0.5));
        },
        [] {});
  }
};

// Type-2 output (reference minfft.c:714-725, 763-774): real-DFT unpacking,
// then y_n = 2 Re(V_n e_n), y_{N-n} = -2 Im(V_n e_n) (DCT-2; DST-2 maps the
// same values to reversed positions).  t1 = w_4N^n (n < N/2), t2 = w_N^k.
struct StoreDCT2 {
  static __device__ __forceinline__ void emit(real* out, int64_t s, int n, int N, bool dst, cpx V, cpx e) {
    const cpx q = cmul(V, e);
    if (!dst) {
      out[int64_t(n) * s] = 2 * q.x;
      out[int64_t(N - n) * s] = -2 * q.y;
    } else {
      out[int64_t(n - 1) * s] = -2 * q.y;
      out[int64_t(N - n - 1) * s] = 2 * q.x;
    }
  }
  // emit() for V2 = 2V (from unpack_pair2)
  static __device__ __forceinline__ void emit2(real* out, int64_t s, int n, int N, bool dst, cpx V2, cpx e) {
    const cpx q = cmul(V2, e);
    if (!dst) {
      out[int64_t(n) * s] = q.x;
      out[int64_t(N - n) * s] = -q.y;
    } else {
      out[int64_t(n - 1) * s] = -q.y;
      out[int64_t(N - n - 1) * s] = q.x;
    }
  }
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets&,
                                             cpx (&v)[R]) {
    __syncthreads();
    scatter_natural<L, R>(v, x.j, x.c, t);
    __syncthreads();
    if (!x.active) return;
    real* out = static_cast<real*>(p.out) + x.oout;
    if (p.out_k == 1)
      rotate<true, L, R>(p, out, 1, x, t);
    else
      rotate<false, L, R>(p, out, p.out_k, x, t);
  }
  // The four outputs of the pair (k, L-k), k = j + i*TPT: positions k, N-k,
  // L-k and L+k (one less for DST-2, which swaps each two of one value).
  template <bool kUnit, int L, int R>
  static __device__ __forceinline__ void rotate(const AxisParams& p, real* out, int64_t s, const Ctx& x,
                                                const Tile& t) {
    constexpr int N = 2 * L, TPT = L / R;
    const bool dst = (p.flags & F_DST) != 0;
    if (dst) out -= s;
    const real r2 = real(1.414213562373095048801688724209698079);
    const T23Roots<L, R> t23(p.t1, x.j);
    const RftRoots<L, R> rft(p.t2, x.j);
    Walk<real, kUnit, TPT> lo(out + int64_t(x.j) * s, s), up(out + int64_t(L + x.j) * s, s);
    Walk<real, kUnit, -TPT> hi(out + int64_t(N - x.j) * s, s), dn(out + int64_t(L - x.j) * s, s);
    auto put = [&](real* a, real* b, cpx q) {  // y_n = Re, y_(N-n) = -Im
      *a = dst ? -q.y : q.x;
      *b = dst ? q.x : -q.y;
    };
    const PairSlots<L, R> at(t, x.c, x.j);
    pair_loop<L, R>(
        x,
        [&](int i, int k) {
          const cpx za = at.at(i);
          if (k == 0) {
            const real v0 = za.x + za.y, vl = za.x - za.y;
            *(dst ? hi.q : lo.q) = 2 * v0;
            *up.q = r2 * vl;
          } else {
            const cpx q = cmul(cconj(za), w128(8));  // w_4N^(L/2) = w_16
            put(lo.q, hi.q, cmk(2 * q.x, 2 * q.y));
          }
        },
        [&](int i, int) {
          const cpx za = at.at(i), zb = at.mirror(i), f = rft(i), e = t23(i);
          put(lo.q, hi.q, cmul(unpack_one2(za, zb, f), e));
          put(dn.q, up.q, cmul(unpack_mirror2(za, zb, f), t23_mirror(e)));
        },
        [&] { lo.step(), up.step(), hi.step(), dn.step(); });
  }
};

// Split column DFT of a 2-D real DFT with Nr = 4Q rows, forward half.  The
// CTA holds the four rows j + Q*m (transform c = m: batch layout d0 = 4 with
// is0 = Q rows, d1 = Q with is1 = one row, cpb = 4).  After their half-length
// DFTs it applies, column by column, the first radix-4 stage of the length-Nr
// column DFTs across the four rows' spectra X_m,
//   Z_q[j] = w_Nr^(j*q) * sum_m X_m w_4^(m*q),
// and writes Z_q to row j of block q of the output (block stride os0, element
// stride out_k); length-Q DFTs of each block then finish the column DFTs
// (their output p is row q + 4p).  One pass over the spectrum pairs (k, L-k)
// covers all four rows: each thread unpacks the pair for every row (one root
// w_N^k for all four) and stores both columns.  t1 = w_N^k (real-DFT table),
// t2 = w_Nr^n.
struct StoreR2CQ {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets& to,
                                             cpx (&v)[R]) {
    constexpr int NT = 4 * (L / R);  // threads of the CTA (four transforms)
    __syncthreads();
    scatter_natural<L, R>(v, x.j, x.c, t);
    __syncthreads();
    const int64_t jr = umod(udiv(x.b, p.d0), p.d1);  // the CTA's row index j
    const cpx w1 = ldg(p.t2 + jr), w2 = ldg(p.t2 + 2 * jr), w3 = ldg(p.t2 + 3 * jr);
    cpx* out = static_cast<cpx*>(p.out) + to.out_off[0];  // row j of block 0
    const int64_t bs = p.os0;
    // column col of the four rows -> blocks 0..3
    auto emit = [&](int col, const cpx (&X)[4]) {
      const cpx a0 = cadd(X[0], X[2]), a1 = csub(X[0], X[2]), c0 = cadd(X[1], X[3]), c1 = csub(X[1], X[3]);
      const cpx mic1 = cmk(c1.y, -c1.x);  // -i * c1
      cpx* q = out + col;
      q[0] = cadd(a0, c0);
      q[bs] = cmul(cadd(a1, mic1), w1);
      q[2 * bs] = cmul(csub(a0, c0), w2);
      q[3 * bs] = cmul(csub(a1, mic1), w3);
    };
#pragma unroll
    for (int it = 0; it < (L / 2 + NT) / NT; ++it) {
      const int k = threadIdx.x + it * NT;  // pair (k, L-k), k = 0 .. L/2
      if (k <= L / 2) {
        cpx Xa[4], Xb[4];
        if (k == 0) {
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const cpx z = t.s[t.idx(m, 0)];
            Xa[m] = cmk(z.x + z.y, real(0));
            Xb[m] = cmk(z.x - z.y, real(0));  // X_L
          }
          emit(0, Xa);
          emit(L, Xb);
        } else if (2 * k == L) {
#pragma unroll
          for (int m = 0; m < 4; ++m) Xa[m] = cconj(t.s[t.idx(m, k)]);
          emit(k, Xa);
        } else {
          const cpx f = ldg(p.t1 + k);
#pragma unroll
          for (int m = 0; m < 4; ++m) unpack_pair(t.s[t.idx(m, k)], t.s[t.idx(m, L - k)], f, Xa[m], Xb[m]);
          emit(k, Xa);
          emit(L - k, Xb);
        }
      }
    }
  }
};

// Inverse real DFT output: the inverse half-length DFT (conjugate of the
// forward result) read as interleaved reals (reference minfft.c:605,658).
struct StoreC2R {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile&, const TileOffsets&,
                                             cpx (&v)[R]) {
    if (!x.active) return;
    constexpr int TPT = L / R;
    real* out = static_cast<real*>(p.out) + x.oout;
    if (p.flags & F_VEC) {
      cpx* q = reinterpret_cast<cpx*>(out) + x.j;
#pragma unroll
      for (int r = 0; r < R; ++r) q[r * TPT] = cconj(v[r]);
    } else {
      real* q = out + 2 * x.j;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        q[2 * r * TPT] = v[r].x;
        q[2 * r * TPT + 1] = -v[r].y;
      }
    }
  }
};

// Type-3 output (reference minfft.c:821-824, 871-874): the inverse real
// DFT's reals t_i go to y[2i] (i < N/2) and y[2N-1-2i] (i >= N/2, negated
// for DST-3).
struct StoreDCT3 {
  // reals t_2m, t_2m+1 (m = j + r*TPT) go to y[4m], y[4m+2] while r < R/2,
  // else to y[2N-1-4m], y[2N-3-4m] (negated for DST-3)
  template <bool kUnit, int L, int R>
  static __device__ __forceinline__ void spread(real* out, int64_t s, int j, bool dst, const cpx (&v)[R]) {
    constexpr int N = 2 * L, TPT = L / R, m0 = (R / 2) * TPT;
    const real sg = dst ? real(-1) : real(1);
    Walk<real, kUnit, 4 * TPT> a(out + int64_t(4 * j) * s, s), b(out + int64_t(4 * j + 2) * s, s);
#pragma unroll
    for (int r = 0; r < R / 2; ++r, a.step(), b.step()) {
      *a.q = v[r].x;
      *b.q = -v[r].y;
    }
    Walk<real, kUnit, -4 * TPT> c(out + int64_t(2 * N - 1 - 4 * (j + m0)) * s, s),
        d(out + int64_t(2 * N - 3 - 4 * (j + m0)) * s, s);
#pragma unroll
    for (int r = R / 2; r < R; ++r, c.step(), d.step()) {
      *c.q = sg * v[r].x;
      *d.q = sg * -v[r].y;
    }
  }
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets&,
                                             cpx (&v)[R]) {
    real* out = static_cast<real*>(p.out) + x.oout;
    real* gout = out;
    int64_t s = p.out_k;
    bool staged = false;
    if constexpr (L >= 2) {
      if (rows_staged_out(p)) {  // the outputs into the row's shared-memory slot, then the row out whole
        __syncthreads();
        out = tile_row(t, x.c);
        s = 1;
        staged = true;
      }
    }
    const bool dst = (p.flags & F_DST) != 0;
    if constexpr (L >= 2) {
      if (x.active) {
        if (s == 1)
          spread<true, L, R>(out, 1, x.j, dst, v);
        else
          spread<false, L, R>(out, s, x.j, dst, v);
      }
      if (staged) {
        __syncthreads();
        if (x.active) row_s2g<L, R>(gout, out, x.j);
      }
    } else {  // L = 1: y0 = t0, y1 = +-t1
      if (!x.active) return;
      const cpx w = cconj(v[0]);
      out[0] = w.x;
      out[p.out_k] = dst ? -w.y : w.y;
    }
  }
};

// Type-4 post-rotation (reference minfft.c:916-921, 963-968): T_m feeds
// y[2m] = 2 Re(g_2m T_m) and y[N-1-2m] = 2 Re(g_{N-1-2m} conj(T_m)) (Im for
// DST-4), g_q = w_8N^(2q+1) from table t2.
struct StoreT4 {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile&, const TileOffsets&,
                                             cpx (&v)[R]) {
    if (!x.active) return;
    real* out = static_cast<real*>(p.out) + x.oout;
    const bool dst = (p.flags & F_DST) != 0;
    if (p.out_k == 1)
      rotate<true, L, R>(p, out, 1, x.j, dst, v);
    else
      rotate<false, L, R>(p, out, p.out_k, x.j, dst, v);
  }
  template <bool kUnit, int L, int R>
  static __device__ __forceinline__ void rotate(const AxisParams& p, real* out, int64_t s, int j, bool dst,
                                                cpx (&v)[R]) {
    constexpr int N = 2 * L, TPT = L / R;
    Walk<real, kUnit, 2 * TPT> lo(out + int64_t(2 * j) * s, s);
    Walk<real, kUnit, -2 * TPT> hi(out + int64_t(N - 1 - 2 * j) * s, s);
    // t2[q] = w_8N^(2q+1): g_2m = t2[2j] * w_4R^r for m = j + r*TPT, and
    // g_{N-1-2m} = -i conj(g_2m), so that one product A = g_2m T_m gives both
    // outputs: 2 Re(g_{N-1-2m} conj(T_m)) = -2 Im A (Im: -2 Re A)
    const cpx g = cscale(ldg(p.t2 + 2 * j), real(2));
#pragma unroll
    for (int r = 0; r < R; ++r, lo.step(), hi.step()) {
      const cpx gr = kTablesNear && R == 8 && L > R ? cscale(ldg(p.t2 + 2 * (j + r * TPT)), real(2))
                                                    : cmul(g, w128(r * (32 / R)));
      const cpx A = cmul(gr, v[r]);
      *lo.q = dst ? A.y : A.x;
      *hi.q = dst ? -A.x : -A.y;
    }
  }
};

// Type-4 post-rotation fused into the last pass of a Stockham chain over
// HBM along a 1-D line (reference minfft.c:916-921, 963-968): output k of
// sub-DFT b is the line's point m = (its normal offset) + k*out_k, and
// T_m gives y[2m] = 2 Re(g_2m T_m), y[N-1-2m] = 2 Re(g_{N-1-2m} conj(T_m))
// (Im for DST-4), g_q = w_8N^(2q+1) as the product of the coarse and fine
// roots t1, t2 of 8N (kbits fine bits), and g_{N-1-2m} = -i conj(g_2m); y is
// the line's N reals at b2 * k_out_line (the pass's os2 is 0).  As in
// LoadT4Chain the CTA holds mirror pairs of sub-DFTs: y[2m+1] is
// y[N-1-2m'] of the mirror point m' = Lt-1-m (output L-1-k of the partner
// sub-DFT), so each element hands that value to its mirror's thread through
// the tile and writes the pair (y[2m], y[2m+1]) as one vector.
template <template <int, int> class Roots>
struct StoreT4ChainBy {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets&,
                                             cpx (&v)[R]) {
    constexpr int TPT = L / R;
    const int64_t b2 = udiv(x.b, p.d0 * p.d1);
    real* out = static_cast<real*>(p.out) + b2 * p.k_out_line;
    const bool dst = (p.flags & F_DST) != 0;
    const int h = p.cpb / 2;
    const int pc = x.c < h ? x.c + h : x.c - h;  // the mirror sub-DFT's slot
    real* sb = reinterpret_cast<real*>(t.s);
    const bool vec = (reinterpret_cast<uintptr_t>(out) % sizeof(cpx)) == 0;
    // g_2m = w_8N^(4m+1) for m = m0 + r*TPT*out_k
    const Roots<R, 32> gw(p.t1, p.t2, p.kbits, uint32_t(4 * (x.oout + int64_t(x.j) * p.out_k) + 1));
    __syncthreads();  // the last Stockham exchange has finished with the tile
    // a slot holds 2*lp >= 2L reals: the mirror's values below L, its own above
    real* own = sb + x.c * 2 * t.lp + x.j;
    real* put = sb + pc * 2 * t.lp + (L - 1 - x.j);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      // with g_{N-1-2m} = -i conj(g_2m), A = g_2m T_m gives both outputs (StoreT4)
      const cpx A = cmul(gw.at(r), v[r]);
      own[L + r * TPT] = 2 * (dst ? A.y : A.x);
      put[-r * TPT] = -2 * (dst ? A.x : A.y);
    }
    __syncthreads();
    Walk<real, false, TPT> w(out + 2 * (x.oout + int64_t(x.j) * p.out_k), 2 * p.out_k);
#pragma unroll
    for (int r = 0; r < R; ++r, w.step()) {
      const real a = own[L + r * TPT], b = own[r * TPT];
      if (vec) {
        __stcs(reinterpret_cast<cpx*>(w.q), cmk(a, b));
      } else {
        __stcs(w.q, a);
        __stcs(w.q + 1, b);
      }
    }
  }
};
using StoreT4Chain = StoreT4ChainBy<RootProgression>;

// Unpacking of the real DFT (reference minfft.c:547-578; StoreR2C) of output
// point m: X_m, and at m = 0 also X_Lt.  Roots of N (t1, t2, kbits); the
// line's N/2 + 1 complex outputs at line * k_out_line (complex units; the
// pass's os2 is 0, so a transform's output offset is its index in the line).
struct StoreR2CLine {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets&,
                                             cpx (&v)[R]) {
    constexpr int TPT = L / R;
    cpx* out = static_cast<cpx*>(p.out) + udiv(x.b, p.d0 * p.d1) * p.k_out_line;
    const Mirror mi = mirror_spectrum<TPT>(p, x, x.oout);
    const int64_t m0 = x.oout + int64_t(x.j) * p.out_k;
    const RootSteps<R, 64> fw(p.t1, p.t2, p.kbits, uint32_t(m0));
    __syncthreads();  // the last Stockham exchange has finished with the tile
    scatter_mirror<L, R>(v, x, mi, t);
    __syncthreads();
    const cpx* zm = slot_at<TPT>(t, mi.slot, mi.jm);
    Walk<cpx, false, TPT> w(out + m0, p.out_k);
#pragma unroll
    for (int r = 0; r < R; ++r, w.step()) {
      cpx X = cscale(unpack_one2(v[r], zm[nat_off<TPT>(R - 1 - r)], fw.at(r)), real(0.5));
      if (r == 0 && mi.turned) {
        X = cmk(v[0].x + v[0].y, real(0));
        out[p.kn / 2] = cmk(v[0].x - v[0].y, real(0));
      }
      *w.q = X;
    }
  }
};

// Type-2 output (reference minfft.c:714-725, 763-774; StoreDCT2) of output
// point m: y_m = Re(2 V_m e_m) and y_(N-m) = -Im(2 V_m e_m), V_m the real
// DFT's value and e_m = w_4N^m; DST-2 writes the same values to reversed
// positions; at m = 0 y_0 and y_Lt.  Roots of 4N (t1, t2, kbits) for e_m and
// w_N^m; the line's N reals at line * k_out_line.
struct StoreDCT2Line {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets&,
                                             cpx (&v)[R]) {
    constexpr int TPT = L / R;
    real* out = static_cast<real*>(p.out) + udiv(x.b, p.d0 * p.d1) * p.k_out_line;
    const bool dst = (p.flags & F_DST) != 0;
    const int64_t N = p.kn;
    const Mirror mi = mirror_spectrum<TPT>(p, x, x.oout);
    const int64_t m0 = x.oout + int64_t(x.j) * p.out_k;
    __syncthreads();  // the last Stockham exchange has finished with the tile
    scatter_mirror<L, R>(v, x, mi, t);
    __syncthreads();
    const real r2 = real(1.414213562373095048801688724209698079);
    const real y0 = 2 * (v[0].x + v[0].y), yl = r2 * (v[0].x - v[0].y);
    const cpx* zm = slot_at<TPT>(t, mi.slot, mi.jm);
    {
      const RootSteps<R, 64> fw(p.t1, p.t2, p.kbits, uint32_t(4 * m0));
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = unpack_one2(v[r], zm[nat_off<TPT>(R - 1 - r)], fw.at(r));
    }
    const RootSteps<R, 16> ew(p.t1, p.t2, p.kbits, uint32_t(m0));
    const int64_t sa = dst ? -p.out_k : p.out_k;
    Walk<real, false, TPT> wa(dst ? out + (N - 1 - m0) : out + m0, sa);
    Walk<real, false, -TPT> wb(dst ? out + (m0 - 1) : out + (N - m0), sa);
#pragma unroll
    for (int r = 0; r < R; ++r, wa.step(), wb.step()) {
      const cpx e = ew.at(r);
      real a = v[r].x * e.x - v[r].y * e.y, b = -(v[r].x * e.y) - v[r].y * e.x;
      real* pb = wb.q;
      if (r == 0 && mi.turned) {
        a = y0;
        b = yl;
        pb = out + (dst ? N / 2 - 1 : N / 2);
      }
      *wa.q = a;
      *pb = b;
    }
  }
};

// Type-3 de-interleave (reference minfft.c:821-824, 871-874; StoreDCT3) of
// output point m: (t_2m, t_2m+1) go to y[4m], y[4m+2] for m < Lt/2 (k < L/2)
// and, for its mirror Lt-1-m, to y[4m+3], y[4m+1] (negated for DST-3): the
// element of the lower half writes the four reals as one vector.
struct StoreDCT3Line {
  template <int L, int R>
  static __device__ __forceinline__ void run(const AxisParams& p, const Ctx& x, const Tile& t, const TileOffsets&,
                                             cpx (&v)[R]) {
    constexpr int TPT = L / R;
    real* out = static_cast<real*>(p.out) + udiv(x.b, p.d0 * p.d1) * p.k_out_line;
    const real sg = (p.flags & F_DST) ? real(-1) : real(1);
    const Mirror mi = mirror_reflected<TPT>(p, x);
    const bool vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    cpx* put = slot_at<TPT>(t, mi.slot, mi.jm);
    const cpx* get = slot_at<TPT>(t, x.c, x.j);
    __syncthreads();  // the last Stockham exchange has finished with the tile
#pragma unroll
    for (int r = R / 2; r < R; ++r) put[nat_off<TPT>(R - 1 - r)] = v[r];
    __syncthreads();
    Walk<real, false, TPT> w(out + 4 * (x.oout + int64_t(x.j) * p.out_k), 4 * p.out_k);
#pragma unroll
    for (int r = 0; r < R / 2; ++r, w.step()) {
      const cpx u = get[nat_off<TPT>(r)];  // conjugated, as v is
      st_real4(w.q, Real4{{v[r].x, -sg * u.y, -v[r].y, sg * u.x}}, vec);
    }
  }
};

// The fused passes of a 1-D real chain take mirror pairs of sub-DFTs into one
// CTA: with M = d0*d1 sub-DFTs per line, slots c < cpb/2 hold sub-DFTs i of
// the line and slots c + cpb/2 their mirrors, M-1-i for reflected pairs (and
// the type-4 steps), M-i for spectrum pairs, where sub-DFT M/2 sits in the
// mirror slot of sub-DFT 0 (the planner makes cpb even and a divisor of M).
enum MirrorKind : int { kNoMirror = 0, kReflected, kSpectrum };
template <class Op>
struct MirrorPairs {
  static constexpr MirrorKind value = kNoMirror;
};
#define MB_MIRROR(Op, kind)                    \
  template <>                                  \
  struct MirrorPairs<Op> {                     \
    static constexpr MirrorKind value = kind;  \
  }
template <template <int, int> class Roots>
struct MirrorPairs<LoadT4ChainBy<Roots>> {
  static constexpr MirrorKind value = kReflected;
};
template <template <int, int> class Roots>
struct MirrorPairs<StoreT4ChainBy<Roots>> {
  static constexpr MirrorKind value = kReflected;
};
MB_MIRROR(LoadDCT2Line, kReflected);
MB_MIRROR(StoreDCT3Line, kReflected);
MB_MIRROR(LoadDCT3Line, kSpectrum);
MB_MIRROR(LoadC2RLine, kSpectrum);
MB_MIRROR(StoreR2CLine, kSpectrum);
MB_MIRROR(StoreDCT2Line, kSpectrum);
#undef MB_MIRROR

// Batch index of the transform in slot c of a tile (one CTA per tile).
template <MirrorKind kMirror>
__device__ __forceinline__ int64_t tile_batch(const AxisParams& p, int c, int64_t tile) {
  if constexpr (kMirror != kNoMirror) {
    const int64_t M = p.d0 * p.d1;
    const int64_t per_line = udiv(M, p.cpb);  // CTAs per line
    const int64_t line = udiv(tile, per_line), q = tile - line * per_line;
    const int h = p.cpb / 2;
    const int64_t i = q * h + (c < h ? c : c - h);
    if (c < h) return line * M + i;
    if constexpr (kMirror == kReflected) return line * M + (M - 1 - i);
    return line * M + (i == 0 ? M / 2 : M - i);
  } else {
    return tile * p.cpb + c;
  }
}

// ------------------------------------------------------------------ kernel
// Register budget per thread: a radix-R thread holds R complex values; with
// 512-thread CTAs, 16 doubles-complex get 128 registers (1 CTA per SM), and
// every halving of the state doubles the CTAs the budget allows.
template <int R>
struct MinBlocks {
  // double: 128 registers at radix 16, 64 at radix 8 (and below);
  // single: 64 at radix 16, 40 at radix 8, 64 below
  static constexpr int value = sizeof(real) == 8 ? (R >= 16 ? 1 : 2) : (R >= 16 ? 2 : R == 8 ? 3 : 2);
};

// Complex columns of 4096 points in single, of which a CTA holds two: passes
// whose sums are scalar instructions.  Packed sums, ahead everywhere else (8000
// rows of 4096 points 198 us a pair, 213 scalar), cost them up to 5% on arrays
// beyond the L2 -- column passes of the real DFT of 16384 x 2048 166 us scalar, 175
// packed, of 4096 x 16384 368 and 387 -- in as many registers and without spills.
struct LoadCplxScalar : LoadCplx {};

// Load stages that take no shared memory at all: the exchange tile is as the
// CTA's last barrier left it.
template <class Op>
struct KeepsTile {
  static constexpr bool value = std::is_base_of<LoadCplx, Op>::value || std::is_same<Op, LoadR2C>::value ||
                                std::is_same<Op, LoadDCT2>::value || std::is_same<Op, LoadT4>::value;
};

template <int L, int R, class LoadOp, class StoreOp>
__global__ void __launch_bounds__(512, MinBlocks<R>::value) axis_pass_kernel(const AxisParams p) {
  static_assert(R <= L || L < 2, "radix at most the length");
  constexpr int TPT = L / R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int64_t* offs = reinterpret_cast<int64_t*>(smem_raw);
  const int64_t left = p.nbatch - int64_t(blockIdx.x) * p.cpb;
  TileOffsets to{offs, offs + p.cpb, int(left < p.cpb ? left : p.cpb)};
  Tile t{reinterpret_cast<cpx*>(smem_raw + 16 * ((2 * p.cpb * sizeof(int64_t) + 15) / 16)), p.lp};

  constexpr MirrorKind kMirror =
      MirrorPairs<LoadOp>::value != kNoMirror ? MirrorPairs<LoadOp>::value : MirrorPairs<StoreOp>::value;
  // offsets of the CTA's transforms, computed once per transform
  for (int c = threadIdx.x; c < p.cpb; c += blockDim.x) {
    const int64_t b = tile_batch<kMirror>(p, c, blockIdx.x);
    int64_t b0, oi, oo;
    batch_offsets(p, b < p.nbatch ? b : 0, b0, oi, oo);
    to.in_off[c] = oi;
    to.out_off[c] = oo;
  }
  __syncthreads();

  Ctx x;
  if (p.colmode) {
    x.c = threadIdx.x % p.cpb;
    x.j = threadIdx.x / p.cpb;
  } else {
    x.j = threadIdx.x % TPT;
    x.c = threadIdx.x / TPT;
  }
  x.b = tile_batch<kMirror>(p, x.c, blockIdx.x);
  x.active = x.b < p.nbatch;
  x.oin = to.in_off[x.c];
  x.oout = to.out_off[x.c];
  x.b0 = umod(x.b, p.d0);

  // everything above reads kernel parameters only, so it runs while the
  // previous kernel drains
  cpx v[R];
  pdl_wait();
  LoadOp::template run<L, R>(p, x, t, v);
  pdl_release();
  run_passes<L, R, 1, KeepsTile<LoadOp>::value, std::is_same<LoadOp, LoadCplxScalar>::value>(v, x.j, x.c, t, p.tw);
  StoreOp::template run<L, R>(p, x, t, to, v);
}

// Number of bytes of dynamic shared memory the kernel needs for cpb transforms.
inline size_t axis_pass_smem(int L, int R, int cpb, int colmode) {
  return 16 * ((2 * cpb * sizeof(int64_t) + 15) / 16) + size_t(cpb) * tile_pitch(L, R, cpb, colmode) * sizeof(cpx);
}

}  // namespace mb
