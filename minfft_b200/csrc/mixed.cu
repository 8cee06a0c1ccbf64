// Mixed batches: thousands of independent 1-D transforms of any kind and
// power-of-two length, run by one persistent kernel launched from a CUDA
// graph.
//
// Planning (host).  Jobs are grouped by (kind, direction, length).  Each
// group of transforms whose DFT fits in one CTA (4096 points) is cut into
// work items of up to `cpb` transforms (the items of a length-L group use
// L/16 threads per transform, so a 256-thread CTA holds 256*16/L of them).
// Transforms of 8192 points, which take 512 threads, run in a kernel of their
// own beside the persistent one, a CTA each (300 real jobs of 2^14 points in
// double 65.3 us as two passes, 47.2 so; 600 jobs of 2^4 .. 2^14 in single 29.6 and
// 23.3; 20000 of 2^4 .. 2^16 1011 and 955).  A longer transform (2^14 .. 2^16 complex points) is a Stockham chain of
// two passes through a scratch slot, and each pass is cut into tiles of 4096
// points, one work item each, with the kind's pre- and post-processing fused
// into the passes (the *Line and type-4 chain stages of axis_pass.cuh, which
// work on mirror pairs of sub-DFTs).
//
// Execution (device).  Every resident CTA takes the next item from an
// atomic counter until the list is exhausted.  The list interleaves the
// first-pass tiles of later transforms with the last-pass tiles of earlier
// ones, so that a transform's last pass comes more than one grid of items
// after its first (whose tiles are then done) and only about 1.5 grids of
// scratch are live: the scratch stays in the L2, and each long transform
// crosses HBM once each way.  (One CTA per long transform, two passes and
// element-wise sweeps through a private slice, kept 300 MB of scratch live
// and each CTA's phases in sequence: 20000 jobs of 2^4 .. 2^16 points in f32
// took 1102 us, 1056 so.)
//
// Waits.  A last-pass tile waits until its transform's first-pass tiles are
// done, a first-pass tile until the last transform that used its scratch
// slot is.  What an item waits for stands before it in the list, so it has
// been taken by a running CTA, and first-pass tiles of the first users of a
// slot wait for nothing: the waits end whatever the residency.  They are
// bounded all the same: a CTA whose wait runs out sets *status and stops.
// The others go on until they wait for a tile that no longer comes, so the
// launch ends after about twice the limit at most, with its output incomplete.
#include <cuda_runtime.h>
#include <stdio.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "kernel_registry.h"
#include "axis_pass.cuh"
#include "minfft_b200.h"

#define MB_EXPORT extern "C" __attribute__((visibility("default")))

namespace mb {
void set_last_error(int code, const char* msg);
void host_table(int kind, int64_t N, std::vector<cpx>& h);
cudaError_t dev_malloc(void** p, size_t bytes);  // every device allocation of the library (plan.cu)
template <class T>
cudaError_t dev_malloc(T** p, size_t bytes) {
  return dev_malloc(reinterpret_cast<void**>(p), bytes);
}
}  // namespace mb

namespace mb {
namespace mixed {

constexpr int kThreads = 256;
constexpr int kSlots = 21;           // table slots by log2 length, 0 .. 20
constexpr int kSmallMaxLog2L = 12;   // one-CTA DFTs up to 4096 points
constexpr int kWideLog2L = 13;       // DFTs of a 512-thread CTA
constexpr int kWideThreads = 512;
constexpr int kBigMaxLog2L = 16;     // two passes through scratch up to 65536
constexpr int kTilePoints = 16 * kThreads;  // points of a long item's tile
constexpr int kOffsetsBytes = 1024;  // tile offsets of the long-item passes (<= 64 transforms)
constexpr int kMinBlocks = sizeof(real) == 8 ? 2 : 4;  // CTAs per SM: 128 / 64 registers
// Scratch of each long length: 1.7 grids of tiles (1024 in single on a grid of
// 592 CTAs, 512 in double on 296), small enough to stay in the L2 beside the
// streams (20000 jobs in f32: 1056 us with 32 MiB, 1083 with 64, 1085 with 24).
constexpr size_t kSlotBytes = size_t(32) << 20;
constexpr long long kWaitLimit = 1LL << 22;

struct Job {
  const void* in;
  void* out;
  int op;
  int log2n;
};

enum ItemKind : int { kShort = 0, kUnit, kFirst, kLast };

struct __align__(16) Item {
  int kind;
  int combo;
  int log2L;
  int flags;
  int count;  // short items: transforms
  int first;  // short items: index of the first job
  int tile;   // long items: tile of the pass
  int id;     // long items: index of the transform's completion counters
  int dep;    // first-pass tiles: transform whose last pass frees the slot, or -1
  int64_t scratch;  // long items: offset of the slot (complex elements)
  const void* in;   // long items: the job's arrays
  void* out;
};

struct Params {
  const Job* jobs;  // in item order
  const Item* items;
  int nitems;         // of the persistent kernel; the wide transforms' follow
  int nbig;           // long transforms
  unsigned* counter;  // the queue, then nbig counters of finished first-pass tiles and nbig of last-pass tiles
  int* status;        // host-mapped; set when a wait ran out
  // Test hook (zero in normal batches): > 0 limits the waits to that many
  // polls and leaves the first tile of the first long transform uncounted.
  long long withhold;
  cpx* scratch;
  const cpx* tw[kSlots];    // w_L^m, by log2 L
  const cpx* rft[kSlots];   // real-DFT roots, by log2 N
  const cpx* t23[kSlots];   // type-2/3 roots, by log2 N
  const cpx* t4a[kSlots];   // type-4 pre-rotation, by log2 N
  const cpx* t4b[kSlots];   // type-4 post-rotation, by log2 N
  const cpx* sthi[kSlots];  // coarse roots of a long length, by log2 of it
  const cpx* stlo[kSlots];  // fine roots of a long length
  const cpx* sthi1[kSlots];  // the same minus one
  const cpx* stlo1[kSlots];
};

__host__ __device__ constexpr int small_radix(int L) { return L < 16 ? L : 16; }
__host__ __device__ constexpr int log2c(int v) { return v <= 1 ? 0 : 1 + log2c(v / 2); }
__host__ __device__ constexpr int small_cpb(int L) { return kThreads / (L / small_radix(L)); }
__host__ __device__ constexpr int first_bits(int lg) { return (lg + 1) / 2; }  // pass lengths of a long DFT
__host__ __device__ constexpr int root_bits(int lg) { return (lg + 1) / 2; }   // fine bits of a root pair

// ---------------------------------------------------------------- device
template <int L, class LoadOp, class StoreOp, int T = kThreads>
__device__ __noinline__ void run_small(const Params& mp, const Item& it, unsigned char* smem) {
  constexpr int R = small_radix(L);
  constexpr int TPT = L / R;
  constexpr int CPB = T / TPT;
  const int c = threadIdx.x / TPT, j = threadIdx.x % TPT;
  const bool active = c < it.count;
  Job job{};
  if (active) job = mp.jobs[it.first + c];
  const int log2N = (it.combo == K_CPLX) ? it.log2L : it.log2L + 1;
  AxisParams p;
  memset(&p, 0, sizeof(p));
  p.in = job.in;
  p.out = job.out;
  p.nbatch = it.count;
  p.d0 = p.d1 = 1;
  p.in_n = 1;
  p.out_k = 1;
  p.tw = mp.tw[it.log2L];
  p.st_ns = 1;
  p.st_div = 1;
  p.cpb = CPB;
  p.flags = it.flags;
  p.lp = tile_pitch(L, R, CPB, 0);
  switch (it.combo) {
    case K_R2C:
      p.t1 = mp.rft[log2N];
      if ((reinterpret_cast<uintptr_t>(job.in) % sizeof(cpx)) == 0) p.flags |= F_VEC;
      break;
    case K_C2R:
      p.t2 = mp.rft[log2N];
      if ((reinterpret_cast<uintptr_t>(job.out) % sizeof(cpx)) == 0) p.flags |= F_VEC;
      break;
    case K_DCT2:
    case K_DCT3:
      p.t1 = mp.t23[log2N];
      p.t2 = mp.rft[log2N];
      break;
    case K_T4:
      p.t1 = mp.t4a[log2N];
      p.t2 = mp.t4b[log2N];
      break;
    default: break;
  }
  Ctx x;
  x.b = c;
  x.b0 = 0;
  x.oin = 0;
  x.oout = 0;
  x.c = c;
  x.j = j;
  x.active = active;
  Tile t{reinterpret_cast<cpx*>(smem + kOffsetsBytes), p.lp};
  TileOffsets to{nullptr, nullptr, it.count};
  cpx v[R];
  LoadOp::template run<L, R>(p, x, t, v);
  run_passes<L, R, 1, KeepsTile<LoadOp>::value>(v, j, c, t, p.tw);
  StoreOp::template run<L, R>(p, x, t, to, v);
}

// Finished tiles of a long transform's pass, counted in global memory.
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Waits (bounded) until *p reaches n; all threads of the CTA call it.
__device__ __forceinline__ bool tiles_done(const Params& mp, const unsigned* p, unsigned n) {
  bool ok = true;
  if (threadIdx.x == 0) {
    const long long limit = mp.withhold > 0 ? mp.withhold : kWaitLimit;
    long long i = 0;
    while (ld_acquire(p) < n)
      if (++i > limit) {
        ok = false;
        *reinterpret_cast<volatile int*>(mp.status) = 1;
        break;
      }
  }
  return __syncthreads_and(ok) != 0;
}
// Counts one finished tile.  The barrier orders every thread's writes before
// thread 0's release, which is cumulative: no fence of their own.
__device__ __forceinline__ void tile_done(unsigned* p) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// One tile of a pass of a long transform of 2^lg points: CPB sub-DFTs of RP
// points (16 values per thread).  The first pass reads the job's input and
// writes its sub-DFTs contiguously into the scratch slot; the last pass
// reads that with the Stockham pre-twiddle and writes the job's output.
template <int RP, bool kIsLast, class Ld, class St>
__device__ __noinline__ void run_tile(const Params& mp, const Item& it, unsigned char* smem) {
  constexpr int R = 16, TPT = RP / R, CPB = kThreads / TPT;
  static_assert(CPB * 2 * sizeof(int64_t) <= kOffsetsBytes, "offsets region");
  const int lg = it.log2L;
  const int M = (1 << lg) / RP;  // sub-DFTs of the pass
  const int log2N = it.combo == K_CPLX ? lg : lg + 1;
  AxisParams p;
  memset(&p, 0, sizeof(p));
  p.nbatch = M;
  p.d0 = kIsLast ? M : 1;
  p.d1 = kIsLast ? 1 : M;
  p.is0 = p.is1 = 1;
  p.in_n = M;
  p.out_k = kIsLast ? M : 1;
  p.st_ns = kIsLast ? M : 1;
  p.st_div = 1;
  p.tw = mp.tw[log2c(RP)];
  p.cpb = CPB;
  p.colmode = 1;
  p.lp = tile_pitch(RP, R, CPB, 1);
  p.kn = int64_t(1) << log2N;
  // root pairs of the fused step: 2N before and 8N after a type-4 chain, 4N
  // for types 2 and 3, N for the real DFT
  const int lr = it.combo == K_T4                               ? log2N + (kIsLast ? 3 : 1)
                 : (it.combo == K_DCT2 || it.combo == K_DCT3) ? log2N + 2
                                                              : log2N;
  if constexpr (kIsLast) {
    p.in = mp.scratch + it.scratch;
    p.out = it.out;
    p.flags = (it.flags & (F_DST | F_CONJ_OUT)) | F_SRC_SMEM;  // scratch by plain loads: it stays in the L2
    p.st_lobits = root_bits(lg);
    p.st_hi = mp.sthi[lg];
    p.st_lo = mp.stlo[lg];
    p.t1 = mp.sthi1[lr];
    p.t2 = mp.stlo1[lr];
    p.kbits = root_bits(lr);
  } else {
    p.in = it.in;
    p.out = mp.scratch + it.scratch;
    p.flags = (it.flags & (F_DST | F_CONJ_IN)) | F_STAGE_ROWS;
    p.st_lobits = root_bits(lr);
    p.st_hi = mp.sthi1[lr];
    p.st_lo = mp.stlo1[lr];
  }
  constexpr MirrorKind kMirror = MirrorPairs<Ld>::value != kNoMirror ? MirrorPairs<Ld>::value : MirrorPairs<St>::value;
  int64_t* offs = reinterpret_cast<int64_t*>(smem);
  if (!kIsLast && threadIdx.x < CPB) offs[threadIdx.x] = tile_batch<kMirror>(p, threadIdx.x, it.tile) * RP;
  Tile t{reinterpret_cast<cpx*>(smem + kOffsetsBytes), p.lp};
  TileOffsets to{offs, offs, CPB};
  Ctx x;
  x.c = threadIdx.x % CPB;
  x.j = threadIdx.x / CPB;
  x.b = tile_batch<kMirror>(p, x.c, it.tile);
  x.b0 = kIsLast ? x.b : 0;
  x.oin = x.b;
  x.oout = kIsLast ? x.b : x.b * RP;
  x.active = true;
  cpx v[R];
  Ld::template run<RP, R>(p, x, t, v);
  run_passes<RP, R, 1, KeepsTile<Ld>::value>(v, x.j, x.c, t, p.tw);
  St::template run<RP, R>(p, x, t, to, v);
}

template <int RP>
__device__ __forceinline__ void run_first(const Params& mp, const Item& it, unsigned char* smem) {
  switch (it.combo) {
    case K_CPLX: run_tile<RP, false, LoadCplx, StoreCplx>(mp, it, smem); break;
    case K_R2C: run_tile<RP, false, LoadCplx, StoreCplx>(mp, it, smem); break;
    case K_C2R: run_tile<RP, false, LoadC2RLine, StoreCplx>(mp, it, smem); break;
    case K_DCT2: run_tile<RP, false, LoadDCT2Line, StoreCplx>(mp, it, smem); break;
    case K_DCT3: run_tile<RP, false, LoadDCT3Line, StoreCplx>(mp, it, smem); break;
    default: run_tile<RP, false, LoadT4ChainBy<RootSteps>, StoreCplx>(mp, it, smem); break;
  }
}

template <int RP>
__device__ __forceinline__ void run_last(const Params& mp, const Item& it, unsigned char* smem) {
  switch (it.combo) {
    case K_CPLX: run_tile<RP, true, LoadCplx, StoreCplx>(mp, it, smem); break;
    case K_R2C: run_tile<RP, true, LoadCplx, StoreR2CLine>(mp, it, smem); break;
    case K_C2R: run_tile<RP, true, LoadCplx, StoreCplx>(mp, it, smem); break;
    case K_DCT2: run_tile<RP, true, LoadCplx, StoreDCT2Line>(mp, it, smem); break;
    case K_DCT3: run_tile<RP, true, LoadCplx, StoreDCT3Line>(mp, it, smem); break;
    default: run_tile<RP, true, LoadCplx, StoreT4ChainBy<RootSteps>>(mp, it, smem); break;
  }
}

__device__ __forceinline__ bool run_long(const Params& mp, const Item& it, unsigned char* smem) {
  unsigned* firsts = mp.counter + 1;
  unsigned* lasts = firsts + mp.nbig;
  const unsigned tiles = unsigned(1 << it.log2L) / kTilePoints;
  if (it.kind == kFirst) {
    // the slot's previous user has the same length, hence as many tiles
    if (it.dep >= 0 && !tiles_done(mp, lasts + it.dep, tiles)) return false;
    if (first_bits(it.log2L) == 7)
      run_first<128>(mp, it, smem);
    else
      run_first<256>(mp, it, smem);
    if (!(mp.withhold > 0 && it.id == 0 && it.tile == 0)) tile_done(firsts + it.id);
  } else {
    if (!tiles_done(mp, firsts + it.id, tiles)) return false;
    if (it.log2L - first_bits(it.log2L) == 7)
      run_last<128>(mp, it, smem);
    else
      run_last<256>(mp, it, smem);
    tile_done(lasts + it.id);
  }
  return true;
}

// length-1 transforms: y = 2x (type 2), x (type 3), sqrt(2) x (type 4),
// (x, 0) (real DFT), Re z (inverse real DFT), z (complex DFT)
__device__ __noinline__ void run_unit(const Params& mp, const Item& it) {
  for (int c = threadIdx.x; c < it.count; c += blockDim.x) {
    const Job job = mp.jobs[it.first + c];
    switch (job.op) {
      case MINFFT_B200_DFT:
      case MINFFT_B200_INVDFT: *static_cast<cpx*>(job.out) = *static_cast<const cpx*>(job.in); break;
      case MINFFT_B200_REALDFT: *static_cast<cpx*>(job.out) = cmk(*static_cast<const real*>(job.in), real(0)); break;
      case MINFFT_B200_INVREALDFT: *static_cast<real*>(job.out) = static_cast<const cpx*>(job.in)->x; break;
      case MINFFT_B200_DCT2:
      case MINFFT_B200_DST2: *static_cast<real*>(job.out) = 2 * *static_cast<const real*>(job.in); break;
      case MINFFT_B200_DCT3:
      case MINFFT_B200_DST3: *static_cast<real*>(job.out) = *static_cast<const real*>(job.in); break;
      default:
        *static_cast<real*>(job.out) = real(1.414213562373095048801688724209698079) * *static_cast<const real*>(job.in);
        break;
    }
  }
}

template <class Ld, class St>
__device__ __forceinline__ void run_small_any(const Params& mp, const Item& it, unsigned char* smem) {
  switch (it.log2L) {
    case 0: run_small<1, Ld, St>(mp, it, smem); break;
    case 1: run_small<2, Ld, St>(mp, it, smem); break;
    case 2: run_small<4, Ld, St>(mp, it, smem); break;
    case 3: run_small<8, Ld, St>(mp, it, smem); break;
    case 4: run_small<16, Ld, St>(mp, it, smem); break;
    case 5: run_small<32, Ld, St>(mp, it, smem); break;
    case 6: run_small<64, Ld, St>(mp, it, smem); break;
    case 7: run_small<128, Ld, St>(mp, it, smem); break;
    case 8: run_small<256, Ld, St>(mp, it, smem); break;
    case 9: run_small<512, Ld, St>(mp, it, smem); break;
    case 10: run_small<1024, Ld, St>(mp, it, smem); break;
    case 11: run_small<2048, Ld, St>(mp, it, smem); break;
    case 12: run_small<4096, Ld, St>(mp, it, smem); break;
    default: break;
  }
}

__global__ void __launch_bounds__(kThreads, kMinBlocks) mixed_kernel(const __grid_constant__ Params mp) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_item[2];
  __shared__ Item s_desc[2];
  // Thread 0 keeps one index ahead of the item being prepared: while item n
  // runs, the descriptor of item n + 1 is on its way into shared memory and
  // the index of item n + 2 is taken from the queue.
  unsigned ahead = 0;
  auto fetch = [&](int idx, int slot) {
    s_item[slot] = idx;
    if (idx < mp.nitems) {
      const char* src = reinterpret_cast<const char*>(mp.items + idx);
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&s_desc[slot]));
#pragma unroll
      for (int i = 0; i < int(sizeof(Item)); i += 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i), "l"(src + i) : "memory");
    }
  };
  // A batch without long transforms has no waits, so any CTA may have any item:
  // each starts with the one of its own index and goes on with the one a grid
  // later, and only then turns to the counter, whose answer it asks for a whole
  // item ahead.  (Thread 0 holds its CTA's first barrier up until the answer is
  // there, behind a grid of atomics on one address: in single, 300 jobs of
  // 2^4 .. 2^10 points take 14.3 us from the counter alone and 10.3 so, 5000 of 2^10
  // 28.6 with one item dealt and 20.0 so, 9919 of 2^4 .. 2^12 41.5 and 35.2; 11054 of
  // 2^4 .. 2^10 in double 30.6 and 27.1.)
  const unsigned dealt = mp.nbig ? 0u : 2 * gridDim.x;
  if (threadIdx.x == 0) {
    fetch(int(mp.nbig ? atomicAdd(mp.counter, 1u) : blockIdx.x), 0);
    ahead = mp.nbig ? atomicAdd(mp.counter, 1u) : gridDim.x + blockIdx.x;
  }
  for (int n = 0;; ++n) {
    if (threadIdx.x == 0) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (s_item[n & 1] >= mp.nitems) break;
    const Item it = s_desc[n & 1];
    if (threadIdx.x == 0) {
      fetch(int(ahead), (n + 1) & 1);
      ahead = dealt + atomicAdd(mp.counter, 1u);
    }
    bool ok = true;
    if (it.kind >= kFirst) {
      ok = run_long(mp, it, smem);
    } else if (it.kind == kUnit) {
      run_unit(mp, it);
    } else {
      switch (it.combo) {
        case K_CPLX: run_small_any<LoadCplx, StoreCplx>(mp, it, smem); break;
        case K_R2C: run_small_any<LoadR2C, StoreR2C>(mp, it, smem); break;
        case K_C2R: run_small_any<LoadC2R, StoreC2R>(mp, it, smem); break;
        case K_DCT2: run_small_any<LoadDCT2, StoreDCT2>(mp, it, smem); break;
        case K_DCT3: run_small_any<LoadDCT3, StoreDCT3>(mp, it, smem); break;
        default: run_small_any<LoadT4, StoreT4>(mp, it, smem); break;
      }
    }
    if (!ok) break;
  }
}

// One transform of 8192 points per CTA.
__global__ void __launch_bounds__(kWideThreads, kMinBlocks / 2) wide_kernel(const __grid_constant__ Params mp) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int L = 1 << kWideLog2L;
  const Item it = mp.items[mp.nitems + blockIdx.x];
  switch (it.combo) {
    case K_CPLX: run_small<L, LoadCplx, StoreCplx, kWideThreads>(mp, it, smem); break;
    case K_R2C: run_small<L, LoadR2C, StoreR2C, kWideThreads>(mp, it, smem); break;
    case K_C2R: run_small<L, LoadC2R, StoreC2R, kWideThreads>(mp, it, smem); break;
    case K_DCT2: run_small<L, LoadDCT2, StoreDCT2, kWideThreads>(mp, it, smem); break;
    case K_DCT3: run_small<L, LoadDCT3, StoreDCT3, kWideThreads>(mp, it, smem); break;
    default: run_small<L, LoadT4, StoreT4, kWideThreads>(mp, it, smem); break;
  }
}

size_t wide_smem() {
  return kOffsetsBytes + 16 * ((tile_pitch(1 << kWideLog2L, 16, 1, 0) * sizeof(cpx) + 15) / 16);
}

// shared memory of the persistent kernel: offsets + the largest tile of any item
size_t kernel_smem() {
  size_t m = 0;
  for (int lg = 0; lg <= kSmallMaxLog2L; ++lg) {
    const int L = 1 << lg;
    const int cpb = small_cpb(L);
    m = std::max(m, size_t(cpb) * tile_pitch(L, small_radix(L), cpb, 0) * sizeof(cpx));
  }
  for (int rp : {128, 256}) {  // long items' tiles
    const int cpb = kThreads / (rp / 16);
    m = std::max(m, size_t(cpb) * tile_pitch(rp, 16, cpb, 1) * sizeof(cpx));
  }
  return kOffsetsBytes + 16 * ((m + 15) / 16);
}

}  // namespace mixed
}  // namespace mb

// ==================================================================== host
using mb::cpx;
using mb::real;
using namespace mb::mixed;

namespace {
std::atomic<long long> g_withhold{0};  // test hook: batches planned from now on (Params::withhold)
}

struct minfft_b200_mixed {
  int device = 0;
  int count = 0;
  std::vector<Job> jobs;
  std::vector<Item> items;  // the persistent kernel's, then the wide transforms'
  int nwide = 0;
  Params params;
  void* d_jobs = nullptr;
  void* d_items = nullptr;
  unsigned* d_counter = nullptr;
  size_t counter_bytes = 0;
  cpx* d_scratch = nullptr;
  int* h_status = nullptr;  // host-mapped: set by a kernel whose bounded wait ran out
  int64_t slot_base[kSlots] = {};  // scratch of each long length (complex elements)
  int slots[kSlots] = {};
  std::vector<void*> tables;
  int grid = 0;
  int per_sm = 1;
  size_t smem = 0;
  int split = 1;  // jobs per short item = slots / split
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

namespace {

bool ok(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return true;
  char buf[256];
  snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
  mb::set_last_error(e == cudaErrorMemoryAllocation ? MINFFT_B200_ENOMEM : MINFFT_B200_ECUDA, buf);
  return false;
}

int fail(int code, const char* msg) {
  mb::set_last_error(code, msg);
  return code;
}

int ilog2i(int64_t v) {
  int r = 0;
  while ((int64_t(1) << r) < v) ++r;
  return r;
}

int combo_of(int op) {
  switch (op) {
    case MINFFT_B200_DFT:
    case MINFFT_B200_INVDFT: return mb::K_CPLX;
    case MINFFT_B200_REALDFT: return mb::K_R2C;
    case MINFFT_B200_INVREALDFT: return mb::K_C2R;
    case MINFFT_B200_DCT2:
    case MINFFT_B200_DST2: return mb::K_DCT2;
    case MINFFT_B200_DCT3:
    case MINFFT_B200_DST3: return mb::K_DCT3;
    default: return mb::K_T4;
  }
}

int flags_of(int op) {
  if (op == MINFFT_B200_INVDFT) return mb::F_CONJ_IN | mb::F_CONJ_OUT;
  if (op == MINFFT_B200_DST2 || op == MINFFT_B200_DST3 || op == MINFFT_B200_DST4) return mb::F_DST;
  return 0;
}

const cpx* upload(minfft_b200_mixed* m, int kind, int64_t N) {
  std::vector<cpx> h;
  mb::host_table(kind, N, h);
  void* d = nullptr;
  if (!ok(mb::dev_malloc(&d, h.size() * sizeof(cpx)), "cudaMalloc(table)")) return nullptr;
  m->tables.push_back(d);
  if (!ok(cudaMemcpy(d, h.data(), h.size() * sizeof(cpx), cudaMemcpyHostToDevice), "cudaMemcpy(table)"))
    return nullptr;
  return static_cast<const cpx*>(d);
}

void release_graph(minfft_b200_mixed* m) {
  if (m->exec) cudaGraphExecDestroy(m->exec);
  if (m->graph) cudaGraphDestroy(m->graph);
  m->exec = nullptr;
  m->graph = nullptr;
}

// Cut the job groups into items (short groups: slots/split jobs per item),
// order them, upload, and capture counter reset + kernel in a graph.
bool build_items(minfft_b200_mixed* m) {
  std::map<std::tuple<int, int, int, int>, std::vector<int>> groups;  // (long, combo, flags, log2L) -> jobs
  std::vector<Item> wide;
  for (int i = 0; i < m->count; ++i) {
    const Job& j = m->jobs[i];
    const int combo = combo_of(j.op);
    const int64_t n = int64_t(1) << j.log2n;
    if (n == 1) {
      groups[std::make_tuple(0, -1, 0, 0)].push_back(i);
      continue;
    }
    const int lgL = combo == mb::K_CPLX ? j.log2n : j.log2n - 1;
    groups[std::make_tuple(lgL > kWideLog2L ? 1 : 0, combo, flags_of(j.op), lgL)].push_back(i);
  }
  std::vector<std::pair<double, Item>> its;  // short items by cost
  std::vector<Item> longs;                   // one prototype per long transform
  std::vector<Job> order;
  for (auto& g : groups) {
    const int combo = std::get<1>(g.first), flags = std::get<2>(g.first), lgL = std::get<3>(g.first);
    const std::vector<int>& js = g.second;
    Item it{};
    it.combo = combo;
    it.log2L = lgL;
    it.flags = flags;
    it.dep = -1;
    if (std::get<0>(g.first)) {
      for (int i : js) {
        const Job& j = m->jobs[i];
        Item l = it;
        l.in = j.in;
        l.out = j.out;
        // the inverse real DFT's chain ends conjugated, as the complex inverse's does
        if (combo == mb::K_C2R) l.flags |= mb::F_CONJ_OUT;
        longs.push_back(l);
      }
      continue;
    }
    const int L = 1 << lgL;
    const int per = combo < 0 ? kThreads : lgL == kWideLog2L ? 1 : std::max(1, small_cpb(L) / m->split);
    for (size_t s = 0; s < js.size(); s += per) {
      it.kind = combo < 0 ? kUnit : kShort;
      it.count = int(std::min<size_t>(per, js.size() - s));
      it.first = int(order.size());
      for (int k = 0; k < it.count; ++k) order.push_back(m->jobs[js[s + k]]);
      if (lgL == kWideLog2L && combo >= 0) {
        wide.push_back(it);
        continue;
      }
      its.push_back(std::make_pair(double(L) * std::max(1, lgL) * it.count, it));  // cost: points processed
    }
  }
  std::stable_sort(its.begin(), its.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
  std::stable_sort(longs.begin(), longs.end(), [](const Item& a, const Item& b) { return a.log2L > b.log2L; });
  // The list: first-pass tiles until the oldest transform's are `lag` items
  // back (or its length's slots are used up), then that transform's
  // last-pass tiles; short items fill the lag once the long ones run out,
  // and the rest follow, largest first.
  m->items.clear();
  const size_t lag = size_t(m->grid) + size_t(m->grid) / 2;
  struct Open {
    int id;
    size_t end;  // list position after its first-pass tiles
  };
  std::deque<Open> open;
  std::map<int, std::vector<int>> users;  // log2L -> transforms in slot order
  std::map<int, int> live;                // log2L -> slots in use by open transforms
  size_t next = 0, nshort = 0;
  auto emit = [&](int id, int kind) {
    const int tiles = (1 << longs[id].log2L) / kTilePoints;
    for (int t = 0; t < tiles; ++t) {
      Item it = longs[id];
      it.kind = kind;
      it.tile = t;
      it.id = id;
      if (kind == kLast) it.dep = -1;
      m->items.push_back(it);
    }
  };
  while (next < longs.size() || !open.empty()) {
    const bool old = !open.empty() && m->items.size() - open.front().end >= lag;
    if (next < longs.size() && !old && live[longs[next].log2L] < m->slots[longs[next].log2L]) {
      Item& l = longs[next];
      std::vector<int>& u = users[l.log2L];
      const int S = m->slots[l.log2L], k = int(u.size());
      l.scratch = m->slot_base[l.log2L] + int64_t(k % S) * (int64_t(1) << l.log2L);
      l.dep = k >= S ? u[k - S] : -1;
      u.push_back(int(next));
      ++live[l.log2L];
      emit(int(next), kFirst);
      open.push_back(Open{int(next), m->items.size()});
      ++next;
    } else if (!old && next == longs.size() && nshort < its.size()) {
      m->items.push_back(its[nshort++].second);
    } else {
      emit(open.front().id, kLast);
      --live[longs[open.front().id].log2L];
      open.pop_front();
    }
  }
  while (nshort < its.size()) m->items.push_back(its[nshort++].second);
  const int nbig = int(longs.size()), nitems = int(m->items.size());
  m->items.insert(m->items.end(), wide.begin(), wide.end());
  m->nwide = int(wide.size());

  if (m->d_jobs) cudaFree(m->d_jobs);
  if (m->d_items) cudaFree(m->d_items);
  if (m->d_counter) cudaFree(m->d_counter);
  m->d_jobs = m->d_items = nullptr;
  m->d_counter = nullptr;
  m->counter_bytes = (1 + 2 * size_t(nbig)) * sizeof(unsigned);
  if (!ok(mb::dev_malloc(&m->d_jobs, std::max<size_t>(1, order.size()) * sizeof(Job)), "cudaMalloc(jobs)") ||
      !ok(mb::dev_malloc(&m->d_items, std::max<size_t>(1, m->items.size()) * sizeof(Item)), "cudaMalloc(items)") ||
      !ok(mb::dev_malloc(&m->d_counter, m->counter_bytes), "cudaMalloc(counter)"))
    return false;
  if (!order.empty() && !ok(cudaMemcpy(m->d_jobs, order.data(), order.size() * sizeof(Job), cudaMemcpyHostToDevice),
                            "cudaMemcpy(jobs)"))
    return false;
  if (!m->items.empty() &&
      !ok(cudaMemcpy(m->d_items, m->items.data(), m->items.size() * sizeof(Item), cudaMemcpyHostToDevice),
          "cudaMemcpy(items)"))
    return false;
  m->params.jobs = static_cast<const Job*>(m->d_jobs);
  m->params.items = static_cast<const Item*>(m->d_items);
  m->params.nitems = nitems;
  m->params.nbig = nbig;
  m->params.withhold = g_withhold.load();
  m->params.counter = m->d_counter;
  // graph: reset the queue and the tile counters, run the persistent kernel;
  // beside them the wide transforms' kernel, which starts first (the persistent
  // CTAs take the SMs as its own leave them)
  release_graph(m);
  if (!ok(cudaGraphCreate(&m->graph, 0), "cudaGraphCreate")) return false;
  void* args[1] = {&m->params};
  auto kernel = [&](const void* fn, int grid, int threads, size_t smem, const cudaGraphNode_t* after) {
    cudaKernelNodeParams k = {};
    k.func = const_cast<void*>(fn);
    k.gridDim = dim3(grid);
    k.blockDim = dim3(threads);
    k.sharedMemBytes = unsigned(smem);
    k.kernelParams = args;
    cudaGraphNode_t node;
    return ok(cudaGraphAddKernelNode(&node, m->graph, after, after ? 1 : 0, &k), "cudaGraphAddKernelNode");
  };
  if (m->nwide && !kernel((const void*)wide_kernel, m->nwide, kWideThreads, wide_smem(), nullptr)) return false;
  if (nitems) {
    cudaMemsetParams z = {};
    z.dst = m->d_counter;
    z.elementSize = sizeof(unsigned);
    z.width = m->counter_bytes / sizeof(unsigned);
    z.height = 1;
    cudaGraphNode_t node;
    if (!ok(cudaGraphAddMemsetNode(&node, m->graph, nullptr, 0, &z), "cudaGraphAddMemsetNode") ||
        !kernel((const void*)mixed_kernel, m->grid, kThreads, m->smem, &node))
      return false;
  }
  return ok(cudaGraphInstantiate(&m->exec, m->graph, 0), "cudaGraphInstantiate");
}

}  // namespace

MB_EXPORT void minfft_b200_mixed_free(minfft_b200_mixed* m) {
  if (!m) return;
  release_graph(m);
  for (void* t : m->tables) cudaFree(t);
  cudaFree(m->d_jobs);
  cudaFree(m->d_items);
  cudaFree(m->d_counter);
  cudaFree(m->d_scratch);
  if (m->h_status) cudaFreeHost(m->h_status);
  delete m;
}

MB_EXPORT minfft_b200_mixed* minfft_b200_mixed_plan(int count, const minfft_b200_job* jobs) {
  if (count < 1 || !jobs) {
    fail(MINFFT_B200_EINVAL, "mixed plan: need at least one job");
    return nullptr;
  }
  minfft_b200_mixed* m = new (std::nothrow) minfft_b200_mixed();
  if (!m) {
    fail(MINFFT_B200_ENOMEM, "mixed plan: host allocation failed");
    return nullptr;
  }
  m->count = count;
  m->jobs.resize(count);
  std::vector<int> need_tw(kSlots, 0), need_st(kSlots, 0), need_st1(kSlots, 0), nlong(kSlots, 0);
  std::vector<int> need_kind(kSlots * mb::K_COUNT, 0);
  for (int i = 0; i < count; ++i) {
    const minfft_b200_job& j = jobs[i];
    const int64_t n = j.n;
    if (j.op < MINFFT_B200_DFT || j.op > MINFFT_B200_DST4 || n < 1 || (n & (n - 1)) || !j.in || !j.out) {
      char buf[160];
      snprintf(buf, sizeof(buf), "mixed plan: job %d has a bad transform code, length or pointer", i);
      fail(MINFFT_B200_EINVAL, buf);
      minfft_b200_mixed_free(m);
      return nullptr;
    }
    const int combo = combo_of(j.op);
    const int lgn = ilog2i(n);
    const int lgL = (combo == mb::K_CPLX) ? lgn : std::max(lgn - 1, 0);
    if (lgL > kBigMaxLog2L) {
      fail(MINFFT_B200_EINVAL, "mixed plan: lengths above 65536 complex points (131072 real) are not supported");
      minfft_b200_mixed_free(m);
      return nullptr;
    }
    // complex arrays are accessed as aligned pairs; real arrays of a real DFT
    // (or its inverse) of more than 16384 reals are required to be aligned so too
    const bool pairs = lgL > 13;
    const bool cin = combo == mb::K_CPLX || combo == mb::K_C2R || (combo == mb::K_R2C && pairs);
    const bool cout = combo == mb::K_CPLX || combo == mb::K_R2C || (combo == mb::K_C2R && pairs);
    if ((cin && reinterpret_cast<uintptr_t>(j.in) % sizeof(cpx)) ||
        (cout && reinterpret_cast<uintptr_t>(j.out) % sizeof(cpx))) {
      fail(MINFFT_B200_EINVAL, "mixed plan: complex data must be aligned to its size");
      minfft_b200_mixed_free(m);
      return nullptr;
    }
    m->jobs[i] = Job{j.in, j.out, j.op, lgn};
    if (n == 1) continue;
    if (lgL > kWideLog2L) {
      ++nlong[lgL];
      need_tw[first_bits(lgL)] = need_tw[lgL - first_bits(lgL)] = 1;
      need_st[lgL] = 1;  // the last pass's pre-twiddle; need_st1: the fused steps' roots (run_tile)
      if (combo == mb::K_R2C || combo == mb::K_C2R) need_st1[lgn] = 1;
      if (combo == mb::K_DCT2 || combo == mb::K_DCT3) need_st1[lgn + 2] = 1;
      if (combo == mb::K_T4) need_st1[lgn + 1] = need_st1[lgn + 3] = 1;
      continue;
    }
    need_tw[lgL] = 1;
    need_kind[combo * kSlots + lgn] = 1;
  }
  if (!ok(cudaGetDevice(&m->device), "cudaGetDevice")) {
    minfft_b200_mixed_free(m);
    return nullptr;
  }
  Params& P = m->params;
  memset(&P, 0, sizeof(P));
  bool good = true;
  for (int lg = 0; lg < kSlots && good; ++lg) {
    const int64_t L = int64_t(1) << lg;
    if (need_tw[lg]) good = (P.tw[lg] = upload(m, mb::tables::TB_TW, L)) != nullptr;
    if (good && need_st[lg]) {
      good = (P.sthi[lg] = upload(m, mb::tables::TB_STHI, L)) && (P.stlo[lg] = upload(m, mb::tables::TB_STLO, L));
    }
    if (good && need_st1[lg])
      good = (P.sthi1[lg] = upload(m, mb::tables::TB_STHI1, L)) && (P.stlo1[lg] = upload(m, mb::tables::TB_STLO1, L));
    for (int combo = 1; combo < mb::K_COUNT && good; ++combo) {
      if (!need_kind[combo * kSlots + lg]) continue;
      const int64_t N = L;
      if (combo == mb::K_R2C || combo == mb::K_C2R || combo == mb::K_DCT2 || combo == mb::K_DCT3)
        if (!P.rft[lg]) good = (P.rft[lg] = upload(m, mb::tables::TB_RFT, N)) != nullptr;
      if (good && (combo == mb::K_DCT2 || combo == mb::K_DCT3) && !P.t23[lg])
        good = (P.t23[lg] = upload(m, mb::tables::TB_T23, N)) != nullptr;
      if (good && combo == mb::K_T4 && !P.t4a[lg])
        good = (P.t4a[lg] = upload(m, mb::tables::TB_T4PRE, N)) && (P.t4b[lg] = upload(m, mb::tables::TB_T4POST, N));
    }
  }
  int sms = 148;
  if (good) good = ok(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device), "device query");
  m->smem = kernel_smem();
  if (good)
    good = ok(cudaFuncSetAttribute((const void*)mixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(m->smem)),
              "cudaFuncSetAttribute") &&
           ok(cudaFuncSetAttribute((const void*)wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(wide_smem())),
              "cudaFuncSetAttribute");
  int occ = 1;
  if (good)
    good = ok(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)mixed_kernel, kThreads, m->smem),
              "occupancy query");
  m->per_sm = std::max(1, occ);
  m->grid = sms * m->per_sm;
  // scratch slots of each long length, in kSlotBytes
  int64_t scratch = 0;
  for (int lg = kWideLog2L + 1; lg <= kBigMaxLog2L; ++lg) {
    const size_t bytes = (size_t(1) << lg) * sizeof(cpx);
    m->slots[lg] = int(std::min<size_t>(nlong[lg], kSlotBytes / bytes));
    m->slot_base[lg] = scratch;
    scratch += int64_t(m->slots[lg]) << lg;
  }
  if (good && scratch > 0) good = ok(mb::dev_malloc(&m->d_scratch, size_t(scratch) * sizeof(cpx)), "cudaMalloc(scratch)");
  if (good)
    good = ok(cudaHostAlloc(reinterpret_cast<void**>(&m->h_status), sizeof(int), cudaHostAllocMapped),
              "cudaHostAlloc(status)");
  if (good) {
    *m->h_status = 0;
    good = ok(cudaHostGetDevicePointer(reinterpret_cast<void**>(&P.status), m->h_status, 0), "status address");
  }
  P.scratch = m->d_scratch;
  if (good) good = build_items(m);
  if (!good) {
    minfft_b200_mixed_free(m);
    return nullptr;
  }
  return m;
}

MB_EXPORT int minfft_b200_mixed_execute(minfft_b200_mixed* m, void* stream) {
  if (!m || !m->exec) return fail(MINFFT_B200_EINVAL, "mixed execute: NULL plan");
  if (*static_cast<volatile int*>(m->h_status)) {
    *m->h_status = 0;
    return fail(MINFFT_B200_ETIMEOUT, "mixed execute: an earlier run gave up waiting for a pass of a long job");
  }
  return ok(cudaGraphLaunch(m->exec, static_cast<cudaStream_t>(stream)), "cudaGraphLaunch") ? MINFFT_B200_OK
                                                                                             : MINFFT_B200_ECUDA;
}

MB_EXPORT int minfft_b200_mixed_items(const minfft_b200_mixed* m) { return m ? int(m->items.size()) : -1; }

// Time the plan's tile shapes (jobs per short work item: all slots, 1/2,
// 1/4, 1/8 of them) and persistent grid sizes (1 .. max CTAs per SM), keep
// the fastest.  Runs the batch several times (outputs are overwritten).
MB_EXPORT int minfft_b200_mixed_autotune(minfft_b200_mixed* m, int reps) {
  if (!m) return fail(MINFFT_B200_EINVAL, "mixed autotune: NULL plan");
  if (reps < 1) reps = 3;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
  const int max_per_sm = m->per_sm;
  cudaStream_t st;
  if (!ok(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "cudaStreamCreate")) return MINFFT_B200_ECUDA;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  int best_split = m->split, best_per = m->per_sm;
  auto grid_for = [&](int per) { return sms * per; };
  for (int split : {1, 2, 4, 8}) {
    for (int per = 1; per <= max_per_sm; ++per) {
      m->split = split;
      m->grid = grid_for(per);
      if (!build_items(m)) continue;
      cudaGraphLaunch(m->exec, st);
      cudaEventRecord(e0, st);
      for (int r = 0; r < reps; ++r) cudaGraphLaunch(m->exec, st);
      cudaEventRecord(e1, st);
      cudaEventSynchronize(e1);
      float ms = 0;
      if (cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess && ms > 0 && ms < best) {
        best = ms;
        best_split = split;
        best_per = per;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(st);
  m->split = best_split;
  m->grid = grid_for(best_per);
  return build_items(m) ? MINFFT_B200_OK : MINFFT_B200_ECUDA;
}

MB_EXPORT int minfft_b200_test_mixed_withhold(long long polls) {
  if (polls < 0) return fail(MINFFT_B200_EINVAL, "poll count must be >= 0");
  g_withhold.store(polls);
  return MINFFT_B200_OK;
}
