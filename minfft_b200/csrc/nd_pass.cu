// Small multi-dimensional transforms in one launch.
//
// A 2-D or 3-D transform of a few thousand points runs in less time than its
// launches take: one launch per axis costs the host 2.4 us and the GPU about
// as much.  Here a cluster of kNdCluster CTAs per array runs all axes, with a
// cluster barrier (release / acquire, which orders the global writes of one
// step before the reads of the next) where the launches ended.  Each step is
// the axis pass's own load stage, Stockham passes and store stage
// (axis_pass.cuh), radix 8, its transforms dealt out over the CTAs; the array
// stays in the L2 between the steps.  The root tables are copied to shared
// memory before the wait for the previous kernel, so that no step waits for
// the L2 on their account.  (One CTA per array with the array in its shared
// memory was measured first: 7.5 us for a DCT-2 of 64 x 64 in f32, against
// 6.4 as two launches and 5.2 so -- a thousand instructions per warp in
// sequence on one SM, a quarter of them waiting to be fetched.)
//
// In place is safe within a step: a transform's loads are all done before its
// first store, and transforms do not overlap; a step whose input and output
// differ in size never has them in one buffer (build_program).
#define MB_TABLES_GENERIC 1
#include "nd_pass.h"

#include "kernel_registry.h"

namespace mb {

namespace {

constexpr int nd_radix(int L) { return L < 8 ? L : 8; }
// Pitch between the transforms of the exchange tile: odd, so that adjacent
// transforms (columns) fall on different banks whatever their length.
__host__ __device__ constexpr int nd_pitch(int L) { return padded_len(L) | 1; }
// Exchange tile of a CTA: 8 values per thread (fewer below 8 points), padded.
__host__ __device__ constexpr int nd_tile_elems(int threads) { return threads * 9; }
constexpr bool nd_tile_fits(int L) {
  return (64 / (L / nd_radix(L))) * nd_pitch(L) <= nd_tile_elems(64);
}
static_assert(nd_tile_fits(2) && nd_tile_fits(8) && nd_tile_fits(16) && nd_tile_fits(32) && nd_tile_fits(64) &&
                  nd_tile_fits(128),
              "every length's tile fits");

template <int LG, class LoadOp, class StoreOp>
__device__ __noinline__ void nd_axis(const NdAxis& a, const cpx* tables, const void* src, void* dst, int vec, int rank,
                                     cpx* tile) {
  constexpr int L = 1 << LG, R = nd_radix(L), TPT = L / R;
  const int cpb = blockDim.x / TPT;
  AxisParams p;
  memset(&p, 0, sizeof(p));
  p.in = src;
  p.out = dst;
  p.nbatch = a.nb;
  p.d0 = a.inner;
  p.d1 = 1;
  p.in_n = p.out_k = a.inner;
  p.tw = tables;
  p.t1 = tables + a.n_tw;
  p.t2 = tables + a.n_tw + a.n_t1;
  p.st_ns = p.st_div = 1;
  p.cpb = cpb;
  p.flags = a.flags | vec;
  // rows: threads of one transform adjacent; columns: transforms adjacent
  const bool col = a.inner > 1;
  p.colmode = col ? 1 : 0;
  p.lp = nd_pitch(L);
  Tile t{tile, p.lp};
  TileOffsets to{nullptr, nullptr, cpb};
  Ctx x;
  x.c = col ? threadIdx.x % cpb : threadIdx.x / TPT;
  x.j = col ? threadIdx.x / cpb : threadIdx.x % TPT;
  for (int base = rank * cpb; base < a.nb; base += kNdCluster * cpb) {
    const int b = base + x.c;
    x.b = b;
    x.active = b < a.nb;
    const int b1 = x.active ? b / a.inner : 0, b0 = x.active ? b - b1 * a.inner : 0;
    x.b0 = b0;
    x.oin = b0 + b1 * a.in_row;
    x.oout = b0 + b1 * a.out_row;
    cpx v[R];
    LoadOp::template run<L, R>(p, x, t, v);
    run_passes<L, R, 1, KeepsTile<LoadOp>::value>(v, x.j, x.c, t, p.tw);
    StoreOp::template run<L, R>(p, x, t, to, v);
    __syncthreads();  // the tile is free
  }
}

template <class LoadOp, class StoreOp>
__device__ __forceinline__ void nd_step(const NdAxis& a, const cpx* tables, const void* src, void* dst, int vec,
                                        int rank, cpx* tile) {
  switch (a.log2L) {
    case 0: nd_axis<0, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
    case 1: nd_axis<1, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
    case 2: nd_axis<2, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
    case 3: nd_axis<3, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
    case 4: nd_axis<4, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
    case 5: nd_axis<5, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
    case 6: nd_axis<6, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
    default: nd_axis<7, LoadOp, StoreOp>(a, tables, src, dst, vec, rank, tile); break;
  }
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Ld1/St1: the first step's stages; LdM/StM: the steps between; LdN/StN: the
// last step's.  kIn, kMid, kOut: whether the buffers hold complex values.
template <class Ld1, class St1, class LdM, class StM, class LdN, class StN, bool kIn, bool kMid, bool kOut>
__global__ void __cluster_dims__(kNdCluster, 1, 1) __launch_bounds__(kNdMaxThreads, 1)
    nd_pass_kernel(const __grid_constant__ NdParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  cpx* tile = reinterpret_cast<cpx*>(smem);
  cpx* tables = tile + nd_tile_elems(blockDim.x);
  const int64_t i = blockIdx.x / kNdCluster;
  const int rank = blockIdx.x % kNdCluster;
  const char* in = static_cast<const char*>(p.in) + i * p.in_stride * int(kIn ? sizeof(cpx) : sizeof(real));
  char* mid = static_cast<char*>(p.mid) + i * p.mid_stride * int(kMid ? sizeof(cpx) : sizeof(real));
  char* out = static_cast<char*>(p.out) + i * p.out_stride * int(kOut ? sizeof(cpx) : sizeof(real));
  {
    cpx* q = tables;
    auto copy = [&](const cpx* src, int n) {
      for (int e = threadIdx.x; e < n; e += blockDim.x) q[e] = __ldg(src + e);
      q += n;
    };
    for (int k = 0; k < p.naxes; ++k) {
      copy(p.ax[k].tw, p.ax[k].n_tw);
      copy(p.ax[k].t1, p.ax[k].n_t1);
      copy(p.ax[k].t2, p.ax[k].n_t2);
    }
  }
  __syncthreads();
  pdl_wait();
  auto next = [&](int k) { return p.ax[k].n_tw + p.ax[k].n_t1 + p.ax[k].n_t2; };
  nd_step<Ld1, St1>(p.ax[0], tables, in, mid, p.flags, rank, tile);
  pdl_release();
  tables += next(0);
  cluster_barrier();
  for (int k = 1; k + 1 < p.naxes; ++k) {
    nd_step<LdM, StM>(p.ax[k], tables, mid, mid, 0, rank, tile);
    tables += next(k);
    cluster_barrier();
  }
  nd_step<LdN, StN>(p.ax[p.naxes - 1], tables, mid, out, p.flags, rank, tile);
}

}  // namespace

const void* nd_kernel(int first_combo, int last_combo) {
  if (first_combo == K_R2C)
    return (const void*)nd_pass_kernel<LoadR2C, StoreR2C, LoadCplx, StoreCplx, LoadCplx, StoreCplx, false, true, true>;
  if (last_combo == K_C2R)
    return (const void*)nd_pass_kernel<LoadCplx, StoreCplx, LoadCplx, StoreCplx, LoadC2R, StoreC2R, true, true, false>;
  switch (first_combo) {
    case K_CPLX:
      return (const void*)nd_pass_kernel<LoadCplx, StoreCplx, LoadCplx, StoreCplx, LoadCplx, StoreCplx, true, true,
                                         true>;
    case K_DCT2:
      return (const void*)nd_pass_kernel<LoadDCT2, StoreDCT2, LoadDCT2, StoreDCT2, LoadDCT2, StoreDCT2, false, false,
                                         false>;
    case K_DCT3:
      return (const void*)nd_pass_kernel<LoadDCT3, StoreDCT3, LoadDCT3, StoreDCT3, LoadDCT3, StoreDCT3, false, false,
                                         false>;
    case K_T4:
      return (const void*)nd_pass_kernel<LoadT4, StoreT4, LoadT4, StoreT4, LoadT4, StoreT4, false, false, false>;
    default: return nullptr;
  }
}

size_t nd_smem(int threads, int table_elems) {
  return size_t(nd_tile_elems(threads) + table_elems) * sizeof(cpx);
}

}  // namespace mb
