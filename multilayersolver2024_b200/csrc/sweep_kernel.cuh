// sweep_kernel.cuh -- the kernel of sweep.cuh (instantiated by flow_fp32.cu and
// flow_fp64.cu).
#pragma once

#include "sweep.cuh"

namespace mlx {

// `iterations` sweeps of one layer's elastic tets.
template <typename R, int MAT, bool DAMP>
__global__ void __launch_bounds__(kSweepThreads) k_sweep(TetData<R> td, SweepArgs<R> a, R4<R>* __restrict__ pos,
                                                         const R4<R>* __restrict__ oldp, R inv_h2, R inv_h) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __shared__ int turn, last;
  if (threadIdx.x == 0) turn = 0;
  const unsigned base = __ldcg(&a.state->base);
  const int T = td.T;
  const int G = gridDim.x, mine = (a.n_chunks - (int)blockIdx.x + G - 1) / G;
  __syncthreads();
  bool ok = true;
  for (int it = 0; it < a.iterations && ok; ++it) {
    const unsigned at = base + (unsigned)it * (unsigned)a.D;
    // chunk j of this CTA is always warp j mod nw's, so a tet's multipliers
    // stay with one thread
    for (int j = threadIdx.x >> 5; j < mine; j += nw) {
      const int q = blockIdx.x + j * G, n = it * mine + j;
      const int2 ch = a.chunks[q];
      const bool active = lane < ch.y;
      // (the lanes past the end load the chunk's last tet and write nothing)
      const int i = ch.x + min(lane, ch.y - 1), s = a.list ? a.list[i] : i;
      TetRest<R, MAT> r;
      load_rest<R, MAT>(td, s, r);
      const ushort4 cw = a.corner[s];
      const R4<R> m4 = a.minv[s];
      R minv[4] = {m4.x, m4.y, m4.z, m4.w};
      const int4 v = r.v;
      const int vk[4] = {v.x, v.y, v.z, v.w};
      const unsigned word[4] = {cw.x, cw.y, cw.z, cw.w};
      unsigned want[4], need = 0;
      V3<R> X[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        want[k] = at + (word[k] & kSweepRank);
        if (it == 0 && (word[k] & kSweepRank) == 0) {
          const R4<R> p = ldcg_r4(pos + vk[k]);
          X[k] = {p.x, p.y, p.z};
        } else if (active) {
          need |= 1u << k;
        }
      }
      ok = sweep_turn(&turn, n - a.gate, a.error) && sweep_acquire(a.rec, v, want, need, X, a.error);
      if (!ok) break;
      if (lane == 0) atomicAdd(&turn, 1);
      if (active) {
        R lnew[num_lambda<MAT>()];
        tet_update<R, MAT, DAMP>(r, X, minv, oldp, inv_h2, inv_h, lnew);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (!(word[k] & kSweepLast)) {
            sweep_release(a.rec + vk[k], X[k], want[k] + 1);
            continue;
          }
          if (a.pins && (word[k] & kSweepPinned)) {
            // xi(pinnedDOFs) = pinnedx (xpbdLayer3D.m:333)
            const int* pa = a.pin_at + 3 * (size_t)vk[k];
            if (pa[0] >= 0) X[k].x = a.pin_vals[pa[0]];
            if (pa[1] >= 0) X[k].y = a.pin_vals[pa[1]];
            if (pa[2] >= 0) X[k].z = a.pin_vals[pa[2]];
          }
          if (it + 1 < a.iterations) sweep_release(a.rec + vk[k], X[k], at + (unsigned)a.D);
          else stcg_r4(pos + vk[k], make_r4<R>(X[k].x, X[k].y, X[k].z, minv[k]));
        }
#pragma unroll
        for (int l = 0; l < num_lambda<MAT>(); ++l) td.lambda[(size_t)l * T + s] = lnew[l];
      }
      __syncwarp();
    }
  }
  // the next launch's base, once every CTA has read this one's
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&a.state->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  unsigned next = base + (unsigned)a.iterations * (unsigned)a.D;
  if (next >= 0u - (unsigned)(2 * kSweepMaxTags)) {
    ulonglong2* p = reinterpret_cast<ulonglong2*>(a.rec);
    const size_t n = (size_t)a.N * (sizeof(SweepRec<R>) / sizeof(ulonglong2));
    for (size_t i = threadIdx.x; i < n; i += blockDim.x) p[i] = make_ulonglong2(0, 0);
    next = 0;
  }
  if (threadIdx.x == 0) {
    a.state->ticket = 0;
    a.state->base = next;
  }
}

template <typename R> static const void* sweep_kernel_of(int mat_kind, bool damp) {
  switch (mat_kind) {
    case MAT_NH: return (const void*)k_sweep<R, MAT_NH, false>;
    case MAT_STVK_BLOCKS:
      return damp ? (const void*)k_sweep<R, MAT_STVK_BLOCKS, true> : (const void*)k_sweep<R, MAT_STVK_BLOCKS, false>;
    default:
      return damp ? (const void*)k_sweep<R, MAT_STVK_LAME, true> : (const void*)k_sweep<R, MAT_STVK_LAME, false>;
  }
}

}  // namespace mlx
