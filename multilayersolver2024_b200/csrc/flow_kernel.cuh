// flow_kernel.cuh -- the kernel of flow.cuh (instantiated by flow_fp32.cu and
// flow_fp64.cu, one translation unit each).
#pragma once

#include "flow.cuh"

namespace mlx {

// `iterations` sweeps of one layer's elastic tets.  Dynamic shared memory:
// a.slots records, then an mbarrier per chunk.  CT: with device-detected
// contacts.
template <typename R, int MAT, bool DAMP, bool CT>
__global__ void __launch_bounds__(flow_threads<R>(), 1)
    k_flow(TetData<R> td, FlowArgs<R> a, R4<R>* __restrict__ pos, const R4<R>* __restrict__ oldp, R inv_h2, R inv_h,
           DevContacts dc) {
  constexpr uint32_t kRec = sizeof(R4<R>);
  extern __shared__ __align__(16) unsigned char fl_smem[];
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const unsigned rank = cluster_rank();
  const uint32_t rec = smem_u32(fl_smem), bars = rec + (uint32_t)a.slots * kRec;
  const int q0 = a.part_off[blockIdx.x], mine = a.part_off[blockIdx.x + 1] - q0;
  for (int j = threadIdx.x; j < mine; j += blockDim.x) {
    const int4 ch = a.chunks[q0 + j];
    const unsigned local = ch.w & 0xffff, none = (unsigned)ch.w >> 16;
    flow_bar_init(bars + 8 * j, 1 + local);
    if (none) flow_arrive(bars + 8 * j, none);
    flow_arm(bars + 8 * j, (unsigned)ch.z * kRec);
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  cluster_arrive();
  cluster_wait();
  const int T = td.T;
  bool ok = true;
  for (int it = 0; it < a.iterations && ok; ++it) {
    const bool first = it == 0, final = it + 1 == a.iterations;
    for (int j = threadIdx.x >> 5; j < mine; j += nw) {
      const int4 ch = a.chunks[q0 + j];
      const int n = ch.y;
      const bool active = lane < n;
      // (the lanes past the end load the chunk's last tet and write nothing)
      const int i = ch.x + min(lane, n - 1), s = a.list ? a.list[i] : i;
      TetRest<R, MAT> r;
      load_rest<R, MAT>(td, s, r);
      const FlowCorner fc = a.corner[s];
      const int vk[4] = {r.v.x, r.v.y, r.v.z, r.v.w};
      ok = flow_wait(bars + 8 * j, it & 1, a.error);
      if (!ok) break;
      // (no record of the next phase can arrive before this warp's results leave)
      if (lane == 0 && !final) flow_arm(bars + 8 * j, (unsigned)(4 * n - (ch.w & 0xffff)) * kRec);
      R4<R> p[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (first && (fc.c[k].x & (kFlowFirst << 16))) p[k] = ldcg_r4(pos + vk[k]);
        else p[k] = flow_ld(rec + (fc.c[k].x & 0xffffu) * kRec, R());
      }
      __syncwarp();
      if (active) {
        if (CT) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (fc.c[k].x & (kFlowBefore << 16)) flow_contacts<R>(dc, vk[k], p[k], oldp, a.h, a.contact_resistance);
        }
        V3<R> X[4];
        R minv[4], lnew[num_lambda<MAT>()];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          X[k] = {p[k].x, p[k].y, p[k].z};
          minv[k] = p[k].w;
        }
        tet_update<R, MAT, DAMP>(r, X, minv, oldp, inv_h2, inv_h, lnew);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          p[k] = make_r4<R>(X[k].x, X[k].y, X[k].z, minv[k]);
          const unsigned word = fc.c[k].x >> 16, to = fc.c[k].y;
          if (word & kFlowLast) {
            if (CT && (word & (a.after == 1 ? kFlowFree : kFlowAfter)))
              flow_contacts<R>(dc, vk[k], p[k], oldp, a.h, a.contact_resistance);
            if (a.pins && (word & kFlowPinned)) {
              // xi(pinnedDOFs) = pinnedx (xpbdLayer3D.m:333)
              const int* pa = a.pin_at + 3 * (size_t)vk[k];
              if (pa[0] >= 0) p[k].x = a.pin_vals[pa[0]];
              if (pa[1] >= 0) p[k].y = a.pin_vals[pa[1]];
              if (pa[2] >= 0) p[k].z = a.pin_vals[pa[2]];
            }
            if (final) {
              stcg_r4(pos + vk[k], p[k]);
              continue;
            }
          }
          const uint32_t dst = rec + (to & 0x3fffu) * kRec, bar = bars + ((to >> 14) & 0x3fffu) * 8;
          if ((to >> 28) == rank) {
            flow_st(dst, p[k]);
            flow_arrive(bar, 1);
          } else {
            flow_push(mapa_rank(dst, to >> 28), mapa_rank(bar, to >> 28), p[k]);
          }
        }
#pragma unroll
        for (int l = 0; l < num_lambda<MAT>(); ++l) td.lambda[(size_t)l * T + s] = lnew[l];
      }
      __syncwarp();
    }
  }
  // no CTA leaves while another may still write into its shared memory
  cluster_arrive();
  cluster_wait();
}

template <typename R, bool CT> static const void* flow_kernel_of(int mat_kind, bool damp) {
  switch (mat_kind) {
    case MAT_NH: return (const void*)k_flow<R, MAT_NH, false, CT>;
    case MAT_STVK_BLOCKS:
      return damp ? (const void*)k_flow<R, MAT_STVK_BLOCKS, true, CT> : (const void*)k_flow<R, MAT_STVK_BLOCKS, false, CT>;
    default:
      return damp ? (const void*)k_flow<R, MAT_STVK_LAME, true, CT> : (const void*)k_flow<R, MAT_STVK_LAME, false, CT>;
  }
}

}  // namespace mlx
