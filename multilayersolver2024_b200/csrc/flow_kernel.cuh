// flow_kernel.cuh -- the kernel of flow.cuh (instantiated by flow_fp32.cu and
// flow_fp64.cu, one translation unit each).
#pragma once

#include "flow.cuh"

namespace mlx {

// `iterations` sweeps of one layer's elastic tets.  Dynamic shared memory:
// a.slots records, then an mbarrier per chunk.  CT: with device-detected
// contacts.
template <typename R, int MAT, bool DAMP, bool CT, int TH>
__global__ void __launch_bounds__(TH, 1)
    k_flow(TetData<R> td, FlowArgs<R> a, R4<R>* __restrict__ pos, const R4<R>* __restrict__ oldp, R inv_h2, R inv_h,
           DevContacts dc) {
  pdl_launch_dependents();
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
  pdl_wait();  // (so far only what the layer's build wrote has been read)
  const int T = td.T;
  bool ok = true;
  for (int it = 0; it < a.iterations && ok; ++it) {
    const bool first = it == 0, final = it + 1 == a.iterations;
    for (int j = threadIdx.x >> 5; j < mine; j += nw) {
      const int4 ch = a.chunks[q0 + j];
      const int n = ch.y & 63;
      const bool active = lane < n;
      // (the planes repeat the chunk's last tet past the end)
      const size_t q = (size_t)(q0 + j);
      int s = 0;
      if (first || final) {
        const int i = ch.x + min(lane, n - 1);
        s = a.list ? a.list[i] : i;
      }
      TetRest<R, MAT> r;
      StvkPre<R> pre;
      {
        constexpr int P = flow_planes<MAT>();
        const R4<R>* rp = a.rest + q * (P * 32) + lane;
        R w[4 * P];
#pragma unroll
        for (int c = 0; c < P; ++c) {
          const R4<R> v = rp[32 * c];
          w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
        }
#pragma unroll
        for (int c = 0; c < 9; ++c) r.G[c] = w[c];
        constexpr int m0 = MAT == MAT_NH ? 9 : 14;
#pragma unroll
        for (int c = 0; c < mat_stride(MAT); ++c) r.mat[c] = w[m0 + c];
        if constexpr (MAT != MAT_NH) {
          const R m[4] = {w[9], w[10], w[11], w[12]};
          r.vol = w[13];
          stvk_pre<R>(m, r.G, pre);
        }
      }
      FlowCorner fc;
      {
        const uint4 c0 = a.corner[q * 64 + lane], c1 = a.corner[q * 64 + 32 + lane];
        fc.c[0] = make_uint2(c0.x, c0.y);
        fc.c[1] = make_uint2(c0.z, c0.w);
        fc.c[2] = make_uint2(c1.x, c1.y);
        fc.c[3] = make_uint2(c1.z, c1.w);
      }
      r.v = make_int4(0, 0, 0, 0);
      const bool pins = a.pins && (ch.y & kFlowChunkPins);
      if (first || final || CT || DAMP || pins) r.v = a.vid[q * 32 + lane];
      const int vk[4] = {r.v.x, r.v.y, r.v.z, r.v.w};
      R* lam = first ? td.lambda + s : a.lambda + q * (32 * num_lambda<MAT>()) + lane;
      const size_t ls = first ? (size_t)T : 32;
#pragma unroll
      for (int l = 0; l < num_lambda<MAT>(); ++l) r.lam[l] = lam[l * ls];
      // what does not depend on the records: the first tets' positions, and
      // the pinned values brought close
      R4<R> p[4];
      if (first) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (fc.c[k].x & (kFlowFirst << 16)) p[k] = ldcg_r4(pos + vk[k]);
      }
      if (pins) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if ((fc.c[k].x & (kFlowLast << 16)) && (fc.c[k].x & (kFlowPinned << 16))) {
            const int* pa = a.pin_at + 3 * (size_t)vk[k];
            const int i0 = max(max(pa[0], pa[1]), pa[2]);
            asm volatile("prefetch.global.L1 [%0];" ::"l"(a.pin_vals + i0));
          }
      }
      unsigned mb = 0, ma = 0;  // corners with contacts before / after the projection
      FlowContact ahead;
      if (CT) {
        const unsigned mark = a.after == 1 ? kFlowFree : kFlowAfter;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned word = fc.c[k].x >> 16;
          if (a.after == 2 && (word & kFlowBefore)) mb |= 1u << k;
          if ((word & kFlowLast) && (word & mark)) ma |= 1u << k;
        }
        ahead = flow_contact_ahead<R>(dc, active ? mb | ma : 0, vk, oldp, a.h);
      }
      ok = flow_wait(bars + 8 * j, it & 1, a.error);
      if (!ok) break;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (!first || !(fc.c[k].x & (kFlowFirst << 16))) p[k] = flow_ld(rec + (fc.c[k].x & 0xffffu) * kRec, R());
      // (no record of the next phase can arrive before this warp's results leave)
      if (lane == 0 && !final) flow_arm(bars + 8 * j, (unsigned)(4 * n - (ch.w & 0xffff)) * kRec);
      __syncwarp();
      if (active) {
        if (CT && mb) flow_contacts<R>(dc, mb, ahead, vk, p, oldp, a.h, a.contact_resistance);
        V3<R> X[4];
        R minv[4], lnew[num_lambda<MAT>()];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          X[k] = {p[k].x, p[k].y, p[k].z};
          minv[k] = p[k].w;
        }
        tet_update<R, MAT, DAMP>(r, X, minv, oldp, inv_h2, inv_h, lnew, &pre);
#pragma unroll
        for (int k = 0; k < 4; ++k) p[k] = make_r4<R>(X[k].x, X[k].y, X[k].z, minv[k]);
        if (CT && ma) flow_contacts<R>(dc, ma, ahead, vk, p, oldp, a.h, a.contact_resistance);
        if (pins) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if ((fc.c[k].x & (kFlowLast << 16)) && (fc.c[k].x & (kFlowPinned << 16))) {
              // xi(pinnedDOFs) = pinnedx (xpbdLayer3D.m:333)
              const int* pa = a.pin_at + 3 * (size_t)vk[k];
              if (pa[0] >= 0) p[k].x = a.pin_vals[pa[0]];
              if (pa[1] >= 0) p[k].y = a.pin_vals[pa[1]];
              if (pa[2] >= 0) p[k].z = a.pin_vals[pa[2]];
            }
        }
        if (final) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned to = fc.c[k].y;
            if (fc.c[k].x & (kFlowLast << 16)) stcg_r4(pos + vk[k], p[k]);
            else flow_send(rec + (to & 0x3fffu) * kRec, bars + ((to >> 14) & 0x3fffu) * 8, to >> 28, rank, p[k]);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned to = fc.c[k].y;
            flow_send(rec + (to & 0x3fffu) * kRec, bars + ((to >> 14) & 0x3fffu) * 8, to >> 28, rank, p[k]);
          }
        }
#pragma unroll
        for (int l = 0; l < num_lambda<MAT>(); ++l) {
          if (final) td.lambda[(size_t)l * T + s] = lnew[l];
          else a.lambda[q * (32 * num_lambda<MAT>()) + 32 * l + lane] = lnew[l];
        }
      }
      __syncwarp();
    }
  }
  // no CTA leaves while another may still write into its shared memory: every
  // record sent was waited for, unless a wait gave up -- then the stores in
  // flight get time to land once nothing sends any more
  cluster_arrive();
  cluster_wait();
  if (*reinterpret_cast<volatile int*>(a.error)) __nanosleep(200000);
}

// The rest and vertex planes of one layer: chunk blockIdx.x, lane threadIdx.x.
template <typename R, int MAT>
__global__ void __launch_bounds__(32) k_flow_pack(TetData<R> td, const int4* __restrict__ chunks,
                                                  const int* __restrict__ list, const double* __restrict__ mass3,
                                                  R4<R>* __restrict__ rest, int4* __restrict__ vid) {
  constexpr int P = flow_planes<MAT>(), m0 = MAT == MAT_NH ? 9 : 14;
  const int4 ch = chunks[blockIdx.x];
  const int lane = threadIdx.x, i = ch.x + min(lane, (ch.y & 63) - 1), s = list ? list[i] : i, T = td.T;
  const size_t q = blockIdx.x;
  R w[4 * P];
#pragma unroll
  for (int c = 0; c < 4 * P; ++c) w[c] = 0;
  const int4 v = td.vid[s];
#pragma unroll
  for (int c = 0; c < 9; ++c) w[c] = td.dminv[(size_t)c * T + s];
  if constexpr (MAT != MAT_NH) {
    w[9] = (R)(1.0 / mass3[3 * v.x]);
    w[10] = (R)(1.0 / mass3[3 * v.y]);
    w[11] = (R)(1.0 / mass3[3 * v.z]);
    w[12] = (R)(1.0 / mass3[3 * v.w]);
    w[13] = td.vol[s];
  }
#pragma unroll
  for (int c = 0; c < mat_stride(MAT); ++c) w[m0 + c] = td.mat[(size_t)c * T + s];
#pragma unroll
  for (int c = 0; c < P; ++c)
    rest[q * (P * 32) + 32 * c + lane] = make_r4<R>(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
  vid[q * 32 + lane] = v;
}

template <typename R> static const void* flow_pack_kernel_of(int mat_kind) {
  switch (mat_kind) {
    case MAT_NH: return (const void*)k_flow_pack<R, MAT_NH>;
    case MAT_STVK_ISO: return (const void*)k_flow_pack<R, MAT_STVK_ISO>;
    case MAT_STVK_BLOCKS: return (const void*)k_flow_pack<R, MAT_STVK_BLOCKS>;
    default: return (const void*)k_flow_pack<R, MAT_STVK_LAME>;
  }
}

template <typename R, bool CT, int TH> static const void* flow_kernel_of(int mat_kind, bool damp) {
  switch (mat_kind) {
    case MAT_NH: return (const void*)k_flow<R, MAT_NH, false, CT, TH>;
    case MAT_STVK_ISO: return (const void*)k_flow<R, MAT_STVK_ISO, false, CT, TH>;
    case MAT_STVK_BLOCKS:
      return damp ? (const void*)k_flow<R, MAT_STVK_BLOCKS, true, CT, TH>
                  : (const void*)k_flow<R, MAT_STVK_BLOCKS, false, CT, TH>;
    default:
      return damp ? (const void*)k_flow<R, MAT_STVK_LAME, true, CT, TH>
                  : (const void*)k_flow<R, MAT_STVK_LAME, false, CT, TH>;
  }
}

}  // namespace mlx
