// flow.cuh -- the projectGS loop of one layer as a dataflow over vertex
// versions, records pushed through (distributed) shared memory.
//
// Every tet reads and writes each of its four vertices once per sweep, so the
// Gauss-Seidel order of the colours (xpbdLayer3D.m:357-378) is one chain per
// vertex: the tets at a vertex in colour order, each reading the record the
// one before it wrote.  Here a tet writes its four corners straight into the
// shared memory of the CTA that projects each vertex's next tet, and every
// store counts on an mbarrier of the chunk of 32 tets that the next tet
// belongs to: a store and an arrive inside the CTA, st.async and its bytes
// across CTAs.  A warp sleeps on its chunk's mbarrier until all of the chunk's
// records are there: no barrier, fence, poll or launch separates the colours,
// and colours overlap wherever the vertices allow.
//
// Layout.  The mesh's elements are cut into G groups of whole connected
// components, one thread-block cluster of CS CTAs each, and a group's
// elements into CS parts, one per CTA rank.  A CTA has one slot (x, y, z, 1/m)
// per vertex its tets touch.  A vertex's versions form one chain, so a slot is
// never overwritten before it was read.  Per layer and corner the host fixes
// the slot that is read, the rank, slot and chunk of the vertex's next tet and
// the corner word (below).  A vertex's first tet of the first iteration reads
// the position array and its last tet of the last iteration writes it, so a
// launch begins and ends there.
//
// A CTA's tets are cut into chunks of at most 32 of one colour, in colour
// order; chunk j is warp j mod nw's in every iteration, so a tet's
// multipliers stay with one thread.  The CTAs of a cluster are co-scheduled
// and every warp works in order, so the first unfinished chunk can always
// run.  A chunk's barrier is armed for iteration it + 1 before iteration it's
// results leave the warp, and whatever arrives for it + 1 depends on those.
// A wait that lasts kWaitNs sets the error flag and ends the launch.
//
// What bounds it: a vertex's chain, one projection (~1,200 cycles for a
// Neo-Hookean tet), its stores' way to the next CTA and the wake-up per tet,
// ~0.9 us per colour on meshes whose chunks leave the SMs idle; above ~100
// chunks per CTA the warps share the SM (~250 cycles per chunk).  Whole
// recorded steps, us per sweep of this path / colour launches (B200,
// Neo-Hookean FP32): 27,648 tets on 16 CTAs 33 / 61, 98,304 tets 43 / 68;
// other sizes, materials and precisions: sweep_times.h.  Variants, the sweeps
// alone: polling the records' versions instead of mbarriers 33 us against 29 on
// the 27,648 tets (the polls take the shared-memory pipe from the
// projections), st.async inside the CTA too 45 against 41 on the 98,304 (it
// goes out to the network and back), the rest data gathered per tet instead of
// read from chunk planes 58 against 41 there.
// Bulk copies of the rest data into shared memory and prefetches of the next
// chunk's lines into L1 or L2 gave nothing, two or four smaller CTAs per SM
// neither.
//
// The per-vertex phases of an iteration join the chain: the contacts of a
// vertex run where their phase falls between two of its tets (before the tet
// that follows, or after the last), the pinned DOFs after the last.
#pragma once

#include "cluster.cuh"
#include "common.cuh"
#include "contacts.cuh"
#include "persistent.cuh"
#include "tet_kernels.cuh"

namespace mlx {

template <typename R> __host__ __device__ constexpr int flow_threads() { return sizeof(R) == 4 ? 512 : 256; }
// corner word, marks of the vertex at this tet: first and last of the layer's
// tets at the vertex (in colour order), pinned DOFs, contacts before this tet
// or after it (contact colouring), no body
constexpr unsigned kFlowFirst = 1, kFlowLast = 2, kFlowPinned = 4, kFlowBefore = 8, kFlowAfter = 16, kFlowFree = 32;
constexpr int kFlowMaxSlots = 1 << 14, kFlowMaxChunks = 1 << 14;

constexpr int kFlowChunkPins = 64;  // a pinned vertex's last tet is in the chunk

// corner of a tet: x = slot it is read from | corner word << 16, y = where the
// vertex's next tet reads it: rank << 28 | chunk << 14 | slot
struct FlowCorner {
  uint2 c[4];
};

// Rest data of a tet in the chunk planes: DmInv (9), for StVK the corners'
// inverse masses (4) and the volume, then the material.
template <int MAT> __host__ __device__ constexpr int flow_planes() {
  return ((MAT == MAT_NH ? 9 : 14) + mat_stride(MAT) + 3) / 4;
}
inline int flow_planes_of(int mat) {
  switch (mat) {
    case MAT_NH: return flow_planes<MAT_NH>();
    case MAT_STVK_ISO: return flow_planes<MAT_STVK_ISO>();
    case MAT_STVK_BLOCKS: return flow_planes<MAT_STVK_BLOCKS>();
    default: return flow_planes<MAT_STVK_LAME>();
  }
}

template <typename R> struct FlowArgs {
  const int* part_off;      // [G CS + 1] chunks of each part
  // first position in the list (sorted id if no list); tets, kFlowChunkPins, colour << 8;
  // records that other CTAs send for iteration 0; records that come from this
  // CTA, those of them that no tet sends for iteration 0 << 16
  const int4* chunks;
  const int* list;          // layer's elastic tets, NULL = identity
  // per chunk, lane-interleaved planes of 32 vectors: rest data
  // (flow_planes), corners (2 planes) and vertex ids
  const R4<R>* rest;
  const uint4* corner;
  const int4* vid;
  R* lambda;                // [chunk][multiplier][32] between the first and the last iteration
  const int* pin_at;        // [3N] index into pin_vals or -1
  const R* pin_vals;
  int* error;
  int cs, slots, iterations;
  int pins;                 // apply the pinned DOFs at the end of every iteration
  int after;                // contacts after the last tet: 0 none, 1 all, 2 those marked kFlowAfter
  double h, contact_resistance;
};

// Sends a record to slot address `a` of CTA `to` of the cluster and counts it
// on the mbarrier at `bar` there: a store and an arrive inside this CTA,
// st.async and its bytes otherwise (predicated: the lanes of a warp differ,
// and two branches per corner cost more than the instructions).
__device__ __forceinline__ void flow_send(uint32_t a, uint32_t bar, unsigned to, unsigned rank, float4 v) {
  asm volatile(
      "{.reg .pred l; .reg .b32 ra, rb;\n"
      "setp.eq.u32 l, %6, %7;\n"
      "@l st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n"
      "@l mbarrier.arrive.release.cta.shared::cta.b64 _, [%5], 1;\n"
      "@!l mapa.shared::cluster.u32 ra, %0, %6;\n"
      "@!l mapa.shared::cluster.u32 rb, %5, %6;\n"
      "@!l st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [ra], {%1, %2, %3, %4}, [rb];}" ::"r"(a),
      "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar), "r"(to), "r"(rank)
      : "memory");
}
__device__ __forceinline__ void flow_send(uint32_t a, uint32_t bar, unsigned to, unsigned rank, double4 v) {
  asm volatile(
      "{.reg .pred l; .reg .b32 ra, rb;\n"
      "setp.eq.u32 l, %6, %7;\n"
      "@l st.shared.v2.f64 [%0], {%1, %2};\n"
      "@l st.shared.v2.f64 [%0 + 16], {%3, %4};\n"
      "@l mbarrier.arrive.release.cta.shared::cta.b64 _, [%5], 1;\n"
      "@!l mapa.shared::cluster.u32 ra, %0, %6;\n"
      "@!l mapa.shared::cluster.u32 rb, %5, %6;\n"
      "@!l st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [ra], {%1, %2}, [rb];\n"
      "@!l st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [ra + 16], {%3, %4}, [rb];}" ::"r"(a),
      "d"(v.x), "d"(v.y), "d"(v.z), "d"(v.w), "r"(bar), "r"(to), "r"(rank)
      : "memory");
}
__device__ __forceinline__ void flow_bar_init(uint32_t bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void flow_arrive(uint32_t bar, unsigned n) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
// completes the barrier's phase once `bytes` have arrived in it
__device__ __forceinline__ void flow_arm(uint32_t bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool flow_try(uint32_t bar, unsigned parity) {
  unsigned ok;
  asm volatile("{.reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
__device__ __forceinline__ float4 flow_ld(uint32_t a, float) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double4 flow_ld(uint32_t a, double) {
  double4 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.z), "=d"(v.w) : "r"(a + 16) : "memory");
  return v;
}

// Waits (a whole warp) for the phase of a chunk's records, at most kWaitNs;
// false when it gave up or another wait has.
__device__ __forceinline__ bool flow_wait(uint32_t bar, unsigned parity, int* error) {
  unsigned spins = 0;
  unsigned long long t0 = 0;
  while (!__all_sync(0xffffffffu, flow_try(bar, parity))) {
    if ((++spins & 63u) != 0) continue;
    bool over = *reinterpret_cast<volatile int*>(error) != 0;
    const unsigned long long t = global_ns();
    if (t0 == 0) t0 = t;
    if (t - t0 > kWaitNs) {
      atomicExch(error, 1);
      over = true;
    }
    if (__any_sync(0xffffffffu, over)) return false;
  }
  return true;
}

// A vertex record in registers, for the contact projection.
template <typename R> struct FlowPos {
  R4<R>* p;
  __device__ __forceinline__ R4<R> ld(int) const { return *p; }
  __device__ __forceinline__ void st(int, R4<R> x) const { *p = x; }
};

// What the contact of one corner does not need the record for, gathered while
// the warp waits: the chain of loads (index, mask, step-start position,
// obstacle, multiplier) and the contact's geometry took ~2,000 cycles after
// the record had arrived.  Covers the tet's first marked corner; k < 0: none,
// i < 0: no contact, `one`: a single obstacle (n, c, aT and lam hold).
struct FlowContact {
  int k, i, f, one;
  D3 n, c;
  double aT, lam;
};
template <typename R>
__device__ __forceinline__ FlowContact flow_contact_ahead(const DevContacts& dc, unsigned m, const int (&vk)[4],
                                                          const R4<R>* __restrict__ x0, double h) {
  FlowContact a;
  a.k = -1;
  a.i = -1;
  a.f = a.one = 0;
  a.n = a.c = d3(0, 0, 0);
  a.aT = a.lam = 0;
  if (!m) return a;
  a.k = __ffs(m) - 1;
  const int v = a.k == 0 ? vk[0] : a.k == 1 ? vk[1] : a.k == 2 ? vk[2] : vk[3];
  a.i = dc.cidx[v];
  if (a.i < 0) return a;
  const unsigned mask = dc.mask[v];
  const R4<R> s = x0[v];
  a.f = __ffs(mask) - 1;
  a.one = (mask & (mask - 1)) == 0;
  if (!a.one) return a;
  double comp;
  obstacle_contact(dc.obs[a.f], (double)s.x, (double)s.y, (double)s.z, a.n, a.c, comp);
  a.aT = comp / (h * h);
  a.lam = dc.lambda[(size_t)a.i * dc.nobs + a.f];
  return a;
}

// The device-detected elastic contacts of the corners marked in m.  One
// corner of a tet at a time, whichever it is: the lanes of a warp rarely mark
// more than one, and a pass per corner index would run the projection four
// times.
template <typename R>
__device__ __forceinline__ void flow_contacts(const DevContacts& dc, unsigned m, const FlowContact& a,
                                              const int (&vk)[4], R4<R> (&p)[4], const R4<R>* __restrict__ x0, double h,
                                              double resistance) {
  while (m) {
    const int k = __ffs(m) - 1;
    m &= m - 1;
    const int v = k == 0 ? vk[0] : k == 1 ? vk[1] : k == 2 ? vk[2] : vk[3];
    const int i = k == a.k ? a.i : dc.cidx[v];
    if (i < 0) continue;
    R4<R> q = k == 0 ? p[0] : k == 1 ? p[1] : k == 2 ? p[2] : p[3];
    if (k == a.k && a.one) {
      // elastic_contacts_of_vertex with one obstacle
      const D3 x = d3((double)q.x, (double)q.y, (double)q.z);
      const double minv = (double)q.w;
      double phi = dot(a.n, x - a.c);
      if (phi > 0) phi = 0;
      const double C = resistance * phi;
      const double dl = (-C - a.aT * a.lam) / (2 * minv + a.aT);
      dc.lambda[(size_t)i * dc.nobs + a.f] = a.lam + dl;
      const D3 xn = d3(x.x + minv * (dl * a.n.x), x.y + minv * (dl * a.n.y), x.z + minv * (dl * a.n.z));
      q = make_r4<R>((R)xn.x, (R)xn.y, (R)xn.z, q.w);
    } else {
      elastic_contacts_of_vertex<R>(dc, i, FlowPos<R>{&q}, x0, h, resistance);
    }
    if (k == 0) p[0] = q;
    if (k == 1) p[1] = q;
    if (k == 2) p[2] = q;
    if (k == 3) p[3] = q;
  }
}

// k_flow_pack of a precision and material: fills the chunk planes.
const void* flow_pack_kernel_fp32(int mat_kind);
const void* flow_pack_kernel_fp64(int mat_kind);
inline const void* flow_pack_kernel(bool fp64, int mat_kind) {
  return fp64 ? flow_pack_kernel_fp64(mat_kind) : flow_pack_kernel_fp32(mat_kind);
}
// k_flow of a precision and material (flow_fp32.cu, flow_fp64.cu); `ct`: with
// device-detected contacts, `small`: at most 256 threads (FP32: twice the
// registers, none spilled; StVK with contacts always so).
const void* flow_kernel_fp32(int mat_kind, bool damp, bool ct, bool small);
const void* flow_kernel_fp64(int mat_kind, bool damp, bool ct);
inline const void* flow_kernel(bool fp64, int mat_kind, bool damp, bool ct, bool small) {
  return fp64 ? flow_kernel_fp64(mat_kind, damp, ct) : flow_kernel_fp32(mat_kind, damp, ct, small);
}

}  // namespace mlx
