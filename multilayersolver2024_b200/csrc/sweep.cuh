// sweep.cuh -- the colour sweep of projectGS as one launch, ordered by
// per-vertex versions instead of a launch (or a barrier) per colour.
//
// Every tet reads and writes each of its four vertices once per sweep, so the
// Gauss-Seidel order of the colours (xpbdLayer3D.m:357-378) is one chain per
// vertex: the tets at a vertex in colour order, each reading the record the
// one before it wrote.  A record carries its version in the same 16-byte word
// as the position; a tet polls the four records until they hold the versions
// it needs, projects, and writes the next versions.  The 16-byte accesses are
// single (ld / st.relaxed.gpu.b128), so position and version arrive together
// and no fence, barrier or launch separates the colours.  Each version of a
// record is read by exactly one tet (the next writer), so nothing is
// overwritten before it was read.
//
// Versions: with D the largest number of the layer's tets at a vertex, the
// tet of rank k at a vertex waits in iteration `it` for tag
// base + it D + k and leaves base + it D + k + 1; the vertex's last tet leaves
// base + (it + 1) D, what rank 0 of the next iteration waits for.  Rank 0 of
// the first iteration reads the position array and the last tet of the last
// iteration writes it, so a launch begins and ends with the position array
// and the records are scratch.  `base` lives on the device and grows by
// iterations * D per launch, so a tag left by an earlier launch never matches
// (before the 32-bit counter wraps the last CTA clears the records).
//
// The layer's tets are cut into chunks of 32 of one colour, in colour order,
// dealt to the CTAs in turn; chunk j of a CTA is warp j mod nw's in every
// iteration, so a tet's multipliers stay with one thread.  All CTAs are
// resident (cooperative launch) and each warp works in order, so the first
// unfinished chunk can always run.  At most `gate` chunks of a CTA wait for
// records at a time (in order): polls of records that are far from ready only
// slow the others down.  A wait that lasts kWaitNs sets the error flag and
// ends the launch.
//
// What bounds it: the chain of a vertex, one projection (~1,200 cycles) and
// one way through L2 (~2,000 cycles under load) per tet.  For components that
// would keep one cluster of flow.cuh busy longer: 393,216 Neo-Hookean tets in
// FP32 take 75 us per sweep of a fixed loop here, 96 with a launch per colour,
// 138 on one cluster; one iteration per launch (a monitored loop, its monitor
// included) 97, 96 and 172, so that takes the colour launches; FP64 147, 128
// and 201 (three words a record), so FP64 does not come here.  Above 1.3 M tets
// the records and rest data leave L2 (3.5 M: 290, colours 218).  Variants on
// the 393,216, the sweeps alone (62 us): chunks of 16 tets 81, records padded
// to a sector or a line 62 to 72, a pause between polls +2.
#pragma once

#include "common.cuh"
#include "persistent.cuh"
#include "tet_kernels.cuh"

namespace mlx {

constexpr int kSweepThreads = 256;
// corner word: rank of the tet among the layer's tets at the vertex, in
// colour order; kSweepLast marks the vertex's last tet, kSweepPinned a vertex
// with pinned DOFs
constexpr int kSweepLast = 0x8000, kSweepPinned = 0x4000, kSweepRank = 0x3fff;
// launches whose tags could span more than this take the colour launches
constexpr long long kSweepMaxTags = 1ll << 28;

// one vertex's record: (x, y, z, tag), or for FP64 three words (value, tag)
template <typename R> struct SweepRec;
template <> struct SweepRec<float> {
  ulonglong2 w;
};
template <> struct SweepRec<double> {
  ulonglong2 w[3];
};

struct SweepState {
  unsigned base, ticket;
};

template <typename R> struct SweepArgs {
  const int2* chunks;       // [n_chunks] first position in the list (sorted id if no list), tets
  const int* list;          // layer's elastic tets, NULL = identity
  const ushort4* corner;    // [T] corner words, sorted ids
  const R4<R>* minv;        // [T] inverse masses of the corners, sorted ids
  SweepRec<R>* rec;         // [N]
  SweepState* state;
  int* error;
  const int* pin_at;        // [3N] index into pin_vals or -1
  const R* pin_vals;
  int n_chunks, iterations, D, N;
  int gate;                 // chunks of a CTA that may wait for records at a time
  int pins;                 // apply the pinned DOFs at the end of every iteration
};

__device__ __forceinline__ void sweep_st(ulonglong2* p, unsigned long long lo, unsigned long long hi) {
  asm volatile("{.reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t;}" ::"l"(p), "l"(lo), "l"(hi)
               : "memory");
}

// the four records' words of a poll, loaded together where `need` has the
// corner's bit
__device__ __forceinline__ void sweep_ld4(const ulonglong2* p0, const ulonglong2* p1, const ulonglong2* p2,
                                          const ulonglong2* p3, unsigned need, ulonglong2 (&w)[4]) {
  asm volatile(
      "{.reg .pred a, b, c, d; .reg .b128 t0, t1, t2, t3; .reg .b32 m;\n"
      "and.b32 m, %12, 1; setp.ne.u32 a, m, 0;\n"
      "and.b32 m, %12, 2; setp.ne.u32 b, m, 0;\n"
      "and.b32 m, %12, 4; setp.ne.u32 c, m, 0;\n"
      "and.b32 m, %12, 8; setp.ne.u32 d, m, 0;\n"
      "mov.b128 t0, {%0, %1}; mov.b128 t1, {%2, %3}; mov.b128 t2, {%4, %5}; mov.b128 t3, {%6, %7};\n"
      "@a ld.relaxed.gpu.global.b128 t0, [%8];\n"
      "@b ld.relaxed.gpu.global.b128 t1, [%9];\n"
      "@c ld.relaxed.gpu.global.b128 t2, [%10];\n"
      "@d ld.relaxed.gpu.global.b128 t3, [%11];\n"
      "mov.b128 {%0, %1}, t0; mov.b128 {%2, %3}, t1; mov.b128 {%4, %5}, t2; mov.b128 {%6, %7}, t3;}"
      : "+l"(w[0].x), "+l"(w[0].y), "+l"(w[1].x), "+l"(w[1].y), "+l"(w[2].x), "+l"(w[2].y), "+l"(w[3].x), "+l"(w[3].y)
      : "l"(p0), "l"(p1), "l"(p2), "l"(p3), "r"(need)
      : "memory");
}

// Bounded wait of a whole warp: false once the wait has lasted kWaitNs or
// another one has.
__device__ __forceinline__ bool sweep_wait_on(unsigned spins, unsigned long long& t0, int* error) {
  if ((spins & 1023u) != 0) return true;
  bool over = *reinterpret_cast<volatile int*>(error) != 0;
  const unsigned long long t = global_ns();
  if (t0 == 0) t0 = t;
  if (t - t0 > kWaitNs) {
    atomicExch(error, 1);
    over = true;
  }
  return !__any_sync(0xffffffffu, over);
}

// Waits until more than `after` chunks of this CTA have their records.
__device__ __forceinline__ bool sweep_turn(const int* turn, int after, int* error) {
  unsigned spins = 0;
  unsigned long long t0 = 0;
  while (__any_sync(0xffffffffu, *reinterpret_cast<const volatile int*>(turn) <= after))
    if (!sweep_wait_on(++spins, t0, error)) return false;
  return true;
}

// Waits for the records of the corners in `need` to reach their tags.
__device__ __forceinline__ bool sweep_acquire(const SweepRec<float>* rec, const int4& v, const unsigned (&want)[4],
                                              unsigned need, V3<float> (&X)[4], int* error) {
  ulonglong2 w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = make_ulonglong2(0, 0);
  const unsigned got0 = need;
  unsigned spins = 0;
  unsigned long long t0 = 0;
  while (__any_sync(0xffffffffu, need != 0)) {
    sweep_ld4(&rec[v.x].w, &rec[v.y].w, &rec[v.z].w, &rec[v.w].w, need, w);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if ((unsigned)(w[k].y >> 32) == want[k]) need &= ~(1u << k);
    if (!sweep_wait_on(++spins, t0, error)) return false;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if ((got0 >> k) & 1u)
      X[k] = {__uint_as_float((unsigned)w[k].x), __uint_as_float((unsigned)(w[k].x >> 32)),
              __uint_as_float((unsigned)w[k].y)};
  return true;
}
__device__ __forceinline__ bool sweep_acquire(const SweepRec<double>* rec, const int4& v, const unsigned (&want)[4],
                                              unsigned need, V3<double> (&X)[4], int* error) {
  ulonglong2 w[3][4];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) w[c][k] = make_ulonglong2(0, 0);
  const unsigned got0 = need;
  unsigned n[3] = {need, need, need}, spins = 0;
  unsigned long long t0 = 0;
  while (__any_sync(0xffffffffu, (n[0] | n[1] | n[2]) != 0)) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      sweep_ld4(&rec[v.x].w[c], &rec[v.y].w[c], &rec[v.z].w[c], &rec[v.w].w[c], n[c], w[c]);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (w[c][k].y == want[k]) n[c] &= ~(1u << k);
    if (!sweep_wait_on(++spins, t0, error)) return false;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if ((got0 >> k) & 1u)
      X[k] = {__longlong_as_double(w[0][k].x), __longlong_as_double(w[1][k].x), __longlong_as_double(w[2][k].x)};
  return true;
}

__device__ __forceinline__ void sweep_release(SweepRec<float>* r, V3<float> x, unsigned tag) {
  sweep_st(&r->w, (unsigned long long)__float_as_uint(x.x) | ((unsigned long long)__float_as_uint(x.y) << 32),
           (unsigned long long)__float_as_uint(x.z) | ((unsigned long long)tag << 32));
}
__device__ __forceinline__ void sweep_release(SweepRec<double>* r, V3<double> x, unsigned tag) {
  sweep_st(&r->w[0], __double_as_longlong(x.x), tag);
  sweep_st(&r->w[1], __double_as_longlong(x.y), tag);
  sweep_st(&r->w[2], __double_as_longlong(x.z), tag);
}

// k_sweep of a precision and material (flow_fp32.cu, flow_fp64.cu).
const void* sweep_kernel_fp32(int mat_kind, bool damp);
const void* sweep_kernel_fp64(int mat_kind, bool damp);
inline const void* sweep_kernel(bool fp64, int mat_kind, bool damp) {
  return fp64 ? sweep_kernel_fp64(mat_kind, damp) : sweep_kernel_fp32(mat_kind, damp);
}

}  // namespace mlx
