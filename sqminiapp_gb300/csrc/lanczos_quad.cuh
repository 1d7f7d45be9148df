// lanczos_quad.cuh -- FP32 Lanczos kernel with split stencil passes over aligned quads.
//
// Same recurrence and operator as lanczos_kernel.cuh (src/lsdft_scf.cc:119-147 with
// H = -1/2 Lap (12th-order FD, Dirichlet cube, src/lsdft_initObjs.cc:393-475) + diag(Veff)
// + the Kleinman-Bylander projectors of the atom images that meet the cube,
// src/lsdft_matvec.cc:25-149); FP32 vectors, corrected operator, full projector records.
//
// Layout.  P and U are both [nz][ny][pitch] floats in shared memory, pitch = 4*ceil(nx/4),
// planes a multiple of all banks apart (quad_plane_floats): every row starts on a 16-byte boundary
// and holds whole float4 quads; the pad columns [nx, pitch) and plane pads stay zero.  There are no
// zero rows or columns between rows: neighbours outside the cube are never loaded (x: the quad loads
// are predicated off at the row ends; y and z: a quad of zeros stands for them).  A point's P and U
// indices are the same, z*PS + y*pitch + x.
//
// Stencil, split by axis so that two of the three axes come from registers:
//   pass A  a thread owns one quad (x..x+3) of row y over a z-range and walks z with a
//           13-plane register ring (one float4 load per plane); the x neighbours of the quad
//           are four aligned float4 loads of the same row; it adds the diagonal (Veff, read as
//           one aligned float4 from a quad-aligned copy of the padded potential; the stencil's
//           own diagonal is left out, see Scaling) and forms U <- s (Veff + Dz + Dx) P - gamma U;
//   pass B  a thread owns one quad of plane z over a y-range and walks y with a 13-row
//           register ring: U += s Dy P.
// Consecutive threads own consecutive quads in pass A; pass B's columns are dealt to the lanes by the
// bank they begin in: hardly any bank conflicts in either.
//
// Projector list.  Its unit is (image, column of quads, four planes): T_l of four quads above one
// another (zero outside the support), and one word with the image, the first plane and the place of
// the unit's partial sums; chi_lm = T_l P_lm(x,y,z) is formed while streaming, over a column with the
// same x and y for every plane.  A thread owns one column over a range of planes and all its units
// (dealt out by bank and number, so that the lanes of a warp have equally many and read eight banks at
// once): no two threads meet on a quad, the scatter needs no atomics, and every run gives the same result.  The list is built once per
// node and lives in the SM's tensor memory, which this kernel does not need for anything else
// (tcgen05.ld: no L2 round trip, no shared memory); what exceeds its 512 columns goes to a slice of
// global scratch.  The gather writes four (s+p) partial sums per unit, ordered by atom, to shared
// memory where they fit, else to the scratch slice.
//   Before, a list of points (20 bytes each) was streamed from L2 twice a step: 2 x 148 of 591
// instructions per quad-warp and step, and the atomics of the scatter.
//
// Per Lanczos step (v_k = s_k P with s_k a power of two, U = v_{k-1}), four CTA barriers:
//   1  projector gather c = chi^T P (partial sums per unit)  ||  pass A
//   2  pass B  ||  alpha = Gamma s c (and <P, V_nl P>)  -> per-warp partials of <P, H P>
//   3  projector scatter U += chi alpha  ||  every warp reduces the a_k partials
//   4  w = U - a_k v, P <- w, U <- v  -> per-warp partials of b_k^2
// After barrier 4 every warp reduces the b partials itself (the same tree in every warp, so
// every thread sees the same b_k and takes the same branch).  a_k and b_k^2 are summed per
// thread in FP32 with Kahan compensation, then across threads as double-float pairs (an FP32
// head and tail added with error-free transformations, about 48 bits of significand): GB300's
// FP64 pipe runs at a small fraction of its FP32 rate, so the step loop keeps FP64 out of its
// critical path and converts to double only to store a_k and b_k.
//
// Scaling.  The vector is never normalised: v_k = s_k P_k with s_k the power of two that brings
// |v_k| into [1, 2), so no element is rounded by the scaling, and
//   a_k = <P,HP> / |P|^2,   w = H v_k - a_k v_k - gamma_k v_{k-1},   P <- w,
//   b_k = |w| / |v_k|,      gamma_{k+1} = s_{k+1} |w|^2 / |v_k|^2
// with a_k and gamma_k as double-floats (head and tail applied).  Normalising by a rounded 1/b_k left
// |v_k| off by 1e-7 and so a_k by twice that of its 18 + V: that, not the stencil's rounding, was
// most of the FP32 error (weights 6e-6 -> 4e-7 and the lowest Ritz value 5e-7 -> 5e-8 Ha on a 27^3
// cube without projectors).  What was left came from the stencil's constant diagonal (18 at h = 0.5,
// where Veff is below 1): the start vector's H v and its a_0 were rounded at that size.  The recurrence
// runs on H - hshift, which has the same vectors, b_k and weights, and hshift is added to a_k in FP64.
// Restated on the CPU, 144 nodes of 27^3 and 40 steps: relative error of a node's weights 1.1e-6 -> 2.3e-7
// (root mean square), 2.6e-6 -> 5.6e-7 (largest), at no cost.
//
// Memory traffic.  Pass A reads Veff from L2 one plane ahead.  Nodes after the first round come
// from a device-side queue.
//
// CTA pair (PAIR, lanczos_quad_pair_kernel): one node per cluster of two CTAs for cubes whose
// P and U do not fit one CTA.  The cube is split in z (PairPlanes); each CTA owns its planes of
// U and of the list and holds P on its planes plus the 6 the z stencil reads from the peer's
// side, which the peer stores there in its update phase (distributed shared memory).  Barriers
// 2 and 4 become cluster barriers; c is exchanged per slot after phase 2 and a_k, b_k are
// summed from both CTAs' partials in rank order, so both CTAs take every branch together.
#pragma once

#include <cooperative_groups.h>

#include "lanczos_kernel.cuh"
#include "tc5.cuh"

namespace sq {
namespace lq {

using lk::O;
using lk::W;
using lk::kMaxWarps;

// Blackwell packed FP32 (PTX .f32x2, sm_100+): two lanes of float2 per instruction.
__device__ __forceinline__ unsigned long long as_u64(float2 a) {
  return *reinterpret_cast<unsigned long long *>(&a);
}
__device__ __forceinline__ float2 as_f2(unsigned long long r) {
  return *reinterpret_cast<float2 *>(&r);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {  // a*b + c
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(as_u64(a)), "l"(as_u64(b)), "l"(as_u64(c)));
  return as_f2(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(as_u64(a)), "l"(as_u64(b)));
  return as_f2(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(as_u64(a)), "l"(as_u64(b)));
  return as_f2(d);
}
__device__ __forceinline__ float2 lo(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 splat(float c) { return make_float2(c, c); }

// Shared memory by byte address (cvta_shared): whole quads, and loads that a lane may skip (the
// registers keep their values).  As C++ expressions the skipped loads of the stencil passes
// became real branches, and the moves around them a third of all issued instructions.
__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ float4 lds_quad(unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
// at a + OFS, the offset in the instruction
template <int OFS> __device__ __forceinline__ void lds_quad_if(bool on, unsigned a, float4 &v) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%4+%6];\n\t}"
      : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
      : "r"(a), "r"((int)on), "n"(OFS)
      : "memory");
}
template <int OFS> __device__ __forceinline__ void lds_pair_if(bool on, unsigned a, float2 &v) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\t@p ld.shared.v2.f32 {%0, %1}, [%2+%4];\n\t}"
      : "+f"(v.x), "+f"(v.y)
      : "r"(a), "r"((int)on), "n"(OFS)
      : "memory");
}
__device__ __forceinline__ void sts_quad_if(bool on, unsigned a, float4 v) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p st.shared.v4.f32 [%4], {%0, %1, %2, %3};\n\t}" ::"f"(v.x),
      "f"(v.y), "f"(v.z), "f"(v.w), "r"(a), "r"((int)on)
      : "memory");
}
// a quad of global memory, or zeros
__device__ __forceinline__ float4 ldg_quad_if(bool on, const float4 *g) {
  float4 v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
      "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
      : "l"(g), "r"((int)on));
  return v;
}

// Kahan-compensated FP32 running sum.
struct Kahan {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

// Double-float value hi + lo (|lo| <= ulp(hi)/2) and its sum (Knuth's TwoSum, then a
// renormalising FastTwoSum).
struct DF {
  float hi, lo;
};
__device__ __forceinline__ DF df_add(DF x, DF y) {
  const float s = x.hi + y.hi;
  const float bb = s - x.hi;
  float e = (x.hi - (s - bb)) + (y.hi - bb);
  e += x.lo + y.lo;
  const float h = s + e;
  return DF{h, e - (h - s)};
}
__device__ __forceinline__ DF df_of(const Kahan &k) {  // s - c, renormalised
  const float h = k.s - k.c;
  return DF{h, -k.c - (h - k.s)};
}
__device__ __forceinline__ DF df_warp_sum(DF v) {  // the same butterfly in every lane
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    DF w;
    w.hi = __shfl_xor_sync(0xffffffffu, v.hi, o);
    w.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
    v = df_add(v, w);
  }
  return v;
}
// Quotient of two double-floats as a double-float (relative error about 2^-45).
__device__ __forceinline__ DF df_div(DF x, DF y) {
  const float q = x.hi / y.hi;
  const float r = fmaf(-q, y.hi, x.hi) + (x.lo - q * y.lo);
  return DF{q, r / y.hi};
}
// The power of two s with s^2 n in [1, 4) (n a normal number above zero).
__device__ __forceinline__ float unit_scale(float n) {
  const int e = ((__float_as_int(n) >> 23) & 255) - 127;
  return __int_as_float((127 - (e >> 1)) << 23);
}
// Sum of nw per-warp partials red[0..nw), the same tree in every lane of every warp, so every
// thread gets the bit-identical total.
__device__ __forceinline__ DF df_all_reduce(const float2 *red, int nw) {
  const int lane = threadIdx.x & 31;
  const float2 r = lane < nw ? red[lane] : make_float2(0.f, 0.f);
  return df_warp_sum(DF{r.x, r.y});
}

// Floats per z-plane of P and U: ny rows of pitch, rounded up to all 32 banks, so that the bank of a
// quad is that of its column (8 classes of columns) whatever its plane.  A quarter-warp reads or
// writes its 8 quads at once if they are of 8 classes: the list's columns and pass B's are dealt to the
// lanes that way (bank_slot).  Dealt by their number of units alone, over planes whose banks follow
// on one another, a gather and a scatter of 27^3 took 7800 shared-memory wavefronts instead of 3450, of
// 29^3 12000 instead of 4700: 39304 nodes of 27^3 and 40 steps 191.8 -> 179.7 ms, 12001 of 29^3 and 50
// steps 114.4 -> 107.4 ms, 9001 of 33^3 on pairs 115.5 -> 110.7 ms (whole calls).
__host__ __device__ constexpr int quad_plane_floats(int ny, int pitch) {
  return (ny * pitch + 31) / 32 * 32;
}
// The thread of the rank-th column of bank class r: lane r of the rank-th group of 8; what a class has
// beyond the groups goes where others have fewer.  size(r): columns of class r, their sum <= 8 groups.
template <typename FN> __device__ __forceinline__ int bank_slot(int r, int rank, int groups, FN &&size) {
  if (rank < groups) return 8 * rank + r;
  int m = rank - groups;
  for (int i = 0; i < r; i++) m += max(0, size(i) - groups);
  for (int i = 0; i < 8; i++) {
    const int n = size(i), free = max(0, groups - n);
    if (m < free) return 8 * (n + m) + i;
    m -= free;
  }
  return 0;  // not reached
}

// CTA pair (cube split in z at zsplit): CTA r owns planes [zo0, zo1) of P and U and keeps
// P's planes [pz0, pz1) = its own plus O halo planes on the peer's side, which the peer writes.
struct PairPlanes {
  int zo0, zo1, pz0, pz1;
};
__host__ __device__ constexpr PairPlanes pair_planes(int nz, int zsplit, int rank) {
  return rank == 0 ? PairPlanes{0, zsplit, 0, zsplit + O < nz ? zsplit + O : nz}
                   : PairPlanes{zsplit, nz, zsplit - O > 0 ? zsplit - O : 0, nz};
}
// planes of P and of U to allocate: the larger of the two CTAs'
__host__ __device__ constexpr int pair_p_planes(int nz, int zsplit) {
  return (pair_planes(nz, zsplit, 0).pz1 - pair_planes(nz, zsplit, 0).pz0) >
                 (pair_planes(nz, zsplit, 1).pz1 - pair_planes(nz, zsplit, 1).pz0)
             ? pair_planes(nz, zsplit, 0).pz1 - pair_planes(nz, zsplit, 0).pz0
             : pair_planes(nz, zsplit, 1).pz1 - pair_planes(nz, zsplit, 1).pz0;
}
__host__ __device__ constexpr int pair_u_planes(int nz, int zsplit) {
  return zsplit > nz - zsplit ? zsplit : nz - zsplit;
}

// ---- the projector list ----
// A unit of the list is (image, column, kRun planes): the radial values T_l of kRun quads above one
// another, zero outside the support and the run.  A thread owns one column of quads over a range of
// planes ("item") and its units, so no two threads ever meet on a quad.
constexpr int kRun = 4;
constexpr int kListColumns = 512;  // the whole tensor memory of an SM, shared by its CTAs
// Units of a quarter (32 of the 128 lanes): T, the word and (x, y, z) relative to the atom.
__host__ __device__ constexpr int list_units_per_quarter(int columns, int nch) {
  return columns / (4 * kRun * nch + 4);
}
// Plane ranges per column: as many as the threads allow with at least kRun planes each.
__host__ __device__ constexpr int list_chunks(int columns, int planes, int threads) {
  int c = threads / columns < 1 ? 1 : threads / columns;
  while (c > 1 && planes / c < kRun) c--;
  return c;
}
__host__ __device__ constexpr int list_planes(int planes) {  // planes to allocate
  return planes < kRun ? kRun : planes;
}
// Bytes of per-node scratch of the list build: the items in order, unit counts per (image, warp), units
// and runs per item.
__host__ __device__ constexpr int list_scratch_bytes(int max_img, int nw) {
  return 4 * (32 * nw + max_img * nw + 32 * nw);
}
// The radial tables of this kernel hold whole quads: rows of the box's points behind `shift` zeros
// (four copies, shift 0..3: the image's box start modulo 4 picks the one whose quads are the cube's),
// zeros outside the support.  The planes and channels of a column of quads lie next to one another
// ([row][quad][plane][channel]): a unit is one run of memory, half the sectors of a plane by plane
// layout.  Quads of a row, and of a channel.
__host__ __device__ inline int quad_table_row(const TypeDesc &td) { return (td.fx + 6) / 4; }
__host__ __device__ inline int quad_table_channel(const TypeDesc &td) {
  return quad_table_row(td) * td.fy * td.fz;
}

// Tensor memory: a warp reads and writes its own quarter of the lanes.
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float4 (&t)[4]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=f"(t[0].x), "=f"(t[0].y), "=f"(t[0].z), "=f"(t[0].w), "=f"(t[1].x), "=f"(t[1].y),
        "=f"(t[1].z), "=f"(t[1].w), "=f"(t[2].x), "=f"(t[2].y), "=f"(t[2].z), "=f"(t[2].w),
        "=f"(t[3].x), "=f"(t[3].y), "=f"(t[3].z), "=f"(t[3].w)
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(unsigned taddr, const float4 (&t)[4]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"f"(
          t[0].x),
      "f"(t[0].y), "f"(t[0].z), "f"(t[0].w), "f"(t[1].x), "f"(t[1].y), "f"(t[1].z), "f"(t[1].w),
      "f"(t[2].x), "f"(t[2].y), "f"(t[2].z), "f"(t[2].w), "f"(t[3].x), "f"(t[3].y), "f"(t[3].z),
      "f"(t[3].w), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld4(unsigned taddr, float4 &a) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w)
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_st4(unsigned taddr, float4 a) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "f"(a.x),
               "f"(a.y), "f"(a.z), "f"(a.w)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// A barrier of the CTA that also orders the tensor-memory accesses of its warps: a warp's units have other
// places in the next node, where another warp of the same lanes read before.
__device__ __forceinline__ void tmem_sync() {
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
}
// The wait names the registers it guards, so that no use of them moves above it.
template <int N> __device__ __forceinline__ void tmem_wait_ld(float4 (&t)[N][4], float4 &m) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(m.x), "+f"(m.y), "+f"(m.z), "+f"(m.w)::"memory");
#pragma unroll
  for (int c = 0; c < N; c++)
#pragma unroll
    for (int i = 0; i < 4; i++)
      asm volatile("" : "+f"(t[c][i].x), "+f"(t[c][i].y), "+f"(t[c][i].z), "+f"(t[c][i].w));
}

// A unit's word: atom slot (10 bits), first plane from its item's first one (6), place of its partial
// sums (16).  The host plans no list with longer items (kQuadListPlanes): from the cube's first plane the
// field would end at 67 planes, and a cube of 17 x 17 x 69 points fits the SM.
static_assert(kQuadListPlanes <= 63 + kRun, "6 bits hold the last unit's first plane");
__device__ __forceinline__ unsigned unit_word(int slot, int z0, int place) {
  return (unsigned)(slot | (z0 << 10)) | ((unsigned)place << 16);
}
// An image of the node: box point 0 in cube coordinates (z from the first owned plane) as floats,
// its coordinates relative to the atom, its table (in quads), type and atom slot.
struct ImgRow {
  float bx, by, bz, ox;
  float oy, oz;
  int tab, type_slot;
  __device__ __forceinline__ int type() const { return type_slot & 15; }
  __device__ __forceinline__ int slot() const { return type_slot >> 4; }
};
static_assert(kMaxTypes <= 16, "ImgRow packs the type into 4 bits");
static_assert(sizeof(ImgRow) == 32, "two 16-byte loads");
__device__ __forceinline__ ImgRow load_row(const ImgRow *r) {
  const float4 a = reinterpret_cast<const float4 *>(r)[0], b = reinterpret_cast<const float4 *>(r)[1];
  return ImgRow{a.x, a.y, a.z, a.w, b.x, b.y, __float_as_int(b.z), __float_as_int(b.w)};
}

// Products of a unit's T with kRun quads of a column.  gather: the unit's raw sums (times norm() they
// are <chi_lm, P>); scatter: adds sum_lm chi_lm q_lm, q with norm() in it.
template <int MASK> struct UnitChi {
  static constexpr int nch = (MASK & 1) + ((MASK >> 1) & 1) + ((MASK >> 2) & 1) + ((MASK >> 3) & 1);
  static constexpr int nlm = lk::Lm<MASK>::nlm;
  static __device__ __forceinline__ float norm(int) { return 1.f; }
  // FN(channel, rank, harmonic) at (x, y, z)
  template <typename FN>
  static __device__ __forceinline__ void harmonics(float x, float y, float z, FN &&fn) {
    int c = 0;
    auto channel = [&](auto Lc) {
      constexpr int L = decltype(Lc)::value;
      if constexpr (MASK & (1 << L)) {
        lk::solid_harmonics<L, float>(x, y, z, [&](int s, float ylm) { fn(c, lk::Lm<MASK>::rank(s), ylm); });
        c++;
      }
    };
    channel(std::integral_constant<int, 0>{});
    channel(std::integral_constant<int, 1>{});
    channel(std::integral_constant<int, 2>{});
    channel(std::integral_constant<int, 3>{});
  }
  static __device__ __forceinline__ float at(float4 v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
  static __device__ __forceinline__ void gather(const LanczosParams &p, const float4 (&T)[nch][kRun],
                                                const float4 (&v)[kRun], float x, float y, float z,
                                                float (&c)[nlm]) {
#pragma unroll
    for (int s = 0; s < nlm; s++) c[s] = 0.f;
#pragma unroll
    for (int k = 0; k < kRun; k++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float t[nch];
#pragma unroll
        for (int q = 0; q < nch; q++) t[q] = at(v[k], i) * at(T[q][k], i);
        harmonics(fmaf(p.hxf, float(i), x), y, fmaf(p.hzf, float(k), z),
                  [&](int q, int r, float ylm) { c[r] = fmaf(ylm, t[q], c[r]); });
      }
  }
  static __device__ __forceinline__ void scatter(const LanczosParams &p, const float4 (&T)[nch][kRun],
                                                 float4 (&u)[kRun], float x, float y, float z,
                                                 const float (&q)[nlm]) {
#pragma unroll
    for (int k = 0; k < kRun; k++) {
      float r4[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float g[nch];
#pragma unroll
        for (int c = 0; c < nch; c++) g[c] = 0.f;
        harmonics(fmaf(p.hxf, float(i), x), y, fmaf(p.hzf, float(k), z),
                  [&](int c, int r, float ylm) { g[c] = fmaf(ylm, q[r], g[c]); });
#pragma unroll
        for (int c = 0; c < nch; c++) r4[i] = fmaf(at(T[c][k], i), g[c], r4[i]);
      }
      u[k] = make_float4(r4[0], r4[1], r4[2], r4[3]);
    }
  }
};
// s and p channels, two points per instruction: over a column x and y are the same for every plane,
// so their sums are taken once per unit.  Ranks: s, y, z, x.
template <> struct UnitChi<3> {
  static constexpr int nch = 2, nlm = 4;
  static __device__ __forceinline__ float norm(int r) { return r == 0 ? 1.f : 0.488602511902920f; }
  static __device__ __forceinline__ void gather(const LanczosParams &p, const float4 (&T)[nch][kRun],
                                                const float4 (&v)[kRun], float x, float y, float z,
                                                float (&c)[nlm]) {
    float2 s = mul2(lo(T[0][0]), lo(v[0]));
    s = fma2(hi(T[0][0]), hi(v[0]), s);
    float2 t01 = mul2(lo(T[1][0]), lo(v[0])), t23 = mul2(hi(T[1][0]), hi(v[0]));
    float2 sz = mul2(splat(z), add2(t01, t23));
#pragma unroll
    for (int k = 1; k < kRun; k++) {
      s = fma2(lo(T[0][k]), lo(v[k]), s);
      s = fma2(hi(T[0][k]), hi(v[k]), s);
      const float2 a = mul2(lo(T[1][k]), lo(v[k])), b = mul2(hi(T[1][k]), hi(v[k]));
      sz = fma2(splat(fmaf(p.hzf, float(k), z)), add2(a, b), sz);
      t01 = add2(t01, a);
      t23 = add2(t23, b);
    }
    const float2 x01 = make_float2(x, x + p.hxf);
    const float2 x23 = make_float2(fmaf(p.hxf, 2.f, x), fmaf(p.hxf, 3.f, x));
    const float2 sx = fma2(x01, t01, mul2(x23, t23)), t = add2(t01, t23);
    c[0] = s.x + s.y;
    c[1] = y * (t.x + t.y);
    c[2] = sz.x + sz.y;
    c[3] = sx.x + sx.y;
  }
  static __device__ __forceinline__ void scatter(const LanczosParams &p, const float4 (&T)[nch][kRun],
                                                 float4 (&u)[kRun], float x, float y, float z,
                                                 const float (&q)[nlm]) {
    const float2 q0 = splat(q[0]), qx = splat(q[3]), yz = splat(fmaf(q[1], y, q[2] * z));
    const float2 x01 = make_float2(x, x + p.hxf);
    const float2 x23 = make_float2(fmaf(p.hxf, 2.f, x), fmaf(p.hxf, 3.f, x));
    const float2 g01 = fma2(qx, x01, yz), g23 = fma2(qx, x23, yz);
    const float qzh = q[2] * p.hzf;
#pragma unroll
    for (int k = 0; k < kRun; k++) {
      const float2 dz = splat(qzh * float(k));
      const float2 a = k ? add2(g01, dz) : g01, b = k ? add2(g23, dz) : g23;
      const float2 u01 = fma2(lo(T[1][k]), a, fma2(lo(T[0][k]), q0, lo(u[k])));
      const float2 u23 = fma2(hi(T[1][k]), b, fma2(hi(T[0][k]), q0, hi(u[k])));
      u[k] = make_float4(u01.x, u01.y, u23.x, u23.y);
    }
  }
};

// Planes [a, b) of an item's column that an image's support meets.
struct ListRun {
  int a, b;
  __device__ __forceinline__ int units() const { return (max(b - a, 0) + kRun - 1) / kRun; }
};
// Item t of the list: chunk t % chunks of column t / chunks, so that a warp's items lie in few rows.
struct ListItem {
  int index, column;  // t, and the quad index in a plane
  int zb, ze;   // its planes, from the first owned one
  int top;      // units end here: ze, or kRun in a cube of fewer planes (that many are allocated)
  float x, y;   // cube coordinates of the column's first point
  __device__ __forceinline__ ListItem(int t, int chunks, int nq, int planes) {
    column = t / chunks;
    const int chunk = t - column * chunks;
    index = t;
    const int row = column / nq;
    x = float(4 * (column - row * nq));
    y = float(row);
    zb = planes * chunk / chunks;
    ze = planes * (chunk + 1) / chunks;
    top = max(ze, zb + kRun);
  }
  // A run may be longer than the support (T is zero there), but no quad lies outside the image's box.
  __device__ __forceinline__ ListRun run(const LanczosParams &p, const ImgRow *row, float ih) const {
    const ImgRow g = load_row(row);
    const TypeDesc &td = p.types[g.type()];
    const float fx = x - g.bx, fy = y - g.by;
    const float d0 = fmaf(p.hxf, fx, g.ox), d1 = d0 + p.hxf, d2 = d1 + p.hxf, d3 = d2 + p.hxf;
    const float near = fminf(fminf(fabsf(d0), fabsf(d1)), fminf(fabsf(d2), fabsf(d3)));
    const float dy = fmaf(p.hyf, fy, g.oy), rest = td.support_r2_f32 * (1.f + 1e-5f) - near * near - dy * dy;
    const bool meets = rest >= 0.f && fx > -4.f && fx < float(td.fx) && fy >= 0.f && fy < float(td.fy);
    // |oz + hz (z - bz)| <= sqrt(rest), a touch wider
    float half;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(half) : "f"(fmaxf(rest, 0.f)));
    const float low = fmaf(-half - g.oz, ih, -1e-3f), high = fmaf(half - g.oz, ih, 1e-3f);
    const int bz = (int)g.bz;
    ListRun r;
    r.a = max(zb, bz + max(0, (int)ceilf(low)));
    r.b = min(ze, bz + min(td.fz, (int)floorf(high) + 1));
    return meets && r.b > r.a ? r : ListRun{0, 0};
  }
};
// Exclusive scan of n integers in place by one warp; returns their sum.
__device__ __forceinline__ int warp_exclusive_scan(int *v, int n) {
  const int lane = threadIdx.x & 31;
  const int per = (n + 31) / 32, b = min(n, lane * per), e = min(n, b + per);
  int sum = 0;
  for (int i = b; i < e; i++) sum += v[i];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  int at = incl - sum;
  for (int i = b; i < e; i++) {
    const int t = v[i];
    v[i] = at;
    at += t;
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, incl, 31);
}

// Sums of N values over each G lanes; the total of value i goes to fn(i, total) in one of them.  N = 4
// halves the values with the lanes first (G = 32: 6 shuffles instead of 20).
template <int G, int N, typename FN> __device__ __forceinline__ void group_totals(const float (&v)[N], FN &&fn) {
  const int lane = threadIdx.x & 31;
  if constexpr (N == 4) {
    const bool hi = lane & (G / 2), mid = lane & (G / 4);
    float a = hi ? v[2] : v[0], b = hi ? v[3] : v[1];
    a += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], G / 2);
    b += __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], G / 2);
    float c = mid ? b : a;
    c += __shfl_xor_sync(0xffffffffu, mid ? a : b, G / 4);
#pragma unroll
    for (int o = G / 8; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((lane & (G / 4 - 1)) == 0) fn((lane & (G - 1)) / (G / 4), c);
  } else {
#pragma unroll
    for (int s = 0; s < N; s++) {
      float r = v[s];
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
      if ((lane & (G - 1)) == 0) fn(s, r);
    }
  }
}

// PAIR: one node per cluster of two CTAs (the cube split in z, see PairPlanes); else one node
// per CTA.
template <int MASK, int MAXT, bool ISO, bool PAIR>
__device__ __forceinline__ void quad_body(const LanczosParams &p, const float *__restrict__ veffq,
                                          const ImageMeta *__restrict__ images,
                                          const float *__restrict__ tables,
                                          unsigned char *proj_scratch, double *__restrict__ ab_out,
                                          int *__restrict__ status) {
  constexpr int NLM = lk::Lm<MASK>::nlm;
  using Chi = UnitChi<MASK>;
  constexpr int NCH = Chi::nch;
  constexpr int kTCols = 4 * kRun * NCH;  // tensor-memory columns of a unit's T
  constexpr int kPart = (NLM + 3) / 4;    // float4 of a unit's partial sums
  // The arrays of P and U change places every step: the update writes one instead of two of them (the
  // shared-memory data path is what the kernel waits for most).  4864 nodes of 29^3 and 50 steps 40.2 ->
  // 38.6 ms; the 12-warp kernel, which has the registers to read the update's next quads ahead, gains
  // nothing (27^3 20.05 and 20.15 ms); a CTA of a pair holds more planes of P than of U.
  constexpr bool kSwap = !PAIR && MAXT > 384;
  const int nw = blockDim.x >> 5;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nx = p.nx, ny = p.ny, nz = p.nz, pitch = p.pitch;
  const int nq = pitch >> 2;        // quads per row
  const int PS = quad_plane_floats(ny, pitch);  // plane stride (floats)
  const int PS4 = PS >> 2;                       // plane stride (quads)
  const int maxi = p.max_img;
  // planes owned ([zo0, zo1): U and the list) and held of P ([pz0, pz1)); P plane z sits at
  // local plane z - pz0, U plane z at z - zo0
  int cr = 0;  // rank in the CTA pair
  if constexpr (PAIR) cr = (int)cooperative_groups::this_cluster().block_rank();
  const PairPlanes pp = PAIR ? pair_planes(nz, p.zsplit, cr) : PairPlanes{0, nz, 0, nz};
  const int zo0 = pp.zo0, zo1 = pp.zo1, pz0 = pp.pz0, pz1 = pp.pz1, nzo = zo1 - zo0;
  const int ncp = (PAIR ? pair_p_planes(nz, p.zsplit) : list_planes(nz)) * PS;  // floats of P
  const int ncu = (PAIR ? pair_u_planes(nz, p.zsplit) : list_planes(nz)) * PS;  // floats of U
  const int pofs4 = -pz0 * PS4, uofs4 = -zo0 * PS4;  // quad index shifts of planes

  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *P = reinterpret_cast<float *>(smem_raw);
  float *U = P + ncp;
  unsigned char *cur = reinterpret_cast<unsigned char *>(U + ncu);
  float2 *sum_a = reinterpret_cast<float2 *>(cur);  // <P,HP> and |w|^2 of every step, double-floats
  float2 *sum_b = sum_a + 64;
  float2 *red_a = sum_b + 64;  // per-warp double-float partials
  float2 *red_b = red_a + kMaxWarps;
  cur += sizeof(float2) * (2 * kMaxWarps + 128);  // (16-byte multiples so far: alpha is read as float4)
  float *alpha = reinterpret_cast<float *>(cur);
  cur += sizeof(float4) * maxi * kPart;
  // PAIR: the two CTAs' gathered c per (slot, lm), [rank][slot * NLM + lm] (each CTA writes
  // its row into both), the per-warp partials of the projector part of a_k and the two
  // CTAs' capacity flags
  float *cx = reinterpret_cast<float *>(cur);
  float2 *red_n = reinterpret_cast<float2 *>(cur);
  int *xflag = reinterpret_cast<int *>(cur);
  if constexpr (PAIR) {
    cur += sizeof(float) * 2 * maxi * NLM;
    cur += (8 - (reinterpret_cast<uintptr_t>(cur) & 7)) & 7;
    red_n = reinterpret_cast<float2 *>(cur);
    cur += sizeof(float2) * kMaxWarps;
    xflag = reinterpret_cast<int *>(cur);
    cur += sizeof(int) * 4;
  }
  int *img = reinterpret_cast<int *>(cur);
  int *slot_type = img + maxi;
  int *slot_first = slot_type + maxi;    // first image of every slot (images sorted by atom), n_img
  int *slot_base = slot_first + maxi + 1;  // first partial sums of every slot, their number
  int *cnt = slot_base + maxi + 1;  // [0] images, [1] slots, [2] overflow, [3] next node, [4] TMEM
  int *wunits = cnt + 5;            // units of every warp's longest lane
  ImgRow *rows = reinterpret_cast<ImgRow *>(
      (reinterpret_cast<uintptr_t>(wunits + kMaxWarps) + 15) & ~static_cast<uintptr_t>(15));
  float4 *zq = reinterpret_cast<float4 *>(rows + maxi);  // a quad of zeros
  float4 *part_s = zq + 1;                               // [p.part_cap] partial sums
  // scratch of the list build: U, which is cleared after it, if it is large enough
  int *scratch = list_scratch_bytes(maxi, nw) <= 4 * ncu ? reinterpret_cast<int *>(U)
                                                         : reinterpret_cast<int *>(part_s + p.part_cap);

  // this CTA's slice of global scratch: T and words of the units beyond the tensor memory
  // ([batch][lane]), partial sums, the items' runs
  float4 *gT = reinterpret_cast<float4 *>(proj_scratch + (size_t)blockIdx.x * p.proj_bytes_per_cta);
  float4 *gmeta = gT + (size_t)p.list_batches * 32 * kRun * NCH;
  float4 *part_g = gmeta + (size_t)p.list_batches * 32;
  float4 *grun = part_g + (size_t)p.part_total * kPart;
  const float4 *qtables = reinterpret_cast<const float4 *>(tables);

  float4 *P4 = reinterpret_cast<float4 *>(P);
  float4 *U4 = reinterpret_cast<float4 *>(U);
  float4 *P4o = P4 + (zo0 - pz0) * PS4;  // the owned planes of P, indexed as U
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  // byte addresses: P, U, a quad of zeros that stands for every plane and row outside the cube
  const unsigned sP = smem_addr(P), sU = smem_addr(U);
  const unsigned sZ = smem_addr(zq);
  if (threadIdx.x == 0) *zq = zero4;  // the node loop's first barrier comes before its first use
  const int PB = 16 * PS4, RB = 16 * nq;  // bytes of a plane and of a row
  // list items: column (quad xq of row y) and plane range [nzo c / nlc, nzo (c+1) / nlc) of the owned
  const int ncol = nq * ny, nlc = list_chunks(ncol, nzo, blockDim.x), n_item = ncol * nlc;
  if (warp == 0) tc5::tmem_alloc(reinterpret_cast<uint32_t *>(cnt + 4), (uint32_t)p.list_columns);
  tmem_sync();
  const float ihz = 1.f / p.hzf;
  const unsigned tquarter = (unsigned)cnt[4] + ((unsigned)(warp & 3) << 21);  // the warp's lanes

  // pass A: nq consecutive threads own the quads of a row, so consecutive threads touch consecutive
  // quads.  Row yA, z-range [zbA, zeA) of the owned planes
  const int grp = threadIdx.x / nq, ql = threadIdx.x - grp * nq;
  const int nch = p.zchunks, nchB = PAIR ? p.ychunks : p.zchunks;
  const int yA = grp % ny, zcA = grp / ny;
  const int zlen = (nzo + nch - 1) / nch;
  const int zbA = zo0 + min(nzo, zcA * zlen), zeA = min(zo1, zbA + zlen);
  const bool actA = zcA < nch && zbA < zeA;
  // pass B: quad qB of owned plane zB, y-range [ybB, yeB); the columns (y-range, plane, quad) dealt by
  // the bank class of their first row, ranked by y-range, quad, plane
  const int ylen = (ny + nchB - 1) / nchB;
  int colB;
  {
    auto of_class = [&](int c, int r) {  // quads of y-range c in class r
      const int first = (r - c * ylen * nq) & 7;
      return first < nq ? (nq - first + 7) >> 3 : 0;
    };
    scratch[threadIdx.x] = nchB * nzo * nq;
    __syncthreads();
    if ((int)threadIdx.x < nchB * nzo * nq) {
      const int c = grp / nzo, r = (c * ylen * nq + ql) & 7;
      int rank = (ql >> 3) * nzo + grp % nzo;
      for (int i = 0; i < c; i++) rank += of_class(i, r) * nzo;
      scratch[bank_slot(r, rank, (nchB * nzo * nq + 31) / 32 * 4, [&](int i) {  // as few warps as hold them
        int n = 0;
        for (int k = 0; k < nchB; k++) n += of_class(k, i) * nzo;
        return n;
      })] = threadIdx.x;
    }
    __syncthreads();
    colB = scratch[threadIdx.x];
    __syncthreads();
  }
  const int grpB = colB / nq, qB = colB - grpB * nq;
  const int zB = zo0 + grpB % nzo, ycB = grpB / nzo;
  const int ybB = min(ny, ycB * ylen), yeB = min(ny, ybB + ylen);
  const bool actB = ycB < nchB && ybB < yeB;
  // x neighbours of the quad inside the row; lanes of the last quad zero its pad points
  const bool hm1 = ql >= 1, hm2 = ql >= 2, hp1 = ql + 1 < nq, hp2 = ql + 2 < nq;
  const int x0 = 4 * ql;
  const int row4 = yA * nq + ql;  // pass A: quad index of (x0, yA) in a plane
  const bool in1 = x0 + 1 < nx, in2 = x0 + 2 < nx, in3 = x0 + 3 < nx;  // x0 < nx always

  // nodes: the first round one per CTA, then a queue (status[1], zeroed before the launch):
  // per-node cost varies with the atoms near the node, so CTAs take nodes as they finish.
  // PAIR: node i of the cluster sequence, both CTAs alike (no queue).
  const long long n_units = PAIR ? gridDim.x / 2 : gridDim.x;
  const long long unit = PAIR ? blockIdx.x / 2 : blockIdx.x;
  for (long long node = p.node_begin + unit; node < p.node_end;
       node = PAIR ? node + n_units : p.node_begin + n_units + cnt[3]) {
    const int I = (int)(node % p.Nx);
    const int J = (int)((node / p.Nx) % p.Ny);
    const int K = (int)(node / ((long long)p.Nx * p.Ny));
    const int Xs = I - p.nhx, Ys = J - p.nhy, Zs = K - p.nhz;

    // ---- images that meet the cube, in order; every warp looks at its share.  P cleared ----
    const int share = (p.n_images + 32 * nw - 1) / (32 * nw) * 32;
    const int i0 = warp * share, i1 = min(p.n_images, i0 + share);
    auto meets = [&](int i) {
      if (i >= i1) return false;
      const int4 b = *reinterpret_cast<const int4 *>(&images[i]);
      const TypeDesc &td = p.types[b.w];
      return b.x <= Xs + nx - 1 && b.x + td.fx - 1 >= Xs && b.y <= Ys + ny - 1 &&
             b.y + td.fy - 1 >= Ys && b.z <= Zs + nz - 1 && b.z + td.fz - 1 >= Zs;
    };
    {
      int found = 0;
      for (int base = i0; base < i1; base += 32)
        found += __popc(__ballot_sync(0xffffffffu, meets(base + lane)));
      if (lane == 0) wunits[warp] = found;
    }
    for (int e = threadIdx.x; e < (ncp >> 2); e += blockDim.x) P4[e] = zero4;
    __syncthreads();
    {
      int at = 0, count = 0;
      for (int w = 0; w < nw; w++) {
        at += w < warp ? wunits[w] : 0;
        count += wunits[w];
      }
      for (int base = i0; base < i1; base += 32) {
        const bool ok = meets(base + lane);
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        const int pos = at + __popc(m & ((1u << lane) - 1u));
        if (ok && pos < maxi) img[pos] = base + lane;
        at += __popc(m);
      }
      if (threadIdx.x == 0) {
        cnt[0] = min(count, maxi);
        cnt[2] = count > maxi;
      }
    }
    __syncthreads();
    const int n_img = cnt[0];
    if (warp == 0) {  // their rows, and the slots (images are sorted by atom)
      int slots = 0;
      for (int base = 0; base < n_img; base += 32) {
        const int k = base + lane;
        bool start = false;
        ImageMeta m{};
        if (k < n_img) {
          m = images[img[k]];
          start = (k == 0) || images[img[k - 1]].atom != m.atom;
        }
        const unsigned starts = __ballot_sync(0xffffffffu, start);
        const int g = slots + __popc(starts & ((1u << lane) - 1u)) + (start ? 0 : -1);
        if (k < n_img) {
          const TypeDesc &td = p.types[m.type];
          const int shift = (m.bx - Xs) & 3;  // which copy of the table has the cube's quads aligned
          rows[k] = ImgRow{(float)(m.bx - Xs), (float)(m.by - Ys), (float)(m.bz - Zs - zo0), (float)m.ox,
                           (float)m.oy, (float)m.oz,
                           (int)(m.tab_base + (long long)shift * __popc(td.chan_mask) * quad_table_channel(td)),
                           m.type | (g << 4)};
          if (start) {
            slot_type[g] = m.type;
            slot_first[g] = k;
          }
        }
        slots += __popc(starts);
      }
      if (lane == 0) {
        slot_first[slots] = n_img;
        cnt[1] = slots;
      }
    }
    __syncthreads();
    const int n_slot = cnt[1];

    // ---- runs of every item (thread t: item t), kept in the scratch slice; units per (image, warp)
    // and per item.  The warp's lanes share the images whose boxes meet the bounds of its columns; both
    // plane ranges of a column in one warp make those bounds few rows (a warp that held the end of one
    // range and the start of the next took all 63 images, and the CTA waited for it).  The whole build of
    // a node of 27^3 and 63 images: 111K -> 58K cycles, 40 steps 1.36M ----
    int *order = scratch, *kw = order + 32 * nw;
    int *item_units = kw + maxi * nw;
    int2 *runs = reinterpret_cast<int2 *>(grun) + threadIdx.x;  // run i: + i * blockDim.x
    int units = 0;
    {  // and its first unit's place among the warp's of the image
      const bool mine = threadIdx.x < n_item;
      const ListItem it(mine ? threadIdx.x : 0, nlc, nq, nzo);
      const int row = it.column / nq;
      const int r0 = __reduce_min_sync(0xffffffffu, mine ? row : ny), r1 = __reduce_max_sync(0xffffffffu, mine ? row : -1);
      const int z0 = __reduce_min_sync(0xffffffffu, mine ? it.zb : nzo), z1 = __reduce_max_sync(0xffffffffu, mine ? it.ze : 0);
      int n_run = 0;
      for (int base = 0; base < n_img; base += 32) {
        const int k = base + lane;
        bool near = false;
        if (k < n_img) {
          const ImgRow g = load_row(rows + k);
          const TypeDesc &td = p.types[g.type()];
          near = (int)g.by <= r1 && (int)g.by + td.fy > r0 && (int)g.bz < z1 && (int)g.bz + td.fz > z0;
        }
        int total = 0;  // of image k
        auto keep = [&](int k, ListRun r, int place) {
          if (!r.units()) return;
          // planes from the item's first one, as in unit_word
          runs[(size_t)blockDim.x * n_run++] = make_int2(k | ((r.a - it.zb) << 10) | ((r.b - it.zb) << 17), place);
          units += r.units();
        };
        for (unsigned todo = __ballot_sync(0xffffffffu, near); todo;) {  // two images at once
          const int s0 = __ffs(todo) - 1;
          todo &= todo - 1;
          const int s1 = todo ? __ffs(todo) - 1 : 32;
          todo &= todo - 1;
          const ListRun q0 = it.run(p, rows + base + s0, ihz), q1 = it.run(p, rows + base + (s1 & 31), ihz);
          const ListRun r0 = mine ? q0 : ListRun{0, 0}, r1 = mine && s1 < 32 ? q1 : ListRun{0, 0};
          const int n = r0.units() | r1.units() << 16;
          int incl = n;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
          }
          const int all = __shfl_sync(0xffffffffu, incl, 31);
          total = lane == s0 ? all & 0xffff : lane == s1 ? all >> 16 : total;
          incl -= n;
          keep(base + s0, r0, incl & 0xffff);
          keep(base + s1, r1, incl >> 16);
        }
        if (k < n_img) kw[k * nw + warp] = total;
      }
      item_units[threadIdx.x] = units | (n_run << 16);
      order[threadIdx.x] = n_item;
    }
    __syncthreads();

    // ---- items dealt to the lanes by their number of units, the most first: within their bank class;
    // where the classes differ so much that this takes twice as many batches (units of a warp's 32
    // lanes) as the units would fill, or more than there is room for, among all ----
    const int own_units = units;
    int my, w_units, n_part, batch0, batches, quarter0;  // batches before this warp's, units before it in its quarter
    for (int step = 8;; step = 1) {
      if ((int)threadIdx.x < n_item) {
        const int r = step == 1 ? 0 : (int)threadIdx.x / nlc & 7;
        int rank = 0;
        for (int c = r * nlc; c < (r + 1) * nlc; c++)
#pragma unroll 4
          for (int t = c; t < n_item; t += step * nlc) {
            const int n = item_units[t] & 0xffff;
            rank += n > own_units || (n == own_units && t < (int)threadIdx.x);
          }
        if (step == 8)
          rank = bank_slot(r, rank, (int)blockDim.x >> 3, [&](int i) { return nlc * ((ncol - i + 7) >> 3); });
        order[rank] = threadIdx.x;
      }
      if (warp == 0 && step == 8) {  // the places of the partial sums: by image, warp, lane
        __syncwarp();
        const int total = warp_exclusive_scan(kw, n_img * nw);
        for (int g = lane; g < n_slot; g += 32) slot_base[g] = kw[slot_first[g] * nw];
        if (lane == 0) slot_base[n_slot] = total;
      }
      __syncthreads();
      my = order[threadIdx.x];
      units = my < n_item ? item_units[my] & 0xffff : 0;
      w_units = __reduce_max_sync(0xffffffffu, units);
      if (lane == 0) wunits[warp] = w_units;
      __syncthreads();
      batch0 = batches = quarter0 = 0;
      for (int w = 0; w < nw; w++) {
        const int u = wunits[w];
        if (w < warp) {
          batch0 += u;
          if ((w & 3) == (warp & 3)) quarter0 += u;
        }
        batches += u;
      }
      n_part = slot_base[n_slot];
      if (step == 1 || batches <= min(p.list_batches, n_part / 16 + 2 * nw)) break;
      order[threadIdx.x] = n_item;
      __syncthreads();
    }
    const ListItem item(my < n_item ? my : 0, nlc, nq, nzo);
    bool overflow = cnt[2] || batches > p.list_batches || n_part > p.part_total;
    if constexpr (PAIR) {  // both CTAs take the capacity branch together
      if (threadIdx.x == 0) {
        xflag[cr] = overflow;
        *cooperative_groups::this_cluster().map_shared_rank(xflag + cr, cr ^ 1) = overflow;
      }
      cooperative_groups::this_cluster().sync();
      overflow = xflag[0] || xflag[1];
    } else {
      // the next node, read by every thread after this node's last barrier (the previous
      // value was read before the barriers above)
      // (by the last warp, which has the fewest units)
      if (threadIdx.x == blockDim.x - 1) cnt[3] = atomicAdd(status + 1, 1);
    }
    if (overflow) {  // capacity exceeded: report, NaN coefficients
      if (threadIdx.x == 0) atomicOr(status, kStatusCapacity);
      if (cr == 0)
        for (int j = threadIdx.x; j < 2 * p.nqp; j += blockDim.x)
          ab_out[(node - p.node_begin) * 2 * p.nqp + j] = __longlong_as_double(0x7ff8000000000000ll);
      if constexpr (PAIR) cooperative_groups::this_cluster().sync();  // flags read by both
      else __syncthreads();
      continue;
    }
    float4 *part = n_part * kPart <= p.part_cap ? part_s : part_g;
    const int tm_units = max(0, min(w_units, list_units_per_quarter(p.list_columns, NCH) - quarter0));
    const unsigned tmT = tquarter + (unsigned)(quarter0 * kTCols);
    const unsigned tmM = tquarter + (unsigned)(list_units_per_quarter(p.list_columns, NCH) * kTCols + quarter0 * 4);
    float4 *wT = gT + (size_t)batch0 * 32 * kRun * NCH + lane;  // of unit u: + ((u * NCH + c) * kRun + k) * 32
    float4 *wmeta = gmeta + (size_t)batch0 * 32 + lane;         // of unit u: + u * 32

    // ---- the units: word, coordinates and T ----
    {
      const int2 *mine = reinterpret_cast<const int2 *>(grun) + item.index;
      const bool k1 = (int)item.x + 1 < nx, k2 = (int)item.x + 2 < nx, k3 = (int)item.x + 3 < nx;
      const int xq = (int)item.x >> 2;
      const int n_run = my < n_item ? item_units[my] >> 16 : 0;
      int left = 0, a = 0, b = 0, place = 0, cmask = 0, nc = 0;
      const float4 *tq = qtables;  // the column's quad of plane 0 of the box, channel 0
      ImgRow g{};
      int i = 0;
      auto unit = [&](int u, float4 (&T)[NCH][kRun], float4 &meta) {
        meta = make_float4(__uint_as_float(unit_word(0, 0, 0)), 0.f, 0.f, 0.f);
        const bool on = u < units;
        if (on && left == 0) {
          const int2 r = mine[(size_t)blockDim.x * i++];
          const ListRun run{item.zb + ((r.x >> 10) & 127), item.zb + (r.x >> 17)};
          a = run.a;
          b = run.b;
          left = run.units();
          place = r.y + kw[(r.x & 1023) * nw + (item.index >> 5)];
          g = load_row(rows + (r.x & 1023));
          const TypeDesc &td = p.types[g.type()];
          cmask = td.chan_mask;
          nc = __popc(cmask);
          tq = qtables +
               (g.tab + (((int)item.y - (int)g.by) * quad_table_row(td) + xq - ((int)g.bx >> 2)) * td.fz * nc);
        }
        const int z0 = on ? min(a, item.top - kRun) : item.zb;
        if (on)
          meta = make_float4(__uint_as_float(unit_word(g.slot(), z0 - item.zb, place)), fmaf(p.hxf, item.x - g.bx, g.ox),
                             fmaf(p.hyf, item.y - g.by, g.oy), fmaf(p.hzf, float(z0) - g.bz, g.oz));
        const float4 *tz = tq + (z0 - (int)g.bz) * nc;
        int c = 0, ch = 0;
#pragma unroll
        for (int l = 0; l < 4; l++) {
          if (!(MASK & (1 << l))) continue;
          const bool have = on && (cmask & (1 << l));
#pragma unroll
          for (int q = 0; q < kRun; q++)  // planes [a, b) of the unit's
            T[c][q] = ldg_quad_if(have && z0 + q >= a && z0 + q < b, tz + q * nc + ch);
          ch += have ? 1 : 0;
          c++;
        }
        a = on ? z0 + kRun : a;
        place += on;
        left -= on;
      };
      auto store = [&](int u, float4 (&T)[NCH][kRun], float4 meta) {
#pragma unroll
        for (int c = 0; c < NCH; c++)
#pragma unroll
          for (int q = 0; q < kRun; q++) {  // pad points
            T[c][q].y = k1 ? T[c][q].y : 0.f;
            T[c][q].z = k2 ? T[c][q].z : 0.f;
            T[c][q].w = k3 ? T[c][q].w : 0.f;
          }
        __syncwarp();
        if (u < tm_units) {
#pragma unroll
          for (int c = 0; c < NCH; c++) tmem_st16(tmT + (unsigned)(u * kTCols + 16 * c), T[c]);
          tmem_st4(tmM + (unsigned)(4 * u), meta);
        } else {
#pragma unroll
          for (int c = 0; c < NCH; c++)
#pragma unroll
            for (int q = 0; q < kRun; q++) wT[((u * NCH + c) * kRun + q) * 32] = T[c][q];
          wmeta[32 * u] = meta;
        }
      };
      constexpr int kAtOnce = MAXT <= 384 && NCH <= 2 ? 2 : 1;  // units whose table loads are in flight together
      for (int u = 0; u < w_units; u += kAtOnce) {
        float4 T[kAtOnce][NCH][kRun], meta[kAtOnce];
#pragma unroll
        for (int k = 0; k < kAtOnce; k++) unit(u + k, T[k], meta[k]);
#pragma unroll
        for (int k = 0; k < kAtOnce; k++)
          if (u + k < w_units) store(u + k, T[k], meta[k]);
      }
      tmem_wait_st();
    }
    auto load_unit = [&](int u, float4 (&T)[NCH][kRun], float4 &meta) {
      if (u < tm_units) {
#pragma unroll
        for (int c = 0; c < NCH; c++) tmem_ld16(tmT + (unsigned)(u * kTCols + 16 * c), T[c]);
        tmem_ld4(tmM + (unsigned)(4 * u), meta);
        tmem_wait_ld(T, meta);
      } else {
        meta = wmeta[32 * u];
#pragma unroll
        for (int c = 0; c < NCH; c++)
#pragma unroll
          for (int q = 0; q < kRun; q++) T[c][q] = wT[((u * NCH + c) * kRun + q) * 32];
      }
    };
    // the item's first quad in P and U
    const unsigned itemU = 16u * (unsigned)(item.column + item.zb * PS4), itemP = itemU + (unsigned)((zo0 - pz0) * PB);
    unsigned aP0 = sP, aU0 = sU;  // the arrays of P and U (kSwap: they change places every step)
    __syncthreads();  // the scratch in U is read
    for (int e = threadIdx.x; e < (ncu >> 2); e += blockDim.x) U4[e] = zero4;
    {  // v_0: the unit vector at the cube centre, in every CTA that holds that plane of P
      const int zc = (nz - 1) / 2;
      if (threadIdx.x == 0 && zc >= pz0 && zc < pz1)
        P[(zc - pz0) * PS + (ny - 1) / 2 * pitch + (nx - 1) / 2] = 1.f;
    }
    __syncthreads();

    // quad-aligned copy of the padded Veff for this node (copy s: I + s = 0 mod 4)
    const int sh = (4 - (I & 3)) & 3;
    const float4 *vq = reinterpret_cast<const float4 *>(veffq + (size_t)sh * p.vq_copy_stride) +
                       (size_t)((I + sh) >> 2);
    const int VPS4 = p.EY * (p.vq_row >> 2);             // plane stride in quads
    const size_t VRS4 = (size_t)(p.vq_row >> 2);         // row stride in quads

    float sc = 1.f;          // s_k
    DF n2 = {1.f, 0.f};      // |P|^2
    DF gam = {0.f, 0.f};     // gamma_k
    int steps = 0;
    for (int j = 0; j < p.nqp; j++) {
      const float2 sc2 = splat(sc), ngh2 = splat(-gam.hi), ngl2 = splat(-gam.lo);

      // ---- phase 1: projector gather  ||  pass A ----
      for (int u = 0; u < w_units; u++) {
        float4 T[NCH][kRun], meta;
        load_unit(u, T, meta);
        const unsigned w = __float_as_uint(meta.x);
        unsigned a = aP0 + itemP + (unsigned)((int)((w >> 10) & 63u) * PB);
        float4 v[kRun];
#pragma unroll
        for (int i = 0; i < kRun; i++, a += (unsigned)PB) v[i] = lds_quad(a);
        float c[NLM];
        Chi::gather(p, T, v, meta.y, meta.z, meta.w, c);
        if (u < units) {
          float4 *dst = part + (size_t)(w >> 16) * kPart;
#pragma unroll
          for (int i = 0; i < kPart; i++)
            dst[i] = make_float4(c[4 * i], 4 * i + 1 < NLM ? c[4 * i + 1] : 0.f,
                                 4 * i + 2 < NLM ? c[4 * i + 2] : 0.f, 4 * i + 3 < NLM ? c[4 * i + 3] : 0.f);
        }
        __syncwarp();
      }
      Kahan ka;
      if (actA) {
        float2 czs[O + 1], cxs[O + 1];
#pragma unroll
        for (int d = 1; d <= O; d++) {
          czs[d] = splat(p.czf[d]);
          cxs[d] = ISO ? czs[d] : splat(p.cxf[d]);
        }
        const float4 *vrow = vq + (size_t)(K * p.EY + J + yA) * VRS4 + ql + (size_t)zbA * VPS4;
        // the quad at plane zbA + i of P and U, and P's plane 6 further on: all lanes make zlen
        // steps (a uniform loop), those past their range keep nothing and read the x neighbours (aX) of
        // their last plane again: the planes after it may lie beyond P, whose place behind U with
        // kSwap has no array of that size after it
        const unsigned aP = aP0 + 16u * (unsigned)(row4 + zbA * PS4 + pofs4);
        unsigned aX = aP, aN = aP + (unsigned)(O * PB);
        unsigned aU = aU0 + 16u * (unsigned)(row4 + zbA * PS4 + uofs4);
        const int live = zeA - zbA, above = nz - O - zbA;
        float4 ring[W];
#pragma unroll
        for (int q = -O; q < O; q++) {
          const int zq = zbA + q;
          ring[q + O + 1] = lds_quad(zq >= 0 && zq < nz ? aP + (unsigned)(q * PB) : sZ);
        }
        // x neighbours: the upper half of quad q-2, quads q-1 and q+1, the lower half of q+2
        float2 xm2 = make_float2(0.f, 0.f), xp2 = make_float2(0.f, 0.f);
        float4 xm1 = zero4, xp1 = zero4;
        // Veff (from L2) one plane ahead; P and U of a plane as it begins, which the arithmetic of the
        // other warps covers.  With Veff two planes and U one ahead (13 registers more and copies between
        // them) 4864 nodes took 20.5 instead of 20.1 ms at 27^3, 57.0 instead of 54.9 on pairs at 33^3
        float4 dv1 = __ldg(vrow);
        for (int i0 = 0; i0 < zlen; i0 += W) {
#pragma unroll
          for (int s = 0; s < W; s++) {
            const int i = i0 + s;
            if (i >= zlen) break;
            ring[s] = lds_quad(i < above ? aN : sZ);
#define RING(dd) ring[(s + (dd) + O + 1) % W]
            lds_pair_if<-24>(hm2, aX, xm2);
            lds_quad_if<-16>(hm1, aX, xm1);
            lds_quad_if<16>(hp1, aX, xp1);
            lds_pair_if<32>(hp2, aX, xp2);
            const float4 c = RING(0);
            const float4 dv = dv1, uo = lds_quad(i < live ? aU : sZ);
            const int next = min(i + 1, live - 1);
            dv1 = __ldg(vrow + next * VPS4);
            float2 h01 = mul2(lo(dv), lo(c)), h23 = mul2(hi(dv), hi(c));
#pragma unroll
            for (int d = 1; d <= O; d++) {
              h01 = fma2(czs[d], add2(lo(RING(-d)), lo(RING(d))), h01);
              h23 = fma2(czs[d], add2(hi(RING(-d)), hi(RING(d))), h23);
            }
#undef RING
            // x neighbours: e[i] = P[x0 - 6 + i], i = 0..15
            const float e[16] = {xm2.x, xm2.y, xm1.x, xm1.y, xm1.z, xm1.w, c.x,   c.y,
                                 c.z,   c.w,   xp1.x, xp1.y, xp1.z, xp1.w, xp2.x, xp2.y};
#pragma unroll
            for (int d = 1; d <= O; d++) {
              if (d % 2 == 0) {
                h01 = fma2(cxs[d], add2(make_float2(e[6 - d], e[7 - d]), make_float2(e[6 + d], e[7 + d])), h01);
                h23 = fma2(cxs[d], add2(make_float2(e[8 - d], e[9 - d]), make_float2(e[8 + d], e[9 + d])), h23);
              } else {
                h01 = fma2(cxs[d], make_float2(e[6 - d] + e[6 + d], e[7 - d] + e[7 + d]), h01);
                h23 = fma2(cxs[d], make_float2(e[8 - d] + e[8 + d], e[9 - d] + e[9 + d]), h23);
              }
            }
            // zero the pad points; U <- s h - gamma U; a_k partial <P, h>
            h01.y = in1 ? h01.y : 0.f;
            h23.x = in2 ? h23.x : 0.f;
            h23.y = in3 ? h23.y : 0.f;
            const float2 n01 = fma2(sc2, h01, fma2(ngh2, lo(uo), mul2(ngl2, lo(uo))));
            const float2 n23 = fma2(sc2, h23, fma2(ngh2, hi(uo), mul2(ngl2, hi(uo))));
            sts_quad_if(i < live, aU, make_float4(n01.x, n01.y, n23.x, n23.y));
            const float2 pa = fma2(lo(c), h01, mul2(hi(c), h23));
            ka.add(i < live ? pa.x + pa.y : 0.f);
            // (a pair has one range, so all its lanes walk to their end together: the sum is 1% faster there,
            // the product 0.5% in the others; 9001 nodes of 33^3 106.7 -> 105.6 ms, 39304 of 27^3 168.4 -> 167.5)
            if constexpr (PAIR) aX += (unsigned)PB;
            else aX = aP + (unsigned)(next * PB);
            aN += (unsigned)PB;
            aU += (unsigned)PB;
          }
        }
      }
      __syncthreads();

      // ---- phase 2: pass B  ||  alpha = Gamma s c ----
      if (actB) {
        float2 cys[O + 1];
#pragma unroll
        for (int d = 1; d <= O; d++) cys[d] = splat(ISO ? p.czf[d] : p.cyf[d]);
        // the quad at row ybB + i of P and U, and P's row 6 further on; all lanes make ylen steps
        unsigned aP = aP0 + 16u * (unsigned)(zB * PS4 + qB + pofs4 + ybB * nq);
        unsigned aN = aP + (unsigned)(O * RB);
        unsigned aU = aU0 + 16u * (unsigned)(zB * PS4 + qB + uofs4 + ybB * nq);
        const int live = yeB - ybB, above = ny - O - ybB;
        // before the step of row y, ring[j] holds row y - 6 + j (mod W); y + 6 joins at its start
        float4 ring[W];
#pragma unroll
        for (int j = 0; j < W - 1; j++) {
          const int yq = ybB - O + j;
          ring[j] = lds_quad(yq >= 0 && yq < ny ? aP + (unsigned)((j - O) * RB) : sZ);
        }
        for (int i0 = 0; i0 < ylen; i0 += W) {
#pragma unroll
          for (int s = 0; s < W; s++) {
            const int i = i0 + s;
            if (i >= ylen) break;
            ring[(s + W - 1) % W] = lds_quad(i < above ? aN : sZ);
            const float4 uo = lds_quad(i < live ? aU : sZ);
#define RING(dd) ring[(s + (dd) + O) % W]
            float2 h01 = mul2(cys[1], add2(lo(RING(-1)), lo(RING(1))));
            float2 h23 = mul2(cys[1], add2(hi(RING(-1)), hi(RING(1))));
#pragma unroll
            for (int d = 2; d <= O; d++) {
              h01 = fma2(cys[d], add2(lo(RING(-d)), lo(RING(d))), h01);
              h23 = fma2(cys[d], add2(hi(RING(-d)), hi(RING(d))), h23);
            }
            const float4 c = RING(0);
#undef RING
            const float2 n01 = fma2(sc2, h01, lo(uo)), n23 = fma2(sc2, h23, hi(uo));
            sts_quad_if(i < live, aU, make_float4(n01.x, n01.y, n23.x, n23.y));
            const float2 pa = fma2(lo(c), h01, mul2(hi(c), h23));
            ka.add(i < live ? pa.x + pa.y : 0.f);
            aN += (unsigned)RB;
            aU += (unsigned)RB;
          }
        }
      }
      // c of every slot, its units' partial sums in a fixed order; alpha = Gamma_l s c (the harmonics'
      // constants on both sides), <P, V_nl P> = sum Gamma_l c^2.  A warp per slot, or with more slots
      // than warps eight lanes (4864 nodes: 32 atoms, 27^3 24.2 -> 23.2 ms; 4 atoms, 25^3 15.4 against
      // 15.9 with a warp; the pair and the 16-warp kernels lose 2% with eight).
      {
        auto sum_slot = [&](int sl, int first, int step, float (&c)[NLM]) {
#pragma unroll
          for (int s = 0; s < NLM; s++) c[s] = 0.f;
          const int end = sl < n_slot ? slot_base[sl + 1] : 0;
#pragma unroll 4
          for (int j = sl < n_slot ? slot_base[sl] + first : 0; j < end; j += step) {
#pragma unroll
            for (int i = 0; i < kPart; i++) {
              const float4 t = part[(size_t)j * kPart + i];
              c[4 * i] += t.x;
              if (4 * i + 1 < NLM) c[4 * i + 1] += t.y;
              if (4 * i + 2 < NLM) c[4 * i + 2] += t.z;
              if (4 * i + 3 < NLM) c[4 * i + 3] += t.w;
            }
          }
          __syncwarp();
        };
        auto finish = [&](int sl, int r, float total) {
          const float cr_sum = total * Chi::norm(r);
          if constexpr (PAIR) {  // this CTA's part of c, into both CTAs' row cr of cx
            float *x = cx + cr * maxi * NLM + sl * NLM + r;
            *x = cr_sum;
            *cooperative_groups::this_cluster().map_shared_rank(x, cr ^ 1) = cr_sum;
          } else {
            const TypeDesc &td = p.types[slot_type[sl]];
            const int l = p.rank_l[r];
            const float gl = (td.chan_mask & (1 << l)) ? float(td.gamma[l]) : 0.f;
            const float al = gl * cr_sum;
            alpha[sl * 4 * kPart + r] = al * sc * Chi::norm(r);
            ka.add(al * cr_sum);
          }
        };
        float c[NLM];
        if (PAIR || MAXT > 384 || n_slot <= nw) {
          for (int sl = warp; sl < n_slot; sl += nw) {
            sum_slot(sl, lane, 32, c);
            group_totals<32, NLM>(c, [&](int r, float total) { finish(sl, r, total); });
          }
        } else {
          for (int s0 = warp * 4; s0 < n_slot; s0 += nw * 4) {
            const int sl = s0 + (lane >> 3);
            sum_slot(sl, lane & 7, 8, c);
            group_totals<8, NLM>(c, [&](int r, float total) {
              if (sl < n_slot) finish(sl, r, total);
            });
          }
        }
      }
      {
        const DF ap = df_warp_sum(df_of(ka));
        if (lane == 0) red_a[warp] = make_float2(ap.hi, ap.lo);
      }
      if constexpr (PAIR) cooperative_groups::this_cluster().sync();
      else __syncthreads();

      // ---- phase 3: projector scatter U += chi alpha  ||  a_k ----
      if constexpr (PAIR) {
        // alpha from the two CTAs' rows, and <P, V_nl P> = sum Gamma_l c^2 over the slots, the same
        // sum in both CTAs
        Kahan kn;
        for (int e = threadIdx.x; e < n_slot * NLM; e += blockDim.x) {
          const int sl = e / NLM, r = e - sl * NLM;
          const TypeDesc &td = p.types[slot_type[sl]];
          const int l = p.rank_l[r];
          const float gl = (td.chan_mask & (1 << l)) ? float(td.gamma[l]) : 0.f;
          const float cv = cx[e] + cx[maxi * NLM + e];
          alpha[sl * 4 * kPart + r] = gl * cv * sc * Chi::norm(r);
          kn.add(gl * cv * cv);
        }
        const DF np = df_warp_sum(df_of(kn));
        if (lane == 0) red_n[warp] = make_float2(np.hi, np.lo);
        __syncthreads();
      }
      for (int u = 0; u < w_units; u++) {
        float4 T[NCH][kRun], meta;
        load_unit(u, T, meta);
        const unsigned w = __float_as_uint(meta.x);
        const float4 *al = reinterpret_cast<const float4 *>(alpha) + (w & 1023u) * kPart;
        float q[NLM];
#pragma unroll
        for (int i = 0; i < kPart; i++) {
          const float4 t = al[i];
          q[4 * i] = t.x;
          if (4 * i + 1 < NLM) q[4 * i + 1] = t.y;
          if (4 * i + 2 < NLM) q[4 * i + 2] = t.z;
          if (4 * i + 3 < NLM) q[4 * i + 3] = t.w;
        }
        const unsigned a = aU0 + itemU + (unsigned)((int)((w >> 10) & 63u) * PB);
        float4 v[kRun];
#pragma unroll
        for (int i = 0; i < kRun; i++) v[i] = lds_quad(a + (unsigned)(i * PB));
        Chi::scatter(p, T, v, meta.y, meta.z, meta.w, q);
#pragma unroll
        for (int i = 0; i < kRun; i++) sts_quad_if(u < units, a + (unsigned)(i * PB), v[i]);
      }
      DF adf;
      if constexpr (PAIR) {
        // a_k: CTA 0's stencil partials, CTA 1's, then the projector part (fixed order)
        auto cl = cooperative_groups::this_cluster();
        const float2 *ra0 = cr == 0 ? red_a : cl.map_shared_rank(red_a, 0);
        const float2 *ra1 = cr == 1 ? red_a : cl.map_shared_rank(red_a, 1);
        adf = df_add(df_add(df_all_reduce(ra0, nw), df_all_reduce(ra1, nw)), df_all_reduce(red_n, nw));
      } else {
        adf = df_all_reduce(red_a, nw);
      }
      __syncthreads();

      // ---- phase 4: w = U - a_k v, P <- w, U <- v, b_k^2 partial ----
      {
        const DF ak = df_div(adf, n2);
        const float2 nah2 = splat(-ak.hi), nal2 = splat(-ak.lo);
        Kahan kb;
        // owned planes.  PAIR: quads [h0, h1) are the
        // peer's halo planes and also go to its P at e + dpeer.
        const int nown = nzo * PS4;
        int h0 = 0, h1 = 0, dpeer = 0;
        float4 *P4peer = P4;
        if constexpr (PAIR) {
          const PairPlanes pq = pair_planes(nz, p.zsplit, cr ^ 1);
          h0 = (max(zo0, pq.pz0) - zo0) * PS4;
          h1 = (min(zo1, pq.pz1) - zo0) * PS4;
          dpeer = (zo0 - pq.pz0) * PS4;
          P4peer = cooperative_groups::this_cluster().map_shared_rank(P4, cr ^ 1);
        }
        if constexpr (kSwap) {
          // w goes where U was, and P stays as the next U (scaled through gamma)
          const float2 nahs2 = splat(-ak.hi * sc), nals2 = splat(-ak.lo * sc);
          unsigned ap = aP0 + 16u * threadIdx.x, au = aU0 + 16u * threadIdx.x;
          const unsigned step = 16u * blockDim.x;
          for (int e = threadIdx.x; e < nown; e += blockDim.x) {
            const unsigned at = au;
            const float4 pv = lds_quad(ap), uv = lds_quad(au);
            ap += step;
            au += step;
            const float2 w01 = fma2(nals2, lo(pv), fma2(nahs2, lo(pv), lo(uv)));
            const float2 w23 = fma2(nals2, hi(pv), fma2(nahs2, hi(pv), hi(uv)));
            sts_quad_if(true, at, make_float4(w01.x, w01.y, w23.x, w23.y));
            const float2 q = fma2(w01, w01, mul2(w23, w23));
            kb.add(q.x + q.y);
          }
        } else {
          // the next quad's P and U are read before this quad's are written
          float4 npv = zero4, nuv = zero4;
          if (threadIdx.x < nown) {
            npv = P4o[threadIdx.x];
            nuv = U4[threadIdx.x];
          }
          for (int e = threadIdx.x; e < nown; e += blockDim.x) {
            const float4 pv = npv, uv = nuv;
            if (e + (int)blockDim.x < nown) {
              npv = P4o[e + blockDim.x];
              nuv = U4[e + blockDim.x];
            }
            const float2 v01 = mul2(lo(pv), sc2), v23 = mul2(hi(pv), sc2);
            const float2 w01 = fma2(nal2, v01, fma2(nah2, v01, lo(uv)));
            const float2 w23 = fma2(nal2, v23, fma2(nah2, v23, hi(uv)));
            const float4 w4 = make_float4(w01.x, w01.y, w23.x, w23.y);
            P4o[e] = w4;
            if constexpr (PAIR) {
              if (e >= h0 && e < h1) P4peer[e + dpeer] = w4;
            }
            U4[e] = make_float4(v01.x, v01.y, v23.x, v23.y);
            const float2 q = fma2(w01, w01, mul2(w23, w23));
            kb.add(q.x + q.y);
          }
        }
        const DF bp = df_warp_sum(df_of(kb));
        if (lane == 0) red_b[warp] = make_float2(bp.hi, bp.lo);
        if (threadIdx.x == 0) sum_a[j] = make_float2(adf.hi, adf.lo);
      }
      DF b2;
      if constexpr (PAIR) {  // the halo planes and both CTAs' b partials are in place
        auto cl = cooperative_groups::this_cluster();
        cl.sync();
        const float2 *rb0 = cr == 0 ? red_b : cl.map_shared_rank(red_b, 0);
        const float2 *rb1 = cr == 1 ? red_b : cl.map_shared_rank(red_b, 1);
        b2 = df_add(df_all_reduce(rb0, nw), df_all_reduce(rb1, nw));
      } else {
        __syncthreads();
        b2 = df_all_reduce(red_b, nw);
      }
      if (threadIdx.x == 0) sum_b[j] = make_float2(b2.hi, b2.lo);
      steps = j + 1;
      if (!(b2.hi > 0.f) || !isfinite(b2.hi)) {  // breakdown: the Krylov space is invariant
        if (threadIdx.x == 0) atomicOr(status, kStatusBreakdown);
        break;
      }
      // the next vector's scale, the power of two that brings |s P|^2 into [1, 4), and
      // gamma = <s' w, H s P> / |s P|^2 = s' |w|^2 / (s^2 |P|^2)
      const float nsc = unit_scale(b2.hi);
      const DF g = df_div(b2, n2);
      const float gs = kSwap ? nsc / sc : nsc / (sc * sc);  // kSwap: U is P = v / s
      gam = DF{g.hi * gs, g.lo * gs};
      n2 = b2;
      sc = nsc;
      if constexpr (kSwap) {
        const unsigned t = aP0;
        aP0 = aU0;
        aU0 = t;
      }
    }
    __syncthreads();
    if (cr == 0)
      for (int r = threadIdx.x; r < p.nqp; r += blockDim.x) {
        double av = 0.0, bv = 0.0;  // after a breakdown
        if (r < steps) {
          const float2 one = make_float2(1.f, 0.f), np = r ? sum_b[r - 1] : one;
          const double n = (double)np.x + np.y;
          av = ((double)sum_a[r].x + sum_a[r].y) / n + p.hshift;
          bv = sqrt(((double)sum_b[r].x + sum_b[r].y) / n) / (double)(r ? unit_scale(np.x) : 1.f);
        }
        double *o = ab_out + (node - p.node_begin) * 2 * p.nqp;
        o[r] = av;
        o[p.nqp + r] = bv;
      }
    // the next node's units (or the release below) take the places that this node's warps read
    tmem_sync();
  }
  // no CTA of a pair leaves while its peer may still read its shared memory
  if constexpr (PAIR) cooperative_groups::this_cluster().sync();
  if (warp == 0) tc5::tmem_dealloc((unsigned)cnt[4], (uint32_t)p.list_columns);
}

template <int MASK, int MAXT, bool ISO>
__global__ void __launch_bounds__(MAXT, 1)
    lanczos_quad_kernel(const __grid_constant__ LanczosParams p, const float *__restrict__ veffq,
                        const ImageMeta *__restrict__ images, const float *__restrict__ tables,
                        unsigned char *proj_scratch, double *__restrict__ ab_out,
                        int *__restrict__ status) {
  quad_body<MASK, MAXT, ISO, false>(p, veffq, images, tables, proj_scratch, ab_out, status);
}

// One node per cluster of two CTAs (cubes whose P and U do not fit one CTA).
template <int MASK, bool ISO>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
    lanczos_quad_pair_kernel(const __grid_constant__ LanczosParams p,
                             const float *__restrict__ veffq, const ImageMeta *__restrict__ images,
                             const float *__restrict__ tables, unsigned char *proj_scratch,
                             double *__restrict__ ab_out, int *__restrict__ status) {
  quad_body<MASK, 384, ISO, true>(p, veffq, images, tables, proj_scratch, ab_out, status);
}

template <int MASK, int MAXT, bool ISO>
cudaError_t launch_quad_variant(const LanczosParams &p, int grid, int block, size_t smem,
                                cudaStream_t s, const void *veffq, const ImageMeta *images,
                                const void *tables, void *proj_scratch, double *ab, int *status) {
  if (block > MAXT) return cudaErrorInvalidConfiguration;
  auto k = lanczos_quad_kernel<MASK, MAXT, ISO>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<grid, block, smem, s>>>(p, (const float *)veffq, images, (const float *)tables,
                              (unsigned char *)proj_scratch, ab, status);
  return cudaGetLastError();
}

template <int MASK, bool ISO>
cudaError_t launch_quad_pair_variant(const LanczosParams &p, int grid, int block, size_t smem,
                                     cudaStream_t s, const void *veffq, const ImageMeta *images,
                                     const void *tables, void *proj_scratch, double *ab,
                                     int *status) {
  if (block > 384 || grid % 2 != 0) return cudaErrorInvalidConfiguration;
  auto k = lanczos_quad_pair_kernel<MASK, ISO>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<grid, block, smem, s>>>(p, (const float *)veffq, images, (const float *)tables,
                              (unsigned char *)proj_scratch, ab, status);
  return cudaGetLastError();
}

// Clusters of two that can be resident at once for this block and shared-memory size.
template <int MASK, bool ISO>
cudaError_t pair_max_clusters(int block, size_t smem, int *clusters) {
  auto k = lanczos_quad_pair_kernel<MASK, ISO>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2, 1, 1);
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaOccupancyMaxActiveClusters(clusters, (void *)k, &cfg);
}

}  // namespace lq
}  // namespace sq
