// stage_pair_impl.cuh -- z-marching RK stage kernels for sm_100a with two
// x-adjacent cells per thread (templates; instantiated by pair_*.cu).
//
// One RK stage is split along the velocity-stress structure of the equations:
// the velocity part differentiates only the six stresses and the stress part
// only the three velocities.  A CTA of 16 x 8 threads owns a tile of 32 x 8
// (x, y) columns, each thread the cell pair (2t, 2t+1) of its row, and marches
// through a chunk of z-planes; persistent CTAs walk the (tile, z-chunk) items.
// The 32 x 8 tile loads 2.2 halo values per cell and component (64 x 4: 2.8),
// which is what lets three CTAs share an SM, and its 32-cell columns put fewer
// cells into tiles that touch an x layer.
//
// Items come in two lists with kernels of their own.  Lean items hold no PML
// cell and no cell outside the grid: their kernel needs 94-142 registers
// instead of 160-240, so it keeps three (16-bit storage: four) CTAs per SM
// where the one kernel for both kept two (three), and runs both parts of a
// tile side by side (they share the stage input's V and sigma in L2).  The
// march is bound by latency and instruction fetch before it is bound by HBM,
// so resident warps count: at three CTAs the lean launch of the 256x256x128
// hill's inner stage moves 67% of the DRAM peak (52-58% before), that of the
// 600x600x250 one 5.8 TB/s.  Unrolling the march by 2 or
// 5 (no register moves in the z-window) is slower: 14.9 -> 15.2 and 16.5 ms on
// the 600x600x250 hill; four CTAs with two slots too (15.4 ms).
//
// Pairs make every per-cell quantity a float2: the stencil and RHS
// arithmetic runs as packed FFMA2 / FMUL2 / FADD2 (one instruction for both
// cells), and the shared-memory reads, the pointwise operands and the
// global stores are 64-bit accesses.  Only the x-derivative assembles some of
// its operand pairs from neighbouring pairs.
//
// The march runs against the long reach of the z-stencil: a forward stencil
// (reach -1..+3) marches downwards, a backward one (reach -3..+1) upwards, so
// the stencil always needs one plane ahead and three behind.  Each plane
// arrives by TMA (cp.async.bulk.tensor, no multicast) into one slot of a
// shared-memory ring of 3 or 4, on one mbarrier per slot:
//   * the differentiated components with an x/y halo, one 4-D box
//     {40 x, 14 y, 1 z, NC components} (x from -4, y from -3);
//   * the pointwise operands of the plane, boxes {32, 8, 1, n}: the RK
//     registers (FW and/or tW), the media coefficients and the metric.
// A plane is needed one iteration after it lands (its centre enters the
// per-thread register window of five planes) and in the next one (x/y
// stencils, pointwise operands); one or two further planes are in flight.
//
// The per-cell arithmetic is that of the reference's CalDiffmix + CalWavemix
// + Iteration* (src/calculate.cu:4121-4621, 6330-6734); the top three layers'
// velocities come from the traction-image kernel (timg.cu) and point sources
// from a separate tiny kernel (solver.cu).  CFS-PML auxiliaries are read and
// written with 64-bit global accesses (prefetched into L2 by tensor prefetch
// when the plane's slot is issued).
//
// Every mbarrier wait is bounded (about 2 s of %globaltimer).  On expiry the
// CTA leaves the march together (the flag is read after a barrier), records
// an error code in *err, waits (bounded) for its own copies still in flight
// and returns; the host then reports CGFD_ERR_TIMEOUT.  Before issuing any
// copy the CTA checks the alignment of its slots and barriers (error code 2).
#pragma once

#include "cgfd_internal.cuh"
#include "ptx_util.cuh"

#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <vector>

namespace cgfd {
namespace pair {
using namespace ptx;

constexpr int TX = 16, TY = 8, TT = TX * TY;  // threads per CTA
constexpr int NWARP = TT / 32;
constexpr int CX = 2 * TX;                    // cells per tile row
constexpr int HY = TY + 6;                    // halo box rows (y from -3)
constexpr int PWT = CX * TY;                  // values per pointwise tile
// halo box columns per storage type: x from -HOFF, so that the box origin is
// 16-byte aligned (x from -4 for FP32, -8 for 16-bit storage)
template <typename T> struct Halo {
  static constexpr int HOFF = (sizeof(T) == 4) ? 4 : 8;
  static constexpr int HX = CX + 2 * HOFF;
  static constexpr int HPL = HX * HY;  // values per component per halo plane
};
enum { PART_VEL = 0, PART_STR = 1 };
// launches of a stage: the velocity and the stress part of the general items,
// and both parts of the lean ones
enum { GEN_VEL = PART_VEL, GEN_STR = PART_STR, LEAN_BOTH = 2, NLIST = 3 };

// NC: staged (differentiated) components, C0: first of them in a set;
// NS: components the part updates (V: 3, T: 6), S0 their first index;
// NCOEF: media coefficients it reads, COEF0 the first (lam2mu, mu, irho).
template <int PART> struct PartInfo;
template <> struct PartInfo<PART_VEL> {
  static constexpr int NC = 6, C0 = TXX, NS = 3, S0 = VX, NCOEF = 1, COEF0 = 2;
};
template <> struct PartInfo<PART_STR> {
  static constexpr int NC = 3, C0 = VX, NS = 6, S0 = TXX, NCOEF = 2, COEF0 = 0;
};

// Slot layout (byte offsets): halo [NC][HY][HX] of the storage type T, then
// pointwise tiles of PWT values: u0 [NS] (FW, or tW in the final stage) and
// u1 [NS] (tW in the inner stages) of type T, coef [NCOEF] and met [3]
// (zeta_x, zeta_y, zeta_z) of FP32.  Every region starts on 128 B (a tensor
// copy's shared-memory destination must) and the slot stride is a multiple
// of 128 B.
constexpr uint32_t up128(uint32_t b) { return (b + 127u) / 128u * 128u; }
template <typename T, int PART> struct Slot {
  static constexpr int NC = PartInfo<PART>::NC, NS = PartInfo<PART>::NS;
  static constexpr uint32_t HALO_B = (uint32_t)(Halo<T>::HPL * NC * sizeof(T));
  static constexpr uint32_t U0 = up128(HALO_B);
  static constexpr uint32_t U_B = (uint32_t)(NS * PWT * sizeof(T));  // one register set
  static constexpr uint32_t U1 = U0 + up128(U_B);
  static constexpr uint32_t COEF = U1 + up128(U_B);
  static constexpr uint32_t MET = COEF + (uint32_t)(PartInfo<PART>::NCOEF * PWT * 4);
  static constexpr uint32_t BYTES = MET + 3 * PWT * 4;
};
static_assert(Slot<float, PART_VEL>::BYTES % 128 == 0 && Slot<float, PART_STR>::BYTES % 128 == 0,
              "slots");
static_assert(Slot<__half, PART_VEL>::BYTES % 128 == 0 && Slot<__half, PART_STR>::BYTES % 128 == 0,
              "slots");

// Resident CTAs per SM the kernels are compiled for, and ring slots.  General
// FP32: three CTAs at 168 registers with three slots, FA and tA read at the
// update: the 256x256x128 hill 1.69 ms per step against 1.77 with two CTAs,
// four slots and those loads early (the 160x160x80 half-space 0.53, 0.56).
// General 16-bit: three CTAs (four would spill 120-290 B per thread: 1.88
// instead of 1.49 ms).
template <typename T, bool LEAN> struct Res;
template <> struct Res<float, false> { static constexpr int CTAS = 3, NSLOT = 3; };
template <> struct Res<float, true> { static constexpr int CTAS = 3, NSLOT = 3; };
template <> struct Res<__half, false> { static constexpr int CTAS = 3, NSLOT = 4; };
template <> struct Res<__half, true> { static constexpr int CTAS = 4, NSLOT = 3; };
template <> struct Res<__nv_bfloat16, false> : Res<__half, false> {};
template <> struct Res<__nv_bfloat16, true> : Res<__half, true> {};
template <typename T, int LIST> struct Ring {
  static constexpr bool LEAN = LIST == LEAN_BOTH;
  static constexpr int NSLOT = Res<T, LEAN>::NSLOT, CTAS = Res<T, LEAN>::CTAS;
  static constexpr uint32_t BYTES_V = Slot<T, PART_VEL>::BYTES, BYTES_S = Slot<T, PART_STR>::BYTES;
  static constexpr uint32_t BYTES = LIST == GEN_VEL   ? BYTES_V
                                    : LIST == GEN_STR ? BYTES_S
                                    : BYTES_V > BYTES_S ? BYTES_V : BYTES_S;
  static constexpr size_t SMEM = (size_t)NSLOT * BYTES + 128 + 128;  // + barriers, align slack
  // 228 KB of shared memory per SM, 1 KB of it reserved per CTA
  static_assert(CTAS * (SMEM + 1024) <= 233472, "resident CTAs");
};

// Tensor maps of one launch.  halo/u0/u1/coef/met feed the ring; the aux
// maps (per direction: stage input, FA, tA) only drive L2 prefetches.
struct Maps {
  CUtensorMap halo;  // stage input, box {40, 14, 1, NC}
  CUtensorMap u0;    // FW (or tW), box {32, 8, 1, NS}
  CUtensorMap u1;    // tW, box {32, 8, 1, NS}
  CUtensorMap coef;  // media, box {32, 8, 1, NCOEF}
  CUtensorMap met;   // metric, box {32, 8, 1, 3}
  CUtensorMap aux[3][3];  // [direction][ain, afw, ta], box {32, 8, 1, NS}
};

// A work item: the planes [z0, z1) of the tile of columns at (i0, j0).  Packed
// into one 128-bit load: {i0, j0, z0, z1}, planes in 21 bits (grid sides reach
// 2^20 cells), the 11 above them hold 2 * model + part in two halves.
struct Item {
  int i0, j0, z0, z1, model, part;
};
constexpr int ITEM_Z_BITS = 21, ITEM_MODELS = 1 << (2 * (32 - ITEM_Z_BITS) - 1);
__host__ __device__ inline int4 pack_item(const Item &t) {
  const unsigned mp = 2u * (unsigned)t.model + (unsigned)t.part, hi = 32 - ITEM_Z_BITS;
  int4 v;
  v.x = t.i0;
  v.y = t.j0;
  v.z = (int)((unsigned)t.z0 | (mp & ((1u << hi) - 1)) << ITEM_Z_BITS);
  v.w = (int)((unsigned)t.z1 | mp >> hi << ITEM_Z_BITS);
  return v;
}
__host__ __device__ inline Item unpack_item(const int4 &v) {
  const unsigned z = (unsigned)v.z, w = (unsigned)v.w, mask = (1u << ITEM_Z_BITS) - 1;
  const unsigned mp = z >> ITEM_Z_BITS | w >> ITEM_Z_BITS << (32 - ITEM_Z_BITS);
  return Item{v.x, v.y, (int)(z & mask), (int)(w & mask), (int)(mp >> 1), (int)(mp & 1)};
}

// Work list of a launch: packed items ordered by decreasing estimated cost;
// CTAs take them in order from an atomic counter (reset by the last CTA of the
// launch before), so expensive PML items start first and the cheap interior
// items fill the tail.  A batched launch reads each model's stage arguments and
// tensor maps from the device arrays bargs / bmaps (one entry per model).
struct Work {
  const int4 *items[2];  // general, lean
  // per launch: next item, CTAs done; zero between launches
  int *counter;
  int nitems[2];
  int has_aux[3];     // direction has a PML (aux maps valid; single model)
  const StageArgs *bargs;
  const Maps *bmaps;   // [velocity, stress][model]
  int nmodels;
  // bound of every mbarrier wait, and the test hook of cgfd_test_withhold_copy:
  // with withhold >= 0 the halo copy of entry `withhold` (at most the last one)
  // of a list's first velocity item is not issued, so the wait for that plane
  // expires
  unsigned wait_us = WAIT_US;
  int withhold = -1;
};

// ---------------------------- float2 helpers ------------------------------
typedef float2 f2;
__device__ __forceinline__ f2 F2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ f2 S2(float a) { return make_float2(a, a); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f2 neg2(f2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ f2 lds2(const float *p) { return *reinterpret_cast<const f2 *>(p); }
// Reads of the ring: explicit shared-memory loads at 32-bit addresses.  The
// slots are written by tensor copies only, which the compiler does not see as
// stores.
__device__ __forceinline__ f2 lds_f2(uint32_t a) {
  f2 r;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "r"(a));
  return r;
}
__device__ __forceinline__ unsigned lds_u32(uint32_t a) {
  unsigned r;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(r) : "r"(a));
  return r;
}
// a pair of stored values (any storage type) as float2
template <typename T> __device__ __forceinline__ f2 ldp(uint32_t a) {
  if constexpr (sizeof(T) == 4) return lds_f2(a);
  else return Elem<T>::widen(lds_u32(a));
}
// r times a power-of-two component scale; FP32 storage is unscaled
template <typename T> __device__ __forceinline__ float scaled(float r, float s) {
  if constexpr (sizeof(T) == 4) return r;
  else return r * s;
}

// DRP/opt MacCormack 5-point operator on a pair, in the forward form
// (m1 = p - s, c0 = p, p1..p3 = p + s..3s for the marching sign s; r = s/h)
// (raw: h times the derivative; the marching sign S is in the coefficients)
template <int S>
__device__ __forceinline__ f2 drp2_raw(f2 m1, f2 c0, f2 p1, f2 p2, f2 p3) {
  f2 t = mul2(S2(S * CGFD_DA_1), m1);
  t = fma2(S2(S * CGFD_DA0), c0, t);
  t = fma2(S2(S * CGFD_DA1), p1, t);
  t = fma2(S2(S * CGFD_DA2), p2, t);
  return fma2(S2(S * CGFD_DA3), p3, t);
}

// x-derivative (raw) of the pair at ring address p (halo plane), its values C
// already in registers
template <int X, typename T>
__device__ __forceinline__ f2 dx_pair(uint32_t p, f2 C) {
  constexpr int E = sizeof(T);
  if constexpr (X > 0) {
    const f2 La = ldp<T>(p - 2 * E), Lb = ldp<T>(p + 2 * E), Lc = ldp<T>(p + 4 * E);
    return drp2_raw<X>(F2(La.y, C.x), C, F2(C.y, Lb.x), Lb, F2(Lb.y, Lc.x));
  } else {
    const f2 Lz = ldp<T>(p - 4 * E), La = ldp<T>(p - 2 * E), Lb = ldp<T>(p + 2 * E);
    return drp2_raw<X>(F2(C.y, Lb.x), C, F2(La.y, C.x), La, F2(Lz.y, La.x));
  }
}
// y-derivative (raw) of the same
template <int Y, typename T>
__device__ __forceinline__ f2 dy_pair(uint32_t p, f2 C) {
  constexpr uint32_t R = (uint32_t)(Y * Halo<T>::HX * (int)sizeof(T));  // (mod 2^32)
  return drp2_raw<Y>(ldp<T>(p - R), C, ldp<T>(p + R), ldp<T>(p + 2u * R), ldp<T>(p + 3u * R));
}

// masked pair access: bit 0 = first cell, bit 1 = second; p1 is the second
// cell's address (p0 + 1 wherever both bits can be set)
__device__ __forceinline__ f2 ld2(const float *p0, const float *p1, int m) {
  if (m == 3) return *reinterpret_cast<const f2 *>(p0);
  f2 r = F2(0.f, 0.f);
  if (m & 1) r.x = *p0;
  if (m & 2) r.y = *p1;
  return r;
}
__device__ __forceinline__ void st2(float *p0, float *p1, int m, f2 v) {
  if (m == 3) {
    *reinterpret_cast<f2 *>(p0) = v;
  } else {
    if (m & 1) *p0 = v.x;
    if (m & 2) *p1 = v.y;
  }
}
// the same for a field set of storage type T (second cell at p + 1)
template <typename T>
__device__ __forceinline__ f2 ldt2(const T *p, int m) {
  if (m == 3) return Elem<T>::ld2(p);
  f2 r = F2(0.f, 0.f);
  if (m & 1) r.x = Elem<T>::ld(p);
  if (m & 2) r.y = Elem<T>::ld(p + 1);
  return r;
}
template <typename T>
__device__ __forceinline__ void stt2(T *p, int m, f2 v) {
  if (m == 3) {
    Elem<T>::st2(p, v);
  } else {
    if (m & 1) Elem<T>::st(p, v.x);
    if (m & 2) Elem<T>::st(p + 1, v.y);
  }
}

// The per-thread register window of the z-stencil holds the staged
// components as stored: a float2 for FP32, the raw 16-bit pair (one 32-bit
// register) for FP16 / BF16, widened at use.  The widening is exact, so the
// arithmetic is that of a widened window, at half its registers (the 16-bit
// kernels run at 168 registers to fit three CTAs per SM).
template <typename T> struct Win {
  using type = unsigned;
  __device__ __forceinline__ static f2 get(unsigned v) { return Elem<T>::widen(v); }
  __device__ __forceinline__ static unsigned ld(uint32_t a) { return lds_u32(a); }
  // from global memory
  __device__ __forceinline__ static unsigned ldm(const T *p, int m) {
    if (m == 3) return *reinterpret_cast<const unsigned *>(p);
    const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
    return ((m & 1) ? (unsigned)h[0] : 0u) | ((m & 2) ? (unsigned)h[1] << 16 : 0u);
  }
  __device__ __forceinline__ static unsigned zero() { return 0u; }
};
template <> struct Win<float> {
  using type = f2;
  __device__ __forceinline__ static f2 get(f2 v) { return v; }
  __device__ __forceinline__ static type ld(uint32_t a) { return lds_f2(a); }
  __device__ __forceinline__ static type ldm(const float *p, int m) { return ldt2(p, m); }
  __device__ __forceinline__ static type zero() { return S2(0.f); }
};

// 16-bit storage keeps the RK accumulator as its difference from the step
// state, tW - FW: the difference is about a time step's change of the field,
// an order of magnitude below the field, so its FP16/BF16 rounding is that
// much finer (the accumulator's rounding was the largest share of the 16-bit
// storage error).  The final stage then reads FW besides it.
template <typename T> struct TwDelta { static constexpr bool value = sizeof(T) != 4; };
// the second pointwise register set is loaded: inner stages (tW, or the stage
// input under tW elision), and the final stage with the difference form (tW)
template <int KIND, typename T> struct TwoRegs {
  static constexpr bool value = KIND == 1 || (KIND == 2 && TwDelta<T>::value);
};

// RK update of one pair (Iteration*): KIND 0 first stage (u0 = FW; no tW
// under tW elision), 1 inner (u0 = FW, u1 = tW; in the second stage under
// elision u1 = the stage input W and tW = FW + rtw*(W - FW) + bdt*h),
// 2 final (u0 = tW; with the difference form u0 = FW and u1 = tW - FW).
// u0, u1 and the outputs are in stored units; adt, bdt carry the component's
// inverse scale (every set of a component shares its scale, so the rebuild
// and the difference are the same in stored units).
template <int KIND, typename T>
__device__ __forceinline__ void rk_store2(const StageArgs &a, T *out, T *tw, int m, f2 u0, f2 u1,
                                          f2 hh, float adt, float bdt) {
  constexpr bool D = TwDelta<T>::value;
  if (KIND == 0) {
    stt2(out, m, fma2(S2(adt), hh, u0));
    if (!a.tw_skip) stt2(tw, m, D ? mul2(S2(bdt), hh) : fma2(S2(bdt), hh, u0));
  } else if (KIND == 1) {
    stt2(out, m, fma2(S2(adt), hh, u0));
    f2 base = u1;
    if (a.tw_skip && a.rk == 1)
      base = D ? mul2(S2(a.rtw), add2(u1, neg2(u0))) : fma2(S2(a.rtw), add2(u1, neg2(u0)), u0);
    stt2(tw, m, fma2(S2(bdt), hh, base));
  } else {
    stt2(out, m, fma2(S2(bdt), hh, D ? add2(u0, u1) : u0));
  }
}

// ADE auxiliaries of one pair and direction: the stage input ai (FA in the
// first stage, A after) enters the RHS and is loaded before the stencil
// arithmetic.  The update reads FA and tA of one direction right before
// writing A (FA in the final stage) and tA, so that only one direction's
// values are live at the 168 registers that three CTAs per SM leave.
// o0/o1: the cells' indices, m: the cells' mask.
template <int KIND, int N>
struct Aux2 {
  f2 ai[N];
  __device__ __forceinline__ void load(const StageArgs &a, int d, size_t o0, size_t o1, int m,
                                       int c0) {
    const size_t as = a.g.astride[d];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const float *b = a.ain[d] + (c0 + q) * as;
      ai[q] = ld2(b + o0, b + o1, m);
    }
  }
  __device__ __forceinline__ void update(const StageArgs &a, int d, size_t o0, size_t o1, int m,
                                         int c0, const f2 *hh) const {
    const size_t as = a.g.astride[d];
    if constexpr (KIND == 0) {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        float *po = a.aout[d] + (c0 + q) * as, *pt = a.ta[d] + (c0 + q) * as;
        st2(po + o0, po + o1, m, fma2(S2(a.adt), hh[q], ai[q]));
        st2(pt + o0, pt + o1, m, fma2(S2(a.bdt), hh[q], ai[q]));
      }
    } else if constexpr (KIND == 1) {
      // FA and tA together: one memory round trip per direction
      f2 fu[N], tv[N];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const float *b = a.afw[d] + (c0 + q) * as;
        const float *t = a.ta[d] + (c0 + q) * as;
        fu[q] = ld2(b + o0, b + o1, m);
        tv[q] = ld2(t + o0, t + o1, m);
      }
#pragma unroll
      for (int q = 0; q < N; ++q) {
        float *po = a.aout[d] + (c0 + q) * as;
        float *pt = a.ta[d] + (c0 + q) * as;
        st2(po + o0, po + o1, m, fma2(S2(a.adt), hh[q], fu[q]));
        st2(pt + o0, pt + o1, m, fma2(S2(a.bdt), hh[q], tv[q]));
      }
    } else {
      f2 tu[N];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const float *b = a.ta[d] + (c0 + q) * as;
        tu[q] = ld2(b + o0, b + o1, m);
      }
#pragma unroll
      for (int q = 0; q < N; ++q) {
        float *po = a.aout[d] + (c0 + q) * as;
        st2(po + o0, po + o1, m, fma2(S2(a.bdt), hh[q], tu[q]));
      }
    }
  }
};

// Per-pair context of one item (tile column pair), shared by the two parts.
struct Pair {
  int i, j, ix, iy;   // first cell (valid and internal indices)
  int m;              // cells inside the grid (bit mask)
  int mx;             // cells inside an x layer (bit mask)
  bool ypml;          // the row is inside a y layer
  bool kept;          // (16-bit) inside the range of Geom::kx0
  int xa0, xa1, ya;   // auxiliary x indices of the two cells, y index of the row
  f2 iBx, apdx, dbx, bbx;  // x profiles of the two cells (1/B, APD, DB, B)
  float iBy, apdy, dby, bby;
};

// Per-plane quantities of the general (boundary) path.
struct Plane {
  int iz, k;
  size_t c;           // linear index of the first cell
  bool zpml, top, near_top, curved;
  bool met;           // the plane's metric tile was loaded
  float zz;           // zeta_z of the plane when no tile was loaded
  // zeta_z of this thread's pair
  template <typename P> __device__ __forceinline__ f2 zeta_z(const P &pw) const {
    return met ? pw.M(2) : S2(zz);
  }
};

// Pointwise operands of this thread's pair in the current slot (ring
// addresses).
template <typename T>
struct Pw2 {
  uint32_t u0, u1, coef, met;
  __device__ f2 U0(int q) const { return ldp<T>(u0 + q * PWT * (int)sizeof(T)); }
  __device__ f2 U1(int q) const { return ldp<T>(u1 + q * PWT * (int)sizeof(T)); }
  __device__ f2 C(int q) const { return lds_f2(coef + q * PWT * 4); }
  __device__ f2 M(int q) const { return lds_f2(met + q * PWT * 4); }
};

// auxiliary indices of the pair on a plane (X: per cell; Y, Z: the pair is
// contiguous)
struct AuxIdx {
  size_t x0, x1, y, z;
  float iBz, apdz, dbz;
  __device__ AuxIdx() : x0(0), x1(0), y(0), z(0), iBz(1.f), apdz(0.f), dbz(0.f) {}
  __device__ AuxIdx(const StageArgs &a, const Pair &e, const Plane &pl) {
    const Geom &g = a.g;
    iBz = 1.f / a.b[2][pl.iz];
    apdz = a.apd[2][pl.iz];
    dbz = a.db[2][pl.iz];
    const size_t rx = ((size_t)pl.iz * g.nyi + e.iy) * g.nxa;
    x0 = rx + e.xa0;
    x1 = rx + e.xa1;
    y = ((size_t)pl.iz * g.nya + e.ya) * g.px + e.ix;
    const int za = (pl.k < g.nabs[4]) ? pl.k : pl.k - (g.nk - g.nabs[5]) + g.nabs[4];
    z = ((size_t)za * g.nyi + e.iy) * g.px + e.ix;
  }
};

// -------------------------- velocity part ---------------------------------
// dV/dt = (1/rho) (d_xi sigma_x + d_eta sigma_y + zeta . d_zeta sigma), each
// directional part divided by its CFS beta; ADE auxiliaries for V.  The top 3
// layers' velocities come from the traction-image kernel (timg.cu); only
// their z auxiliaries are updated here.
// w[s][q]: staged component s on plane iz + (3 - q) * Z (q = 3: this plane).
template <typename T, int X, int Y, int Z, int KIND, bool LEAN>
__device__ __forceinline__ void vel_pair(const StageArgs &a, const Pair &e, const Plane &pl,
                                         uint32_t hp, const Pw2<T> &pw,
                                         const typename Win<T>::type (&w)[6][5],
                                         float rh) {
  constexpr uint32_t HPB = Halo<T>::HPL * sizeof(T);
  const size_t fs = a.g.fstride;
  auto W = [&](int s, int q) { return Win<T>::get(w[s][q]); };
  // 1/h factors carry the staged component's scale (stored units -> values)
  auto sr = [&](int s) { return S2(scaled<T>(rh, a.sc[TXX + s])); };
  auto dx_raw = [&](int s) { return dx_pair<X, T>(hp + s * HPB, W(s, 3)); };
  auto dy_raw = [&](int s) { return dy_pair<Y, T>(hp + s * HPB, W(s, 3)); };
  auto dz_raw = [&](int s) { return drp2_raw<Z>(W(s, 4), W(s, 3), W(s, 2), W(s, 1), W(s, 0)); };
  auto dx = [&](int s) { return mul2(dx_raw(s), sr(s)); };
  auto dy = [&](int s) { return mul2(dy_raw(s), sr(s)); };
  auto dz = [&](int s) { return mul2(dz_raw(s), sr(s)); };
  T *out = static_cast<T *>(a.out), *tw = static_cast<T *>(a.tw);
  auto adt = [&](int c) { return scaled<T>(a.adt, a.isc[c]); };
  auto bdt = [&](int c) { return scaled<T>(a.bdt, a.isc[c]); };

  if constexpr (LEAN) {
    // components of the stress set: Txx Tyy Tzz Txy Txz Tyz
    constexpr int SX[3] = {0, 3, 4}, SY[3] = {3, 1, 5}, SZ[3] = {4, 5, 2};
    const f2 irho = pw.C(0);
    const f2 ztz = pl.zeta_z(pw);
    f2 hw[3];
    if constexpr (sizeof(T) == 4) {
      // raw derivatives, 1/(rho h) once per component
      const f2 ir = mul2(irho, S2(rh));
      if (pl.curved) {
        const f2 ztx = pw.M(0), zty = pw.M(1);
        f2 z[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) z[q] = dz_raw(q);
#pragma unroll
        for (int q = 0; q < 3; ++q)
          hw[q] = mul2(fma2(ztz, z[SZ[q]],
                            fma2(zty, z[SY[q]], fma2(ztx, z[SX[q]], add2(dx_raw(SX[q]), dy_raw(SY[q]))))),
                       ir);
      } else {
#pragma unroll
        for (int q = 0; q < 3; ++q)
          hw[q] = mul2(fma2(ztz, dz_raw(SZ[q]), add2(dx_raw(SX[q]), dy_raw(SY[q]))), ir);
      }
    } else {
      // scaled derivatives (16-bit storage has a scale per component).  The order
      // of rounding is kept (Geom::kx0): contracted sums inside that range, sums
      // of the rounded products, as in the general path with B = 1, outside it
      const f2 fb = e.kept ? irho : S2(a.one);
      f2 zs[3];
      if (pl.curved) {
        const f2 ztx = pw.M(0), zty = pw.M(1);
        f2 z[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) z[q] = dz(q);
#pragma unroll
        for (int q = 0; q < 3; ++q)
          zs[q] = fma2(ztz, z[SZ[q]], fma2(zty, z[SY[q]], mul2(ztx, z[SX[q]])));
      } else {
#pragma unroll
        for (int q = 0; q < 3; ++q) zs[q] = mul2(ztz, dz(SZ[q]));
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        f2 x = dx(SX[q]), z = zs[q];
        if (!e.kept) {
          x = mul2(x, irho);
          z = mul2(z, irho);
        }
        hw[q] = fma2(z, fb, fma2(x, fb, mul2(dy(SY[q]), irho)));
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
      rk_store2<KIND>(a, out + (VX + q) * fs + pl.c, tw + (VX + q) * fs + pl.c, 3, pw.U0(q),
                      TwoRegs<KIND, T>::value ? pw.U1(q) : S2(0.f), hw[q], adt(VX + q), bdt(VX + q));
    return;
  } else {
  // general path: issue every auxiliary load before the stencil arithmetic
  const AuxIdx ix(a, e, pl);
  const int mx = e.mx, my = e.ypml ? e.m : 0, mz = pl.zpml ? e.m : 0;
  Aux2<KIND, 3> ax, ay, az;
  if (mx) ax.load(a, 0, ix.x0, ix.x1, mx, 0);
  if (my) ay.load(a, 1, ix.y, ix.y + 1, my, 0);
  if (mz) az.load(a, 2, ix.z, ix.z + 1, mz, 0);
  const f2 irho = pw.C(0);
  f2 ztx = S2(0.f), zty = S2(0.f);
  const f2 ztz = pl.zeta_z(pw);
  if (pl.curved) { ztx = pw.M(0); zty = pw.M(1); }
  f2 dxi[3], det[3], dzt[3];
  dxi[0] = dx(0);              // DxTxx
  dxi[1] = dx(3);              // DxTxy
  dxi[2] = dx(4);              // DxTxz
  det[0] = mul2(dy(3), irho);  // DyTxy
  det[1] = mul2(dy(1), irho);  // DyTyy
  det[2] = mul2(dy(5), irho);  // DyTyz
  const f2 DzTzz = dz(2), DzTxz = dz(4), DzTyz = dz(5);
  if (pl.curved) {
    const f2 DzTxx = dz(0), DzTyy = dz(1), DzTxy = dz(3);
    dzt[0] = fma2(ztz, DzTxz, fma2(zty, DzTxy, mul2(ztx, DzTxx)));
    dzt[1] = fma2(ztz, DzTyz, fma2(zty, DzTyy, mul2(ztx, DzTxy)));
    dzt[2] = fma2(ztz, DzTzz, fma2(zty, DzTyz, mul2(ztx, DzTxz)));
  } else {
    dzt[0] = mul2(ztz, DzTxz);
    dzt[1] = mul2(ztz, DzTyz);
    dzt[2] = mul2(ztz, DzTzz);
  }
  const f2 iBy = S2(e.iBy), iBz = S2(ix.iBz);
  f2 hw[3], hax[3], hay[3], haz[3];
  // 16-bit storage: the order of rounding of Geom::kx0 (such a pair has no
  // auxiliaries and B = 1); rows of the range that fill no tile, and models too
  // shallow for lean items, come through here.  Both orders are computed: 0.3-0.6%
  // of a 16-bit step (256x256x128 FP16 30.06 -> 30.22 ms a pass), a branch 1.6-2.8%.
  const bool kept = sizeof(T) != 4 && e.kept && !pl.zpml;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const f2 c = fma2(dzt[q], irho, fma2(dxi[q], irho, det[q]));
    dxi[q] = mul2(dxi[q], irho);
    dzt[q] = mul2(dzt[q], irho);
    const f2 r = fma2(dzt[q], iBz, fma2(det[q], iBy, mul2(dxi[q], e.iBx)));
    hw[q] = kept ? c : r;
  }
  if (mx) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      hw[q] = fma2(neg2(ax.ai[q]), e.iBx, hw[q]);
      hax[q] = fma2(neg2(e.apdx), ax.ai[q], mul2(dxi[q], e.dbx));
    }
  }
  if (my) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      hw[q] = fma2(neg2(ay.ai[q]), iBy, hw[q]);
      hay[q] = fma2(neg2(S2(e.apdy)), ay.ai[q], mul2(det[q], S2(e.dby)));
    }
  }
  if (mz) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      hw[q] = fma2(neg2(az.ai[q]), iBz, hw[q]);
      haz[q] = fma2(neg2(S2(ix.apdz)), az.ai[q], mul2(dzt[q], S2(ix.dbz)));
    }
  }
  // the top 3 layers' velocities (and their x/y auxiliaries) come from the
  // traction-image kernel; only the z auxiliaries are kept here
  const bool xy = !pl.near_top;
  const int mxs = xy ? mx : 0, mys = xy ? my : 0;
  if (mxs) ax.update(a, 0, ix.x0, ix.x1, mxs, 0, hax);
  if (mys) ay.update(a, 1, ix.y, ix.y + 1, mys, 0, hay);
  if (mz) az.update(a, 2, ix.z, ix.z + 1, mz, 0, haz);
  const int ms = xy ? e.m : 0;
#pragma unroll
  for (int q = 0; q < 3; ++q)
    rk_store2<KIND>(a, out + (VX + q) * fs + pl.c, tw + (VX + q) * fs + pl.c, ms, pw.U0(q),
                    TwoRegs<KIND, T>::value ? pw.U1(q) : S2(0.f), hw[q], adt(VX + q), bdt(VX + q));
  }
}

// --------------------------- stress part ----------------------------------
// dsigma/dt from Hooke's law with the velocity gradient in curvilinear form;
// the surface-layer d/dzeta of V comes from the traction-free matrices, the
// next two layers use the 2-point and Gottlieb 2-4 operators (VLOW).
// w[s][q]: velocity component s on plane iz + (3 - q) * Z.

// row r (0, 3, 6) of a surface matrix (9 planes from mv) times (u, v, t)
__device__ __forceinline__ f2 mat_row(const float *mv, size_t plane, int r, f2 u, f2 v, f2 t) {
  return fma2(lds2(mv + (r + 2) * plane), t,
              fma2(lds2(mv + (r + 1) * plane), v, mul2(lds2(mv + r * plane), u)));
}

// the stress rates' parts by direction, in the set order Txx Tyy Tzz Txy Txz Tyz
__device__ __forceinline__ void directional(f2 lam2mu, f2 lambda, f2 miu, f2 ztx, f2 zty, f2 ztz,
                                            const f2 *gx, const f2 *gy, const f2 *gz, f2 *dxi,
                                            f2 *det, f2 *dzt) {
  const f2 tx2 = mul2(ztx, gz[0]), ty2 = mul2(zty, gz[1]), tz2 = mul2(ztz, gz[2]);
  dxi[0] = mul2(lam2mu, gx[0]); det[0] = mul2(lambda, gy[1]);
  dzt[0] = fma2(lambda, tz2, fma2(lambda, ty2, mul2(lam2mu, tx2)));
  dxi[1] = mul2(lambda, gx[0]); det[1] = mul2(lam2mu, gy[1]);
  dzt[1] = fma2(lambda, tz2, fma2(lam2mu, ty2, mul2(lambda, tx2)));
  dxi[2] = mul2(lambda, gx[0]); det[2] = mul2(lambda, gy[1]);
  dzt[2] = fma2(lam2mu, tz2, fma2(lambda, ty2, mul2(lambda, tx2)));
  dxi[3] = mul2(gx[1], miu); det[3] = mul2(gy[0], miu);
  dzt[3] = mul2(fma2(ztx, gz[1], mul2(zty, gz[0])), miu);
  dxi[4] = mul2(gx[2], miu); det[4] = S2(0.f);
  dzt[4] = mul2(fma2(ztx, gz[2], mul2(ztz, gz[0])), miu);
  dxi[5] = S2(0.f); det[5] = mul2(gy[2], miu);
  dzt[5] = mul2(fma2(zty, gz[2], mul2(ztz, gz[1])), miu);
}

// stress rates of the velocity gradient (gx, gy: d/dx and d/dy of Vx, Vy, Vz;
// gz: d/dzeta): lambda times its trace + 2 mu times its diagonal, mu times the
// symmetric sums
__device__ __forceinline__ void hooke(f2 lam, f2 mu, bool curved, f2 ztx, f2 zty, f2 ztz,
                                      const f2 *gx, const f2 *gy, const f2 *gz, f2 *hw) {
  f2 ga = gx[0], gb = gy[1], gxy = add2(gx[1], gy[0]), gxz = gx[2], gyz = gy[2];
  const f2 gc = mul2(ztz, gz[2]), mu2 = add2(mu, mu);
  if (curved) {
    ga = fma2(ztx, gz[0], ga);
    gb = fma2(zty, gz[1], gb);
    gxy = fma2(ztx, gz[1], fma2(zty, gz[0], gxy));
    gxz = fma2(ztx, gz[2], gxz);
    gyz = fma2(zty, gz[2], gyz);
  }
  const f2 tr = mul2(lam, add2(add2(ga, gb), gc));
  hw[0] = fma2(mu2, ga, tr);
  hw[1] = fma2(mu2, gb, tr);
  hw[2] = fma2(mu2, gc, tr);
  hw[3] = mul2(mu, gxy);
  hw[4] = mul2(mu, fma2(ztz, gz[0], gxz));
  hw[5] = mul2(mu, fma2(ztz, gz[1], gyz));
}

template <typename T, int X, int Y, int Z, int KIND, bool LEAN>
__device__ __forceinline__ void str_pair(const StageArgs &a, const Pair &e, const Plane &pl,
                                         uint32_t hp, const Pw2<T> &pw,
                                         const typename Win<T>::type (&w)[3][5],
                                         float rh) {
  constexpr uint32_t HPB = Halo<T>::HPL * sizeof(T);
  const Geom &g = a.g;
  auto W = [&](int s, int q) { return Win<T>::get(w[s][q]); };
  const size_t fs = g.fstride;
  // 1/h factors carry the staged component's scale (stored units -> values)
  auto sr = [&](int s) { return S2(scaled<T>(rh, a.sc[VX + s])); };
  auto dx_raw = [&](int s) { return dx_pair<X, T>(hp + s * HPB, W(s, 3)); };
  auto dy_raw = [&](int s) { return dy_pair<Y, T>(hp + s * HPB, W(s, 3)); };
  auto dz_raw = [&](int s) { return drp2_raw<Z>(W(s, 4), W(s, 3), W(s, 2), W(s, 1), W(s, 0)); };
  auto dx = [&](int s) { return mul2(dx_raw(s), sr(s)); };
  auto dy = [&](int s) { return mul2(dy_raw(s), sr(s)); };
  auto dz = [&](int s) { return mul2(dz_raw(s), sr(s)); };
  T *out = static_cast<T *>(a.out), *tw = static_cast<T *>(a.tw);

  if constexpr (LEAN) {
    // FP32: raw derivatives, the moduli carry 1/h, Hooke's law in its trace form.
    // 16-bit storage has a scale per component, which the derivatives carry with
    // 1/h, and keeps its order of rounding: sums of the rounded products of the
    // three directions, as in the general path with B = 1.
    constexpr bool RAW = sizeof(T) == 4;
    auto gx = [&](int s) { return RAW ? dx_raw(s) : dx(s); };
    auto gy = [&](int s) { return RAW ? dy_raw(s) : dy(s); };
    auto sz = [&](int s) { return RAW ? S2((float)Z) : mul2(S2((float)Z), sr(s)); };
    const f2 DxVx = gx(0), DxVy = gx(1), DxVz = gx(2);
    const f2 DyVx = gy(0), DyVy = gy(1), DyVz = gy(2);
    f2 DzV[3];
    if (pl.iz < g.top - 2) {
#pragma unroll
      for (int q = 0; q < 3; ++q) DzV[q] = RAW ? dz_raw(q) : dz(q);
    } else if (pl.top) {
      const float *mv = a.matv + (size_t)e.iy * g.px + e.ix;
#pragma unroll
      for (int q = 0; q < 3; ++q)
        DzV[q] = add2(mat_row(mv + 9 * g.plane, g.plane, 3 * q, DyVx, DyVy, DyVz),
                      mat_row(mv, g.plane, 3 * q, DxVx, DxVy, DxVz));
    } else if (pl.iz == g.top - 1) {  // 2-point (M22)
#pragma unroll
      for (int q = 0; q < 3; ++q) DzV[q] = mul2(add2(W(q, 2), neg2(W(q, 3))), sz(q));
    } else {  // Gottlieb 2-4 (M24)
#pragma unroll
      for (int q = 0; q < 3; ++q)
        DzV[q] = mul2(fma2(S2(CGFD_MA2), W(q, 1),
                           fma2(S2(CGFD_MA1), W(q, 2), mul2(S2(CGFD_MA0), W(q, 3)))), sz(q));
    }
    const f2 rr = S2(RAW ? rh : 1.f);
    const f2 mu = RAW ? mul2(pw.C(1), rr) : pw.C(1);
    const f2 lam = RAW ? fma2(pw.C(0), rr, neg2(add2(mu, mu))) : fma2(S2(-2.f), mu, pw.C(0));
    const f2 ztz = pl.zeta_z(pw);
    f2 ztx = S2(0.f), zty = S2(0.f);
    if (pl.curved) { ztx = pw.M(0); zty = pw.M(1); }
    const f2 gx3[3] = {DxVx, DxVy, DxVz}, gy3[3] = {DyVx, DyVy, DyVz};
    f2 hw[6];
    if constexpr (RAW) {
      hooke(lam, mu, pl.curved, ztx, zty, ztz, gx3, gy3, DzV, hw);
    } else {
      f2 dxi[6], det[6], dzt[6];
      directional(pw.C(0), lam, mu, ztx, zty, ztz, gx3, gy3, DzV, dxi, det, dzt);
      const f2 one = S2(a.one);  // (add2 of products would be contracted)
#pragma unroll
      for (int q = 0; q < 6; ++q) hw[q] = fma2(dzt[q], one, fma2(det[q], one, dxi[q]));
    }
#pragma unroll
    for (int q = 0; q < 6; ++q)
      rk_store2<KIND>(a, out + (TXX + q) * fs + pl.c, tw + (TXX + q) * fs + pl.c, 3, pw.U0(q),
                      TwoRegs<KIND, T>::value ? pw.U1(q) : S2(0.f), hw[q],
                      scaled<T>(a.adt, a.isc[TXX + q]), scaled<T>(a.bdt, a.isc[TXX + q]));
    return;
  } else {
  // general path: issue every stage-input auxiliary load before the stencil.
  // The stress auxiliaries are kept as one per velocity derivative of the
  // direction (x: d/dx of Vx, Vy, Vz; y: d/dy; z: d/dzeta): each stress's
  // ADE auxiliary is the same linear combination of them, with cell-constant
  // coefficients, as its RHS term is of the derivatives (the ADE is linear),
  // so three values per direction stand for six.
  Aux2<KIND, 3> ax, ay, az;
  const AuxIdx ix(a, e, pl);
  const int mx = e.mx, my = e.ypml ? e.m : 0, mz = pl.zpml ? e.m : 0;
  if (mx) ax.load(a, 0, ix.x0, ix.x1, mx, 3);
  if (my) ay.load(a, 1, ix.y, ix.y + 1, my, 3);
  if (mz) az.load(a, 2, ix.z, ix.z + 1, mz, 3);
  const f2 DxVx = dx(0), DxVy = dx(1), DxVz = dx(2);
  const f2 DyVx = dy(0), DyVy = dy(1), DyVz = dy(2);
  f2 DzVx, DzVy, DzVz;
  // surface matrices of this pair (matVx2Vz: planes 0..8, matVy2Vz: 9..17)
  const float *mv = a.matv + (size_t)e.iy * g.px + e.ix;
  if (pl.top) {
    DzVx = add2(mat_row(mv + 9 * g.plane, g.plane, 0, DyVx, DyVy, DyVz),
                mat_row(mv, g.plane, 0, DxVx, DxVy, DxVz));
    DzVy = add2(mat_row(mv + 9 * g.plane, g.plane, 3, DyVx, DyVy, DyVz),
                mat_row(mv, g.plane, 3, DxVx, DxVy, DxVz));
    DzVz = add2(mat_row(mv + 9 * g.plane, g.plane, 6, DyVx, DyVy, DyVz),
                mat_row(mv, g.plane, 6, DxVx, DxVy, DxVz));
  } else if (pl.iz == g.top - 1) {  // 2-point (M22)
    auto m22 = [&](int s) {
      return mul2(add2(W(s, 2), neg2(W(s, 3))), mul2(S2((float)Z), sr(s)));
    };
    DzVx = m22(0);
    DzVy = m22(1);
    DzVz = m22(2);
  } else if (pl.iz == g.top - 2) {  // Gottlieb 2-4 (M24)
    auto m24 = [&](int s) {
      return mul2(fma2(S2(CGFD_MA2), W(s, 1), fma2(S2(CGFD_MA1), W(s, 2),
                                                  mul2(S2(CGFD_MA0), W(s, 3)))),
                  mul2(S2((float)Z), sr(s)));
    };
    DzVx = m24(0);
    DzVy = m24(1);
    DzVz = m24(2);
  } else {
    DzVx = dz(0);
    DzVy = dz(1);
    DzVz = dz(2);
  }

  const f2 lam2mu = pw.C(0), miu = pw.C(1);
  const f2 lambda = fma2(S2(-2.f), miu, lam2mu);
  f2 ztx = S2(0.f), zty = S2(0.f);
  const f2 ztz = pl.zeta_z(pw);
  if (pl.curved) { ztx = pw.M(0); zty = pw.M(1); }
  const f2 iBy = S2(e.iBy), iBz = S2(ix.iBz);
  f2 hw[6];
  if constexpr (sizeof(T) == 4) {
    // The ADE is linear in the velocity derivatives, so the auxiliaries enter
    // as a correction of the derivatives, (D - a) / B per direction, and
    // Hooke's law is applied once to the corrected gradient: 45 instead of
    // about 100 operations and 36 registers less than the three directional
    // parts and their auxiliary terms of all six stresses.
    f2 gx[3] = {DxVx, DxVy, DxVz}, gy[3] = {DyVx, DyVy, DyVz}, gz[3] = {DzVx, DzVy, DzVz};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (mx) gx[q] = add2(gx[q], neg2(ax.ai[q]));
      if (my) gy[q] = add2(gy[q], neg2(ay.ai[q]));
      if (mz) gz[q] = add2(gz[q], neg2(az.ai[q]));
      gx[q] = mul2(gx[q], e.iBx);
      gy[q] = mul2(gy[q], iBy);
      gz[q] = mul2(gz[q], iBz);
    }
    if (pl.top) {
      // the xi (eta) part of the surface-matrix d/dzeta of V belongs to the x
      // (y) auxiliaries (src/calculate.cu:4479-4491, 4527-4538)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        if (mx) gz[q] = add2(gz[q], neg2(mat_row(mv, g.plane, 3 * q, ax.ai[0], ax.ai[1], ax.ai[2])));
        if (my)
          gz[q] = add2(gz[q], neg2(mat_row(mv + 9 * g.plane, g.plane, 3 * q, ay.ai[0], ay.ai[1],
                                           ay.ai[2])));
      }
    }
    hooke(lambda, miu, pl.curved, ztx, zty, ztz, gx, gy, gz, hw);
  } else {
  f2 dxi[6], det[6], dzt[6];
  {
    const f2 gx[3] = {DxVx, DxVy, DxVz}, gy[3] = {DyVx, DyVy, DyVz}, gz[3] = {DzVx, DzVy, DzVz};
    directional(lam2mu, lambda, miu, ztx, zty, ztz, gx, gy, gz, dxi, det, dzt);
  }

  {
#pragma unroll
    for (int q = 0; q < 6; ++q)
      hw[q] = fma2(dzt[q], iBz, fma2(det[q], iBy, mul2(dxi[q], e.iBx)));
    // surface layer: the ADE auxiliaries also take the xi (eta) part of the
    // surface-matrix d/dzeta of V (src/calculate.cu:4479-4491, 4527-4538)
    auto surf = [&](f2 z1v, f2 z2v, f2 z3v, f2 f, f2 *out) {
      const f2 a1 = mul2(ztx, z1v), a2 = mul2(zty, z2v), a3 = mul2(ztz, z3v);
      out[0] = fma2(f, fma2(lambda, a3, fma2(lambda, a2, mul2(lam2mu, a1))), out[0]);
      out[1] = fma2(f, fma2(lambda, a3, fma2(lam2mu, a2, mul2(lambda, a1))), out[1]);
      out[2] = fma2(f, fma2(lam2mu, a3, fma2(lambda, a2, mul2(lambda, a1))), out[2]);
      out[3] = fma2(f, mul2(fma2(ztx, z2v, mul2(zty, z1v)), miu), out[3]);
      out[4] = fma2(f, mul2(fma2(ztx, z3v, mul2(ztz, z1v)), miu), out[4]);
      out[5] = fma2(f, mul2(fma2(zty, z3v, mul2(ztz, z2v)), miu), out[5]);
    };
    // the six stresses' terms of a vector v of x / y / zeta derivatives of
    // (Vx, Vy, Vz), as dxi / det / dzt are of the derivatives themselves
    // (on the surface layer with the surface-matrix part, scaled by B, which
    // the auxiliary RHS of the reference carries there)
    const float *my2 = mv + 9 * g.plane;
    auto terms_x = [&](const f2 *v, f2 *o) {
      o[0] = mul2(lam2mu, v[0]); o[1] = mul2(lambda, v[0]); o[2] = mul2(lambda, v[0]);
      o[3] = mul2(v[1], miu); o[4] = mul2(v[2], miu); o[5] = S2(0.f);
      if (pl.top)
        surf(mat_row(mv, g.plane, 0, v[0], v[1], v[2]), mat_row(mv, g.plane, 3, v[0], v[1], v[2]),
             mat_row(mv, g.plane, 6, v[0], v[1], v[2]), e.bbx, o);
    };
    auto terms_y = [&](const f2 *v, f2 *o) {
      o[0] = mul2(lambda, v[1]); o[1] = mul2(lam2mu, v[1]); o[2] = mul2(lambda, v[1]);
      o[3] = mul2(v[0], miu); o[4] = S2(0.f); o[5] = mul2(v[2], miu);
      if (pl.top)
        surf(mat_row(my2, g.plane, 0, v[0], v[1], v[2]), mat_row(my2, g.plane, 3, v[0], v[1], v[2]),
             mat_row(my2, g.plane, 6, v[0], v[1], v[2]), S2(e.bby), o);
    };
    auto terms_z = [&](const f2 *v, f2 *o) {
      const f2 tx2 = mul2(ztx, v[0]), ty2 = mul2(zty, v[1]), tz2 = mul2(ztz, v[2]);
      o[0] = fma2(lambda, tz2, fma2(lambda, ty2, mul2(lam2mu, tx2)));
      o[1] = fma2(lambda, tz2, fma2(lam2mu, ty2, mul2(lambda, tx2)));
      o[2] = fma2(lam2mu, tz2, fma2(lambda, ty2, mul2(lambda, tx2)));
      o[3] = mul2(fma2(ztx, v[1], mul2(zty, v[0])), miu);
      o[4] = mul2(fma2(ztx, v[2], mul2(ztz, v[0])), miu);
      o[5] = mul2(fma2(zty, v[2], mul2(ztz, v[1])), miu);
    };
    f2 t[6];
    if (mx) {
      terms_x(ax.ai, t);
#pragma unroll
      for (int q = 0; q < 6; ++q) hw[q] = fma2(neg2(t[q]), e.iBx, hw[q]);
    }
    if (my) {
      terms_y(ay.ai, t);
#pragma unroll
      for (int q = 0; q < 6; ++q) hw[q] = fma2(neg2(t[q]), iBy, hw[q]);
    }
    if (mz) {
      terms_z(az.ai, t);
#pragma unroll
      for (int q = 0; q < 6; ++q) hw[q] = fma2(neg2(t[q]), iBz, hw[q]);
    }
  }
  }
  {
    // one direction at a time: the derivative auxiliaries' RHS
    // (-APD a + DB dV), then their RK update
    f2 ha[3];
    if (mx) {
      ha[0] = fma2(neg2(e.apdx), ax.ai[0], mul2(DxVx, e.dbx));
      ha[1] = fma2(neg2(e.apdx), ax.ai[1], mul2(DxVy, e.dbx));
      ha[2] = fma2(neg2(e.apdx), ax.ai[2], mul2(DxVz, e.dbx));
      ax.update(a, 0, ix.x0, ix.x1, mx, 3, ha);
    }
    if (my) {
      ha[0] = fma2(neg2(S2(e.apdy)), ay.ai[0], mul2(DyVx, S2(e.dby)));
      ha[1] = fma2(neg2(S2(e.apdy)), ay.ai[1], mul2(DyVy, S2(e.dby)));
      ha[2] = fma2(neg2(S2(e.apdy)), ay.ai[2], mul2(DyVz, S2(e.dby)));
      ay.update(a, 1, ix.y, ix.y + 1, my, 3, ha);
    }
    if (mz) {
      ha[0] = fma2(neg2(S2(ix.apdz)), az.ai[0], mul2(DzVx, S2(ix.dbz)));
      ha[1] = fma2(neg2(S2(ix.apdz)), az.ai[1], mul2(DzVy, S2(ix.dbz)));
      ha[2] = fma2(neg2(S2(ix.apdz)), az.ai[2], mul2(DzVz, S2(ix.dbz)));
      az.update(a, 2, ix.z, ix.z + 1, mz, 3, ha);
    }
  }
  const int m = e.m;
#pragma unroll
  for (int q = 0; q < 6; ++q)
    rk_store2<KIND>(a, out + (TXX + q) * fs + pl.c, tw + (TXX + q) * fs + pl.c, m, pw.U0(q),
                    TwoRegs<KIND, T>::value ? pw.U1(q) : S2(0.f), hw[q], scaled<T>(a.adt, a.isc[TXX + q]),
                    scaled<T>(a.bdt, a.isc[TXX + q]));
  }
}

// ------------------------------ the march ---------------------------------
// State of a CTA's ring: the mbarrier phases and the copies in flight.
struct RingState {
  uint32_t ph = 0;    // parity of the next wait, per slot (same in every thread)
  uint32_t pend = 0;  // slots with copies not yet waited for (same in every thread)
};

// One work item of one part.  Returns with every read of the ring done and
// every copy landed, or with *abort_flag set (read after a barrier, so every
// thread sees it).
//
// LEAN items lie inside the layers' inner faces: no auxiliaries, B = 1, every
// cell of the tile valid.
template <typename T, int PART, int X, int Y, int Z, int KIND, bool LEAN>
__device__ __forceinline__ void march(const StageArgs &A, const Maps &M, const Work &wk,
                                      const bool (&aux_on)[3], const Item &it, bool withhold_item,
                                      unsigned char *ring, uint64_t *bars, RingState &rs,
                                      volatile int *abort_flag) {
  using S = Slot<T, PART>;
  constexpr int NSLOT = Res<T, LEAN>::NSLOT;
  constexpr int HOFF = Halo<T>::HOFF, HX = Halo<T>::HX, HPL = Halo<T>::HPL;
  constexpr int NC = PartInfo<PART>::NC, C0 = PartInfo<PART>::C0;
  constexpr int S0 = PartInfo<PART>::S0;
  constexpr int NCOEF = PartInfo<PART>::NCOEF, COEF0 = PartInfo<PART>::COEF0;
  constexpr int DIR = (Z > 0) ? -1 : 1;  // march direction in z
  constexpr int kinda = (KIND == 1) ? 3 : (KIND == 2 ? 2 : 1);  // aux sets read
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int warp = tid >> 5;
  const bool leader = (tid & 31) == 0;
  // this pair inside a halo plane and a pointwise tile (byte offsets)
  const uint32_t sc = (uint32_t)(((ty + 3) * HX + HOFF + 2 * tx) * (int)sizeof(T));
  const uint32_t tc = (uint32_t)(ty * CX + 2 * tx);
  const uint32_t ring32 = su32(ring);
  const Geom &g = A.g;
  const size_t fs = g.fstride;
  const bool flat = A.flat;
  auto met_tile = [&](int p) { return !flat && p >= A.zu_end; };
  // zeta_z of a plane without a metric tile (loaded one plane ahead)
  auto zz_of = [&](int p) { return flat ? 1.f : (p < A.zu_end ? A.zzp[p] : 0.f); };
  const float rh = 1.f / A.h;
  const int zlo = LFD + g.nabs[4], zhi = g.nk + LFD - g.nabs[5];  // z interior [zlo, zhi)
  const int i0 = it.i0, j0 = it.j0, z0 = it.z0;
  // the traction image owns the top three layers' velocities
  const int z1 = (LEAN && PART == PART_VEL) ? min(it.z1, g.top - 2) : it.z1;
  const int n = z1 - z0;                   // planes computed
  if (n <= 0) return;
  const int zf = (DIR > 0) ? z0 : z1 - 1;  // first plane in march order

  // Entry q = 0..n (plane zf + DIR*q; entry n is read for the window only)
  // goes to ring slot q % NSLOT.  The copies of an entry are shared out over
  // the warps' leaders, each of which adds its bytes to the slot's barrier:
  // issued by one thread they held that thread's warp, and at the next
  // barrier the CTA, for the length of five tensor copies and the prefetches.
  auto issue = [&](int q, int s) {
    rs.pend |= 1u << s;
    if (!leader) return;
    unsigned char *slot = ring + (size_t)s * S::BYTES;
    const int p = zf + DIR * q;
    const bool compute = q < n;
    const int cx = XO + i0, cy = LFD + j0;
    fence_proxy_async();
    if (warp == 0) {
      mbar_expect_tx(&bars[s], S::HALO_B);
      const bool withheld =
          PART == PART_VEL && withhold_item && wk.withhold >= 0 && min(wk.withhold, n) == q;
      if (!withheld) tma_load(slot, &M.halo, XO + i0 - HOFF, j0, p, C0, &bars[s]);
    } else if (warp == 1) {
      mbar_expect_tx(&bars[s], compute ? S::U_B : 0u);
      if (compute) tma_load(slot + S::U0, &M.u0, cx, cy, p, S0, &bars[s]);
    } else if (warp == 2) {
      const bool u1 = compute && TwoRegs<KIND, T>::value;
      mbar_expect_tx(&bars[s], u1 ? S::U_B : 0u);
      if (u1) tma_load(slot + S::U1, &M.u1, cx, cy, p, S0, &bars[s]);
    } else {
      const bool met = compute && met_tile(p);
      mbar_expect_tx(&bars[s], (compute ? (uint32_t)(PWT * 4) * NCOEF : 0u) +
                                   (met ? (uint32_t)(PWT * 4) * 3u : 0u));
      if (compute) tma_load(slot + S::COEF, &M.coef, cx, cy, p, COEF0, &bars[s]);
      if (met) tma_load(slot + S::MET, &M.met, cx, cy, p, 0, &bars[s]);
    }
    if constexpr (!LEAN) {
      // the plane's PML auxiliaries into L2 (tile- and plane-uniform presence)
      if (!compute || warp == 0) return;
      const int d = warp - 1;  // direction
      const int c0 = (PART == PART_VEL) ? 0 : 3;
      // (a box may lie partly outside its array -- before it at a high-side layer
      // narrower than the tile, since the low-side layer's cells come first -- and
      // fetches what lies inside; bx is a multiple of 4 values by xaoff)
      const int cxp = max(cx, 0), cyp = max(cy, 0);
      const bool on = aux_on[d] &&
                      (d == 0   ? (i0 < g.nabs[0] || i0 + CX > g.ni - g.nabs[1])
                       : d == 1 ? (j0 < g.nabs[2] || j0 + TY > g.nj - g.nabs[3])
                                : (p < zlo || p >= zhi));
      if (!on) return;
      const int bx = d == 0 ? ((i0 < g.nabs[0]) ? max(i0, 0) : i0 - (g.ni - g.nabs[1]) + g.xaoff)
                            : cxp;
      const int by = d == 1 ? ((j0 < g.nabs[2]) ? max(j0, 0) : j0 - (g.nj - g.nabs[3]) + g.nabs[2]) : cyp;
      const int bz = d == 2 ? ((p - LFD < g.nabs[4]) ? p - LFD
                                                     : p - LFD - (g.nk - g.nabs[5]) + g.nabs[4])
                            : p;
      for (int t = 0; t < kinda; ++t) {
        const int set = (KIND == 2 && t == 1) ? 2 : t;  // final stage: ain, ta
        tma_prefetch(&M.aux[d][set], bx, by, bz, c0);
      }
    }
  };
  for (int q = 0; q < NSLOT; ++q)
    if (q <= n) issue(q, q);
  auto wait = [&](int s) -> bool {  // every thread, in march order
    const bool ok = mbar_wait(&bars[s], (rs.ph >> s) & 1u, wk.wait_us);
    if (ok) {  // an expired wait leaves the copy pending for the drain
      rs.ph ^= 1u << s;
      rs.pend &= ~(1u << s);
    }
    return ok;
  };

  Pair e;
  e.i = i0 + 2 * tx;
  e.j = j0 + ty;
  e.ix = e.i + XO;
  e.iy = e.j + LFD;
  e.m = 3;
  e.kept = A.plain_interior && e.i >= g.kx0 && e.i < g.kx1 && e.j >= g.ky0 && e.j < g.ky1;
  if constexpr (!LEAN) {
    const bool rowok = e.j >= 0 && e.j < g.nj;  // (tile origins may lie left of the grid)
    e.m = (rowok && e.i >= 0 && e.i < g.ni ? 1 : 0) |
          (rowok && e.i + 1 >= 0 && e.i + 1 < g.ni ? 2 : 0);
    auto inx = [&](int i) { return i < g.nabs[0] || i >= g.ni - g.nabs[1]; };
    e.mx = ((e.m & 1) && inx(e.i) ? 1 : 0) | ((e.m & 2) && inx(e.i + 1) ? 2 : 0);
    e.ypml = e.m && (e.j < g.nabs[2] || e.j >= g.nj - g.nabs[3]);
    // xa1 = xa0 + 1 whenever both cells are in a layer (xaoff), and xa0 is
    // even then, so the pair is one aligned 64-bit access
    auto xa = [&](int i) { return (i < g.nabs[0]) ? i : i - (g.ni - g.nabs[1]) + g.xaoff; };
    e.xa0 = xa(e.i);
    e.xa1 = xa(e.i + 1);
    e.ya = (e.j < g.nabs[2]) ? e.j : e.j - (g.nj - g.nabs[3]) + g.nabs[2];
    e.iBx = S2(1.f); e.apdx = S2(0.f); e.dbx = S2(0.f); e.bbx = S2(1.f);
    e.iBy = 1.f; e.apdy = 0.f; e.dby = 0.f; e.bby = 1.f;
    if (e.m & 1) {
      e.bbx.x = A.b[0][e.ix]; e.iBx.x = 1.f / e.bbx.x;
      e.apdx.x = A.apd[0][e.ix]; e.dbx.x = A.db[0][e.ix];
    }
    if (e.m & 2) {
      e.bbx.y = A.b[0][e.ix + 1]; e.iBx.y = 1.f / e.bbx.y;
      e.apdx.y = A.apd[0][e.ix + 1]; e.dbx.y = A.db[0][e.ix + 1];
    }
    if (e.m) {
      e.bby = A.b[1][e.iy]; e.iBy = 1.f / e.bby;
      e.apdy = A.apd[1][e.iy]; e.dby = A.db[1][e.iy];
    }
  }

  // register window: w[c][q] = plane (current) + DIR * (q - 3)
  typename Win<T>::type w[NC][5];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int q = 0; q < 5; ++q) w[c][q] = Win<T>::zero();
  auto push_smem = [&](uint32_t slot) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
      for (int q = 0; q < 4; ++q) w[c][q] = w[c][q + 1];
      w[c][4] = Win<T>::ld(slot + sc + c * (HPL * (int)sizeof(T)));
    }
  };
  // the three planes behind the chunk come straight from global memory
  for (int k = 3; k >= 1; --k) {
    const size_t o = gidx(g, e.ix, e.iy, zf - DIR * k);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
      for (int q = 0; q < 4; ++q) w[c][q] = w[c][q + 1];
      const T *src = static_cast<const T *>(A.in) + (size_t)(C0 + c) * fs + o;
      w[c][4] = e.m ? Win<T>::ldm(src, e.m) : Win<T>::zero();
    }
  }
  // A wait that expires sets the CTA-wide abort flag; the flag is read only
  // after a __syncthreads, so every thread leaves the march together.
  if (!wait(0)) *abort_flag = 1;
  push_smem(ring32);
  __syncthreads();

  size_t c = gidx(g, e.ix, e.iy, zf);
  float zzn = zz_of(zf);
  int s = 0;  // slot of entry q
#pragma unroll 1
  for (int q = 0; q < n; ++q) {
    const float zzc = zzn;
    if (q + 1 < n) zzn = zz_of(zf + DIR * (q + 1));
    const int s1 = s + 1 == NSLOT ? 0 : s + 1;
    if (!wait(s1)) *abort_flag = 1;
    push_smem(ring32 + s1 * S::BYTES);
    // (after an expired wait the plane is computed from what the slot holds and
    // the march is left at the barrier; made to depend on the wait's outcome,
    // this branch was never taken in builds under register pressure)
    int mask = e.m;
    if constexpr (!LEAN) asm volatile("" : "+r"(mask));
    if (mask) {
      const uint32_t slot = ring32 + s * S::BYTES;
      Plane pl;
      pl.iz = zf + DIR * q;
      pl.k = pl.iz - LFD;
      pl.c = c;
      pl.top = (pl.iz == g.top);
      pl.near_top = pl.iz >= g.top - 2;
      pl.zpml = (pl.iz < zlo) || (pl.iz >= zhi);
      pl.curved = pl.iz >= g.con && !flat;
      pl.met = met_tile(pl.iz);
      pl.zz = zzc;
      const Pw2<T> pw{slot + S::U0 + tc * (int)sizeof(T), slot + S::U1 + tc * (int)sizeof(T),
                      slot + S::COEF + tc * 4, slot + S::MET + tc * 4};
      const uint32_t hp = slot + sc;
      if constexpr (PART == PART_VEL)
        vel_pair<T, X, Y, Z, KIND, LEAN>(A, e, pl, hp, pw, w, rh);
      else
        str_pair<T, X, Y, Z, KIND, LEAN>(A, e, pl, hp, pw, w, rh);
    }
    // the slot of entry q is free: refill it with entry q + NSLOT
    __syncthreads();
    if (*abort_flag) return;
    if (q + NSLOT <= n) issue(q + NSLOT, s);
    s = s1;
    c += (DIR > 0) ? g.plane : (size_t)0 - g.plane;
  }
}

// A persistent grid over one part of the general items of a stage, or over
// both parts of the lean ones: there a tile's velocity and stress items follow
// one another in the list, so the two run side by side and share in L2 what
// both read.
template <typename T, int X, int Y, int Z, int KIND, bool B, int LIST>
__global__ void __launch_bounds__(TT, (Ring<T, LIST>::CTAS))
    pair_kernel(const __grid_constant__ Maps maps_v, const __grid_constant__ Maps maps_s,
                const StageArgs a, const Work wk, int *err) {
  using R = Ring<T, LIST>;
  constexpr bool LEAN = R::LEAN;
  constexpr int NSLOT = R::NSLOT;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  // align the ring on the shared-window address itself
  unsigned char *sbase = smem_raw + ((128u - (su32(smem_raw) & 127u)) & 127u);
  unsigned char *ring = sbase;  // NSLOT slots
  uint64_t *bars = reinterpret_cast<uint64_t *>(sbase + (size_t)NSLOT * R::BYTES);
  __shared__ volatile int abort_flag;
  __shared__ volatile int s_next;
  const int tid = threadIdx.y * TX + threadIdx.x;

  if (tid == 0) {
    abort_flag = 0;
    const bool aligned = ((su32(bars) & 7u) == 0) && ((su32(ring) & 127u) == 0);
    if (!aligned) {
      abort_flag = 1;
      if (err) atomicExch(err, 2);
    } else {
      for (int s = 0; s < NSLOT; ++s) mbar_init(&bars[s], NWARP);
      fence_mbar_init();
    }
  }
  __syncthreads();
  RingState rs;
  int *const counter = wk.counter + 2 * LIST;
  if (!abort_flag) {
    for (;;) {
      // the next item, taken only when this CTA is free (a CTA never holds a
      // claim on work while it is still busy)
      if (tid == 0) s_next = atomicAdd(counter, 1);
      __syncthreads();
      const int cur = s_next;
      if (cur >= wk.nitems[LEAN]) break;  // CTA-uniform
      const Item it = unpack_item(wk.items[LEAN][cur]);
      const int part = LEAN ? it.part : LIST, model = B ? it.model : 0;
      // a batched launch reads the item's model's stage arguments in place
      // (global memory, read-only during the launch).  Copied per item into a
      // __shared__ StageArgs and read from there, the 16-bit batched stages
      // behaved as if every component scale were zero (FP32, whose kernels
      // never read the scales, was unaffected); read through a pointer to the
      // copy hidden from the compiler they were correct but 15% slower than
      // in place.
      const StageArgs &A = B ? wk.bargs[model] : a;
      const bool aux_on[3] = {B ? A.ain[0] != nullptr : wk.has_aux[0] != 0,
                              B ? A.ain[1] != nullptr : wk.has_aux[1] != 0,
                              B ? A.ain[2] != nullptr : wk.has_aux[2] != 0};
      if (LIST == GEN_VEL || (LEAN && part == PART_VEL))
        march<T, PART_VEL, X, Y, Z, KIND, LEAN>(A, B ? wk.bmaps[model] : maps_v, wk, aux_on, it,
                                                cur == 0, ring, bars, rs, &abort_flag);
      else if (LIST != GEN_VEL)
        march<T, PART_STR, X, Y, Z, KIND, LEAN>(
            A, B ? wk.bmaps[wk.nmodels + model] : maps_s, wk, aux_on, it, false, ring, bars, rs,
            &abort_flag);
      __syncthreads();  // all reads of the ring done before the next item reuses it
      if (abort_flag) break;
    }
    if (abort_flag && tid == 0) {
      if (err) atomicExch(err, 1);
      // drain: wait (bounded) for copies still in flight before the CTA's
      // shared memory goes away
      for (int s = 0; s < NSLOT; ++s)
        if (rs.pend & (1u << s)) mbar_wait(&bars[s], (rs.ph >> s) & 1u, wk.wait_us);
    }
  }
  // the last CTA to finish resets the counters for the next launch
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(counter + 1, 1) == (int)gridDim.x - 1) {
      counter[0] = 0;
      counter[1] = 0;
    }
  }
}

// Tensor maps of one model's buffers (host side, stage_pair.cu): per field
// set (FW, Wa, Wb, tW) the halo boxes of the two parts and the pointwise
// boxes of V (3) and T (6) components; media, metric; auxiliaries per
// direction and set (FA, A, tA) for V and T components.
struct ModelMaps {
  CUtensorMap haloV[4], haloS[4], ctrV[4], ctrT[4];
  CUtensorMap coefV, coefS, met;
  CUtensorMap auxV[3][3], auxT[3][3];
};

// Launch plan of one solver or of a batch of models.
struct Plan {
  std::vector<ModelMaps> mm;   // one per model
  std::vector<Geom> geoms;
  std::vector<char> plain;     // per model: StageArgs::plain_interior
  Work wk;
  int elem;                    // storage element type of the field sets
  int zchunk = 0;              // planes of the (first model's) interior z-chunks
  int grid[NLIST];             // CTAs per launch (0: no items)
  int sms = 0;                 // of the device
  WorkParams params;
  unsigned long long list_id = 0;  // hash of the lists
  int nmodels = 0;             // 0: single-model plan; else a batch of nmodels
  StageArgs *d_bargs = nullptr;  // batch: [pattern * 4 + stage][model]
  Maps *d_bmaps = nullptr;       // batch: [stage][part][model]
};

// a: the single model's stage arguments (X, Y, Z and the stage kind come
// from it in every case); a batched launch (B) takes each model's arguments
// and maps from wk instead
template <typename T, int X, int Y, int Z, int KIND, bool B, int LIST>
void launch_t(const Plan &pl, const Maps *m, const StageArgs &a, const Work &wk, int *err,
              cudaStream_t s) {
  pair_kernel<T, X, Y, Z, KIND, B, LIST>
      <<<pl.grid[LIST], dim3(TX, TY, 1), Ring<T, LIST>::SMEM, s>>>(m[0], m[1], a, wk, err);
}

template <typename T, int KIND, bool B, int LIST>
void launch_dirs(const Plan &pl, const Maps *m, const StageArgs &a, const Work &wk, int *err,
                 cudaStream_t s) {
  const int code = (a.X > 0 ? 4 : 0) + (a.Y > 0 ? 2 : 0) + (a.Z > 0 ? 1 : 0);
  switch (code) {
    case 0: launch_t<T, -1, -1, -1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
    case 1: launch_t<T, -1, -1, 1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
    case 2: launch_t<T, -1, 1, -1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
    case 3: launch_t<T, -1, 1, 1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
    case 4: launch_t<T, 1, -1, -1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
    case 5: launch_t<T, 1, -1, 1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
    case 6: launch_t<T, 1, 1, -1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
    default: launch_t<T, 1, 1, 1, KIND, B, LIST>(pl, m, a, wk, err, s); break;
  }
}

template <typename T, int KIND, bool B, int LIST>
cudaError_t set_attrs() {
  cudaError_t e = cudaSuccess;
  auto set = [&](const void *f) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)Ring<T, LIST>::SMEM);
  };
  set((const void *)pair_kernel<T, -1, -1, -1, KIND, B, LIST>);
  set((const void *)pair_kernel<T, -1, -1, 1, KIND, B, LIST>);
  set((const void *)pair_kernel<T, -1, 1, -1, KIND, B, LIST>);
  set((const void *)pair_kernel<T, -1, 1, 1, KIND, B, LIST>);
  set((const void *)pair_kernel<T, 1, -1, -1, KIND, B, LIST>);
  set((const void *)pair_kernel<T, 1, -1, 1, KIND, B, LIST>);
  set((const void *)pair_kernel<T, 1, 1, -1, KIND, B, LIST>);
  set((const void *)pair_kernel<T, 1, 1, 1, KIND, B, LIST>);
  return e;
}

// 0: the kernel cannot run on the current device
template <typename T, bool B, int LIST>
int resident_ctas() {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, pair_kernel<T, 1, 1, 1, 1, B, LIST>, TT,
                                                Ring<T, LIST>::SMEM);
  return per * sms;
}

// Entry points per storage type (f: FP32, h: FP16, b: BF16), RK stage kind
// and launch (v, s: general velocity, stress; l: lean), one translation unit each (pair_*.cu).
typedef void (*LaunchFn)(const Plan &, const Maps *, const StageArgs &, const Work &, int *,
                         cudaStream_t);
struct Entry {
  LaunchFn launch[2];     // [batched]
  cudaError_t (*attrs)(); // both forms
  int (*resident[2])();   // [batched] CTAs resident on the device
};
#define CGFD_PAIR_DECL(E) \
  Entry entry_##E##0v(), entry_##E##1v(), entry_##E##2v(), entry_##E##0s(), entry_##E##1s(), \
      entry_##E##2s(), entry_##E##0l(), entry_##E##1l(), entry_##E##2l();
CGFD_PAIR_DECL(f)
CGFD_PAIR_DECL(h)
CGFD_PAIR_DECL(b)
#undef CGFD_PAIR_DECL
template <typename T, int KIND, int LIST>
Entry make_entry() {
  return Entry{{launch_dirs<T, KIND, false, LIST>, launch_dirs<T, KIND, true, LIST>},
               [] {
                 const cudaError_t e = set_attrs<T, KIND, false, LIST>();
                 return e == cudaSuccess ? set_attrs<T, KIND, true, LIST>() : e;
               },
               {[]() -> int { if constexpr (KIND == 1) return resident_ctas<T, false, LIST>(); else return 0; },
                []() -> int { if constexpr (KIND == 1) return resident_ctas<T, true, LIST>(); else return 0; }}};
}

}  // namespace pair
}  // namespace cgfd
