// Element-wise data path: N sources -> reduce -> scale / divide -> cast -> M destinations.
//
// Role of the reference's ReduceOrCopyMulti and its functors
// (src/include/common_kernel.h:490-690, src/include/reduce_kernel.h:15-705), built
// differently: sources and destinations are plain pointers into this GPU's or a
// peer's symmetric heap (no FIFO slots), 16/32-bit floating inputs accumulate in
// fp32 in a fixed rank order so every rank computes bit-identical results, and
// the scale (gradient averaging, user PreMulSum scalar) and the output cast are
// applied in registers before the only store - the "fused scale / cast".
// The 16-byte packs are the unit of every vector access; a range whose pointers
// are not 16-byte aligned takes the scalar path.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "dfccl.h"
#include "platform.h"
#include "types.h"

namespace dfccl {

enum RedOp : int { OP_SUM = 0, OP_PROD = 1, OP_MAX = 2, OP_MIN = 3 };

struct DataArgs {
  int nsrc, ndst;
  const char* src[DF_MAX_RANKS];
  char* dst[DF_MAX_RANKS];
  uint64_t n;            // elements
  double scale;          // 1.0 = none
  int postDiv;           // 0 = none
};

template <int N> struct BitsOf;
template <> struct BitsOf<1> { typedef uint8_t type; };
template <> struct BitsOf<2> { typedef uint16_t type; };
template <> struct BitsOf<4> { typedef uint32_t type; };
template <> struct BitsOf<8> { typedef uint64_t type; };

template <typename T> DF_HD T ld_elem(const T* p) {
  typedef typename BitsOf<sizeof(T)>::type B;
  B b = *(const volatile B*)p;
  T v;
  __builtin_memcpy(&v, &b, sizeof(T));
  return v;
}
template <typename T> DF_HD void st_elem(T* p, T v) {
  typedef typename BitsOf<sizeof(T)>::type B;
  B b;
  __builtin_memcpy(&b, &v, sizeof(T));
  *(volatile B*)p = b;
}

// accumulator type and conversions
template <typename T> struct Elem { typedef T Acc; static DF_HD Acc up(T v) { return v; } static DF_HD T down(Acc a) { return a; } enum { isFloat = 0, isBf16 = 0 }; };
template <> struct Elem<int8_t> { typedef int32_t Acc; static DF_HD Acc up(int8_t v) { return v; } static DF_HD int8_t down(Acc a) { return (int8_t)a; } enum { isFloat = 0, isBf16 = 0 }; };
template <> struct Elem<uint8_t> { typedef uint32_t Acc; static DF_HD Acc up(uint8_t v) { return v; } static DF_HD uint8_t down(Acc a) { return (uint8_t)a; } enum { isFloat = 0, isBf16 = 0 }; };
template <> struct Elem<float> { typedef float Acc; static DF_HD Acc up(float v) { return v; } static DF_HD float down(Acc a) { return a; } enum { isFloat = 1, isBf16 = 0 }; };
template <> struct Elem<double> { typedef double Acc; static DF_HD Acc up(double v) { return v; } static DF_HD double down(Acc a) { return a; } enum { isFloat = 1, isBf16 = 0 }; };
template <> struct Elem<__half> { typedef float Acc; static DF_HD Acc up(__half v) { return __half2float(v); } static DF_HD __half down(Acc a) { return __float2half_rn(a); } enum { isFloat = 1, isBf16 = 0 }; };
template <> struct Elem<__nv_bfloat16> { typedef float Acc; static DF_HD Acc up(__nv_bfloat16 v) { return __bfloat162float(v); } static DF_HD __nv_bfloat16 down(Acc a) { return __float2bfloat16_rn(a); } enum { isFloat = 1, isBf16 = 1 }; };

template <int OP, typename A> DF_HD A red(A a, A b) {
  if (OP == OP_SUM) return a + b;
  if (OP == OP_PROD) return a * b;
  if (OP == OP_MAX) return a > b ? a : b;
  return a < b ? a : b;
}

template <typename Tin, typename Tout, typename A>
DF_HD typename Elem<Tout>::Acc finish(A a, double scale, int postDiv) {
  typedef typename Elem<Tout>::Acc AO;
  if (Elem<Tin>::isFloat) {
    if (scale != 1.0) a = (A)(a * (A)scale);
  } else if (postDiv) {
    a = a / (A)postDiv;
  } else if (scale != 1.0) {
    a = (A)((double)a * scale);
  }
  return (AO)a;
}

DF_HD void st8(void* p, uint2 v) {
#if DF_DEVICE_CODE
  asm volatile("st.relaxed.sys.global.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
#else
  __builtin_memcpy(p, &v, 8);
#endif
}

// ---- 16-byte pack <-> V accumulators, in registers only on the device.  (Going through a local
// array and memcpy is what the host build does; on the device an address-taken array can end up in
// local memory, and a load whose result is stored right away cannot overlap with the next load.)
DF_HD uint32_t packWord(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
DF_HD void setWord(uint4& v, int i, uint32_t w) { if (i == 0) v.x = w; else if (i == 1) v.y = w; else if (i == 2) v.z = w; else v.w = w; }

template <typename T> struct Lane;     // element k of a 16-byte pack <-> accumulator
#if DF_DEVICE_CODE
template <> struct Lane<float> {
  static DF_HD float get(const uint4& v, int k) { return __uint_as_float(packWord(v, k)); }
  static DF_HD void put(uint4& v, int k, float a) { setWord(v, k, __float_as_uint(a)); }
};
template <> struct Lane<int32_t> {
  static DF_HD int32_t get(const uint4& v, int k) { return (int32_t)packWord(v, k); }
  static DF_HD void put(uint4& v, int k, int32_t a) { setWord(v, k, (uint32_t)a); }
};
template <> struct Lane<uint32_t> {
  static DF_HD uint32_t get(const uint4& v, int k) { return packWord(v, k); }
  static DF_HD void put(uint4& v, int k, uint32_t a) { setWord(v, k, a); }
};
template <> struct Lane<__nv_bfloat16> {
  static DF_HD float get(const uint4& v, int k) { uint32_t w = packWord(v, k >> 1); return __uint_as_float((k & 1) ? (w & 0xffff0000u) : (w << 16)); }
  static DF_HD void put(uint4& v, int k, float a) {
    uint32_t h = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a));
    uint32_t w = packWord(v, k >> 1);
    setWord(v, k >> 1, (k & 1) ? ((w & 0x0000ffffu) | (h << 16)) : ((w & 0xffff0000u) | h));
  }
};
template <> struct Lane<__half> {
  static DF_HD float get(const uint4& v, int k) { uint32_t w = packWord(v, k >> 1); return __half2float(__ushort_as_half((unsigned short)((k & 1) ? (w >> 16) : (w & 0xffffu)))); }
  static DF_HD void put(uint4& v, int k, float a) {
    uint32_t h = (uint32_t)__half_as_ushort(__float2half_rn(a));
    uint32_t w = packWord(v, k >> 1);
    setWord(v, k >> 1, (k & 1) ? ((w & 0x0000ffffu) | (h << 16)) : ((w & 0xffff0000u) | h));
  }
};
template <> struct Lane<int8_t> {
  static DF_HD int32_t get(const uint4& v, int k) { return (int32_t)(int8_t)(packWord(v, k >> 2) >> (8 * (k & 3))); }
  static DF_HD void put(uint4& v, int k, int32_t a) { uint32_t sh = 8 * (k & 3), w = packWord(v, k >> 2); setWord(v, k >> 2, (w & ~(0xffu << sh)) | (((uint32_t)a & 0xffu) << sh)); }
};
template <> struct Lane<uint8_t> {
  static DF_HD uint32_t get(const uint4& v, int k) { return (packWord(v, k >> 2) >> (8 * (k & 3))) & 0xffu; }
  static DF_HD void put(uint4& v, int k, uint32_t a) { uint32_t sh = 8 * (k & 3), w = packWord(v, k >> 2); setWord(v, k >> 2, (w & ~(0xffu << sh)) | ((a & 0xffu) << sh)); }
};
template <> struct Lane<double> {
  static DF_HD double get(const uint4& v, int k) { return __hiloint2double((int)packWord(v, 2 * k + 1), (int)packWord(v, 2 * k)); }
  static DF_HD void put(uint4& v, int k, double a) { setWord(v, 2 * k, (uint32_t)__double2loint(a)); setWord(v, 2 * k + 1, (uint32_t)__double2hiint(a)); }
};
template <> struct Lane<int64_t> {
  static DF_HD int64_t get(const uint4& v, int k) { return (int64_t)(((uint64_t)packWord(v, 2 * k + 1) << 32) | packWord(v, 2 * k)); }
  static DF_HD void put(uint4& v, int k, int64_t a) { setWord(v, 2 * k, (uint32_t)(uint64_t)a); setWord(v, 2 * k + 1, (uint32_t)((uint64_t)a >> 32)); }
};
template <> struct Lane<uint64_t> {
  static DF_HD uint64_t get(const uint4& v, int k) { return ((uint64_t)packWord(v, 2 * k + 1) << 32) | packWord(v, 2 * k); }
  static DF_HD void put(uint4& v, int k, uint64_t a) { setWord(v, 2 * k, (uint32_t)a); setWord(v, 2 * k + 1, (uint32_t)(a >> 32)); }
};
#else
template <typename T> struct Lane {
  typedef typename Elem<T>::Acc A;
  static A get(const uint4& v, int k) { T e; __builtin_memcpy(&e, (const char*)&v + k * sizeof(T), sizeof(T)); return Elem<T>::up(e); }
  static void put(uint4& v, int k, A a) { T e = Elem<T>::down(a); __builtin_memcpy((char*)&v + k * sizeof(T), &e, sizeof(T)); }
};
#endif

// ---- whole-pack conversions: V accumulators <-> 16-byte words, few instructions per element
template <typename Tout, typename A, int V>
DF_HD void packAll(uint4* ow, const A* r) {
#if DF_DEVICE_CODE
  if (sizeof(Tout) == 2 && sizeof(A) == 4) {            // bf16 / fp16 from fp32: one convert per pair
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      uint32_t word;
      if (Elem<Tout>::isBf16) { __nv_bfloat162 h = __floats2bfloat162_rn((float)r[k], (float)r[k + 1]); word = *reinterpret_cast<uint32_t*>(&h); }
      else { __half2 h = __floats2half2_rn((float)r[k], (float)r[k + 1]); word = *reinterpret_cast<uint32_t*>(&h); }
      setWord(ow[(k / 2) / 4], (k / 2) % 4, word);
    }
    return;
  }
#endif
  constexpr int VO = 16 / (int)sizeof(Tout);
#pragma unroll
  for (int k = 0; k < V; ++k) Lane<Tout>::put(ow[k / VO], k % VO, (typename Elem<Tout>::Acc)r[k]);
}

// ---- sources that are not 16-byte aligned.  All sources of one call share one misalignment (they are the same offset
// into symmetric buffers), so a logical pack is 16 bytes that straddle two aligned packs: bytes [shift, shift + 16) of
// lo:hi.  The aligned packs are loaded as usual and shifted in registers; in a full trip the upper pack of a thread is
// the lower pack of its neighbour lane and comes by shuffle, so the memory traffic stays that of an aligned copy.
// (Role of the reference's misaligned-load helpers, src/collectives/device/op128.h:40-68.)
DF_HD uint4 shiftPack(const uint4& lo, const uint4& hi, uint32_t shift) {
#if DF_DEVICE_CODE
  const uint32_t bs = (shift & 3u) * 8u;
  uint32_t w0, w1, w2, w3, w4;
  switch (shift >> 2) {
    case 0: w0 = lo.x; w1 = lo.y; w2 = lo.z; w3 = lo.w; w4 = hi.x; break;
    case 1: w0 = lo.y; w1 = lo.z; w2 = lo.w; w3 = hi.x; w4 = hi.y; break;
    case 2: w0 = lo.z; w1 = lo.w; w2 = hi.x; w3 = hi.y; w4 = hi.z; break;
    default: w0 = lo.w; w1 = hi.x; w2 = hi.y; w3 = hi.z; w4 = hi.w; break;
  }
  return make_uint4(__funnelshift_r(w0, w1, bs), __funnelshift_r(w1, w2, bs), __funnelshift_r(w2, w3, bs), __funnelshift_r(w3, w4, bs));
#else
  unsigned char b[32];
  __builtin_memcpy(b, &lo, 16);
  __builtin_memcpy(b + 16, &hi, 16);
  uint4 o;
  __builtin_memcpy(&o, b + shift, 16);
  return o;
#endif
}

// The neighbour lane's pack (the last lane gets its own back); the whole warp calls it.  `at`: where this lane's pack was read.
DF_HD uint4 nextLane(const uint4& v, const char* at) {
#if DF_DEVICE_CODE
  return make_uint4(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1), __shfl_down_sync(0xffffffffu, v.z, 1),
                    __shfl_down_sync(0xffffffffu, v.w, 1));
#else
  return ld16(at + 16);
#endif
}

// Shifted packs without a second load: the aligned packs that a warp of `ws` lanes loads make ws - 1 logical ones, each from a lane's and its
// neighbour's.  (A host thread is a warp of one lane, which reads its neighbour's itself.)  A thread's packs are `first`, first + step, ...
struct ShiftedWalk { uint32_t lane, step; uint64_t first; };
DF_HD ShiftedWalk shiftedWalk(uint32_t tid, uint32_t nt, uint32_t ws) {
  const uint32_t makes = ws > 1 ? ws - 1 : 1, lane = tid % ws;
  ShiftedWalk w;
  w.lane = lane; w.step = nt / ws * makes; w.first = (uint64_t)(tid / ws * makes + lane);
  return w;
}
// The warp whose lane `lane` is at pack q has something to do (the same for its lanes); this lane loads aligned pack q (number nPacks holds
// the end of the last logical one); this lane makes packs of its own.
DF_HD bool shiftedWarpAt(uint64_t q, uint32_t lane, uint64_t nPacks) { return q - lane < nPacks; }
DF_HD bool shiftedLoads(uint64_t q, uint32_t lane, uint64_t nPacks) { return shiftedWarpAt(q, lane, nPacks) && q <= nPacks; }
DF_HD bool shiftedMakes(uint32_t lane, uint32_t ws) { return ws == 1 || lane != ws - 1; }

// U logical packs of one source for this thread; pack u starts `u * strideB` bytes after `s`, `shift` = s & 15.
// SHIFT = false: s is aligned.  FULL: every thread of the block loads all of its U packs (warp shuffles are safe).
template <bool FULL, bool SHIFT, int U>
DF_HD void loadPacks(uint4* out, const char* s, uint32_t strideB, uint32_t shift, uint64_t p0, uint32_t stride, uint64_t nPacks) {
  if (!SHIFT) {
#pragma unroll
    for (int u = 0; u < U; ++u) if (FULL || p0 + (uint64_t)u * stride < nPacks) out[u] = ld16(s + (uint64_t)u * strideB);
    return;
  }
  const char* a = s - shift;                       // aligned; every aligned pack touched holds at least one wanted byte
#if DF_DEVICE_CODE
  if (FULL) {                                      // every load before the first shuffle, which waits for its pack
    uint4 last[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      out[u] = ld16(a + (uint64_t)u * strideB);
      if ((threadIdx.x & 31) == 31) last[u] = ld16(a + (uint64_t)u * strideB + 16);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 hi = nextLane(out[u], nullptr);
      out[u] = shiftPack(out[u], (threadIdx.x & 31) == 31 ? last[u] : hi, shift);
    }
    return;
  }
#endif
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!(FULL || p0 + (uint64_t)u * stride < nPacks)) continue;
    out[u] = shiftPack(ld16(a + (uint64_t)u * strideB), ld16(a + (uint64_t)u * strideB + 16), shift);
  }
}

// First loose element of thread `tid`: the warps that the last, partly filled trip over `nPacks` leaves idle come first, so
// that the ragged end is on its way while that trip still waits for memory.
DF_HD uint64_t looseStart(int tid, int nt, uint64_t nPacks) {
  int used = (int)(nPacks % (uint64_t)nt + 31) & ~31;
  if (used >= nt) used = 0;
  return (uint64_t)(tid >= used ? tid - used : tid + nt - used);
}

// What a pack of sums becomes: scaled or divided, cast, in 16-byte words.
template <typename Tin, typename Tout>
DF_HD void finishPack(uint4* ow, typename Elem<Tin>::Acc* acc, typename Elem<Tin>::Acc mul, bool doMul, int postDiv, double dscale) {
  typedef typename Elem<Tin>::Acc A;
  constexpr int V = 16 / (int)sizeof(Tin), NW = (V * (int)sizeof(Tout) + 15) / 16;
  if (Elem<Tin>::isFloat) {
    if (doMul) {
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] = acc[k] * mul;
    }
  } else if (postDiv) {
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = acc[k] / (A)postDiv;
  } else if (doMul) {
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = (A)((double)acc[k] * dscale);
  }
#pragma unroll
  for (int w = 0; w < NW; ++w) ow[w] = make_uint4(0u, 0u, 0u, 0u);
  packAll<Tout, A, V>(ow, acc);
}
// `wide`: o is 32-byte aligned (looked at for results of 32 bytes only)
template <int OUTB>
DF_HD void storePack(char* o, const uint4* ow, bool wide) {
  if (OUTB == 8) st8(o, make_uint2(ow[0].x, ow[0].y));
  else if (OUTB == 32) st32(o, ow[0], ow[(OUTB + 15) / 16 - 1], wide);
  else {
#pragma unroll
    for (int w = 0; w < OUTB / 16; ++w) st16(o + 16 * w, ow[w]);
  }
}

// One noinline body per (input type, output type, operator): the daemon's register
// budget is the maximum over what it inlines, so the variants stay out of line.
// The hot loop is written for instruction count (it was issue-bound at 150 warp instructions
// per 16-byte pack in its first form): pointers are read from shared memory once per source
// and trip, indices are a base plus compile-time multiples of the stride, the bounds test is
// hoisted out of full trips, the scale is a float decided once, outputs are packed pairwise.
template <typename Tin, typename Tout, int OP, bool FULL, bool SHIFT, int U>
DF_HD void reduceTrip(const DataArgs* a, uint64_t p0, uint64_t nPacks, uint32_t strideB, int nsrc, int ndst,
                      typename Elem<Tin>::Acc mul, bool doMul, int postDiv, double dscale,
                      uint64_t srcOff, uint64_t dstOff, uint32_t shift) {
  typedef typename Elem<Tin>::Acc A;
  constexpr int V = 16 / (int)sizeof(Tin);
  constexpr int OUTB = V * (int)sizeof(Tout);
  constexpr int NW = (OUTB + 15) / 16;
  const uint32_t stride = strideB >> 4;
  const uint64_t off = srcOff + p0 * 16;
  A acc[U][V];
  uint4 cur[U], nxt[U];
  if (U == 1) {
    // a small call is one such trip: four sources at a time, or it would wait for memory once per source (509 bf16 of four
    // ranks: 8.5 us from the arrival to the end of the sum, a round trip each and another four for the ragged end)
    for (int j0 = 0; j0 < nsrc; j0 += 4) {
      uint4 in[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) if (j0 + q < nsrc) loadPacks<FULL, SHIFT, 1>(&in[q], a->src[j0 + q] + off, strideB, shift, p0, stride, nPacks);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (j0 + q >= nsrc) break;
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const A e = (A)Lane<Tin>::get(in[q], k);
          acc[0][k] = j0 + q == 0 ? e : red<OP>(acc[0][k], e);
        }
      }
    }
  } else {
  loadPacks<FULL, SHIFT, U>(cur, a->src[0] + off, strideB, shift, p0, stride, nPacks);
  for (int j = 1; j <= nsrc; ++j) {
    if (j < nsrc) loadPacks<FULL, SHIFT, U>(nxt, a->src[j] + off, strideB, shift, p0, stride, nPacks);
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const A e = (A)Lane<Tin>::get(cur[u], k);
        acc[u][k] = j == 1 ? e : red<OP>(acc[u][k], e);
      }
    }
    if (j < nsrc) {
#pragma unroll
      for (int u = 0; u < U; ++u) cur[u] = nxt[u];
    }
  }
  }
  uint4 ow[U][NW];
#pragma unroll
  for (int u = 0; u < U; ++u) finishPack<Tin, Tout>(ow[u], acc[u], mul, doMul, postDiv, dscale);
  for (int d = 0; d < ndst; ++d) {
    char* o = a->dst[d] + dstOff + p0 * OUTB;
    const bool wide = OUTB == 32 && ((uintptr_t)o & 31) == 0;      // the same for every thread of the block
#pragma unroll
    for (int u = 0; u < U; ++u) if (FULL || p0 + (uint64_t)u * stride < nPacks) storePack<OUTB>(o + (uint64_t)u * stride * OUTB, ow[u], wide);
  }
}

// The unrolled trips of one call, for aligned (SHIFT = false) or uniformly misaligned sources.
template <typename Tin, typename Tout, int OP, bool SHIFT>
DF_HD void reduceTrips(const DataArgs* a, uint64_t nPacks, int nsrc, int ndst, typename Elem<Tin>::Acc mul, bool doMul, int postDiv,
                       double scale, uint64_t srcOff, uint64_t dstOff, uint32_t shift) {
  // The sum carries the traffic; the rarer operators trade speed for code size, shifting takes registers.  (Shifted sums of as many sources
  // as reduceAhead does not take, reduce-scatter of 1 000 003 fp32, four packs with a shuffle behind every load / two with all loads first, us:
  // 3 ranks 45.0 / 36.3, 5 114 / 74, 7 197 / 119; 8 ranks bf16 -> fp32 141 / 91; shorter ones 3 - 20 % less too.)
  constexpr int U = OP == OP_SUM && !SHIFT ? 4 : 2;
  const int tid = df_tid(), nt = df_nthreads();
  // Software-pipelined over the sources inside a trip: the U loads of source j+1 are issued before
  // the U packs of source j are consumed, so up to 2*U 16-byte loads are in flight per thread.
  const uint64_t step = (uint64_t)nt * U;
  const uint32_t strideB = (uint32_t)nt * 16u;
  uint64_t base = 0;
  for (; base + step <= nPacks; base += step)
    reduceTrip<Tin, Tout, OP, true, SHIFT, U>(a, base + tid, nPacks, strideB, nsrc, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, shift);
  // what the unrolled trips leave: one pack per thread per trip, the last trip partly filled
  for (; base + nt <= nPacks; base += nt)
    reduceTrip<Tin, Tout, OP, true, SHIFT, 1>(a, base + tid, nPacks, strideB, nsrc, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, shift);
  if (base + tid < nPacks)
    reduceTrip<Tin, Tout, OP, false, SHIFT, 1>(a, base + tid, nPacks, strideB, nsrc, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, shift);
}

// Sums of N aligned sources, N = 2, 4 or 8: a thread's next 8 / N packs of every source are on their way while the present ones are
// added up and stored.  Bound: what a block's SM has in flight (one block of 480 threads an SM, 64 or 128 of them); in the trips above
// every source is a wait of its own, and a trip's loads are behind the stores of the one before.  us for whole all-reduces from the host
// among N ranks on one GPU, trips / this: 16.8 M values bf16 2 ranks 93.5 / 63.5, fp32 164 / 104, bf16 -> fp32 98.8 / 69.9; 5.2 M bf16
// 4 ranks 41.9 / 38.3, 13.1 M fp32 106.5 / 97.2; 16.8 M fp32 8 ranks 231 / 210; below 1 M the same.  Results twice as wide as their
// operands are mostly stores: among four ranks one pack a source does better than two (13.1 M 80.7 / 76.2, two 79.4), among eight the
// trips stay (170 / 169 - 174).  Copies gain nothing from loads ahead, shorter ones lose 1 - 2 %.
// SHIFT: the sources are `shift` bytes off the 16-byte grid.  The 32 aligned packs that a warp loads make 31 logical ones, each from a
// lane's and its neighbour's (31 of 32 of the traffic is wanted, and no lane has a second load to keep registers for).
// In the trips a shuffle per pack stood between its load and the next one's.  us, reduce-scatter of fp32 and all-gather of bf16 among
// four ranks, pieces off the grid, before / now: 20 003 values 65 / 56, 250 003 66.8 / 54.3, 1 000 003 121 / 76, 2 000 003 194 / 101 (2 000 000,
// on the grid, 93); two ranks 2 000 003 118 / 66.5.
template <typename Tin, typename Tout, int N, bool SHIFT>
DF_HD void reduceAhead(const DataArgs* a, uint64_t nPacks, int ndst, typename Elem<Tin>::Acc mul, bool doMul, int postDiv, double scale,
                       uint64_t srcOff, uint64_t dstOff, uint32_t shift) {
  typedef typename Elem<Tin>::Acc A;
  constexpr int V = 16 / (int)sizeof(Tin), OUTB = V * (int)sizeof(Tout), NW = (OUTB + 15) / 16;
  constexpr int U = N == 4 && NW == 2 ? 1 : 8 / N;
  const uint32_t tid = (uint32_t)df_tid(), nt = (uint32_t)df_nthreads(), ws = (uint32_t)df_warpsize();
  ShiftedWalk w = {0u, nt, tid};
  if (SHIFT) w = shiftedWalk(tid, nt, ws);
  const uint32_t lane = w.lane, step = w.step;             // (from one of a thread's packs to its next)
  const char* src[N];
#pragma unroll
  for (int j = 0; j < N; ++j) src[j] = a->src[j] + srcOff - (SHIFT ? shift : 0);
  uint4 in[U][N];
  auto load = [&](uint64_t p) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t q = p + (uint32_t)u * step;
      if (!(SHIFT ? shiftedLoads(q, lane, nPacks) : q < nPacks)) continue;
#pragma unroll
      for (int j = 0; j < N; ++j) in[u][j] = ld16(src[j] + q * 16);
    }
  };
  uint64_t p = w.first;
  load(p);
#pragma unroll 1
  while (shiftedWarpAt(p, lane, nPacks)) {
    uint4 ow[U][NW];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t q = p + (uint32_t)u * step;
      if (!shiftedWarpAt(q, lane, nPacks)) continue;
      A acc[V];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        uint4 v = in[u][j];
        if (SHIFT) v = shiftPack(v, nextLane(v, src[j] + q * 16), shift);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const A e = (A)Lane<Tin>::get(v, k);
          acc[k] = j == 0 ? e : red<OP_SUM>(acc[k], e);
        }
      }
      finishPack<Tin, Tout>(ow[u], acc, mul, doMul, postDiv, scale);
    }
    const uint64_t q = p;
    p += U * step;
    load(p);
    if (SHIFT && !shiftedMakes(lane, ws)) continue;
#pragma unroll 1
    for (int d = 0; d < ndst; ++d) {
      char* o = a->dst[d] + dstOff + q * OUTB;
      const bool wide = OUTB == 32 && ((uintptr_t)o & 31) == 0;
#pragma unroll
      for (int u = 0; u < U; ++u) if (q + (uint32_t)u * step < nPacks) storePack<OUTB>(o + (uint64_t)u * step * OUTB, ow[u], wide);
    }
  }
}

// How a call's pointers line up.  The vector path needs all sources at one misalignment and all destinations at one
// misalignment (true for equal offsets into symmetric buffers): `head` elements bring the destinations to their alignment, from
// there on the sources are read as packs shifted by `shift` bytes.  Anything else goes element by element (no packs).
struct Lineup { uint64_t head, nPacks; uint32_t shift; };
// Where the sources of a call whose pointers line up stand against the grid of its destinations.
DF_HD uint32_t shiftOf(const DataArgs* a, int esIn, int esOut) {
  const int outB = 16 / esIn * esOut, DA = outB >= 16 ? 16 : outB;
  const uint32_t sphase = (uint32_t)((uintptr_t)a->src[0] & 15), dphase = (uint32_t)((uintptr_t)a->dst[0] & (DA - 1));
  const uint64_t head = ((DA - dphase) & (DA - 1)) / (uint32_t)esOut;
  return (sphase + (uint32_t)(head > a->n ? a->n : head) * esIn) & 15;
}
DF_HD Lineup lineUp(const DataArgs* a, int nsrc, int ndst, uint64_t n, int esIn, int esOut) {
  const int V = 16 / esIn, outB = V * esOut, DA = outB >= 16 ? 16 : outB;          // alignment the vector stores need
  const uint32_t sphase = (uint32_t)((uintptr_t)a->src[0] & 15), dphase = (uint32_t)((uintptr_t)a->dst[0] & (DA - 1));
  bool vec = (dphase & (esOut - 1)) == 0 && (sphase & (esIn - 1)) == 0;
  for (int j = 1; j < nsrc; ++j) vec &= ((uintptr_t)a->src[j] & 15) == sphase;
  for (int j = 1; j < ndst; ++j) vec &= ((uintptr_t)a->dst[j] & (DA - 1)) == dphase;
  Lineup l;
  l.head = vec ? (uint32_t)((DA - dphase) & (DA - 1)) / (uint32_t)esOut : 0;
  if (l.head > n) l.head = n;
  l.shift = (uint32_t)((sphase + l.head * esIn) & 15);
  l.nPacks = vec ? (n - l.head) / (uint32_t)V : 0;
  return l;
}

// Small calls: a pack per thread and trip, four sources at a time, the operator looked at per pack, in as few registers as
// that takes (device/datapath_small.cu): what a call saves of the caller's registers goes to local memory and comes back after
// fences that emptied L1.  509 bf16 of four ranks took 9000 clocks in the bodies for long calls, of which 2500 were the sum.
// False (and nothing done) where the sources straddle packs: shifting them takes registers.
template <typename Tin, typename Tout>
DF_HD_NOINLINE bool reduceSmall(const DataArgs* a, int op) {
  typedef typename Elem<Tin>::Acc A;
  constexpr int V = 16 / (int)sizeof(Tin), OUTB = V * (int)sizeof(Tout), NW = (OUTB + 15) / 16;
  const int tid = df_tid(), nt = df_nthreads(), nsrc = a->nsrc, ndst = a->ndst, postDiv = a->postDiv;
  const uint64_t n = a->n;
  const double scale = a->scale;
  const bool doMul = scale != 1.0;
  const Lineup l = lineUp(a, nsrc, ndst, n, (int)sizeof(Tin), (int)sizeof(Tout));
  if (l.shift && l.nPacks) return false;
  const uint32_t nPacks = (uint32_t)l.nPacks;
  const uint64_t srcOff = l.head * sizeof(Tin), dstOff = l.head * sizeof(Tout);
#pragma unroll 1
  for (uint32_t p = (uint32_t)tid; p < nPacks; p += (uint32_t)nt) {
    A acc[V];
#pragma unroll 1
    for (int j0 = 0; j0 < nsrc; j0 += 4) {
      uint4 in[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) if (j0 + q < nsrc) in[q] = ld16(a->src[j0 + q] + srcOff + p * 16u);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (j0 + q >= nsrc) break;
        if (j0 + q == 0) {
#pragma unroll
          for (int k = 0; k < V; ++k) acc[k] = (A)Lane<Tin>::get(in[q], k);
        } else if (op == OP_SUM) {
#pragma unroll
          for (int k = 0; k < V; ++k) acc[k] = red<OP_SUM>(acc[k], (A)Lane<Tin>::get(in[q], k));
        } else if (sizeof(Tin) == sizeof(Tout)) {        // (casts exist for sums only)
          const bool mx = op == OP_MAX, pr = op == OP_PROD;
#pragma unroll
          for (int k = 0; k < V; ++k) {
            const A e = (A)Lane<Tin>::get(in[q], k);
            acc[k] = pr ? red<OP_PROD>(acc[k], e) : mx ? red<OP_MAX>(acc[k], e) : red<OP_MIN>(acc[k], e);
          }
        }
      }
    }
    uint4 ow[NW];
    finishPack<Tin, Tout>(ow, acc, (A)scale, doMul, postDiv, scale);
#pragma unroll 1
    for (int d = 0; d < ndst; ++d) {
      char* o = a->dst[d] + dstOff + (uint64_t)p * OUTB;
      storePack<OUTB>(o, ow, OUTB == 32 && ((uintptr_t)o & 31) == 0);
    }
  }
  // the head, the ragged tail, or everything when the pointers do not line up: the last warps first, which had no pack
  const uint64_t tail0 = l.head + (uint64_t)nPacks * V;
#pragma unroll 1
  for (uint64_t i = (uint64_t)(nt - 1 - tid); i < l.head + (n - tail0); i += nt) {
    const uint64_t e = i < l.head ? i : tail0 + (i - l.head);
    A acc = A();
#pragma unroll 1
    for (int j0 = 0; j0 < nsrc; j0 += 4) {
      Tin in[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) if (j0 + q < nsrc) in[q] = ld_elem((const Tin*)a->src[j0 + q] + e);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (j0 + q >= nsrc) break;
        const A v = Elem<Tin>::up(in[q]);
        acc = j0 + q == 0 ? v : op == OP_SUM ? red<OP_SUM>(acc, v) : op == OP_PROD ? red<OP_PROD>(acc, v) : op == OP_MAX ? red<OP_MAX>(acc, v) : red<OP_MIN>(acc, v);
      }
    }
    const Tout o = Elem<Tout>::down(finish<Tin, Tout>(acc, scale, postDiv));
    for (int d = 0; d < ndst; ++d) st_elem((Tout*)a->dst[d] + e, o);
  }
  return true;
}

template <typename Tin, typename Tout, bool SHIFT>
DF_HD void reduceAheadOf(const DataArgs* a, uint64_t nPacks, int nsrc, int ndst, typename Elem<Tin>::Acc mul, bool doMul, int postDiv, double scale,
                         uint64_t srcOff, uint64_t dstOff, uint32_t shift) {
  if (nsrc == 2) reduceAhead<Tin, Tout, 2, SHIFT>(a, nPacks, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, shift);
  else if (nsrc == 4) reduceAhead<Tin, Tout, 4, SHIFT>(a, nPacks, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, shift);
  else reduceAhead<Tin, Tout, 8, SHIFT>(a, nPacks, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, shift);
}

// The head, the ragged tail, or everything when the pointers do not line up: element by element.
template <typename Tin, typename Tout, int OP>
DF_HD void reduceLoose(const DataArgs* a, uint64_t head, uint64_t nPacks) {
  typedef typename Elem<Tin>::Acc A;
  const int tid = df_tid(), nt = df_nthreads(), nsrc = a->nsrc, ndst = a->ndst, postDiv = a->postDiv;
  const uint64_t n = a->n, tail0 = head + nPacks * (16 / sizeof(Tin));
  const double scale = a->scale;
  for (uint64_t i = looseStart(tid, nt, nPacks); i < head + (n - tail0); i += nt) {
    const uint64_t e = i < head ? i : tail0 + (i - head);
    A acc = A();
    for (int j0 = 0; j0 < nsrc; j0 += 4) {
      Tin in[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) if (j0 + q < nsrc) in[q] = ld_elem((const Tin*)a->src[j0 + q] + e);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (j0 + q >= nsrc) break;
        acc = j0 + q == 0 ? Elem<Tin>::up(in[q]) : red<OP>(acc, Elem<Tin>::up(in[q]));
      }
    }
    Tout o = Elem<Tout>::down(finish<Tin, Tout>(acc, scale, postDiv));
    for (int d = 0; d < ndst; ++d) st_elem((Tout*)a->dst[d] + e, o);
  }
}

// One body for calls on the 16-byte grid and one for shifted sources: what a body uses of its caller's registers goes to local memory and
// comes back behind fences that emptied L1, and shifting takes most of them.  Bytes of frame, both in one / on the grid: fp32 maximum 248 /
// 16, bf16 maximum 248 / 64, fp32 sum 248 / 160, copies 136 / 16.  us for all-reduces from the host: maxima of fp32 2 ranks 1 M values 28.3 /
// 26.9, 4 ranks 1 M 27.8 / 26.0, 4 M 59.5 / 56.5, fp64 4 ranks 1 M 32.6 / 29.4; broadcast of 2 M bf16 24.6 / 23.8; sums, and shifted sources, the
// same.  (Each lines the pointers up by itself: handed over, the shifted loops took 3 - 7 % longer.)
template <typename Tin, typename Tout, int OP, bool SHIFT>
DF_HD_NOINLINE void reduceBody(const DataArgs* a) {
  const int nsrc = a->nsrc, ndst = a->ndst, postDiv = a->postDiv;
  const double scale = a->scale;
  const bool doMul = scale != 1.0;
  const typename Elem<Tin>::Acc mul = (typename Elem<Tin>::Acc)scale;
  const Lineup l = lineUp(a, nsrc, ndst, a->n, (int)sizeof(Tin), (int)sizeof(Tout));
  const uint64_t srcOff = l.head * sizeof(Tin), dstOff = l.head * sizeof(Tout);
  if (l.nPacks) {
    if (OP == OP_SUM && (nsrc == 2 || nsrc == 4 || (nsrc == 8 && sizeof(Tout) <= sizeof(Tin))))
      reduceAheadOf<Tin, Tout, SHIFT>(a, l.nPacks, nsrc, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, l.shift);
    else reduceTrips<Tin, Tout, OP, SHIFT>(a, l.nPacks, nsrc, ndst, mul, doMul, postDiv, scale, srcOff, dstOff, l.shift);
  }
  reduceLoose<Tin, Tout, OP>(a, l.head, l.nPacks);
}

template <typename Tin, typename Tout, int OP>
DF_HD void reduce_copy(const DataArgs* a) {
  if (shiftOf(a, (int)sizeof(Tin), (int)sizeof(Tout))) reduceBody<Tin, Tout, OP, true>(a);
  else reduceBody<Tin, Tout, OP, false>(a);
}

// Byte copy of one source to M destinations (AllGather, Broadcast, staging).
template <bool FULL, int U>
DF_HD void copyTrip(const DataArgs* a, uint64_t p0, uint64_t nPacks, uint32_t strideB, int ndst, uint64_t off) {
  const uint32_t stride = strideB >> 4;
  uint4 raw[U];
  loadPacks<FULL, false, U>(raw, a->src[0] + off + p0 * 16, strideB, 0, p0, stride, nPacks);
  for (int d = 0; d < ndst; ++d) {
    char* o = a->dst[d] + off + p0 * 16;
#pragma unroll
    for (int u = 0; u < U; ++u) if (FULL || p0 + (uint64_t)u * stride < nPacks) st16(o + (uint64_t)u * strideB, raw[u]);
  }
}

DF_HD void copyTrips(const DataArgs* a, uint64_t nPacks, int ndst, uint64_t off) {
  constexpr int U = 8;
  const int tid = df_tid(), nt = df_nthreads();
  const uint64_t step = (uint64_t)nt * U;
  const uint32_t strideB = (uint32_t)nt * 16u;
  uint64_t base = 0;
  for (; base + step <= nPacks; base += step) copyTrip<true, U>(a, base + tid, nPacks, strideB, ndst, off);
  for (; base + nt <= nPacks; base += nt) copyTrip<true, 1>(a, base + tid, nPacks, strideB, ndst, off);
  if (base + tid < nPacks) copyTrip<false, 1>(a, base + tid, nPacks, strideB, ndst, off);
}

DF_HD void copyShifted(const DataArgs* a, uint64_t nPacks, int ndst, uint64_t off, uint32_t shift) {
  constexpr int U = 8;
  const uint32_t ws = (uint32_t)df_warpsize();
  const ShiftedWalk w = shiftedWalk((uint32_t)df_tid(), (uint32_t)df_nthreads(), ws);
  const char* s = a->src[0] + off - shift;
#pragma unroll 1
  for (uint64_t p = w.first; shiftedWarpAt(p, w.lane, nPacks); p += U * w.step) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t q = p + (uint32_t)u * w.step;
      if (shiftedLoads(q, w.lane, nPacks)) raw[u] = ld16(s + q * 16);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t q = p + (uint32_t)u * w.step;
      if (ws > 1 || shiftedWarpAt(q, w.lane, nPacks)) raw[u] = shiftPack(raw[u], nextLane(raw[u], s + q * 16), shift);
    }
    if (!shiftedMakes(w.lane, ws)) continue;
#pragma unroll 1
    for (int d = 0; d < ndst; ++d) {
      char* o = a->dst[d] + off + p * 16;
#pragma unroll
      for (int u = 0; u < U; ++u) if (p + (uint32_t)u * w.step < nPacks) st16(o + (uint64_t)u * w.step * 16, raw[u]);
    }
  }
}

// Small copies, in the body of the kernel.
DF_HD void copySmall(const DataArgs* a) {
  const int tid = df_tid(), nt = df_nthreads(), ndst = a->ndst;
  const uint64_t n = a->n;
  const Lineup l = lineUp(a, 1, ndst, n, 1, 1);
  const uint32_t nPacks = (uint32_t)l.nPacks;
  const char* src = a->src[0] + l.head - l.shift;
#pragma unroll 1
  for (uint32_t p = (uint32_t)tid; p < nPacks; p += (uint32_t)nt) {
    uint4 v = ld16(src + p * 16u);
    if (l.shift) v = shiftPack(v, ld16(src + p * 16u + 16), l.shift);
#pragma unroll 1
    for (int d = 0; d < ndst; ++d) st16(a->dst[d] + l.head + p * 16u, v);
  }
  const uint64_t tail0 = l.head + (uint64_t)nPacks * 16;
#pragma unroll 1
  for (uint64_t i = (uint64_t)(nt - 1 - tid); i < l.head + (n - tail0); i += nt) {
    const uint64_t e = i < l.head ? i : tail0 + (i - l.head);
    const uint8_t b = ld_elem((const uint8_t*)a->src[0] + e);
    for (int d = 0; d < ndst; ++d) st_elem((uint8_t*)a->dst[d] + e, b);
  }
}

#ifdef DF_DATAPATH_IMPL
DF_HD void copyLoose(const DataArgs* a, uint64_t head, uint64_t nPacks) {
  const int nt = df_nthreads(), ndst = a->ndst;
  const uint64_t nbytes = a->n, tail0 = head + nPacks * 16;
  for (uint64_t i = looseStart(df_tid(), nt, nPacks); i < head + (nbytes - tail0); i += nt) {
    const uint64_t e = i < head ? i : tail0 + (i - head);
    uint8_t b = ld_elem((const uint8_t*)a->src[0] + e);
    for (int d = 0; d < ndst; ++d) st_elem((uint8_t*)a->dst[d] + e, b);
  }
}
template <bool SHIFT>
DF_HD void copyBody(const DataArgs* a) {
  const int ndst = a->ndst;
  Lineup l = {0, 0, 0};
  if (ndst) l = lineUp(a, 1, ndst, a->n, 1, 1);
  if (l.nPacks) {
    if (SHIFT) copyShifted(a, l.nPacks, ndst, l.head, l.shift);
    else copyTrips(a, l.nPacks, ndst, l.head);
  }
  copyLoose(a, l.head, l.nPacks);
}
__host__ __device__ void copy_on_grid(const DataArgs* a) { copyBody<false>(a); }
__host__ __device__ void copy_shifted(const DataArgs* a) { copyBody<true>(a); }
#else
__host__ __device__ void copy_on_grid(const DataArgs* a);
__host__ __device__ void copy_shifted(const DataArgs* a);
#endif
// (the caller chooses: a body between it and these would have a frame of its own, a round trip to L2 on the way back)
DF_HD void copy_multi(const DataArgs* a) {
  if (a->ndst && shiftOf(a, 1, 1)) copy_shifted(a); else copy_on_grid(a);
}

DF_HD int dtypeSize(int t) {
  switch (t) {
    case ncclInt8: case ncclUint8: return 1;
    case ncclFloat16: case ncclBfloat16: return 2;
    case ncclInt32: case ncclUint32: case ncclFloat32: return 4;
    default: return 8;
  }
}

#ifdef DF_DATAPATH_IMPL
template <typename T>
DF_HD void reduce_same(int op, const DataArgs* a) {
  switch (op) {
    case OP_SUM: reduce_copy<T, T, OP_SUM>(a); break;
    case OP_PROD: reduce_copy<T, T, OP_PROD>(a); break;
    case OP_MAX: reduce_copy<T, T, OP_MAX>(a); break;
    default: reduce_copy<T, T, OP_MIN>(a); break;
  }
}

// Returns false when the (in, out, op) combination is not instantiated.
__host__ __device__ bool reduce_dispatch(int inType, int outType, int op, const DataArgs* a) {
  if (inType == outType) {
    switch (inType) {
#ifndef DF_FAST_BUILD
      case ncclInt8: reduce_same<int8_t>(op, a); return true;
      case ncclUint8: reduce_same<uint8_t>(op, a); return true;
      case ncclInt32: reduce_same<int32_t>(op, a); return true;
      case ncclUint32: reduce_same<uint32_t>(op, a); return true;
      case ncclInt64: reduce_same<int64_t>(op, a); return true;
      case ncclUint64: reduce_same<uint64_t>(op, a); return true;
      case ncclFloat16: reduce_same<__half>(op, a); return true;
      case ncclFloat64: reduce_same<double>(op, a); return true;
#endif
      case ncclFloat32: reduce_same<float>(op, a); return true;
      case ncclBfloat16: reduce_same<__nv_bfloat16>(op, a); return true;
      default: return false;
    }
  }
  if (op != OP_SUM) return false;   // fused casts exist for the gradient path only
  if (inType == ncclBfloat16 && outType == ncclFloat32) { reduce_copy<__nv_bfloat16, float, OP_SUM>(a); return true; }
  if (inType == ncclFloat16 && outType == ncclFloat32) { reduce_copy<__half, float, OP_SUM>(a); return true; }
  if (inType == ncclFloat32 && outType == ncclBfloat16) { reduce_copy<float, __nv_bfloat16, OP_SUM>(a); return true; }
  if (inType == ncclFloat32 && outType == ncclFloat16) { reduce_copy<float, __half, OP_SUM>(a); return true; }
  return false;
}

#else
// Defined once, in device/datapath.cu (relocatable device code): every kernel of the library calls the
// same out-of-line bodies instead of compiling its own copy of the 44 variants.
// Returns false when the (in, out, op) combination is not instantiated.
__host__ __device__ bool reduce_dispatch(int inType, int outType, int op, const DataArgs* a);
#endif

#ifdef DF_DATAPATH_SMALL_IMPL
// (comparisons, the gradients' types first, and not a jump table: see nextPhase)
__host__ __device__ bool reduce_small(int inType, int outType, int op, const DataArgs* a) {
  if (inType == outType) {
    if (inType == ncclBfloat16) return reduceSmall<__nv_bfloat16, __nv_bfloat16>(a, op);
    if (inType == ncclFloat32) return reduceSmall<float, float>(a, op);
#ifndef DF_FAST_BUILD
    if (inType == ncclFloat16) return reduceSmall<__half, __half>(a, op);
    if (inType == ncclInt32) return reduceSmall<int32_t, int32_t>(a, op);
    if (inType == ncclInt8) return reduceSmall<int8_t, int8_t>(a, op);
    if (inType == ncclUint8) return reduceSmall<uint8_t, uint8_t>(a, op);
    if (inType == ncclUint32) return reduceSmall<uint32_t, uint32_t>(a, op);
    if (inType == ncclInt64) return reduceSmall<int64_t, int64_t>(a, op);
    if (inType == ncclUint64) return reduceSmall<uint64_t, uint64_t>(a, op);
    if (inType == ncclFloat64) return reduceSmall<double, double>(a, op);
#endif
    return false;
  }
  if (op != OP_SUM) return false;
  if (inType == ncclBfloat16 && outType == ncclFloat32) return reduceSmall<__nv_bfloat16, float>(a, op);
  if (inType == ncclFloat16 && outType == ncclFloat32) return reduceSmall<__half, float>(a, op);
  if (inType == ncclFloat32 && outType == ncclBfloat16) return reduceSmall<float, __nv_bfloat16>(a, op);
  if (inType == ncclFloat32 && outType == ncclFloat16) return reduceSmall<float, __half>(a, op);
  return false;
}
#else
__host__ __device__ bool reduce_small(int inType, int outType, int op, const DataArgs* a);
#endif

// Calls of at most this many packs per thread and source go through the small bodies.  bf16 -> fp32 among four ranks, us, limit
// 2 / 4 / 8: 0.9 M values 24.2 / 24.1 / 24.2, 1.3 M 28.6 / 26.7 / 26.7, 1.9 M 32.2 / 30.7 / 30.2, 2.6 M 35.9 / 36 / 34.4, 3.7 M 42.1 / 42.2 /
// 40.3: the small body is the better one at this limit, and a little beyond it.
#define DF_SMALL_TRIPS 4
// What the step engine calls.
DF_HD bool reduce_block(int inType, int outType, int esIn, int op, const DataArgs* a) {
  const bool small = a->n * (uint64_t)esIn <= (uint64_t)df_nthreads() * 16u * DF_SMALL_TRIPS;
  if (small && reduce_small(inType, outType, op, a)) return true;
  return reduce_dispatch(inType, outType, op, a);
}
DF_HD void copy_block(const DataArgs* a) {
  if (a->n <= (uint64_t)df_nthreads() * 16u * DF_SMALL_TRIPS) copySmall(a); else copy_multi(a);
}

// Host-callable check used at prepare time.
inline bool reduceSupported(int inType, int outType, int op) {
  if (inType < 0 || inType >= ncclNumTypes || outType < 0 || outType >= ncclNumTypes) return false;
  if (inType == outType) return op >= OP_SUM && op <= OP_MIN;
  if (op != OP_SUM) return false;
  return ((inType == ncclBfloat16 || inType == ncclFloat16) && outType == ncclFloat32) ||
         (inType == ncclFloat32 && (outType == ncclBfloat16 || outType == ncclFloat16));
}

}  // namespace dfccl
