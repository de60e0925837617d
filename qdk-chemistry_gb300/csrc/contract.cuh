// The direct sigma's contraction on the fifth-generation tensor cores, from
// operands split into 16-bit parts:
//   E[r][Jb] = sum_k Vp[k][r] C[Ja_k, Jb]          one CTA per alpha string Ia
//   sigma[Ia, Ib] += the entries of E that string Ib needs (the walk)
// (the terms are listed at k_ds_opposite_mm in direct.cu).  Rows r:
//   r < mr          the orbital pair {p < q}: one row serves the excitations
//                   p -> q and q -> p, so V(..|pq) = V(..|qp) is required
//   mr + p, p < n   the other spin's occupied orbital p
//   mr + n          the string-only part of the alpha singles
// With R = mr + n + 1 <= 128 rows E is one 128-lane tile (n <= 15).
//
// Two forms of the same kernel:
//  * FP32 (S = 3 parts): x = b0 + b1 + b2 in bfloat16, 24 bits, the six
//    products down to 2^-24 summed in one FP32 accumulator.
//  * FP64 (S = 7 parts): Vp and C as 63-bit fixed point, seven balanced
//    9-bit digits each, stored as whole numbers in fp16 (|digit| <= 256).
//    Products of digits i and j weigh 2^-9(i+j+2); those of one i + j = g
//    share an accumulator.  A digit product is at most 2^16, so an
//    accumulator holds at most (g + 1) 2^16 K, below 2^24 for K <= 51 and
//    g <= 4: whole numbers that FP32 sums exactly, in any order.  g = 5 and 6
//    weigh 2^-63 and less, where FP32 rounding does not matter; g >= 7 is
//    left out.  C rows carry one exponent each (the largest of the row), which
//    is folded into Vp; the pair rows and the others have one exponent each
//    per alpha string.  E is put together as a 64-bit integer in units of
//    2^-57 of that exponent, the walk sums integers (96 bits), and a sigma
//    element is rounded to FP64 once.
//
// Why this layout: Vp (the A operand) lives in TMEM, written once per alpha
// string, so the MMAs read only the C digits from shared memory (N = 64: 2 KB
// per 32 clocks, a quarter of the shared-memory rate); C digit rows are
// contiguous along Jb, which the MN-major B operand takes as they are, so the
// gather of the K rows is plain 16-byte asynchronous copies.  Accumulators
// are 64-column slots used in turn, one per group in flight, so the products of
// the next chunk run under the read-out and the walk of this one.
//
// What bounds it: the walk (random reads of E, two barriers a chunk) and, in
// FP64, the read-out before it; the products take 33 of 129 us (FP32, 12
// orbitals, 854 thousand determinants) and 2.5 of 5.6 ms (FP64, 14 orbitals,
// 11.8 million).  The forms it replaced took 312 us (TF32 x 3, the walk over
// twice as many rows) and 65 ms (element by element on the FP64 pipe).
#pragma once
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace qdkgb {
namespace ct {

constexpr int kCols = 64;      // beta strings per chunk
constexpr int kPitch = 68;     // E row pitch (elements): 16-byte rows, four banks apart
constexpr int kLoadWarps = 3;  // warps that gather the C digits
constexpr uint32_t kSpin = 1u << 22;
constexpr int kWidth = 9;      // digit width of the FP64 form
constexpr int kUnit = 57;      // E's unit of the FP64 form: 2^-57 of the class exponent
constexpr int kHead = 48;      // words before a chunk's tasks: the bounds of 16 warps' tasks, at 32 those of 8 warps'
constexpr int kNoExp = -5000;  // exponent of an all-zero row

// D[tmem] (+)= A[tmem] B[smem], kind::f16 (A and B of one 16-bit type)
__device__ __forceinline__ void mma_f16_ts(uint32_t dtmem, uint32_t atmem, uint64_t b, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(dtmem),
      "r"(atmem), "l"(b), "r"(idesc), "r"(accumulate));
}
// instruction descriptor, kind::f16: FP32 accumulator, A and B fp16 (0) or
// bf16 (1), A K-major, B MN-major (bit 16)
constexpr uint32_t idesc_f16(int M, int N, int type) {
  return (1u << 4) | ((uint32_t)type << 7) | ((uint32_t)type << 10) | (1u << 16) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}
// two 32-bit columns of the lane this thread owns
__device__ __forceinline__ void tmem_st2(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_addr(b)) : "memory");
}
// a wait that ends early once another role of the CTA has timed out
__device__ __forceinline__ bool wait(uint64_t* b, uint32_t parity, volatile int* fail) {
  for (int i = 0; i < 64; ++i) {
    if (tc::mbar_wait(b, parity, kSpin / 64)) return true;
    if (*fail) return false;
  }
  *fail = 1;
  return false;
}

// the exponent e with |x| < 2^e (kNoExp for zero and denormals, which are
// below every bit that counts here beside a normal number of the same row);
// 1025 for infinities and NaN
__device__ __forceinline__ int exp_above(double x) {
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  return e ? e - 1022 : kNoExp;
}
// x 2^s rounded to a 64-bit integer (|x 2^s| < 2^62), integer arithmetic only
__device__ __forceinline__ int64_t fixed_point(double x, int s) {
  const int64_t b = __double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff);
  int64_t m = e ? ((b & 0xfffffffffffffll) | (1ll << 52)) : 0;
  const int sh = e - 1075 + s;
  if (sh >= 0)
    m = sh > 62 ? 0 : m << sh;
  else
    m = sh < -60 ? 0 : (m + (1ll << (-sh - 1))) >> -sh;
  return b < 0 ? -m : m;
}
// v 2^e
__device__ __forceinline__ double scale2(double v, int e) {
  const int h = __double2hiint(v), x = (h >> 20) & 0x7ff;
  if (x == 0 || x == 0x7ff) return v;  // zero (denormals do not arise from whole numbers)
  if (x + e > 0 && x + e < 0x7ff) return __hiloint2double(h + (e << 20), __double2loint(v));
  return ldexp(v, e);
}
// q 2^e rounded to FP64, to even as (double)q is, by integer instructions: a
// conversion from 64-bit integers is several FP64 ones, 16 clocks a warp each
// (a tile of k_dense64 took 17 us for its 16,384).
static __device__ __noinline__ double whole_scaled_far(int64_t q, int e) { return ldexp((double)q, e); }
__device__ __forceinline__ double whole_scaled(int64_t q, int e) {
  if (q == 0) return 0.;
  const uint64_t u = q < 0 ? 0ull - (uint64_t)q : (uint64_t)q;
  const int lz = __clzll((long long)u);
  const uint64_t m = u << lz, rest = m & 0x7ff;
  uint64_t b = (m >> 11) + (uint64_t)(rest > 0x400 || (rest == 0x400 && (m & 0x800)));  // 2^52 .. 2^53
  const int x = 1085 - lz + e;  // the exponent field, less the one that b's bit 52 adds
  if (x < 0 || x > 2044) return whole_scaled_far(q, e);
  b += (uint64_t)x << 52;
  return __longlong_as_double((long long)(b | (q < 0 ? 1ull << 63 : 0ull)));
}
// balanced digits of q, most significant first: q = sum_i d[i] 2^(W (S-1-i))
template <int S, int W>
__device__ __forceinline__ void digits(int64_t q, int* d) {
#pragma unroll
  for (int i = S - 1; i > 0; --i) {
    const int64_t r = ((q + (1 << (W - 1))) & ((1 << W) - 1)) - (1 << (W - 1));
    d[i] = (int)r;
    q = (q - r) >> W;
  }
  d[0] = (int)q;
}
__device__ __forceinline__ uint32_t pack_f16(int a, int b) {
  const __half2 h = __floats2half2_rn((float)a, (float)b);
  return *(const uint32_t*)&h;
}
// x = p[0] + p[1] + p[2] in bfloat16
__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16* p) {
  p[0] = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(p[0]);
  p[1] = __float2bfloat16_rn(r);
  p[2] = __float2bfloat16_rn(r - __bfloat162float(p[1]));
}
__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 a, __nv_bfloat16 b) {
  return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}

// C (na x nb) into its parts, rows padded with zeros to nbp (a multiple of
// 64): out[s][Ia][nbp], bfloat16 (FP32 form).  grid: (rows, instances).
__global__ void __launch_bounds__(256)
    k_ct_split32(int nb, int nbp, int64_t part, const float* __restrict__ C, uint16_t* __restrict__ out,
                 int64_t cstride, int64_t ostride, const int* __restrict__ act) {
  if (act && !act[blockIdx.y]) return;
  C += blockIdx.y * cstride + (int64_t)blockIdx.x * nb;
  out += blockIdx.y * ostride + (int64_t)blockIdx.x * nbp;
  for (int j = 2 * threadIdx.x; j < nbp; j += 512) {
    __nv_bfloat16 a[3], b[3];
    split_bf16(j < nb ? C[j] : 0.f, a);
    split_bf16(j + 1 < nb ? C[j + 1] : 0.f, b);
#pragma unroll
    for (int s = 0; s < 3; ++s) *(uint32_t*)(out + s * part + j) = pack_bf16(a[s], b[s]);
  }
}
// the same for the FP64 form (fp16 digits): rexp[Ia] the row's exponent;
// *bad set when the row holds an infinity or NaN
__global__ void __launch_bounds__(256)
    k_ct_split64(int nb, int nbp, int64_t part, const double* __restrict__ C, uint16_t* __restrict__ out,
                 int* __restrict__ rexp, int* __restrict__ bad) {
  __shared__ int red[8];
  C += (int64_t)blockIdx.x * nb;
  out += (int64_t)blockIdx.x * nbp;
  int e = kNoExp;
  for (int j = threadIdx.x; j < nb; j += 256) e = max(e, exp_above(C[j]));
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, red[w]);
  if (threadIdx.x == 0) {
    rexp[blockIdx.x] = e == kNoExp ? kNoExp : e + 1;
    if (e > 1024) *bad = 1;
  }
  // |C| 2^-(e + 1) < 1/2
  for (int j = 2 * threadIdx.x; j < nbp; j += 512) {
    int a[7], b[7];
    digits<7, kWidth>(e != kNoExp && j < nb ? fixed_point(C[j], 63 - (e + 1)) : 0, a);
    digits<7, kWidth>(e != kNoExp && j + 1 < nb ? fixed_point(C[j + 1], 63 - (e + 1)) : 0, b);
#pragma unroll
    for (int s = 0; s < 7; ++s) *(uint32_t*)(out + s * part + j) = pack_f16(a[s], b[s]);
  }
}

// the operands of the contraction (instance strides as DsInst in direct.cu)
template <typename T>
struct Args {
  int na, nb, nbp, nsa, n, mr, R, kpad, seg_bytes;
  int64_t part;              // elements between the parts of C
  const int32_t *a_sJ, *a_svo, *rs_of, *seg;
  const T *a_sA, *a_W, *V2;  // V2[pq][R]
  const uint16_t *walk, *Cs;
  const int* rexp;
  const double* D;
  const T* C;
  T* sigma;
  const int* bad;            // FP64: non-finite input, leave the work to the plain form
  unsigned* fault;
  // FP64: alpha strings from `full` on are split over `split` CTAs each, by
  // chunks (row_plan); their sums meet in part_lo / part_hi [CTA][nb] and
  // part_count [string][arrived, failed] (zero before and after)
  int full, split;
  uint64_t* part_lo;
  int32_t* part_hi;
  unsigned* part_count;
};

// How the na alpha strings of the FP64 form go over `slots` SMs: whole ones in
// full waves, those of a last, partly filled wave in `split` pieces of their
// chunks (the pieces' sums are whole numbers and add exactly).  A CTA's start
// and end take as long as about three chunks (12 orbitals: 17 + 4 thousand
// clocks beside 8 thousand a chunk).  924 strings on 152 SMs were seven waves,
// the last with 12 CTAs: 486 -> 447 us.  The FP32 form, two CTAs to an SM, has
// its last wave's SMs to itself and lost by it (139.1 -> 146.6 us a sigma).
struct RowPlan {
  int full, split;
};
inline RowPlan row_plan(int na, int nchunk, int slots) {
  const int rem = na % slots;
  RowPlan best{na, 1};
  int least = 1 << 30;
  for (int s = 1; rem > 0 && s <= nchunk; ++s) {
    const int waves = (int)(((int64_t)rem * s + slots - 1) / slots), cost = waves * (3 + (nchunk + s - 1) / s);
    if (cost < least) {
      least = cost;
      best = s > 1 ? RowPlan{na - rem, s} : RowPlan{na, 1};
    }
  }
  return best;
}

template <typename T>
struct Form;
template <>
struct Form<float> {
  static constexpr int S = 3, G = 1, EpiWarps = 8, MinBlocks = 2, Tmem = 256;
  using E = float;
};
template <>
struct Form<double> {
  static constexpr int S = 7, G = 7, EpiWarps = 16, MinBlocks = 1, Tmem = 512;
  using E = int64_t;
};
// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
  return p != 0;
}

// Shared memory: two C digit buffers, E (R + 1 rows, the last one zero), the
// sigma row's accumulators, the chunk's walk lists, the K rows' strings.
template <typename T>
struct Smem {
  int b_bytes, off_e, off_acc, off_hi, off_list, off_j, total;
  __host__ __device__ Smem(int kpad, int R, int nb, int seg_bytes) {
    b_bytes = Form<T>::S * kpad * 128;
    off_e = 2 * b_bytes;
    off_acc = off_e + (((R + 1) * kPitch * (int)sizeof(T) + 15) & ~15);
    const int nb4 = (nb + 3) & ~3;
    off_hi = off_acc + nb4 * (int)sizeof(T);
    off_list = off_hi + (sizeof(T) == 8 ? nb4 * 4 : 0);
    off_j = off_list + ((seg_bytes + 15) & ~15);
    total = off_j + 3 * kpad * 4 + 64;
  }
};

// KS: K padded to 16 KS.  The accumulator ring takes the TMEM columns that
// Vp's parts leave.
template <typename T, int KS>
__global__ void __launch_bounds__((Form<T>::EpiWarps + 1 + kLoadWarps) * 32, Form<T>::MinBlocks)
    k_contract(Args<T> g) {
  using F = Form<T>;
  constexpr bool kF64 = sizeof(T) == 8;
  constexpr int S = F::S, G = F::G, kEpi = F::EpiWarps * 32, kPad = 16 * KS;
  constexpr int kSl = (F::Tmem - S * KS * 8) / kCols < 7 ? (F::Tmem - S * KS * 8) / kCols : 7;
  static_assert(kSl >= 2 && (!kF64 || kSl >= 4), "accumulator slots");
  // FP64: group gi of a chunk goes to slot gi % kSl.  A wait that need not
  // wait costs 90 clocks on an idle SM and 350 here, so there are few: the
  // read-out waits once for the first kSl groups and once for the rest, the
  // products wait for the read-out of each group whose slot is used again in
  // the chunk (kRe of them), of the last group in slot 0, and of the last.
  constexpr int kRe = kF64 ? (G > kSl ? G - kSl : 0) : 0;
  constexpr int kFirst = kRe > 0 ? kSl : 0;  // the last group in slot 0
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[2], empty[2], accfull[kSl], accempty[kSl], reuse[kF64 ? G : 1], listfull, done;
  __shared__ uint32_t tslot;
  __shared__ int fail_, last_, mexp[2];
  volatile int* fail = &fail_;
  if (kF64 && g.bad && *g.bad) return;
  const Smem<T> L(kPad, g.R, g.nb, g.seg_bytes);
  typename F::E* E = (typename F::E*)(smem + L.off_e);
  T* facc = (T*)(smem + L.off_acc);                    // FP32: the sums
  uint64_t* lo = (uint64_t*)(smem + L.off_acc);        // FP64: bits 0-63 ..
  int32_t* hi = (int32_t*)(smem + L.off_hi);           // .. and 64-95
  const uint16_t* list = (const uint16_t*)(smem + L.off_list);
  int32_t* Jrow = (int32_t*)(smem + L.off_j);
  int32_t* kvo = Jrow + kPad;
  int32_t* kexp = kvo + kPad;
  const bool whole = !kF64 || (int)blockIdx.x < g.full;
  const int piece = whole ? 0 : (int)(blockIdx.x - g.full);  // among the split strings' CTAs
  const int64_t Ia = whole ? (int64_t)blockIdx.x : g.full + piece / g.split;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = g.nsa + 1, n = g.n;
  const int chunks = (g.nb + kCols - 1) / kCols, mine = whole ? 0 : piece % g.split;
  const int chunk0 = whole ? 0 : mine * chunks / g.split;
  const int nchunk = whole ? chunks : (mine + 1) * chunks / g.split - chunk0;
  if (warp == 0) tc::tmem_alloc(&tslot, F::Tmem);
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&full[i], kLoadWarps);
      tc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < kSl; ++i) {
      tc::mbar_init(&accfull[i], 1);
      tc::mbar_init(&accempty[i], F::EpiWarps);
    }
    for (int i = 0; i < (kF64 ? G : 1); ++i) tc::mbar_init(&reuse[i], F::EpiWarps);
    tc::mbar_init(&listfull, 1);
    tc::mbar_init(&done, 1);
    tc::mbar_init_fence();
    fail_ = 0;
    mexp[0] = mexp[1] = kNoExp;
  }
  for (int k = tid; k < kPad; k += blockDim.x) {
    const int32_t J = k < g.nsa ? g.a_sJ[Ia * g.nsa + k] : (int32_t)Ia;
    Jrow[k] = J;
    kvo[k] = k < g.nsa ? g.a_svo[Ia * g.nsa + k] : 0;
    kexp[k] = kF64 && k < K ? g.rexp[J] : kNoExp;
  }
  // rows of C past K stay zero in both digit buffers
  for (int i = tid; i < 2 * S * (kPad - K) * 8; i += blockDim.x) {
    const int b = i & 7, x = i >> 3, k = K + x % (kPad - K), s = x / (kPad - K);  // s: buffer and part
    *(float4*)(smem + s * kPad * 128 + (k >> 3) * 1024 + b * 128 + (k & 7) * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int i = tid; i < g.nb; i += blockDim.x) {
    if (kF64) {
      lo[i] = 0;
      hi[i] = 0;
    } else {
      facc[i] = (T)(g.sigma[Ia * g.nb + i] + (T)g.D[Ia * g.nb + i] * g.C[Ia * g.nb + i]);
    }
  }
  for (int i = tid; i < kPitch; i += blockDim.x) E[g.R * kPitch + i] = 0;
  tc::fence_proxy_async();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tslot, tacc = tmem + S * KS * 8;

  // ---- the A operand: lane r, part s, K rows 2c and 2c + 1 in column s kpad/2 + c
  if (warp < F::EpiWarps) {
    const int q = warp & 3, r = q * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16);
    const int cls = r < g.mr ? 0 : 1;
    constexpr int kPer = F::EpiWarps / 4, kCnt = kPad / kPer;  // warps that share a lane quadrant: kCnt K each
    const int k0 = (warp >> 2) * kCnt;
    // all loads first: one latency for the lot
    T val[kCnt];
#pragma unroll
    for (int i = 0; i < kCnt; ++i) {
      const int k = k0 + i;
      T v = 0;
      if (r < g.R && k < K) {
        if (k == g.nsa) {
          if (r < g.mr) v = __ldg(g.a_W + (int64_t)__ldg(g.rs_of + r) * g.na + Ia);
        } else {
          const int vo = kvo[k];
          v = r == g.R - 1 ? __ldg(g.a_sA + Ia * g.nsa + k)
                           : __ldg(g.V2 + (int64_t)((vo & 0xff) + n * ((vo >> 8) & 0xff)) * g.R + r);
          v = (vo >> 16) ? -v : v;
        }
      }
      val[i] = v;
    }
    if constexpr (kF64) {
      // the largest exponent of each class, C's row exponents folded in
      int e = kNoExp;
#pragma unroll
      for (int i = 0; i < kCnt; ++i) {
        const int ev = exp_above(val[i]), ke = kexp[k0 + i];
        if (ev != kNoExp && ke != kNoExp) e = max(e, ev + ke);
      }
      const int e0 = __reduce_max_sync(0xffffffffu, cls == 0 ? e : kNoExp);
      const int e1 = __reduce_max_sync(0xffffffffu, cls == 1 ? e : kNoExp);
      if (lane == 0) {
        atomicMax(&mexp[0], e0);
        atomicMax(&mexp[1], e1);
      }
      asm volatile("bar.sync 1, %0;\n" ::"r"(kEpi) : "memory");
      if (tid == 0) {
        // |Vp| 2^-M < 1/2; at most 2^24 between the classes, so that the 96-bit sums hold both
        const int m0 = mexp[0] + 1, m1 = mexp[1] + 1;
        mexp[0] = max(m0, m1 - 24);
        mexp[1] = max(m1, m0 - 24);
      }
      asm volatile("bar.sync 1, %0;\n" ::"r"(kEpi) : "memory");
      const int M = mexp[cls];
#pragma unroll
      for (int j = 0; j < kCnt / 4; ++j) {
        uint32_t u[7][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          int a[7], b[7];
          const int i = 4 * j + 2 * h, ka = kexp[k0 + i], kb = kexp[k0 + i + 1];
          digits<7, kWidth>(ka == kNoExp ? 0 : fixed_point(val[i], 63 - M + ka), a);
          digits<7, kWidth>(kb == kNoExp ? 0 : fixed_point(val[i + 1], 63 - M + kb), b);
#pragma unroll
          for (int s = 0; s < 7; ++s) u[s][h] = pack_f16(a[s], b[s]);
        }
#pragma unroll
        for (int s = 0; s < 7; ++s) tmem_st2(tl + s * KS * 8 + (k0 + 4 * j) / 2, u[s]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < kCnt / 4; ++j) {
        uint32_t u[3][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          __nv_bfloat16 a[3], b[3];
          split_bf16(val[4 * j + 2 * h], a);
          split_bf16(val[4 * j + 2 * h + 1], b);
#pragma unroll
          for (int s = 0; s < 3; ++s) u[s][h] = pack_bf16(a[s], b[s]);
        }
#pragma unroll
        for (int s = 0; s < 3; ++s) tmem_st2(tl + s * KS * 8 + (k0 + 4 * j) / 2, u[s]);
      }
    }
    tmem_st_wait();
    tc::fence_before();
  }
  __syncthreads();
  tc::fence_after();

  if (warp >= F::EpiWarps + 1) {
    // ---- loaders: the chunk's digit rows
    const int lt = tid - (F::EpiWarps + 1) * 32;
    constexpr int kLt = kLoadWarps * 32;
    constexpr int items = S * kPad * 8;
    for (int c = 0; c < nchunk; ++c) {
      const int buf = c & 1;
      if (c >= 2 && !wait(&empty[buf], (uint32_t)((c / 2 - 1) & 1), fail)) break;
      const uint32_t dst = tc::smem_addr(smem + buf * L.b_bytes);
      const uint16_t* src = g.Cs + (chunk0 + c) * kCols;
      // item i: 16 bytes at 16 i; part i / (8 kPad), K row i % 8 of block (i / 64) % (kPad / 8), strings 8 ((i / 8) % 8) ..
#pragma unroll 4
      for (int i = lt; i < items; i += kLt) {
        const int s = i / (8 * kPad), x = i - s * (8 * kPad), k = ((x >> 6) << 3) | (x & 7);
        if (k < K)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16 * i),
                       "l"(src + s * g.part + (int64_t)Jrow[k] * g.nbp + ((x >> 3) & 7) * 8)
                       : "memory");
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[buf]);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  } else if (warp == F::EpiWarps) {
    // ---- MMA issue: the whole warp follows, one lane issues.  The groups of
    // a chunk run from the largest (g = 6: seven products) down, so that the
    // slots filled during the walk of the chunk before hold most of the work.
    constexpr uint32_t idesc = idesc_f16(128, kCols, kF64 ? 0 : 1);
    int slot = 0;
    uint32_t round = 0;
    bool ok = true;
    auto all_wait = [&](uint64_t* b, uint32_t parity) {
      if (ok) ok = __all_sync(0xffffffffu, wait(b, parity, fail));
    };
    for (int c = 0; c < nchunk && ok; ++c) {
      const int buf = c & 1;
      all_wait(&full[buf], (uint32_t)((c / 2) & 1));
      // MN-major: 8 x 8 core matrices, 128 bytes between 8-string blocks, 1024 between 8-row blocks
      const uint64_t db = tc::desc(tc::smem_addr(smem + buf * L.b_bytes), 1024, 128);
#pragma unroll
      for (int gi = 0; gi < G; ++gi) {
        if constexpr (kF64) {
          if (gi >= kSl) all_wait(&reuse[gi - kSl], (uint32_t)(c & 1));
          if (c > 0 && gi == 0) all_wait(&reuse[kFirst], (uint32_t)((c - 1) & 1));
          if (c > 0 && gi == 1 && kFirst != G - 1) all_wait(&reuse[G - 1], (uint32_t)((c - 1) & 1));
          slot = gi % kSl;
        } else {
          if (round > 0) all_wait(&accempty[slot], (round - 1) & 1);
        }
        if (ok) {
          tc::fence_after();
          if (elect_one()) {
            const uint32_t d = tacc + (uint32_t)(slot * kCols);
            const int p0 = kF64 ? G - 1 - gi : 0, p1 = kF64 ? G - 1 - gi : 2;
#pragma unroll
            for (int p = p0; p <= p1; ++p)
#pragma unroll
              for (int i = 0; i <= p; ++i)
#pragma unroll
                for (int ks = 0; ks < KS; ++ks)
                  mma_f16_ts(d, tmem + (uint32_t)(i * KS * 8 + 8 * ks), db + (uint64_t)((p - i) * kPad * 8 + 128 * ks),
                             idesc, (p == p0 && i == 0 && ks == 0) ? 0u : 1u);
            if (!kF64) tc::commit(&accfull[slot]);
            if (kF64 && gi == min(kSl, G) - 1) tc::commit(&accfull[0]);
            if (kF64 && kRe > 0 && gi == G - 1) tc::commit(&accfull[1]);
            if (gi == G - 1) tc::commit(&empty[buf]);
          }
          __syncwarp();
        }
        if (!kF64 && ++slot == kSl) {
          slot = 0;
          ++round;
        }
      }
    }
    if (elect_one()) tc::commit(&done);
    __syncwarp();
    tc::mbar_wait(&done, 0, kSpin);  // every product has ended before TMEM is given back
  } else {
    // ---- read-out and walk
    const int q = warp & 3, r = q * 32 + lane;
    constexpr int kBlk = F::EpiWarps / 4, kW = kCols / kBlk;  // columns per warp
    const int col0 = (warp >> 2) * kW;
    const uint32_t tl = tacc + ((uint32_t)(q * 32) << 16) + (uint32_t)col0;
    int slot = 0;
    uint32_t round = 0;
    bool ok = true;
    int shp = 0, sho = 0;
    if (kF64) {
      const int u = min(mexp[0], mexp[1]);
      shp = mexp[0] - u;
      sho = mexp[1] - u;
    }
    // the walk lists of a chunk: one bulk copy (TMA), completing on listfull
    auto load_list = [&](int c) {
      const int u0 = __ldg(g.seg + chunk0 + c), bytes = 2 * (__ldg(g.seg + chunk0 + c + 1) - u0);
      tc::mbar_expect_tx(&listfull, (uint32_t)bytes);
      tc::bulk_g2s(smem + L.off_list, g.walk + u0, (uint32_t)bytes, &listfull);
    };
    if (tid == 0) load_list(0);
    for (int c = 0; c < nchunk; ++c) {
      typename F::E ev[kW];
      if constexpr (kF64) {
        static_assert(kW == 16, "one TMEM load per group");
        float low[16];
        constexpr int64_t kMagic = 0x4b400000;
        // units of 2^-57: group gr weighs 2^(57 - 9 (gr + 2)).  Groups 6 and 5
        // meet in FP32 (below one unit and 2^-6 of a sum); |group 0| <= 2^16 K
        // <= 2^22 and that pair become integers by the 1.5 2^23 addition
        // (their bits, kMagic taken off), the others by a conversion.
        auto take = [&](int gi, const float* v) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float x = v[j];
            if (gi == 0) low[j] = x * 0x1p-15f;
            if (gi == 1)
              ev[j] = (int64_t)(uint64_t)__float_as_uint(fmaf(x, 0x1p-6f, low[j]) + 12582912.f) - kMagic;
            if (gi == 2) ev[j] += (int64_t)__float2int_rn(x) * (1 << 3);
            if (gi == 3) ev[j] += (int64_t)__float2int_rn(x) * (1 << 12);
            if (gi == 4) ev[j] += (int64_t)__float2int_rn(x) * (1 << 21);
            if (gi == 5) ev[j] += (int64_t)__float2int_rn(x) * (1 << 30);
            if (gi == 6) ev[j] += (int64_t)(((uint64_t)__float_as_uint(x + 12582912.f) - kMagic) << 39);
          }
        };
        auto freed = [&](int gi) {
          if (gi < kRe || gi == kFirst || gi == G - 1) {
            tc::fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&reuse[gi]);
          }
        };
        if (ok) ok = __all_sync(0xffffffffu, wait(&accfull[0], (uint32_t)(c & 1), fail));
        tc::fence_after();
#pragma unroll
        for (int gi = 0; gi < G; ++gi) {
          if (kRe > 0 && gi == kSl) {
            if (ok) ok = __all_sync(0xffffffffu, wait(&accfull[1], (uint32_t)(c & 1), fail));
            tc::fence_after();
          }
          // two groups under one wait for TMEM, not across the second wait above
          const int first = gi < kSl ? 0 : kSl, past = gi < kSl ? min(kSl, G) : G;
          if ((gi - first) & 1) continue;
          float v0[16], v1[16];
          if (gi + 1 < past) {
            tc::tmem_ld16x2(tl + (uint32_t)(gi % kSl * kCols), tl + (uint32_t)((gi + 1) % kSl * kCols), v0, v1);
            freed(gi);
            freed(gi + 1);
            take(gi, v0);
            take(gi + 1, v1);
          } else {
            tc::tmem_ld16(tl + (uint32_t)(gi % kSl * kCols), v0);
            freed(gi);
            take(gi, v0);
          }
        }
      } else {
        if (ok) ok = __all_sync(0xffffffffu, wait(&accfull[slot], round & 1, fail));
        tc::fence_after();
#pragma unroll
        for (int h = 0; h < kW; h += 16) tc::tmem_ld16(tl + (uint32_t)(slot * kCols + h), ev + h);
        tc::fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&accempty[slot]);
        if (++slot == kSl) {
          slot = 0;
          ++round;
        }
      }
      if (r < g.R) {
        typename F::E* e = E + r * kPitch + col0;
#pragma unroll
        for (int j = 0; j < kW; j += (kF64 ? 2 : 4)) {
          if constexpr (kF64)
            *(longlong2*)(e + j) = make_longlong2(ev[j], ev[j + 1]);
          else
            *(float4*)(e + j) = make_float4(ev[j], ev[j + 1], ev[j + 2], ev[j + 3]);
        }
      }
      if (ok) ok = __all_sync(0xffffffffu, wait(&listfull, (uint32_t)(c & 1), fail));
      asm volatile("bar.sync 1, %0;\n" ::"r"(kEpi) : "memory");
      if (ok) {
        // tasks: 32 strings each, one lane per string, dealt to the warps by
        // the host (head[w] .. head[w + 1] are warp w's)
        const int nt = list[F::EpiWarps == 16 ? 16 : 32 + 8];
        const uint16_t* head = list + (F::EpiWarps == 16 ? 0 : 32);
        const uint16_t* order = list + kHead + (F::EpiWarps == 16 ? 0 : (nt + 7) & ~7);
        const uint16_t* task = list + kHead + 2 * ((nt + 7) & ~7);
        const uint16_t* tgt = task + 4 * nt + ((4 * nt) & 4);
        const uint16_t* ent = tgt + 32 * nt + lane;
        for (int at = head[warp]; at < head[warp + 1]; ++at) {
          const int t = order[at];
          const uint16_t* p = ent + 32 * (int)task[4 * t];
          const int steps = task[4 * t + 1], own = task[4 * t + 2];
          const int ib = tgt[32 * t + lane];
          if constexpr (kF64) {
            uint64_t sl = 0;
            int32_t sh = 0;
            auto sum = [&](int cnt) {
              uint32_t x0 = 0, x1 = 0, x2 = 0;
              int neg = 0;
#pragma unroll 4
              for (int i = 0; i < cnt; ++i) {
                const uint32_t w = *p;
                p += 32;
                const int m = -(int)(w >> 15);
                const int64_t e = E[w & 0x7fff] ^ (int64_t)m;
                const uint32_t a0 = (uint32_t)e, a1 = (uint32_t)(e >> 32), a2 = (uint32_t)((int)a1 >> 31);
                asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %4;\n addc.u32 %2, %2, %5;\n"
                    : "+r"(x0), "+r"(x1), "+r"(x2)
                    : "r"(a0), "r"(a1), "r"(a2));
                neg -= m;
              }
              asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, 0;\n addc.u32 %2, %2, 0;\n"
                  : "+r"(x0), "+r"(x1), "+r"(x2)
                  : "r"((uint32_t)neg));
              sl = (uint64_t)x0 | ((uint64_t)x1 << 32);
              sh = (int32_t)x2;
            };
            uint64_t tl64 = 0;
            int32_t th = 0;
            auto add_shifted = [&](int s) {
              const uint64_t a = sl << s;
              const int32_t b = (int32_t)(((uint32_t)sh << s) | (s ? (uint32_t)(sl >> (64 - s)) : 0u));
              const uint64_t old = tl64;
              tl64 += a;
              th += b + (tl64 < old ? 1 : 0);
            };
            sum(steps);
            add_shifted(shp);
            if (own) {
              sum(own);
              add_shifted(sho);
            }
            if (ib != 0xffff) {
              const uint64_t old = lo[ib];
              const uint64_t now = old + tl64;
              lo[ib] = now;
              hi[ib] += th + (now < old ? 1 : 0);
            }
          } else {
            float s = ib != 0xffff ? facc[ib] : 0.f;
#pragma unroll 4
            for (int i = 0; i < steps + own; ++i) {
              const uint32_t w = *p;
              p += 32;
              s += __int_as_float(__float_as_int(E[w & 0x7fff]) ^ (int)((w >> 15) << 31));
            }
            if (ib != 0xffff) facc[ib] = s;
          }
        }
      }
      asm volatile("bar.sync 1, %0;\n" ::"r"(kEpi) : "memory");  // E and the list free
      if (ok && tid == 0 && c + 1 < nchunk) load_list(c + 1);
    }
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    bool finish = true;
    if (!whole) {
      // this piece's sums out; the string's last CTA adds the pieces
      const int row = piece / g.split;
      for (int i = tid; i < g.nb; i += kEpi) {
        g.part_lo[(int64_t)piece * g.nb + i] = lo[i];
        g.part_hi[(int64_t)piece * g.nb + i] = hi[i];
      }
      __threadfence();
      asm volatile("bar.sync 1, %0;\n" ::"r"(kEpi) : "memory");
      if (tid == 0) {
        unsigned* cnt = g.part_count + 2 * row;
        if (!ok) atomicOr(cnt + 1, 1u);
        __threadfence();
        int state = atomicAdd(cnt, 1u) == (unsigned)g.split - 1 ? 1 : 0;
        __threadfence();
        if (state) {
          if (atomicExch(cnt + 1, 0u)) state = 2;
          *cnt = 0u;
        }
        last_ = state;
      }
      asm volatile("bar.sync 1, %0;\n" ::"r"(kEpi) : "memory");
      finish = last_ > 0;
      if (last_ == 2) ok = false;
      if (finish) {
        __threadfence();
        const int64_t p0 = (int64_t)row * g.split * g.nb;
        for (int i = tid; i < g.nb; i += kEpi) {
          uint64_t sl = 0;
          int32_t sh = 0;
          for (int k = 0; k < g.split; ++k) {
            const uint64_t a = __ldcg(g.part_lo + p0 + (int64_t)k * g.nb + i);
            sl += a;
            sh += __ldcg(g.part_hi + p0 + (int64_t)k * g.nb + i) + (sl < a ? 1 : 0);
          }
          lo[i] = sl;
          hi[i] = sh;
        }
      }
    }
    for (int i = tid; finish && i < g.nb; i += kEpi) {
      const int64_t at = Ia * g.nb + i;
      if constexpr (kF64) {
        // the integer once to FP64, then its unit
        const int64_t l = (int64_t)lo[i];
        const int32_t h = hi[i];
        const int e = min(mexp[0], mexp[1]) - kUnit;
        double v = (int64_t)h == (l >> 63) ? whole_scaled(l, e) : scale2((double)h * 0x1p64 + (double)(uint64_t)l, e);
        v += fma(g.D[at], g.C[at], g.sigma[at]);
        g.sigma[at] = ok ? v : nan;
      } else {
        g.sigma[at] = ok ? facc[i] : (float)nan;
      }
    }
    if (!ok && tid == 0) {
      // a list copy may be in flight: both phases' ends are bounded waits
      tc::mbar_wait(&listfull, 0, kSpin / 4);
      tc::mbar_wait(&listfull, 1, kSpin / 4);
      atomicOr(g.fault, 1u);
    }
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == 0) tc::tmem_free(tmem, F::Tmem);
}

// ---------------------------------------------------------------- same-spin part
// y = H_aa C + C H_bb^T in FP64 from 16-bit digits (S = 7 balanced 8-bit digits,
// 56 bits, whole numbers in fp16, |digit| <= 128): two dense products of 128 x
// 64 tiles, seven accumulators (i + j = g) of 64 TMEM columns.  A row of H has
// few elements (its doubles and singles), so an accumulator holds at most
// (g + 1) 2^14 m with m the row's elements inside the K range summed in it:
// below 2^24 for g <= 4 while 5 m <= 1024.  The K range is cut (`flush` K
// blocks) so that this holds, and the accumulators go to 64-bit integers in
// units of 2^-54 in between; g = 5, 6 weigh 2^-56 and less.  One exponent per
// row of H, per row of C (second product) and per column of C (first).
constexpr int kDnM = 128, kDnN = 64, kDnK = 32, kDnS = 7, kDnW = 8, kDnUnit = 54;
constexpr int kDnA = kDnS * kDnM * kDnK * 2, kDnB = kDnS * kDnN * kDnK * 2;  // bytes of a K block
constexpr int kDnStages = 2, kDnEpi = 8, kDnThreads = (2 + kDnEpi) * 32;
constexpr int kDnMaxRow = 204;  // elements of an H row in one flush range

// element (r, k) of an operand of `rows`-row tiles: its fp16 offset in part 0
// (blocks of rows x 32 K, the seven parts of a block contiguous; inside a
// part 8-row x 8-K core matrices, K fastest)
__device__ __forceinline__ int64_t dn_off(int r, int k, int rows, int nkb) {
  const int64_t blk = (int64_t)(r / rows) * nkb + k / kDnK;
  const int rr = r % rows, kk = k % kDnK;
  return blk * kDnS * rows * kDnK + ((rr >> 3) * (kDnK / 8) + (kk >> 3)) * 64 + (rr & 7) * 8 + (kk & 7);
}

// One spin's dense same-spin matrix as digits: row i holds its doubles and,
// with ns > 0, the singles' string-only part.  out zeroed before.  One CTA per row.
__global__ void __launch_bounds__(128)
    k_dn_matrix(int nd, int ns, const int32_t* __restrict__ dJ, const double* __restrict__ dval,
                const int32_t* __restrict__ sJ, const int32_t* __restrict__ svo, const double* __restrict__ sA, int rows,
                int nkb, uint16_t* __restrict__ out, int* __restrict__ rexp) {
  __shared__ int red[4];
  const int64_t i = blockIdx.x;
  auto value = [&](int m) {
    if (m < nd) return dval[i * nd + m];
    const double v = sA[i * ns + m - nd];
    return (svo[i * ns + m - nd] >> 16) ? -v : v;
  };
  int e = kNoExp;
  for (int m = threadIdx.x; m < nd + ns; m += 128) e = max(e, exp_above(value(m)));
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
  e = max(max(red[0], red[1]), max(red[2], red[3])) + 1;
  if (threadIdx.x == 0) rexp[i] = e;
  if (e <= kNoExp + 1) return;
  for (int m = threadIdx.x; m < nd + ns; m += 128) {
    const int k = m < nd ? dJ[i * nd + m] : sJ[i * ns + m - nd];
    int d[kDnS];
    digits<kDnS, kDnW>(fixed_point(value(m), kDnS * kDnW - e), d);
    const int64_t o = dn_off((int)i, k, rows, nkb);
#pragma unroll
    for (int s = 0; s < kDnS; ++s) out[o + (int64_t)s * rows * kDnK] = __half_as_ushort(__int2half_rn(d[s]));
  }
}

// exponents of the columns of C (na x nb) by atomic maximum (cexp preset far
// below any exponent).  grid: (column blocks of 32, row splits)
__global__ void __launch_bounds__(256) k_dn_colexp(int na, int nb, const double* __restrict__ C, int* __restrict__ cexp) {
  __shared__ int red[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, col = blockIdx.x * 32 + tx;
  int e = kNoExp;
  if (col < nb)
    for (int r = blockIdx.y * 8 + ty; r < na; r += 8 * gridDim.y) e = max(e, exp_above(C[(int64_t)r * nb + col]));
  red[ty][tx] = e;
  __syncthreads();
  if (ty == 0 && col < nb) {
    for (int w = 1; w < 8; ++w) e = max(e, red[w][tx]);
    atomicMax(&cexp[col], e + 1);
  }
}

// C into both digit operands: A form (rows Ia, K = Jb, exponents rexp of the
// rows) and B form (rows Jb, K = Ja, exponents cexp of the columns).  A CTA
// takes a 32 x 32 tile of C; eight K of one row are one 16-byte store.
__global__ void __launch_bounds__(256)
    k_dn_split(int na, int nb, const double* __restrict__ C, const int* __restrict__ rexp,
               const int* __restrict__ cexp, int nkb1, int nkb2, int napad, int nbpad, uint16_t* __restrict__ outA,
               uint16_t* __restrict__ outB) {
  __shared__ double t[32][33];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  for (int i = threadIdx.x; i < 1024; i += 256) {
    const int r = r0 + (i >> 5), cc = c0 + (i & 31);
    t[i >> 5][i & 31] = r < na && cc < nb ? C[(int64_t)r * nb + cc] : 0.;
  }
  __syncthreads();
  // threads 0-127 the A form, 128-255 the B form: row x, K 8 y .. 8 y + 7
  const int form = threadIdx.x >> 7, x = threadIdx.x & 31, y = (threadIdx.x >> 5) & 3;
  const int row = form ? c0 + x : r0 + x, k0 = (form ? r0 : c0) + 8 * y;
  const int rows = form ? kDnN : kDnM, nkb = form ? nkb1 : nkb2;
  if (row >= (form ? nbpad : napad) || k0 >= nkb * kDnK) return;
  const int e = row < (form ? nb : na) ? (form ? cexp[row] : rexp[row]) : kNoExp;
  uint32_t u[kDnS][4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    int a[kDnS], b[kDnS];
    const int k = 8 * y + 2 * h;
    const double va = form ? t[k][x] : t[x][k], vb = form ? t[k + 1][x] : t[x][k + 1];
    digits<kDnS, kDnW>(e > kNoExp + 1 ? fixed_point(va, kDnS * kDnW - e) : 0, a);
    digits<kDnS, kDnW>(e > kNoExp + 1 ? fixed_point(vb, kDnS * kDnW - e) : 0, b);
#pragma unroll
    for (int s = 0; s < kDnS; ++s) u[s][h] = pack_f16(a[s], b[s]);
  }
  uint16_t* o = (form ? outB : outA) + dn_off(row, k0, rows, nkb);
#pragma unroll
  for (int s = 0; s < kDnS; ++s) *(uint4*)(o + s * rows * kDnK) = make_uint4(u[s][0], u[s][1], u[s][2], u[s][3]);
}

struct DenseArgs {
  int M, N, nkb1, nkb2, flush;
  const uint16_t *a1, *b1, *a2, *b2;  // H_aa (A form), C (B form), C (A form), H_bb (B form)
  const int *ea1, *eb1, *ea2, *eb2;   // exponents: rows of a1 / a2, columns of b1 / b2
  double* out;
  const int* bad;
  unsigned* fault;
  int zsplit;                  // CTAs per tile, each with a range of the K blocks
  unsigned long long* zsum;    // their sums [tile][product][column][row] (whole numbers; zero before and after)
  unsigned* zcount;            // per tile: arrived, failed (zero before and after)
};

// CTAs per tile: as many as the idle SMs allow, with two K blocks each at
// least.  252 strings are eight tiles of sixteen blocks: one CTA each 38.8 us,
// eight each 29 us; 462 are 32 tiles: 58 and 37 us.
inline int dense_split(int64_t tiles, int nblk, int sms) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(sms / tiles, nblk / 2));
}

// USE: 0 reads A and keeps it in the collector, 1 takes it from there, 2 for
// the last time
template <int USE>
__device__ __forceinline__ void mma_f16_ss(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
#define QDKGB_MMA_SS(op)                                                              \
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"                         \
               " tcgen05.mma.cta_group::1.kind::f16.collector::a::" op " [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem), \
               "l"(a), "l"(b), "r"(idesc), "r"(accumulate))
  if (USE == 0) QDKGB_MMA_SS("fill");
  if (USE == 1) QDKGB_MMA_SS("use");
  if (USE == 2) QDKGB_MMA_SS("lastuse");
#undef QDKGB_MMA_SS
}

// warp 0 lane 0 fills a two-stage ring with bulk copies (both operands' seven
// parts of a K block, 84 KB), warp 1 lane 0 issues the 56 products of a block,
// warps 2-9 take the accumulators at the end of every flush range.  Two
// products of 3432 strings: 3.7 ms (24.4 ms element by element), 57 clocks a
// 128 x 64 x 16 product where the tensor cores need 32: L2 feeds 84 KB per K
// block and SM.  With A read from shared memory for each product 4.5 ms.
__global__ void __launch_bounds__(kDnThreads, 1) k_dense64(DenseArgs g) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kDnStages], empty[kDnStages], accfull, accempty;
  __shared__ uint32_t tslot;
  __shared__ int fail_, last_;
  volatile int* fail = &fail_;
  if (*g.bad) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rb = blockIdx.y, nbk = blockIdx.x;
  if (warp == 0) tc::tmem_alloc(&tslot, 512);
  if (tid == 0) {
    for (int s = 0; s < kDnStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(&accfull, 1);
    tc::mbar_init(&accempty, kDnEpi);
    tc::mbar_init_fence();
    fail_ = 0;
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tslot;
  const int nblk_all = g.nkb1 + g.nkb2;
  const int blk0 = (int)blockIdx.z * nblk_all / g.zsplit, nblk = ((int)blockIdx.z + 1) * nblk_all / g.zsplit;
  // the flush ranges end at multiples of `flush` blocks of each product and at its last
  auto range_end = [&](int b) {
    return (b < g.nkb1 ? ((b + 1) % g.flush == 0 || b + 1 == g.nkb1)
                       : ((b - g.nkb1 + 1) % g.flush == 0 || b + 1 == nblk_all)) ||
           b + 1 == nblk;
  };
  if (warp == 0) {
    if (lane == 0) {
      for (int b = blk0; b < nblk; ++b) {
        const int l = b - blk0, s = l % kDnStages;
        if (l >= kDnStages && !wait(&empty[s], (uint32_t)((l / kDnStages - 1) & 1), fail)) break;
        const bool p2 = b >= g.nkb1;
        const int kb = p2 ? b - g.nkb1 : b, nkb = p2 ? g.nkb2 : g.nkb1;
        unsigned char* st = smem + s * (kDnA + kDnB);
        tc::mbar_expect_tx(&full[s], (uint32_t)(kDnA + kDnB));
        tc::bulk_g2s(st, (const unsigned char*)(p2 ? g.a2 : g.a1) + ((int64_t)rb * nkb + kb) * kDnA, kDnA, &full[s]);
        tc::bulk_g2s(st + kDnA, (const unsigned char*)(p2 ? g.b2 : g.b1) + ((int64_t)nbk * nkb + kb) * kDnB, kDnB,
                     &full[s]);
      }
    }
  } else if (warp == 1) {
    {
      constexpr uint32_t idesc = idesc_f16(kDnM, kDnN, 0) & ~(1u << 16);  // both operands K-major
      bool ok = true;
      uint32_t first = 1, ranges = 0;
      int b = blk0;
      for (; b < nblk; ++b) {
        const int l = b - blk0, s = l % kDnStages;
        ok = __all_sync(0xffffffffu, wait(&full[s], (uint32_t)((l / kDnStages) & 1), fail));
        if (ok && first && ranges > 0) ok = __all_sync(0xffffffffu, wait(&accempty, (ranges - 1) & 1, fail));
        if (!ok) break;
        tc::fence_after();
        const uint32_t st = tc::smem_addr(smem + s * (kDnA + kDnB));
        const uint64_t da = tc::desc(st, 128, 512), db = tc::desc(st + kDnA, 128, 512);
        const bool last = range_end(b);
        if (elect_one()) {
          const uint32_t acc0 = first ? 0u : 1u;
          // each part of A against all its parts of B in turn, so that A is read
          // from shared memory once per part and not once per product
#pragma unroll
          for (int ks = 0; ks < kDnK / 16; ++ks)
#pragma unroll
            for (int i = 0; i < kDnS; ++i) {
              const uint64_t ai = da + (uint64_t)(i * (kDnM * kDnK * 2 / 16) + ks * 16);
#pragma unroll
              for (int j = 0; j < kDnS - i; ++j) {
                const uint32_t acc = (i == 0 && ks == 0) ? acc0 : 1u, dt = tmem + 64 * (i + j);
                const uint64_t bj = db + (uint64_t)(j * (kDnN * kDnK * 2 / 16) + ks * 16);
                if (j == 0)
                  mma_f16_ss<0>(dt, ai, bj, idesc, acc);
                else if (j < kDnS - 1 - i)
                  mma_f16_ss<1>(dt, ai, bj, idesc, acc);
                else
                  mma_f16_ss<2>(dt, ai, bj, idesc, acc);
              }
            }
          tc::commit(&empty[s]);
          if (last) tc::commit(&accfull);
        }
        __syncwarp();
        first = last ? 1 : 0;
        ranges += last ? 1 : 0;
      }
      if (!ok) {  // let the products in flight end before TMEM is given back
        if (elect_one()) tc::commit(&accfull);
        __syncwarp();
        tc::mbar_wait(&accfull, ranges & 1, kSpin);
        // copies in flight: the stages filled or being filled
        for (int f = b - blk0 + 1; f < nblk - blk0 && f < b - blk0 + kDnStages; ++f)
          tc::mbar_wait(&full[f % kDnStages], (uint32_t)((f / kDnStages) & 1), kSpin);
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2, row = rb * kDnM + q * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(32 * half);
    const int c0 = nbk * kDnN + 32 * half;
    bool ok = true;
    uint32_t ranges = 0;
    double v[32];
    int64_t acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      v[j] = 0.;
      acc[j] = 0;
    }
    unsigned long long* z1 =
        g.zsum + ((int64_t)(rb * gridDim.x + nbk) * 2 * kDnN + 32 * half) * kDnM + q * 32 + lane;
    unsigned long long* z2 = z1 + kDnN * kDnM;
    const int er1 = row < g.M ? g.ea1[row] - kDnUnit : 0, er2 = row < g.M ? g.ea2[row] - kDnUnit : 0;
    for (int b = blk0; b < nblk; ++b) {
      if (!range_end(b)) continue;
      if (ok) ok = __all_sync(0xffffffffu, wait(&accfull, ranges & 1, fail));
      ++ranges;
      if (!ok) break;
      tc::fence_after();
#pragma unroll
      for (int gr = 0; gr < kDnS; ++gr)
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          float x[16];
          tc::tmem_ld16(tl + 64 * gr + h, x);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            // group gr weighs 2^(54 - 8 (gr + 2)) units
            if (gr == 0) acc[h + j] += (int64_t)(__float2int_rn(x[j]) << 8) * (1 << 30);
            if (gr == 1) acc[h + j] += (int64_t)__float2int_rn(x[j]) * (1 << 30);
            if (gr == 2) acc[h + j] += (int64_t)__float2int_rn(x[j]) * (1 << 22);
            if (gr == 3) acc[h + j] += (int64_t)__float2int_rn(x[j]) * (1 << 14);
            if (gr == 4) acc[h + j] += (int64_t)__float2int_rn(x[j]) * (1 << 6);
            if (gr == 5) acc[h + j] += (int64_t)__float2int_rn(x[j] * 0x1p-2f);
            if (gr == 6) acc[h + j] += (int64_t)__float2int_rn(x[j] * 0x1p-10f);
          }
        }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&accempty);
      if (b + 1 == g.nkb1 || b + 1 == nblk) {
        const bool second = b >= g.nkb1;
        const int er = second ? er2 : er1;
        const int* eb = second ? g.eb2 : g.eb1;
        unsigned long long* z = second ? z2 : z1;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (acc[j] != 0 && row < g.M && c0 + j < g.N) {
            if (g.zsplit > 1)
              atomicAdd(z + j * kDnM, (unsigned long long)acc[j]);
            else
              v[j] += whole_scaled(acc[j], er + eb[c0 + j]);
          }
          acc[j] = 0;
        }
      }
    }
    bool finish = true;
    if (g.zsplit > 1) {
      // the tile's last CTA takes the sums and leaves zeros
      __threadfence();
      asm volatile("bar.sync 1, %0;\n" ::"r"(kDnEpi * 32) : "memory");
      if (tid == 64) {
        unsigned* cnt = g.zcount + 2 * (rb * gridDim.x + nbk);
        if (!ok) atomicOr(cnt + 1, 1u);
        __threadfence();
        int state = atomicAdd(cnt, 1u) == (unsigned)g.zsplit - 1 ? 1 : 0;
        __threadfence();
        if (state) {
          if (atomicExch(cnt + 1, 0u)) state = 2;
          *cnt = 0u;
        }
        last_ = state;
      }
      asm volatile("bar.sync 1, %0;\n" ::"r"(kDnEpi * 32) : "memory");
      finish = last_ > 0;
      if (last_ == 2) ok = false;
      if (finish && row < g.M) {
        __threadfence();
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 8) {
          // eight columns' loads together (columns past N hold zeros)
          int64_t s1[8], s2[8];
          int b1[8], b2[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            s1[j] = (int64_t)__ldcg(z1 + (j0 + j) * kDnM);
            s2[j] = (int64_t)__ldcg(z2 + (j0 + j) * kDnM);
            const int col = min(c0 + j0 + j, g.N - 1);
            b1[j] = g.eb1[col];
            b2[j] = g.eb2[col];
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (s1[j] != 0) v[j0 + j] += whole_scaled(s1[j], er1 + b1[j]);
            if (s2[j] != 0) v[j0 + j] += whole_scaled(s2[j], er2 + b2[j]);
            z1[(j0 + j) * kDnM] = 0ull;
            z2[(j0 + j) * kDnM] = 0ull;
          }
        }
      }
    }
    if (finish && row < g.M)
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (c0 + j < g.N)
          g.out[(int64_t)row * g.N + c0 + j] = ok ? v[j] : __longlong_as_double(0x7ff8000000000000ll);
    if (!ok && lane == 0) atomicOr(g.fault, 1u);
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == 0) tc::tmem_free(tmem, 512);
}

// The FP64 sigma element by element, for inputs with infinities or NaN (which
// have no fixed-point form): runs only when *bad is set.  One CTA per alpha
// string, a thread per beta string.
struct PlainArgs {
  int64_t na, nb;
  int n, nsa, nda, nsb, ndb;
  const int32_t *a_sJ, *a_svo, *a_dJ, *b_sJ, *b_svo, *b_dJ;
  const double *a_sA, *a_dval, *a_W, *b_sA, *b_dval, *b_W, *V, *D;
  const int* bad;
};
__global__ void __launch_bounds__(256) k_plain64(PlainArgs g, const double* __restrict__ C, double* __restrict__ out) {
  if (!*g.bad) return;
  const int64_t Ia = blockIdx.x;
  const int n2 = g.n * g.n;
  auto pair = [&](int32_t vo) { return (vo & 0xff) + g.n * ((vo >> 8) & 0xff); };
  for (int64_t Ib = threadIdx.x; Ib < g.nb; Ib += blockDim.x) {
    double s = g.D[Ia * g.nb + Ib] * C[Ia * g.nb + Ib];
    for (int m = 0; m < g.nda; ++m) s += g.a_dval[Ia * g.nda + m] * C[(int64_t)g.a_dJ[Ia * g.nda + m] * g.nb + Ib];
    for (int m = 0; m < g.ndb; ++m) s += g.b_dval[Ib * g.ndb + m] * C[Ia * g.nb + g.b_dJ[Ib * g.ndb + m]];
    for (int l = 0; l < g.nsb; ++l) {
      const int32_t vo = g.b_svo[Ib * g.nsb + l];
      const double h = g.b_sA[Ib * g.nsb + l] + g.a_W[(int64_t)pair(vo) * g.na + Ia];
      s += ((vo >> 16) ? -h : h) * C[Ia * g.nb + g.b_sJ[Ib * g.nsb + l]];
    }
    for (int k = 0; k < g.nsa; ++k) {
      const int32_t vo = g.a_svo[Ia * g.nsa + k];
      const double* row = C + (int64_t)g.a_sJ[Ia * g.nsa + k] * g.nb;
      double t = (g.a_sA[Ia * g.nsa + k] + g.b_W[(int64_t)pair(vo) * g.nb + Ib]) * row[Ib];
      for (int l = 0; l < g.nsb; ++l) {
        const int32_t wo = g.b_svo[Ib * g.nsb + l];
        const double h = g.V[pair(vo) + (int64_t)n2 * pair(wo)];
        t += ((wo >> 16) ? -h : h) * row[g.b_sJ[Ib * g.nsb + l]];
      }
      s += (vo >> 16) ? -t : t;
    }
    out[Ia * g.nb + Ib] = s;
  }
}

// 1: some V(pq|rs) and V(pq|sr) differ as FP64, 2: as FP32 too (B integral
// sets, V column-major)
__global__ void k_ct_symmetry(const double* __restrict__ V, int n, int64_t tot, int* __restrict__ flag) {
  const int64_t n2 = (int64_t)n * n, n4 = n2 * n2;
  int f = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = i / n4, u = i - b * n4, pq = u % n2, rs = u / n2, r = rs % n, s = rs / n;
    if (r >= s) continue;
    const double x = V[i], y = V[b * n4 + pq + n2 * (s + n * r)];
    if (!(x == y)) f |= 1;
    if (!((float)x == (float)y)) f |= 2;
  }
  if (f) atomicOr(flag, f);
}
// V2[pq][R] (see Args): the pair rows V(pq, rs_r), then V(p p | pq); the last row unused
template <typename T>
__global__ void k_ct_v2(const double* __restrict__ V, const int32_t* __restrict__ rs_of, int n, int mr, int R,
                        T* __restrict__ V2) {
  const int64_t n2 = (int64_t)n * n, tot = n2 * R;
  V += blockIdx.y * n2 * n2;
  V2 += blockIdx.y * tot;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pq = i / R;
    const int r = (int)(i - pq * R);
    V2[i] = r < mr ? (T)V[pq + n2 * rs_of[r]] : r < mr + n ? (T)V[(r - mr) * (int64_t)(n + 1) + n2 * pq] : (T)0;
  }
}

}  // namespace ct
}  // namespace qdkgb
