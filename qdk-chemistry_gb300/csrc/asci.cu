// ASCI determinant search on the device (replaces asci_search /
// asci_contributions_constraint, include/macis/asci/determinant_search.hpp:
// 349-1123, with the contribution formulas of determinant_contributions.hpp:
// 93-297 and the fast diagonals of src/macis/hamiltonian_generator/
// fast_diagonals.ipp:52-127).
//
// GPU design: a few CTAs per core determinant P enumerate every single and
// double excitation Q of P by rows (one beta single, or one pair of occupied
// orbitals, against all its partners), evaluate c_P <Q|H|P>
// and the fast diagonal E0 - H_QQ exactly as the reference does, drop
// |c h| < h_el_tol, and accumulate into an open-addressing hash table keyed by
// the full (alpha, beta) pair (128-bit atomicCAS, then exact fixed-point
// integer atomics of c h; see Table below).  That replaces the reference's
// constraint partitioning plus sort-and-accumulate: every Q's contributions
// meet in one slot.  The core itself is marked and drops out.  Then |rv| =
// |sum / (E0 - H_QQ)| is pruned (|rv| > rv_prune_tol), the k-th largest |rv|
// is found by a radix select on the bit patterns (four 16-bit digits), and
// every candidate with |rv| >= that value is kept - the reference's
// tie-inclusive top-k.  Sums and diagonals do not depend on the order of the
// atomics, so a search repeated on the same input selects the same set with
// the same scores; they agree with the reference's (whose unstable sort
// fixes its own order) to rounding, and the selected sets are identical
// unless two scores tie to the last bits at the cutoff.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "host_parallel.h"
#include "internal.h"

namespace qdkgb {

namespace {

typedef unsigned __int128 u128;
constexpr u128 kEmpty = ~(u128)0;
constexpr int kAsciWarps = 8;
constexpr int kMaxOrb = 64;

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdULL;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ULL;
  x ^= x >> 33;
  return x;
}

// A target's accumulated c <Q|H|P> is kept in fixed point, two 64-bit words
// per slot: x = hi 2^-32 + lo 2^-76 with hi = rint(x 2^32) and lo the rest
// in units of 2^-76 (the split is exact).  Integer additions are exact and
// associative, so the sum - and the selection made from it - does not depend
// on the order in which the atomics land (FP64 atomics would).  |x| < 2^20
// and up to 2^19 contributions per target keep both words in range.  The
// slot's diagonal E0 - H_QQ (the fast diagonal, computed from each
// contributing P, equal up to rounding) is the largest bit pattern among its
// contributors (atomicMax on the bits: order-independent as well); core
// determinants set it to kCoreMark and drop out of the candidates.
constexpr long long kCoreMark = 0x7fffffffffffffffLL;
constexpr long long kHdEmpty = (long long)0x8000000000000000ULL;
constexpr double kFixHi = 4294967296.0;               // 2^32
constexpr double kFixLo = 75557863725914323419136.0;  // 2^76

// A slot's key and sums share one 32-byte sector: a contribution touches two
// sectors at random (this and hd) instead of three.
struct __align__(32) Slot {
  u128 key;
  long long hi, lo;
};
struct Table {
  Slot* slot;
  long long* hd;  // bit pattern of E0 - H_QQ, or kCoreMark
  uint64_t cap;   // slots (any number: the hash is scaled to it)
  int* err;  // set when a probe sequence runs past kMaxProbe (the table is too full): the pass is redone larger
};
constexpr uint64_t kMaxProbe = 4096;

__device__ __forceinline__ double table_sum(const Table& t, uint64_t i) {
  return (double)t.slot[i].hi * (1.0 / kFixHi) + (double)t.slot[i].lo * (1.0 / kFixLo);
}
__device__ __forceinline__ bool table_core(const Table& t, uint64_t i) { return t.hd[i] == kCoreMark; }

// |x| as an ordered integer: comparisons off the FP64 pipe
__device__ __forceinline__ uint64_t magnitude(double x) {
  return (uint64_t)__double_as_longlong(x) & 0x7fffffffffffffffULL;
}
constexpr uint64_t kBits2p19 = (uint64_t)(1023 + 19) << 52, kBits2p20 = (uint64_t)(1023 + 20) << 52;
constexpr uint64_t kBitsInf = (uint64_t)2047 << 52;

__device__ __forceinline__ u128 table_key(uint64_t qa, uint64_t qb) { return ((u128)qb << 64) | (u128)qa; }
__device__ __forceinline__ uint64_t table_home(const Table& t, uint64_t qa, uint64_t qb) {
  return __umul64hi(mix64(qa * 0x9e3779b97f4a7c15ULL ^ mix64(qb)), t.cap);
}
// the key's slot, inserted if need be, when its home h held `old` before an
// exchange; -1 when the probe limit is reached
__device__ __forceinline__ int64_t table_slot(const Table& t, u128 key, uint64_t h, u128 old) {
  for (uint64_t probe = 1; old != kEmpty && old != key; ++probe) {
    if (probe >= t.cap || probe >= kMaxProbe) {
      *t.err = 1;
      return -1;
    }
    if (++h == t.cap) h = 0;
    old = atomicCAS(&t.slot[h].key, kEmpty, key);
  }
  return (int64_t)h;
}

// Adds ch to the target's sum and meets its diagonal with diag(), which is
// worked out while the exchange at the target's home slot is under way.
template <class Diag>
__device__ __forceinline__ void table_add(const Table& t, uint64_t qa, uint64_t qb, double ch, Diag diag) {
  const u128 key = table_key(qa, qb);
  const uint64_t home = table_home(t, qa, qb);
  const u128 old = atomicCAS(&t.slot[home].key, kEmpty, key);
  const double hd = diag();
  // Adding 1.5 x 2^(52 - s) rounds to units of 2^-s (to even, as rint does)
  // and leaves the integer in the low bits: four FP64 operations instead of
  // two roundings, two conversions and their scalings.
  constexpr double kHiM = 1572864.0, kLoM = 6755399441055744.0;  // 1.5 x 2^20, 1.5 x 2^52
  const double t1 = __dadd_rn(ch, kHiM);
  const double rest = __dsub_rn(ch, __dsub_rn(t1, kHiM));
  long long hi = __double_as_longlong(t1) - __double_as_longlong(kHiM);
  long long lo = __double_as_longlong(__fma_rn(rest, kFixLo, kLoM)) - __double_as_longlong(kLoM);
  const int64_t h = table_slot(t, key, home, old);
  if (h < 0) return;
  if (magnitude(ch) >= kBits2p19) {
    if (magnitude(ch) >= kBits2p20) {  // outside the fixed-point range (or not finite)
      *t.err = 2;
      return;
    }
    const double h1 = rint(ch * kFixHi);
    hi = (long long)h1;
    lo = (long long)rint((ch - h1 * (1.0 / kFixHi)) * kFixLo);
  }
  atomicAdd((unsigned long long*)&t.slot[h].hi, (unsigned long long)hi);
  atomicAdd((unsigned long long*)&t.slot[h].lo, (unsigned long long)lo);
  atomicMax(t.hd + h, (long long)__double_as_longlong(hd));
}

__device__ __forceinline__ void table_add_core(const Table& t, uint64_t qa, uint64_t qb) {
  const u128 key = table_key(qa, qb);
  const uint64_t home = table_home(t, qa, qb);
  const int64_t h = table_slot(t, key, home, atomicCAS(&t.slot[home].key, kEmpty, key));
  if (h >= 0) atomicMax(t.hd + h, kCoreMark);
}

struct CoreArgs {
  Integrals I;
  int n;
  int64_t ncore;
  const uint64_t* ca;
  const uint64_t* cb;
  const double* cc;
  double E0;
  double h_el_tol;
  Table T;
  uint32_t npass = 1, pass = 0;  // targets whose part_of() == pass are inserted (npass > 1: PT2 passes)
  bool just_singles = false;     // the search's just_singles: single excitations only
  int nslice = 1;                // CTAs per core determinant
  // |x| >= h_el_tol
  __device__ __forceinline__ bool keeps(double x) const {
    const uint64_t m = magnitude(x);
    return (h_el_tol <= 0. || m >= (uint64_t)__double_as_longlong(h_el_tol)) && m <= kBitsInf && h_el_tol == h_el_tol;
  }
};

// part of the target space of a determinant in a split into npass passes (a
// hash independent of the table slot)
__device__ __forceinline__ uint32_t part_of(uint64_t qa, uint64_t qb, uint32_t npass) {
  return (uint32_t)(mix64(qb * 0x9e3779b97f4a7c15ULL ^ mix64(qa + 0x632be59bd9b4e019ULL)) % npass);
}

__device__ __forceinline__ double G2at(const Integrals& I, uint32_t p, uint32_t q) {
  return ld(I.G2 + p + (size_t)I.n * q);
}
__device__ __forceinline__ double V2at(const Integrals& I, uint32_t p, uint32_t q) {
  return ld(I.V2 + p + (size_t)I.n * q);
}
// Number of distinct target determinants of an enumeration (every single
// and double of every core determinant, and the core itself) as a
// HyperLogLog sketch: 2^kHllBits registers hold the largest leading-zero rank
// of a 64-bit hash per bucket (block-local in shared memory, merged with
// atomicMax).  Sizes the hash table to the targets instead of the
// contributions (relative error ~1.04 / 2^(kHllBits/2)).
constexpr int kHllBits = 12, kHllRegs = 1 << kHllBits;
__device__ __forceinline__ void hll_add(unsigned* reg, uint64_t qa, uint64_t qb) {
  const uint64_t h = mix64(qb * 0xbf58476d1ce4e5b9ULL ^ mix64(qa + 0x94d049bb133111ebULL));
  const unsigned idx = (unsigned)(h >> (64 - kHllBits));
  const uint64_t w = h << kHllBits;
  const unsigned rank = w ? (unsigned)__clzll(w) + 1u : (unsigned)(64 - kHllBits + 1);
  if (reg[idx] < rank) atomicMax(reg + idx, rank);
}

// What a CTA holds of its core determinant, sized by the determinant's own
// counts: singles as (occupied, virtual, sign) and their two G2 elements,
// pairs of occupied and of virtual orbitals, and before them the terms of the
// diagonal element.  41 KB for 64 orbitals half occupied, 105 KB at most (all
// of them occupied).
__host__ __device__ inline size_t asci_smem(bool count, int n, int ka, int kb, bool just_singles) {
  const size_t ns = (size_t)ka * (n - ka) + (size_t)kb * (n - kb);
  const size_t np = just_singles ? 0
                                 : ((size_t)ka * (ka - 1) + (size_t)(n - ka) * (n - ka - 1) + (size_t)kb * (kb - 1) +
                                    (size_t)(n - kb) * (n - kb - 1)) /
                                       2;
  const size_t terms = (size_t)ka + kb + (size_t)ka * ka + (size_t)kb * kb + (size_t)ka * kb;
  const size_t head = count ? kHllRegs * sizeof(unsigned) : (ns * 16 > terms * 8 ? ns * 16 : (terms * 8 + 15) / 16 * 16);
  return head + 2 * (ns + np) + 16;
}

// Singles and doubles of every core determinant: inserted with their
// contributions and diagonals (COUNT: into the sketch `regs`).  nslice CTAs
// per determinant, a warp per row, lanes along the row: an alpha-beta row is
// one beta single against every alpha single (integrals contiguous in the
// lanes' index, the row's share of the diagonal loaded once), a same-spin row
// one pair of occupied orbitals against every pair of virtual ones.  A warp
// per determinant left most of the chip idle at the usual few thousand core
// determinants, and spent 64-bit divisions on every target.  The order of the
// FP64 operations of each contribution and diagonal is the reference's.
//
// Four searches from up to 1,000 of 8+8 electrons in 40 orbitals (141 million
// contributions above the threshold in the largest): 62.8 -> 17.6 ms, the
// sketch 6.3 -> 0.6.  What bounds it: the FP64 pipe for 60% of the time (23
// instructions a contribution, of which 14 are the diagonal, whose rounding
// the selection between spin-flipped twins depends on), and the round trips
// to a table that no cache holds.  Looking at the slot before the exchange
// cost more than the exchanges it saved.
template <bool COUNT>
__global__ void __launch_bounds__(kAsciWarps * 32, 4) k_asci_enum(CoreArgs A, unsigned* __restrict__ regs) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double ea[kMaxOrb], eb[kMaxOrb], hdiag_s;
  __shared__ uint8_t oa[kMaxOrb], va[kMaxOrb], ob[kMaxOrb], vb[kMaxOrb];
  __shared__ double pend_ch[COUNT ? 1 : kAsciWarps][64];
  __shared__ uint16_t pend_x[COUNT ? 1 : kAsciWarps][64];
  constexpr int kThreads = kAsciWarps * 32;
  const int tid = threadIdx.x, lane = tid & 31;
  const Integrals& I = A.I;
  const int n = A.n;
  const size_t nn = (size_t)n;
  const int64_t ip = blockIdx.x / A.nslice;
  const int slice = (int)(blockIdx.x % A.nslice);
  const uint64_t Pa = A.ca[ip], Pb = A.cb[ip];
  const double c = A.cc[ip];
  const int ka = popc64(Pa), kb = popc64(Pb), na_v = n - ka, nb_v = n - kb;
  const int nsa = ka * na_v, nsb = kb * nb_v;
  const int pa_o = ka * (ka - 1) / 2, pb_o = kb * (kb - 1) / 2;
  const int pa_v = na_v * (na_v - 1) / 2, pb_v = nb_v * (nb_v - 1) / 2;
  const int terms = ka + kb + ka * ka + kb * kb + ka * kb;
  double2* sg = reinterpret_cast<double2*>(dyn);  // (G2(a, i), G2(i, a)) per single, beta's after alpha's
  unsigned* hll = reinterpret_cast<unsigned*>(dyn);
  const size_t head =
      COUNT ? kHllRegs * sizeof(unsigned)
            : (size_t)max(16 * (nsa + nsb), (terms * 8 + 15) / 16 * 16);
  uint16_t* sgl = reinterpret_cast<uint16_t*>(dyn + head);  // i | a << 6 | sign << 12
  uint16_t* pao = sgl + nsa + nsb;                          // i | j << 6, i < j
  uint16_t *pav = pao + pa_o, *pbo = pav + pa_v, *pbv = pbo + pb_o;

  if (tid < n) {
    const uint64_t below = (1ull << tid) - 1ull;
    const int x = popc64(Pa & below), y = popc64(Pb & below);
    if ((Pa >> tid) & 1)
      oa[x] = tid;
    else
      va[tid - x] = tid;
    if ((Pb >> tid) & 1)
      ob[y] = tid;
    else
      vb[tid - y] = tid;
  }
  if (COUNT)
    for (int i = tid; i < kHllRegs; i += kThreads) hll[i] = 0u;
  __syncthreads();
  // orbital energies (single_orbital_ens, fast_diagonals.ipp:30-50) and the
  // terms of the diagonal element in me_diag's order
  if (!COUNT) {
    if (tid < 2 * kMaxOrb) {
      const bool alpha = tid < kMaxOrb;
      const int i = tid & (kMaxOrb - 1);
      const uint8_t *same = alpha ? oa : ob, *other = alpha ? ob : oa;
      const int ks = alpha ? ka : kb, ko = alpha ? kb : ka;
      if (i < n) {
        double e = ld(I.T + i + nn * i);
#pragma unroll 4
        for (int x = 0; x < ks; ++x) {
          const uint32_t q = same[x];
          e += G2at(I, i, q) + G2at(I, q, i);
        }
        e -= G2at(I, i, i);
#pragma unroll 4
        for (int x = 0; x < ko; ++x) e += V2at(I, i, other[x]);
        (alpha ? ea : eb)[i] = e;
      }
    } else {
      double* term = reinterpret_cast<double*>(dyn);
      for (int t = tid - 2 * kMaxOrb; t < terms; t += kThreads - 2 * kMaxOrb) {
        int x = t;
        const double* src;
        if (x < ka)
          src = I.T + oa[x] + nn * oa[x];
        else if ((x -= ka) < kb)
          src = I.T + ob[x] + nn * ob[x];
        else if ((x -= kb) < ka * ka)
          src = I.G2 + nn * oa[x / ka] + oa[x % ka];
        else if ((x -= ka * ka) < kb * kb)
          src = I.G2 + nn * ob[x / kb] + ob[x % kb];
        else {
          x -= kb * kb;
          src = I.V2 + nn * ob[x / ka] + oa[x % ka];
        }
        term[t] = ld(src);
      }
    }
  }
  // singles and pairs
  for (int x = tid; x < nsa + nsb; x += kThreads) {
    const bool alpha = x < nsa;
    const int y = alpha ? x : x - nsa, nv = alpha ? na_v : nb_v;
    const uint32_t i = (alpha ? oa : ob)[y / nv], a = (alpha ? va : vb)[y % nv];
    sgl[x] = (uint16_t)(i | (a << 6) | (excitation_sign_odd(alpha ? Pa : Pb, a, i) ? 1u << 12 : 0u));
  }
  if (!A.just_singles) {
    // pairs (x, y), x < y: y runs fastest, rows x of K - 1 - x entries
    auto pairs = [&](uint16_t* out, const uint8_t* list, int K) {
      for (int t = tid; t < K * K; t += kThreads) {
        const int x = t / K, y = t % K;
        if (y > x) out[x * (2 * K - x - 1) / 2 + y - x - 1] = (uint16_t)(list[x] | (list[y] << 6));
      }
    };
    pairs(pao, oa, ka);
    pairs(pav, va, na_v);
    pairs(pbo, ob, kb);
    pairs(pbv, vb, nb_v);
  }
  __syncthreads();
  if (!COUNT) {
    if (tid == 0) {
      const double* term = reinterpret_cast<const double*>(dyn);
      double h = 0.;
#pragma unroll 8
      for (int t = 0; t < terms; ++t) h += term[t];
      hdiag_s = h;
    }
    __syncthreads();
    for (int x = tid; x < nsa + nsb; x += kThreads) {
      const uint32_t i = sgl[x] & 63, a = (sgl[x] >> 6) & 63;
      sg[x] = make_double2(G2at(I, a, i), G2at(I, i, a));
    }
    __syncthreads();
  }
  const double hdiag = COUNT ? 0. : hdiag_s;

  // the core determinant itself: marked, removed later
  if (slice == 0 && tid == 0) {
    if (COUNT)
      hll_add(hll, Pa, Pb);
    else if (A.npass == 1 || part_of(Pa, Pb, A.npass) == A.pass)
      table_add_core(A.T, Pa, Pb);
  }
  auto add = [&](uint64_t qa, uint64_t qb, double ch, auto diag) {
    if (A.npass == 1 || part_of(qa, qb, A.npass) == A.pass) table_add(A.T, qa, qb, ch, diag);
  };
  // A row's N contributions ch(x), those that the threshold keeps gathered
  // until a warp full of them (or the row's end) goes on to full(x, ch).
  auto gather = [&](int N, auto contribution, auto full) {
    double* qc = pend_ch[COUNT ? 0 : tid >> 5];
    uint16_t* qx = pend_x[COUNT ? 0 : tid >> 5];
    int held = 0;
    for (int x0 = 0; x0 < N; x0 += 32) {
      const int x = x0 + lane;
      const double ch = x < N ? contribution(x) : 0.;
      const bool keep = x < N && A.keeps(ch);
      const unsigned m = __ballot_sync(QDKGB_FULL_MASK, keep);
      if (keep) {
        const int p = held + __popc(m & ((1u << lane) - 1u));
        qc[p] = ch;
        qx[p] = (uint16_t)x;
      }
      held += __popc(m);
      __syncwarp();
      const bool last = x0 + 32 >= N;
      while (held >= 32 || (last && held > 0)) {
        if (lane < held) full((int)qx[lane], qc[lane]);
        __syncwarp();
        held -= 32;
        if (lane < held) {
          qc[lane] = qc[32 + lane];
          qx[lane] = qx[32 + lane];
        }
        __syncwarp();
      }
      held = max(held, 0);
    }
  };
  const int r_os = A.just_singles || nsa == 0 ? 0 : nsb;
  const int r_aa = A.just_singles ? 0 : pa_o, r_bb = A.just_singles ? 0 : pb_o;
  const int nrows = r_os + r_aa + r_bb + 2;
  for (int r = slice * kAsciWarps + (tid >> 5); r < nrows; r += A.nslice * kAsciWarps) {
    if (r < r_os) {
      // append_os_doubles_asci_contributions (determinant_contributions.hpp:226-297)
      const uint32_t sb = sgl[nsa + r], j = sb & 63, b = (sb >> 6) & 63;
      const uint64_t qb = (Pb ^ (1ull << j)) | (1ull << b);
      const double* Vb = I.V + nn * nn * (b + nn * j);
      double ebb, ebj, gbj, gjb;
      if (!COUNT) ebb = eb[b], ebj = eb[j], gbj = sg[nsa + r].x, gjb = sg[nsa + r].y;
      if (COUNT) {
        for (int x = lane; x < nsa; x += 32) {
          const uint32_t sa = sgl[x];
          hll_add(hll, (Pa ^ (1ull << (sa & 63))) | (1ull << ((sa >> 6) & 63)), qb);
        }
        continue;
      }
      gather(
          nsa,
          [&](int x) {
            const uint32_t sa = sgl[x];
            return c * ld(Vb + ((sa >> 6) & 63) + nn * (sa & 63));
          },
          [&](int x, double ch) {
            const uint32_t sa = sgl[x], i = sa & 63, a = (sa >> 6) & 63;
            add((Pa ^ (1ull << i)) | (1ull << a), qb, ((sa ^ sb) >> 12) & 1 ? -ch : ch, [&] {
              const double hdq = hdiag + ea[a] + ebb - ea[i] - ebj + V2at(I, i, j) + V2at(I, a, b) - sg[x].x -
                                 sg[x].y - gbj - gjb - V2at(I, a, j) - V2at(I, i, b);
              return A.E0 - hdq;
            });
          });
    } else if (r < r_os + r_aa + r_bb) {
      // append_ss_doubles_asci_contributions (determinant_contributions.hpp:149-210)
      const bool alpha = r < r_os + r_aa;
      const uint32_t po = alpha ? pao[r - r_os] : pbo[r - r_os - r_aa];
      const uint16_t* pv = alpha ? pav : pbv;
      const int npv = alpha ? pa_v : pb_v;
      const uint32_t i = po & 63, j = po >> 6;
      const uint64_t same = alpha ? Pa : Pb;
      const double* eps = alpha ? ea : eb;
      const uint64_t ij = (1ull << i) | (1ull << j);
      if (COUNT) {
        for (int x = lane; x < npv; x += 32) {
          const uint64_t ex = same ^ (ij | (1ull << (pv[x] & 63)) | (1ull << (pv[x] >> 6)));
          hll_add(hll, alpha ? ex : Pa, alpha ? Pb : ex);
        }
        continue;
      }
      gather(
          npv,
          [&](int x) {
            const uint32_t a = pv[x] & 63, b = pv[x] >> 6;
            return c * (Vat(I, b, j, a, i) - Vat(I, b, i, a, j));
          },
          [&](int x, double ch) {
            const uint32_t a = pv[x] & 63, b = pv[x] >> 6;
            const uint64_t fullex = ij | (1ull << a) | (1ull << b);
            const uint64_t ex = same ^ fullex;
            // doubles_sign(state_same, ex_det, full_ex): bra = P, ket = Q
            SingleEx s1 = single_ex(same, ex, fullex);
            const uint64_t f1 = (1ull << s1.o) | (1ull << s1.v);
            SingleEx s2 = single_ex(same, ex ^ f1, fullex ^ f1);
            add(alpha ? ex : Pa, alpha ? Pb : ex, s1.neg != s2.neg ? -ch : ch, [&] {
              const double hdq = hdiag + eps[a] + eps[b] - eps[i] - eps[j] + G2at(I, i, j) + G2at(I, j, i) +
                                 G2at(I, a, b) + G2at(I, b, a) - G2at(I, a, i) - G2at(I, i, a) - G2at(I, b, i) -
                                 G2at(I, i, b) - G2at(I, a, j) - G2at(I, j, a) - G2at(I, b, j) - G2at(I, j, b);
              return A.E0 - hdq;
            });
          });
    } else {
      // append_singles_asci_contributions (determinant_contributions.hpp:93-133)
      const bool alpha = r == r_os + r_aa + r_bb;
      const int x0 = alpha ? 0 : nsa, ns = alpha ? nsa : nsb;
      const uint64_t same = alpha ? Pa : Pb, other = alpha ? Pb : Pa;
      const double* eps = alpha ? ea : eb;
      for (int x = lane; x < ns; x += 32) {
        const uint32_t s1 = sgl[x0 + x], i = s1 & 63, a = (s1 >> 6) & 63;
        const uint64_t ex = (same ^ (1ull << i)) | (1ull << a);
        const uint64_t qa = alpha ? ex : Pa, qb = alpha ? Pb : ex;
        if (COUNT) {
          hll_add(hll, qa, qb);
          continue;
        }
        double h = ld(I.T + a + nn * i);
        const double* G = I.G_red + nn * (a + nn * i);
        const double* Vr = I.V_red + nn * (a + nn * i);
        for (uint64_t m = same; m; m &= m - 1) h += ld(G + low_bit(m));
        for (uint64_t m = other; m; m &= m - 1) h += ld(Vr + low_bit(m));
        if (A.keeps(c * h)) {
          if ((s1 >> 12) & 1) h = -h;
          add(qa, qb, c * h, [&] {
            const double hdq = hdiag + eps[a] - eps[i] - sg[x0 + x].x - sg[x0 + x].y;
            return A.E0 - hdq;
          });
        }
      }
    }
  }
  if (COUNT) {
    __syncthreads();
    for (int i = tid; i < kHllRegs; i += kThreads)
      if (hll[i] > __ldcg(regs + i)) atomicMax(regs + i, hll[i]);
  }
}

// The enumeration's launch shape: enough CTAs per core determinant to fill
// the chip several times over (a determinant's tables are made by each of its
// CTAs, so no more than that), and the shared memory of the largest one.
struct EnumShape {
  unsigned grid;
  size_t smem_count, smem;
};
EnumShape enum_shape(const Context* c, CoreArgs& A, const uint64_t* ca, const uint64_t* cb) {
  EnumShape e{0, 0, 0};
  int rows = 1;
  for (int64_t i = 0; i < A.ncore; ++i) {
    const int ka = __builtin_popcountll(ca[i]), kb = __builtin_popcountll(cb[i]);
    e.smem_count = std::max(e.smem_count, asci_smem(true, A.n, ka, kb, A.just_singles));
    e.smem = std::max(e.smem, asci_smem(false, A.n, ka, kb, A.just_singles));
    rows = std::max(rows, A.just_singles ? 2 : kb * (A.n - kb) + ka * (ka - 1) / 2 + kb * (kb - 1) / 2 + 2);
  }
  const int64_t fill = ((int64_t)c->sm_count * 32 + A.ncore - 1) / A.ncore;
  A.nslice = (int)std::max<int64_t>(1, std::min<int64_t>(fill, (rows + kAsciWarps - 1) / kAsciWarps));
  if (A.ncore * A.nslice > 0x7fffffff) throw Error(QDKGB_ERR_UNSUPPORTED, "ASCI: more than 2^31 core determinants");
  e.grid = (unsigned)(A.ncore * A.nslice);
  // above the default 48 KB only from about 40 electrons of each spin (their
  // diagonal's terms)
  set_max_dynamic_smem((const void*)k_asci_enum<true>, (int)e.smem_count);
  set_max_dynamic_smem((const void*)k_asci_enum<false>, (int)e.smem);
  return e;
}

// candidates: finite score with |rv| > prune; key = bit pattern of |rv|.  A
// CTA gathers the filled slots of a stretch in shared memory (half the table
// is empty) and then divides with all lanes busy; one addition to the global
// count per stretch (one per warp was a queue at that counter: 1.4 ms a search
// over up to 130 million slots, 0.83 so).
constexpr int kExtractSlots = 2048;
__global__ void __launch_bounds__(256) k_asci_extract(Table T, uint64_t cap, double prune, uint64_t* __restrict__ keys,
                                                      uint64_t* __restrict__ slots,
                                                      unsigned long long* __restrict__ count) {
  __shared__ uint16_t list[kExtractSlots];
  __shared__ uint64_t skey[kExtractSlots];
  __shared__ unsigned nlist, nkeep;
  __shared__ unsigned long long base;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  for (uint64_t i0 = (uint64_t)blockIdx.x * kExtractSlots; i0 < cap; i0 += (uint64_t)gridDim.x * kExtractSlots) {
    if (threadIdx.x == 0) nlist = nkeep = 0;
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kExtractSlots / 256; ++t) {
      const unsigned x = t * 256 + threadIdx.x;
      const bool full = i0 + x < cap && T.slot[i0 + x].key != kEmpty && !table_core(T, i0 + x);
      const unsigned m = __ballot_sync(QDKGB_FULL_MASK, full);
      unsigned p = 0;
      if (lane == 0 && m) p = atomicAdd(&nlist, (unsigned)__popc(m));
      p = __shfl_sync(QDKGB_FULL_MASK, p, 0);
      if (full) list[p + __popc(m & below)] = (uint16_t)x;
    }
    __syncthreads();
    const unsigned nl = nlist;
    unsigned mine[kExtractSlots / 256];  // position among the kept ones
#pragma unroll
    for (int t = 0; t < kExtractSlots / 256; ++t) {
      const unsigned y = t * 256 + threadIdx.x;
      mine[t] = ~0u;
      if (t * 256 >= nl) continue;
      bool take = false;
      double arv = 0.;
      if (y < nl) {
        arv = fabs(table_sum(T, i0 + list[y]) / __longlong_as_double(T.hd[i0 + list[y]]));
        take = arv > prune;
        skey[y] = (uint64_t)__double_as_longlong(arv);
      }
      const unsigned m = __ballot_sync(QDKGB_FULL_MASK, take);
      unsigned p = 0;
      if (lane == 0 && m) p = atomicAdd(&nkeep, (unsigned)__popc(m));
      p = __shfl_sync(QDKGB_FULL_MASK, p, 0);
      if (take) mine[t] = p + __popc(m & below);
    }
    __syncthreads();
    if (threadIdx.x == 0) base = nkeep ? atomicAdd(count, (unsigned long long)nkeep) : 0ull;
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kExtractSlots / 256; ++t) {
      const unsigned y = t * 256 + threadIdx.x;
      if (mine[t] == ~0u) continue;
      keys[base + mine[t]] = skey[y];
      slots[base + mine[t]] = i0 + list[y];
    }
    __syncthreads();
  }
}

// histogram (2^width bins, block-local in shared memory) of the digit at
// `shift` among keys whose higher digits equal `prefix`
constexpr int kRadixBits = 11;
__global__ void k_radix_hist(const uint64_t* __restrict__ keys, uint64_t n, int shift, int width, uint64_t prefix,
                             uint64_t hi_mask, unsigned long long* __restrict__ hist) {
  __shared__ unsigned int sh[1 << kRadixBits];
  const int nb = 1 << width;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const uint64_t dm = (uint64_t)nb - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    if ((k & hi_mask) == prefix) atomicAdd(sh + ((k >> shift) & dm), 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    if (sh[i]) atomicAdd(hist + i, (unsigned long long)sh[i]);
}

__global__ void k_asci_select(const uint64_t* __restrict__ keys, const uint64_t* __restrict__ slots, uint64_t n,
                              uint64_t kth, Table T, uint64_t* __restrict__ oa, uint64_t* __restrict__ ob,
                              unsigned long long* __restrict__ count) {
  const int lane = threadIdx.x & 31;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < n; i0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = i0 + threadIdx.x;
    const bool take = i < n && keys[i] >= kth;
    const unsigned m = __ballot_sync(QDKGB_FULL_MASK, take);
    unsigned long long base = 0;
    if (lane == 0 && m) base = atomicAdd(count, (unsigned long long)__popc(m));
    base = __shfl_sync(QDKGB_FULL_MASK, base, 0);
    if (take) {
      const unsigned long long p = base + __popc(m & ((1u << lane) - 1u));
      const u128 key = T.slot[slots[i]].key;
      oa[p] = (uint64_t)key;
      ob[p] = (uint64_t)(key >> 64);
    }
  }
}

// PT2 terms of the filled slots: sum^2 / (E0 - H_QQ) over finite sums (the
// wavefunction's own determinants carry an infinite sum), per block
__global__ void __launch_bounds__(256) k_pt2_sum(Table T, uint64_t cap, double* __restrict__ partial,
                                                 unsigned long long* __restrict__ count) {
  __shared__ double rs[8];
  __shared__ unsigned long long rc[8];
  double s = 0.;
  unsigned long long m = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (uint64_t)gridDim.x * blockDim.x) {
    if (T.slot[i].key != kEmpty && !table_core(T, i)) {
      const double v = table_sum(T, i);
      s += v * v / __longlong_as_double(T.hd[i]);
      ++m;
    }
  }
  s = warp_sum(s);
  for (int d = 16; d > 0; d >>= 1) m += __shfl_xor_sync(QDKGB_FULL_MASK, m, d);
  if ((threadIdx.x & 31) == 0) {
    rs[threadIdx.x >> 5] = s;
    rc[threadIdx.x >> 5] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.;
    unsigned long long u = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      t += rs[w];
      u += rc[w];
    }
    partial[blockIdx.x] = t;
    count[blockIdx.x] = u;
  }
}

__global__ void k_fill_empty(Table T, uint64_t cap) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (uint64_t)gridDim.x * blockDim.x) {
    T.slot[i] = Slot{kEmpty, 0, 0};
    T.hd[i] = kHdEmpty;
  }
}

int64_t binom64(int n, int k) {
  if (k < 0 || k > n) return 0;
  long double r = 1;
  for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
  return (int64_t)std::llround(r);
}

// Slots per estimated distinct target: the table is at most half full, two to
// three probes (in one or two 128-byte lines) for a new target.  Rounded up
// to a power of two from 2.5, as it was, a search allocated, filled and read
// up to 2.5 times as many.
constexpr double kSlotsPerTarget = 2.;

// HyperLogLog estimate of the distinct targets of an enumeration over the
// core list already on the device in A (small-range correction by linear
// counting); `regs` is kHllRegs device words of scratch
double distinct_targets(Context* c, const CoreArgs& A, const EnumShape& es, unsigned* regs) {
  QDKGB_CUDA(cudaMemsetAsync(regs, 0, kHllRegs * sizeof(unsigned), c->stream));
  k_asci_enum<true><<<es.grid, kAsciWarps * 32, es.smem_count, c->stream>>>(A, regs);
  QDKGB_CHECK_LAUNCH();
  std::vector<unsigned> h(kHllRegs);
  QDKGB_CUDA(cudaMemcpyAsync(h.data(), regs, kHllRegs * sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream));
  QDKGB_CUDA(cudaStreamSynchronize(c->stream));
  const double m = kHllRegs;
  double z = 0.;
  int zeros = 0;
  for (unsigned r : h) {
    z += std::ldexp(1., -(int)r);
    zeros += r == 0;
  }
  double e = 0.7213 / (1. + 1.079 / m) * m * m / z;
  if (e <= 2.5 * m && zeros > 0) e = m * std::log(m / zeros);
  return e;
}

}  // namespace

// Returns the new determinant list (top-k candidates followed by the core).
void asci_search_gpu(Context* c, int64_t ncore, const uint64_t* ca, const uint64_t* cb, const double* cc, double E0,
                     int64_t ndets_max, double h_el_tol, double rv_prune_tol, std::vector<uint64_t>& out_a,
                     std::vector<uint64_t>& out_b, int64_t* n_candidates, bool just_singles) {
  NvtxRange nvtx_range("qdkgb.asci_search");
  if (!c->have_ints) throw Error(QDKGB_ERR_STATE, "integrals not set");
  if (ncore <= 0) throw Error(QDKGB_ERR_INVALID, "empty core");
  const int n = c->norb;
  {
    uint64_t u = 0;
    for (int64_t i = 0; i < ncore; ++i) u |= ca[i] | cb[i];
    if (n < 64 && (u >> n)) throw Error(QDKGB_ERR_INVALID, "a determinant occupies an orbital beyond the integrals' norb");
  }
  // table capacity from the number of contributions (a bound on distinct targets)
  int64_t total = ncore;
  for (int64_t i = 0; i < ncore; ++i) {
    const int ka = __builtin_popcountll(ca[i]), kb = __builtin_popcountll(cb[i]);
    const int64_t sa = (int64_t)ka * (n - ka), sb = (int64_t)kb * (n - kb);
    total += sa + sb + sa * sb + binom64(ka, 2) * binom64(n - ka, 2) + binom64(kb, 2) * binom64(n - kb, 2);
  }
  ScopedBuffers<10> scratch(c);
  DeviceBuffer &bslot = scratch.b[0], &bhll = scratch.b[1], &bhd = scratch.b[2], &bck = scratch.b[3],
               &bcs = scratch.b[4], &bcnt = scratch.b[5], &berr = scratch.b[6], &bcore = scratch.b[7],
               &bout = scratch.b[8], &bhist = scratch.b[9];
  uint64_t* dcore = dev_array<uint64_t>(c, bcore, 3 * ncore);
  QDKGB_CUDA(cudaMemcpyAsync(dcore, ca, ncore * 8, cudaMemcpyHostToDevice, c->stream));
  QDKGB_CUDA(cudaMemcpyAsync(dcore + ncore, cb, ncore * 8, cudaMemcpyHostToDevice, c->stream));
  QDKGB_CUDA(cudaMemcpyAsync(dcore + 2 * ncore, cc, ncore * 8, cudaMemcpyHostToDevice, c->stream));
  int* err = dev_array<int>(c, berr, 1);
  unsigned long long* cnt = dev_array<unsigned long long>(c, bcnt, 2);
  QDKGB_CUDA(cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned long long), c->stream));
  CoreArgs A;
  A.I = integrals_view(c);
  A.n = n;
  A.ncore = ncore;
  A.ca = dcore;
  A.cb = dcore + ncore;
  A.cc = (const double*)(dcore + 2 * ncore);
  A.E0 = E0;
  A.h_el_tol = h_el_tol;
  A.just_singles = just_singles;
  // table: kSlotsPerTarget x the estimated distinct targets (at most 1.5 x the
  // contributions); an overflowing enumeration is redone with twice the slots
  const EnumShape es = enum_shape(c, A, ca, cb);
  const double est = distinct_targets(c, A, es, dev_array<unsigned>(c, bhll, kHllRegs));
  uint64_t cap = (uint64_t)(std::min((double)(total + total / 2), kSlotsPerTarget * est + 2. * (double)ncore) + 1024.);
  size_t freeb = 0, totb = 0;
  QDKGB_CUDA(cudaMemGetInfo(&freeb, &totb));
  const size_t slot_bytes = 16 + 16 + 8 + 16;  // key, fixed-point sum, hd, candidate key + slot
  if (cap * slot_bytes > freeb / 2) throw Error(QDKGB_ERR_OOM, "ASCI search: hash table does not fit in device memory");
  for (;;) {
    A.T = Table{dev_array<Slot>(c, bslot, cap), dev_array<long long>(c, bhd, cap), cap, err};
    const unsigned fb = (unsigned)std::min<uint64_t>((cap + 255) / 256, (uint64_t)c->sm_count * 64);
    QDKGB_CUDA(cudaMemsetAsync(err, 0, sizeof(int), c->stream));
    k_fill_empty<<<fb, 256, 0, c->stream>>>(A.T, cap);
    QDKGB_CHECK_LAUNCH();
    k_asci_enum<false><<<es.grid, kAsciWarps * 32, es.smem, c->stream>>>(A, nullptr);
    QDKGB_CHECK_LAUNCH();
    int herr = 0;
    QDKGB_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    QDKGB_CUDA(cudaStreamSynchronize(c->stream));
    if (herr == 2) throw Error(QDKGB_ERR_UNSUPPORTED, "ASCI: a contribution |c H| >= 2^20 is outside the accumulator range");
    if (!herr) break;
    if ((cap << 1) * slot_bytes > freeb / 2) throw Error(QDKGB_ERR_OOM, "ASCI search: hash table overflow");
    cap <<= 1;
  }
  const unsigned fb = (unsigned)std::min<uint64_t>((cap + 255) / 256, (uint64_t)c->sm_count * 64);
  uint64_t* ckeys = dev_array<uint64_t>(c, bck, cap);
  uint64_t* cslots = dev_array<uint64_t>(c, bcs, cap);
  k_asci_extract<<<(unsigned)std::min<uint64_t>((cap + kExtractSlots - 1) / kExtractSlots, (uint64_t)c->sm_count * 32), 256, 0,
                   c->stream>>>(A.T, cap, rv_prune_tol, ckeys, cslots, cnt);
  QDKGB_CHECK_LAUNCH();
  int herr = 0;
  unsigned long long ncand = 0;
  QDKGB_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  QDKGB_CUDA(cudaMemcpyAsync(&ncand, cnt, sizeof(ncand), cudaMemcpyDeviceToHost, c->stream));
  QDKGB_CUDA(cudaStreamSynchronize(c->stream));
  if (herr == 2) throw Error(QDKGB_ERR_UNSUPPORTED, "ASCI: a contribution |c H| >= 2^20 is outside the accumulator range");
  if (herr) throw Error(QDKGB_ERR_OOM, "ASCI search: hash table overflow");
  if (n_candidates) *n_candidates = (int64_t)ncand;
  const int64_t topk = ndets_max - ncore;
  uint64_t kth = 0;  // keep everything
  if (topk <= 0) {
    kth = ~0ull;  // keep nothing but the core
  } else if ((int64_t)ncand > topk) {
    // radix select of the topk-th largest key, digits from the top
    unsigned long long* hist = dev_array<unsigned long long>(c, bhist, 1 << kRadixBits);
    uint64_t prefix = 0, hi_mask = 0;
    int64_t k = topk;
    std::vector<unsigned long long> h(1 << kRadixBits);
    const unsigned hb = (unsigned)std::min<uint64_t>((ncand + 255) / 256, (uint64_t)c->sm_count * 32);
    for (int top = 64; top > 0;) {
      const int width = std::min(kRadixBits, top);
      const int shift = top - width;
      const int nb = 1 << width;
      QDKGB_CUDA(cudaMemsetAsync(hist, 0, nb * 8, c->stream));
      k_radix_hist<<<hb, 256, 0, c->stream>>>(ckeys, ncand, shift, width, prefix, hi_mask, hist);
      QDKGB_CHECK_LAUNCH();
      QDKGB_CUDA(cudaMemcpyAsync(h.data(), hist, nb * 8, cudaMemcpyDeviceToHost, c->stream));
      QDKGB_CUDA(cudaStreamSynchronize(c->stream));
      int64_t acc = 0;
      int d = nb - 1;
      for (; d >= 0; --d) {
        if (acc + (int64_t)h[d] >= k) break;
        acc += (int64_t)h[d];
      }
      if (d < 0) d = 0;
      k -= acc;
      prefix |= (uint64_t)d << shift;
      hi_mask |= ((uint64_t)nb - 1) << shift;
      top = shift;
    }
    kth = prefix;
  }
  uint64_t* dout = dev_array<uint64_t>(c, bout, 2 * std::max<uint64_t>(ncand, 1));
  QDKGB_CUDA(cudaMemsetAsync(cnt + 1, 0, sizeof(unsigned long long), c->stream));
  unsigned long long nsel = 0;
  if (ncand > 0 && kth != ~0ull) {
    const unsigned sb = (unsigned)std::min<uint64_t>((ncand + 255) / 256, (uint64_t)c->sm_count * 32);
    k_asci_select<<<sb, 256, 0, c->stream>>>(ckeys, cslots, ncand, kth, A.T, dout, dout + ncand, cnt + 1);
    QDKGB_CHECK_LAUNCH();
    QDKGB_CUDA(cudaMemcpyAsync(&nsel, cnt + 1, sizeof(nsel), cudaMemcpyDeviceToHost, c->stream));
    QDKGB_CUDA(cudaStreamSynchronize(c->stream));
  }
  out_a.resize(nsel + ncore);
  out_b.resize(nsel + ncore);
  if (nsel) {
    QDKGB_CUDA(cudaMemcpyAsync(out_a.data(), dout, nsel * 8, cudaMemcpyDeviceToHost, c->stream));
    QDKGB_CUDA(cudaMemcpyAsync(out_b.data(), dout + ncand, nsel * 8, cudaMemcpyDeviceToHost, c->stream));
  }
  QDKGB_CUDA(cudaStreamSynchronize(c->stream));
  std::copy(ca, ca + ncore, out_a.begin() + nsel);
  std::copy(cb, cb + ncore, out_b.begin() + nsel);
}

// asci_pt2_constraint (include/macis/asci/pt2.hpp:59-565) on the device:
// E_PT2 = sum over the determinants Q outside the wavefunction of
// (sum_P c_P <Q|H|P>)^2 / (E0 - H_QQ), single contributions with
// |c_P <Q|H|P>| < pt2_tol dropped (determinant_contributions.hpp:49-55,
// mask_constraints.hpp:400-670).  The enumeration of the search runs over the
// whole wavefunction (each determinant inserted with an infinite score, so
// that it drops out), into the hash table; the reference's constraint split
// (there for MPI / OpenMP balance and memory) becomes a split of the target
// space by a hash into passes when the table for every contribution would
// not fit in half of the free device memory.  Every Q lies in one part of
// either split, so the sums are the same.
double asci_pt2_gpu(Context* c, int64_t nd, const uint64_t* a, const uint64_t* b, const double* C, double E0,
                    double pt2_tol, int64_t max_slots, int64_t* npt2) {
  NvtxRange nvtx_range("qdkgb.asci_pt2");
  if (!c->have_ints) throw Error(QDKGB_ERR_STATE, "integrals not set");
  if (nd <= 0) throw Error(QDKGB_ERR_INVALID, "empty wavefunction");
  for (int64_t i = 1; i < nd; ++i)
    if (a[i] < a[i - 1] || (a[i] == a[i - 1] && b[i] < b[i - 1]))
      throw Error(QDKGB_ERR_INVALID, "PT2 Only Works with Sorted Wfns");
  const int n = c->norb;
  {
    uint64_t u = 0;
    for (int64_t i = 0; i < nd; ++i) u |= a[i] | b[i];
    if (n < 64 && (u >> n)) throw Error(QDKGB_ERR_INVALID, "a determinant occupies an orbital beyond the integrals' norb");
  }
  int64_t total = nd;
  for (int64_t i = 0; i < nd; ++i) {
    const int ka = __builtin_popcountll(a[i]), kb = __builtin_popcountll(b[i]);
    const int64_t sa = (int64_t)ka * (n - ka), sb = (int64_t)kb * (n - kb);
    total += sa + sb + sa * sb + binom64(ka, 2) * binom64(n - ka, 2) + binom64(kb, 2) * binom64(n - kb, 2);
  }
  ScopedBuffers<6> scratch(c);
  DeviceBuffer &bslot = scratch.b[0], &bhll = scratch.b[1], &bhd = scratch.b[2], &berr = scratch.b[3],
               &bcore = scratch.b[4], &bpart = scratch.b[5];
  uint64_t* dcore = dev_array<uint64_t>(c, bcore, 3 * nd);
  QDKGB_CUDA(cudaMemcpyAsync(dcore, a, nd * 8, cudaMemcpyHostToDevice, c->stream));
  QDKGB_CUDA(cudaMemcpyAsync(dcore + nd, b, nd * 8, cudaMemcpyHostToDevice, c->stream));
  QDKGB_CUDA(cudaMemcpyAsync(dcore + 2 * nd, C, nd * 8, cudaMemcpyHostToDevice, c->stream));
  int* err = dev_array<int>(c, berr, 1);
  CoreArgs A;
  A.I = integrals_view(c);
  A.n = n;
  A.ncore = nd;
  A.ca = dcore;
  A.cb = dcore + nd;
  A.cc = (const double*)(dcore + 2 * nd);
  A.E0 = E0;
  A.h_el_tol = pt2_tol;
  // table: kSlotsPerTarget x the estimated distinct targets (at most 1.5 x the
  // contributions), split into passes when it exceeds half the free memory or
  // max_slots; a pass whose probing overflows is redone with twice the slots
  const EnumShape es = enum_shape(c, A, a, b);
  const double est = distinct_targets(c, A, es, dev_array<unsigned>(c, bhll, kHllRegs));
  const uint64_t need =
      (uint64_t)(std::min((double)(total + total / 2), kSlotsPerTarget * est + 2. * (double)nd) + 1024.);
  size_t freeb = 0, totb = 0;
  QDKGB_CUDA(cudaMemGetInfo(&freeb, &totb));
  const size_t slot_bytes = 16 + 16 + 8;  // key, fixed-point sum, E0 - H_QQ
  const size_t budget = freeb / 2;
  const uint64_t slot_max = max_slots > 0 ? std::max<uint64_t>((uint64_t)max_slots, 1024) : ~0ull;
  auto fits = [&](uint64_t cp) { return cp * slot_bytes <= budget && cp <= slot_max; };
  uint64_t cap = need;
  if (!fits(need))
    for (cap = 1024; cap < need && fits(cap << 1);) cap <<= 1;
  const uint64_t npass = std::max<uint64_t>(1, (need + cap - 1) / cap);
  if (npass > 0xffffffffull) throw Error(QDKGB_ERR_OOM, "ASCI PT2: too many passes for the device memory");
  A.npass = (uint32_t)npass;
  const unsigned sb = (unsigned)std::min<uint64_t>((need + 255) / 256, (uint64_t)c->sm_count * 8);
  double* partial = (double*)dev_alloc(c, bpart, (size_t)sb * 16 + 64);
  unsigned long long* pcount = (unsigned long long*)(partial + sb);
  std::vector<double> hp(sb);
  std::vector<unsigned long long> hc(sb);
  double ept2 = 0.;
  int64_t count = 0;
  for (uint64_t pass = 0; pass < npass; ++pass) {
    A.pass = (uint32_t)pass;
    for (;;) {
      A.T = Table{dev_array<Slot>(c, bslot, cap), dev_array<long long>(c, bhd, cap), cap, err};
      const unsigned fb = (unsigned)std::min<uint64_t>((cap + 255) / 256, (uint64_t)c->sm_count * 64);
      QDKGB_CUDA(cudaMemsetAsync(err, 0, sizeof(int), c->stream));
      k_fill_empty<<<fb, 256, 0, c->stream>>>(A.T, cap);
      QDKGB_CHECK_LAUNCH();
      k_asci_enum<false><<<es.grid, kAsciWarps * 32, es.smem, c->stream>>>(A, nullptr);
      QDKGB_CHECK_LAUNCH();
      k_pt2_sum<<<sb, 256, 0, c->stream>>>(A.T, cap, partial, pcount);
      QDKGB_CHECK_LAUNCH();
      int herr = 0;
      QDKGB_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
      QDKGB_CUDA(cudaMemcpyAsync(hp.data(), partial, sb * 8, cudaMemcpyDeviceToHost, c->stream));
      QDKGB_CUDA(cudaMemcpyAsync(hc.data(), pcount, sb * 8, cudaMemcpyDeviceToHost, c->stream));
      QDKGB_CUDA(cudaStreamSynchronize(c->stream));
      if (herr == 2) throw Error(QDKGB_ERR_UNSUPPORTED, "ASCI: a contribution |c H| >= 2^20 is outside the accumulator range");
    if (!herr) break;
      if (!fits(cap << 1)) throw Error(QDKGB_ERR_OOM, "ASCI PT2: hash table overflow");
      cap <<= 1;
    }
    for (unsigned i = 0; i < sb; ++i) {
      ept2 += hp[i];
      count += (int64_t)hc[i];
    }
  }
  if (npt2) *npt2 = count;
  return ept2;
}

}  // namespace qdkgb

// ---------------------------------------------------------------- drivers
namespace qdkgb {

namespace {

struct HDet {
  uint64_t a, b;
};
inline bool hspin_less(const HDet& x, const HDet& y) { return x.a != y.a ? x.a < y.a : x.b < y.b; }
inline bool hdet_eq(const HDet& x, const HDet& y) { return x.a == y.a && x.b == y.b; }



// Wall time of the ASCI phases (synchronised: each phase ends in a host
// sync anyway), accumulated into Context::asci_phase_s.
struct PhaseClock {
  Context* c;
  std::chrono::steady_clock::time_point t;
  explicit PhaseClock(Context* ctx) : c(ctx) {
    QDKGB_CUDA(cudaStreamSynchronize(c->stream));
    t = std::chrono::steady_clock::now();
  }
  void lap(int phase) {
    QDKGB_CUDA(cudaStreamSynchronize(c->stream));
    const auto now = std::chrono::steady_clock::now();
    c->asci_phase_s[phase] += std::chrono::duration<double>(now - t).count();
    t = now;
  }
};

// The list the context's FP64 CSR was last built for, so that the next
// iteration patches that matrix instead of rebuilding it (asci_iter's
// incremental build, include/macis/solvers/incremental_h_build.hpp:38-356).
struct HPatchCache {
  std::vector<uint64_t> a, b;
  double thresh = 0.;
  bool valid = false;
};

bool patch_disabled() {
  const char* e = std::getenv("QDKGB_ASCI_FULL_BUILD");
  return e && e[0] && e[0] != '0';
}

// selected_ci_diag (selected_ci_diag.hpp:111-158) on the device for a list
// sorted by spin_comparator; X is the guess (empty: diagonal guess) and the
// eigenvector on return.  With a cache holding the previous list, the FP64
// CSR is patched from the previous one (bit-identical to a rebuild).
double sci_diag_gpu(Context* c, const qdkgb_asci_settings& S, const qdkgb_davidson_settings& ci, double matel_tol,
                    const std::vector<HDet>& dets, std::vector<double>& X, HPatchCache* cache) {
  const int64_t n = (int64_t)dets.size();
  std::vector<uint64_t> a(n), b(n);
  for (int64_t i = 0; i < n; ++i) {
    a[i] = dets[i].a;
    b[i] = dets[i].b;
  }
  const bool mixed = ci.precision == QDKGB_PREC_MIXED;
  // the previous CSR leaves the context before the determinant space is reset
  ScopedBuffers<3> old(c);
  const bool have_old = cache && cache->valid && !mixed && !patch_disabled() && c->H.valid && !c->op_direct &&
                        !c->H.structured && c->H.storage == QDKGB_H_FP64 && c->H.thresh == matel_tol &&
                        c->H.n == (int64_t)cache->a.size() && cache->thresh == matel_tol;
  if (have_old) {
    std::swap(old.b[0], c->H.rowptr);
    std::swap(old.b[1], c->H.colind);
    std::swap(old.b[2], c->H.val);
  }
  if (cache) cache->valid = false;
  PhaseClock clock(c);
  build_det_space(c, n, a.data(), b.data());
  clock.lap(1);
  bool patched = false;
  if (have_old && !c->fci)
    patched = build_hamiltonian_patched(c, matel_tol, cache->a, cache->b, old.b[0], old.b[1], old.b[2],
                                        S.min_patch_overlap);
  for (DeviceBuffer& x : old.b) dev_free(c, x);
  if (patched)
    ++c->asci_patches;
  else
    build_hamiltonian(c, matel_tol, mixed ? QDKGB_H_SPLIT32 : QDKGB_H_FP64);
  clock.lap(2);
  if (cache && !mixed) {
    cache->a.swap(a);
    cache->b.swap(b);
    cache->thresh = matel_tol;
    cache->valid = true;
  }
  qdkgb_davidson_settings s = ci;
  s.nroots = 1;  // the ASCI iterations solve for the lowest root, as the reference's do
  s.use_guess = X.empty() ? 0 : 1;
  X.resize(n, 0.);
  if (!s.use_guess) std::fill(X.begin(), X.end(), 0.);
  double E = 0.;
  davidson(c, &s, &E, X.data(), nullptr, true);
  clock.lap(3);
  return E;
}

// asci_iter (include/macis/asci/iteration.hpp:50-226)
double asci_iter_gpu(Context* c, const qdkgb_asci_settings& S, const qdkgb_davidson_settings& ci, double matel_tol,
                     int64_t ndets_max, double E0, std::vector<HDet>& wfn, std::vector<double>& X, int64_t* ncand,
                     HPatchCache* cache) {
  NvtxRange nvtx_range("qdkgb.asci_iter");
  ++c->asci_iters;
  // the list and vector in spin order, for the warm start's merge scan (the
  // list arrives in that order from the previous iteration)
  std::vector<HDet> sorted_wfn;
  std::vector<double> sorted_X;
  if (S.warm_start) {
    if (std::is_sorted(wfn.begin(), wfn.end(), hspin_less)) {
      sorted_wfn = wfn;
      sorted_X = X;
    } else {
      struct DC {
        HDet d;
        double c;
      };
      std::vector<DC> v(wfn.size());
      for (size_t i = 0; i < v.size(); ++i) v[i] = {wfn[i], X[i]};
      parallel_sort(v, [](const DC& x, const DC& y) { return hspin_less(x.d, y.d); });
      sorted_wfn.resize(v.size());
      sorted_X.resize(v.size());
      for (size_t i = 0; i < v.size(); ++i) {
        sorted_wfn[i] = v[i].d;
        sorted_X[i] = v[i].c;
      }
    }
  }
  if (wfn.size() > 1) {
    // reorder_ci_on_coeff (determinant_sort.hpp:45-64): std::sort of the
    // indices by |C| descending.  The (|C|, index) pairs go through the same
    // std::sort with the same comparisons, so ties come out in the
    // reference's order; the pairs sit together in memory.
    struct KI {
      double k;
      size_t i;
    };
    std::vector<KI> idx(wfn.size());
    for (size_t i = 0; i < idx.size(); ++i) idx[i] = {std::fabs(X[i]), i};
    std::sort(idx.begin(), idx.end(), [](const KI& x, const KI& y) { return x.k > y.k; });
    std::vector<HDet> w2(wfn.size());
    std::vector<double> x2(wfn.size());
    for (size_t i = 0; i < idx.size(); ++i) {
      w2[i] = wfn[idx[i].i];
      x2[i] = X[idx[i].i];
    }
    wfn.swap(w2);
    X.swap(x2);
  }
  size_t nkeep = 0;
  if (S.core_selection_fixed) {
    nkeep = std::min<size_t>((size_t)S.ncdets_max, wfn.size());
  } else {
    if (!(S.core_selection_threshold >= 2.220446049250313e-16 && S.core_selection_threshold <= 1.0))
      throw Error(QDKGB_ERR_INVALID, "core_selection_threshold must be in [epsilon, 1.0]");
    double w = 0.;
    for (size_t i = 0; i < wfn.size(); ++i) {
      w += X[i] * X[i];
      nkeep++;
      if (w >= S.core_selection_threshold) break;
    }
  }
  if (wfn.size() > 1) {  // reorder_ci_on_alpha of the core (determinant_sort.hpp:66-90)
    std::vector<size_t> idx(nkeep);
    for (size_t i = 0; i < nkeep; ++i) idx[i] = i;
    std::sort(idx.begin(), idx.end(), [&](size_t i, size_t j) { return hspin_less(wfn[i], wfn[j]); });
    std::vector<HDet> w2(nkeep);
    std::vector<double> x2(nkeep);
    for (size_t i = 0; i < nkeep; ++i) {
      w2[i] = wfn[idx[i]];
      x2[i] = X[idx[i]];
    }
    std::copy(w2.begin(), w2.end(), wfn.begin());
    std::copy(x2.begin(), x2.end(), X.begin());
  }
  std::vector<uint64_t> ca(nkeep), cb(nkeep);
  for (size_t i = 0; i < nkeep; ++i) {
    ca[i] = wfn[i].a;
    cb[i] = wfn[i].b;
  }
  std::vector<uint64_t> na, nb;
  {
    PhaseClock clock(c);
    asci_search_gpu(c, (int64_t)nkeep, ca.data(), cb.data(), X.data(), E0, ndets_max, S.h_el_tol, S.rv_prune_tol,
                    na, nb, ncand, S.just_singles != 0);
    clock.lap(0);
  }
  wfn.resize(na.size());
  for (size_t i = 0; i < na.size(); ++i) wfn[i] = {na[i], nb[i]};
  parallel_sort(wfn, hspin_less);
  std::vector<double> Xl;
  if (S.warm_start) {
    Xl.assign(wfn.size(), 0.);
    for (size_t i = 0, k = 0; i < wfn.size() && k < sorted_wfn.size();) {
      if (hspin_less(sorted_wfn[k], wfn[i])) {
        ++k;
      } else if (hspin_less(wfn[i], sorted_wfn[k])) {
        ++i;
      } else {
        Xl[i++] = sorted_X[k++];
      }
    }
    double nrm = 0.;
    for (double x : Xl) nrm += x * x;
    nrm = std::sqrt(nrm);
    if (nrm < std::max(S.min_warm_start_overlap, 2.220446049250313e-16))
      Xl.clear();
    else
      for (double& x : Xl) x /= nrm;
  }
  const double E = sci_diag_gpu(c, S, ci, matel_tol, wfn, Xl, cache);
  X = Xl;
  return E;
}

}  // namespace

void asci_run(Context* c, const qdkgb_asci_settings& S, const qdkgb_davidson_settings& ci, double matel_tol,
              std::vector<uint64_t>& a, std::vector<uint64_t>& b, std::vector<double>& X, double& E0, bool grow,
              bool refine, double* E_grow) {
  // the growth settings as get_asci_settings_ checks them
  // (cpp/src/qdk/chemistry/algorithms/microsoft/macis_base.cpp:101-124)
  if (!(S.grow_factor > 1.0)) throw Error(QDKGB_ERR_INVALID, "grow_factor must be > 1.0");
  if (!(S.min_grow_factor > 1.0)) throw Error(QDKGB_ERR_INVALID, "min_grow_factor must be > 1.0");
  if (S.min_grow_factor > S.grow_factor) throw Error(QDKGB_ERR_INVALID, "min_grow_factor must be <= grow_factor");
  if (!(S.growth_backoff_rate > 0.0 && S.growth_backoff_rate < 1.0))
    throw Error(QDKGB_ERR_INVALID, "growth_backoff_rate must be in (0, 1)");
  if (!(S.growth_recovery_rate > 1.0)) throw Error(QDKGB_ERR_INVALID, "growth_recovery_rate must be > 1.0");
  for (double& t : c->asci_phase_s) t = 0.;
  c->asci_iters = 0;
  c->asci_patches = 0;
  c->asci_rot.clear();
  HPatchCache cache;
  std::vector<HDet> wfn(a.size());
  for (size_t i = 0; i < a.size(); ++i) wfn[i] = {a[i], b[i]};
  int64_t ncand = 0;
  if (grow) {
    // asci_grow (include/macis/asci/grow.hpp:45-268), without rotations
    size_t prev = wfn.size();
    double gf = S.grow_factor;
    while ((int64_t)wfn.size() < S.ntdets_max) {
      // taper (grow.hpp:97-107): a step that would pass ntdets_max at the
      // current factor uses max(min_grow_factor, taper_grow_factor) instead
      double eff = gf;
      if (S.taper_grow_factor > 0. && (int64_t)std::ceil((double)wfn.size() * gf) > S.ntdets_max)
        eff = std::max(S.min_grow_factor, S.taper_grow_factor);
      int64_t nnew = std::min<int64_t>(
          std::max<int64_t>(S.ntdets_min, (int64_t)std::ceil((double)wfn.size() * eff)), S.ntdets_max);
      if (nnew <= (int64_t)wfn.size()) {
        nnew = std::min<int64_t>((int64_t)wfn.size() + 1, S.ntdets_max);
        if (nnew <= (int64_t)wfn.size()) break;
      }
      const double E = asci_iter_gpu(c, S, ci, matel_tol, nnew, E0, wfn, X, &ncand, &cache);
      if ((int64_t)wfn.size() < nnew) {
        gf = std::max(S.min_grow_factor, gf * S.growth_backoff_rate);
        if (wfn.size() <= prev) break;
      } else {
        gf = std::min(S.grow_factor, gf * S.growth_recovery_rate);
      }
      prev = wfn.size();
      if (S.grow_with_rot && (int64_t)wfn.size() >= S.rot_size_start) {
        // natural-orbital rotation (grow.hpp:163-252): the spin-summed 1-RDM
        // of the current wavefunction (the context holds its list), its
        // natural orbitals, the integrals rotated to them, and the list
        // rediagonalised from the diagonal guess in the new orbitals (the
        // iteration's energy is kept, as the reference keeps it)
        const int n = c->norb;
        std::vector<double> aa((size_t)n * n, 0.), bb((size_t)n * n, 0.), ordm((size_t)n * n), U;
        rdms_spin_dep(c, X.data(), aa.data(), bb.data(), nullptr, nullptr, nullptr);
        for (size_t i = 0; i < ordm.size(); ++i) ordm[i] = aa[i] + bb[i];
        natural_orbitals(n, ordm, U);
        rotate_integrals(c, U);
        if (c->asci_rot.empty()) {
          c->asci_rot = U;
        } else {
          std::vector<double> R((size_t)n * n, 0.);
          for (int j = 0; j < n; ++j)
            for (int k = 0; k < n; ++k) {
              const double u = U[k + (size_t)n * j];
              for (int i = 0; i < n; ++i) R[i + (size_t)n * j] += c->asci_rot[i + (size_t)n * k] * u;
            }
          c->asci_rot.swap(R);
        }
        cache.valid = false;  // the integrals changed
        std::vector<double> Xr;
        sci_diag_gpu(c, S, ci, matel_tol, wfn, Xr, nullptr);
        X.swap(Xr);
      }
      E0 = E;
    }
  }
  if (E_grow) *E_grow = E0;
  if (refine) {
    // asci_refine (include/macis/asci/refine.hpp:44-237)
    int64_t ndets = (int64_t)wfn.size();
    bool converged = false;
    double prev_dE = 0.;
    int osc = 0;
    int64_t max_iter = S.max_refine_iter, ext = 0;
    std::vector<HDet> prev_wfn;
    for (int64_t iter = 0; iter < max_iter; ++iter) {
      const double E = asci_iter_gpu(c, S, ci, matel_tol, ndets, E0, wfn, X, &ncand, &cache);
      if ((int64_t)wfn.size() != ndets) {
        ndets = (int64_t)wfn.size();
        if (ndets < S.ntdets_min) break;
      }
      const double dE = E - E0;
      if (std::fabs(dE) < S.refine_energy_tol) {
        E0 = E;
        converged = true;
        break;
      }
      if (iter > 0 && prev_dE * dE < 0 && std::fabs(prev_dE + dE) < S.refine_energy_tol) {
        osc++;
        if (osc >= 2 && !prev_wfn.empty()) {
          std::vector<HDet> uni;
          std::set_union(prev_wfn.begin(), prev_wfn.end(), wfn.begin(), wfn.end(), std::back_inserter(uni),
                         hspin_less);
          std::vector<double> Xu(uni.size(), 0.);
          for (size_t i = 0; i < wfn.size(); ++i) {
            auto it = std::lower_bound(uni.begin(), uni.end(), wfn[i], hspin_less);
            if (it != uni.end() && hdet_eq(*it, wfn[i])) Xu[it - uni.begin()] = X[i];
          }
          const double Eu = sci_diag_gpu(c, S, ci, matel_tol, uni, Xu, &cache);
          const int64_t e = std::min<int64_t>(osc, S.max_refine_iter - ext);
          if (e > 0) {
            max_iter += e;
            ext += e;
          }
          wfn = uni;
          X = Xu;
          ndets = (int64_t)wfn.size();
          E0 = Eu;
          prev_wfn.clear();
          osc = 0;
          prev_dE = 0.;
          continue;
        }
      } else {
        osc = 0;
      }
      prev_dE = dE;
      prev_wfn = wfn;
      E0 = E;
    }
    if (!converged) throw Error(QDKGB_ERR_NOT_CONVERGED, "ASCI Refine did not converge");
  }
  a.resize(wfn.size());
  b.resize(wfn.size());
  for (size_t i = 0; i < wfn.size(); ++i) {
    a[i] = wfn[i].a;
    b[i] = wfn[i].b;
  }
}

}  // namespace qdkgb
