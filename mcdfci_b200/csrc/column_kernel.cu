// Column kernel: Hamiltonian column generation fused with the hash-table
// z-update; G CTAs per picked determinant.
//
// Replaces, per iteration, HamiltonianMolecule::get_column (src/hamiltonian.h:
// 412-424, called at src/solver.h:717-739) and stage 1 of
// WaveFunctionCuckoo::update_z_and_get_sub (src/wavefunction.h:468-552): for
// every connected determinant D' of column c (value H = <D'|H|D_c>):
//
//   dz = H * dx_c
//   if |dz * scale| > z_threshold: upsert z[D'] += dz   (insert {x=0, z=dz} if absent)
//   else:                          z[D'] += dz only if D' is present
//   new_z_c += H * x[D'];  dot += dz * x[D']
//   candidate score |x[D'] * xss + z[D']| (value right after this update)
//
// and keeps, per column, the `estimate` (m) candidates with the largest score,
// as the reference's per-thread priority queue does (src/wavefunction.h:544-551).
//
// Work decomposition.  The connected determinants of any determinant in a
// fixed (n_alpha, n_beta) sector form the same index space, so entry e of a
// column is decoded arithmetically from the occupied/virtual orbital lists:
//   e = 0                       diagonal
//   [off1, off2)  alpha singles  (i occ, a vir)
//   [off2, off3)  beta singles
//   [off3, off4)  alpha-alpha doubles  (occupied pair, virtual pair)
//   [off4, off5)  beta-beta doubles
//   [off5, total) alpha-beta doubles   (ia, ib, aa, ab), ab fastest so that
//                 consecutive threads read consecutive integral-table entries
// CTA g of the column's G CTAs takes the g-th contiguous slice, in blocks of
// kRounds entries per thread.
//
// What bounds it.  Every entry touches one pseudo-random slot of a table far
// larger than L2.  Measured on 524,288 random slots of a 17 GB table: one
// 32-byte load each 15 us, an atomic add that returns the old z after it 17 us,
// but 65 us when x is loaded from the sector while its atomic is in flight
// (33 us without the load).  So a probe reads key and x in one load, and the
// add comes later with no load beside it.  Per launch, before (a 16-byte key
// load, then x and the atomic together; sorted warp lists) and after: 24
// orbitals 6a5b, k = 32, m = 64: 70.8 us and 46.1 us; 42 orbitals 24a23b,
// k = 64, m = 128: 1,757 us and 1,272 us; 12 orbitals 6a6b, k = 1, m = 100
// (the lists alone): 34.7 us and 19.8 us.
//
// A block has two phases.  The first needs only the picked determinant: it
// decodes every entry, reads its matrix element and probes the table for its
// slot, one record per entry in shared memory.  The second needs dx: it adds
// to z (inserting where the rule says so) and scores the entry.
//
// Overlap.  Launches of up to four waves of CTAs beside the leader's SM
// (column_overlaps) are enqueued with programmatic dependent launch: the first
// CTAs start while the leader runs.  It publishes its picks before it builds
// and solves the subspace problem, and the CTAs probe their first block
// meanwhile, then wait for its end.  Keys do
// not change while the leader runs; x does, on the picked determinants, so the
// slots that a small filter of these holds have x read again.  What was read
// before the wait is compared with the final picks after it.  The leader in
// turn is launched to start when the column CTAs have, and waits for their
// end, which hides its launch.  Per solve, launched one after the other and
// overlapped: 7 orbitals, k = 8, 600 iterations 18.6 and 16.8 ms; 12 orbitals,
// k = 32, 256 iterations 10.7 and 10.3 ms; 24 orbitals, k = 32, 256 iterations
// 20.8 and 19.3 ms (with the launch overlapped but the probes after the wait,
// 21.9 ms).
//
// Candidates.  The keys of a block and the CTA's list so far (at most m) are
// reduced to the m largest by a radix selection over the whole CTA
// (cta_select): a histogram per pass and one barrier, no sort, since nothing
// downstream depends on the order of a candidate list.  Of equal keys at the
// m-th place the larger determinants stay, whichever warp comes first.  Each CTA's list goes
// to global memory with its sums, and the last CTA of the column to finish
// (atomic ticket) selects the column's m from the G lists and adds the sums
// in a fixed order.  A full list's smallest key is a lower bound of the
// column's m-th largest; the CTAs share the best such bound, and keys below
// it are dropped before the selection.
#include "device_common.cuh"
#include <algorithm>
#include <cstddef>

#include "kernels.h"
#include "select.cuh"

namespace mcd {
namespace {

constexpr int kNT = 256;
constexpr int kW = kNT / 32;
constexpr int kRounds = 4;               // entries per thread and block
constexpr int kBlock = kNT * kRounds;

struct Prelude {
  uint64_t a, b;
  int na, nb, va, vb, nocc;
  int ca_occ, cb_occ, ca_vir, cb_vir;
  int off2, off3, off4, off5, total;
  unsigned char occA[64], occB[64], virA[64], virB[64], occso[128];
};

// Built by one full warp.
__device__ void build_prelude(Prelude& P, Det d, int norb) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  int na = 0, nb = 0, va = 0, vb = 0;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const int p = lane + 32 * half;
    const bool inr = p < norb;
    const bool oa = inr && ((d.a >> p) & 1ull);
    const bool ob = inr && ((d.b >> p) & 1ull);
    const bool xa = inr && !oa, xb = inr && !ob;
    unsigned m = __ballot_sync(~0u, oa);
    if (oa) P.occA[na + __popc(m & lt)] = (unsigned char)p;
    na += __popc(m);
    m = __ballot_sync(~0u, ob);
    if (ob) P.occB[nb + __popc(m & lt)] = (unsigned char)p;
    nb += __popc(m);
    m = __ballot_sync(~0u, xa);
    if (xa) P.virA[va + __popc(m & lt)] = (unsigned char)p;
    va += __popc(m);
    m = __ballot_sync(~0u, xb);
    if (xb) P.virB[vb + __popc(m & lt)] = (unsigned char)p;
    vb += __popc(m);
  }
  int nocc = 0;
#pragma unroll 1
  for (int j = 0; j < 4; ++j) {
    const int s = lane + 32 * j;
    const int p = s >> 1;
    const bool o = p < norb && ((((s & 1) ? d.b : d.a) >> p) & 1ull);
    const unsigned m = __ballot_sync(~0u, o);
    if (o) P.occso[nocc + __popc(m & lt)] = (unsigned char)s;
    nocc += __popc(m);
  }
  if (lane == 0) {
    P.a = d.a;
    P.b = d.b;
    P.na = na;
    P.nb = nb;
    P.va = va;
    P.vb = vb;
    P.nocc = nocc;
    P.ca_occ = na * (na - 1) / 2;
    P.cb_occ = nb * (nb - 1) / 2;
    P.ca_vir = va * (va - 1) / 2;
    P.cb_vir = vb * (vb - 1) / 2;
    P.off2 = 1 + na * va;
    P.off3 = P.off2 + nb * vb;
    P.off4 = P.off3 + P.ca_occ * P.ca_vir;
    P.off5 = P.off4 + P.cb_occ * P.cb_vir;
    P.total = P.off5 + na * nb * va * vb;
  }
  __syncwarp();
}

// Pair index t -> (i, j), i < j, with t = j(j-1)/2 + i.
__device__ __forceinline__ void pair_decode(int t, int& i, int& j) {
  int jj = static_cast<int>((1.0f + sqrtf(8.0f * static_cast<float>(t) + 1.0f)) * 0.5f);
#pragma unroll 1
  while (jj * (jj - 1) / 2 > t) --jj;
#pragma unroll 1
  while ((jj + 1) * jj / 2 <= t) ++jj;
  j = jj;
  i = t - jj * (jj - 1) / 2;
}

// Single p->r of spin s (0 alpha, 1 beta): h_pr + sum over occupied
// spin-orbitals k (interleaved order) of <pk||rk>, as
// get_single_excitation sums it (src/hamiltonian.h:343-347).
__device__ __forceinline__ double single_value(const HamDev& h, const Prelude& P, int s, int p, int r) {
  const int n = h.norb;
  const size_t base = (static_cast<size_t>(s) * n + p) * n + r;
  const double* st = h.st + base * h.nso;
  double v = __ldg(h.sh + base);
  // Eight loads in flight, added in order.
#pragma unroll 1
  for (int x0 = 0; x0 < P.nocc; x0 += 8) {
    double t[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) t[j] = x0 + j < P.nocc ? __ldg(st + P.occso[x0 + j]) : 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (x0 + j < P.nocc) v += t[j];
  }
  return v;
}

// An excitation packed into 27 bits: orbitals p, q, r, s (6 bits each) and the
// kind.  kXAlpha, kXBeta: p -> r; kXAlphaAlpha, kXBetaBeta: p -> r and q -> s;
// kXAlphaBeta: alpha p -> r with beta q -> s; kXDiag: none.
enum : unsigned { kXDiag = 0, kXAlpha, kXBeta, kXAlphaAlpha, kXBetaBeta, kXAlphaBeta };

// The determinant (a, b) after packed excitation x.
__device__ __forceinline__ void apply_x(unsigned x, uint64_t& a, uint64_t& b) {
  const unsigned kind = (x >> 24) & 7u;
  const uint64_t m1 = (1ull << (x & 63u)) ^ (1ull << ((x >> 12) & 63u));
  const uint64_t m2 = (1ull << ((x >> 6) & 63u)) ^ (1ull << ((x >> 18) & 63u));
  // p = r (kXDiag) and q = s (the singles) leave the strings as they are.
  const bool beta1 = kind == kXBeta || kind == kXBetaBeta, beta2 = kind >= kXBetaBeta;
  a ^= (beta1 ? 0ull : m1) ^ (beta2 ? 0ull : m2);
  b ^= (beta1 ? m1 : 0ull) ^ (beta2 ? m2 : 0ull);
}

// Entry e of the column of P's determinant: the packed excitation with its
// flags, (a2, b2) and the value, whose sign kXNegative turns.  kXAny: the entry
// may exist, kXKeep: it is kept whatever its value (the diagonal and singles,
// as get_single_excitation does; doubles are stored by the reference only with
// a non-zero table value).  Leaving sign and test to the caller lets it start
// the hash probe before the table value arrives.  One path for all kinds after
// the orbitals are decoded: the code stays small, since the leader and this
// kernel take turns in the instruction caches.
constexpr unsigned kXNegative = 1u << 29, kXKeep = 1u << 30, kXAny = 1u << 31;

__device__ __forceinline__ void gen_entry(const HamDev& h, const Prelude& P, int e, double hdiag, unsigned& x,
                                          uint64_t& a2, uint64_t& b2, double& v) {
  const int n = h.norb;
  int p = 0, q = 0, r = 0, s = 0;
  unsigned kind = kXDiag;
  const double* val = nullptr;
  if (e >= P.off5) {
    const unsigned vb = P.vb, va = P.va, nb = P.nb;
    const unsigned t0 = e - P.off5, t1 = t0 / vb, t2 = t1 / va, t3 = t2 / nb;
    p = P.occA[t3];
    q = P.occB[t2 - t3 * nb];
    r = P.virA[t1 - t2 * va];
    s = P.virB[t0 - t1 * vb];
    kind = kXAlphaBeta;
    val = h.wab + ((static_cast<size_t>(p) * n + q) * n + r) * n + s;
  } else if (e >= P.off3) {  // same-spin doubles
    const bool beta = e >= P.off4;
    const unsigned t = e - (beta ? P.off4 : P.off3);
    const unsigned cv = beta ? P.cb_vir : P.ca_vir;
    const unsigned char* occ = beta ? P.occB : P.occA;
    const unsigned char* vir = beta ? P.virB : P.virA;
    const unsigned op = t / cv, vp = t - op * cv;
    int i, j, ri, sj;
    pair_decode(op, i, j);
    pair_decode(vp, ri, sj);
    p = occ[i];
    q = occ[j];
    r = vir[ri];
    s = vir[sj];
    kind = beta ? kXBetaBeta : kXAlphaAlpha;
    const size_t np = static_cast<size_t>(h.npair);
    val = h.vss + ((beta ? np : 0) + pair_index(p, q)) * np + pair_index(r, s);
  } else if (e > 0) {
    const bool beta = e >= P.off2;
    const unsigned t = e - (beta ? P.off2 : 1);
    const unsigned nv = beta ? P.vb : P.va;
    const unsigned i = t / nv;
    p = (beta ? P.occB : P.occA)[i];
    r = (beta ? P.virB : P.virA)[t - i * nv];
    kind = beta ? kXBeta : kXAlpha;
  }
  x = static_cast<unsigned>(p) | (static_cast<unsigned>(q) << 6) | (static_cast<unsigned>(r) << 12) |
      (static_cast<unsigned>(s) << 18) | (kind << 24);
  v = hdiag;
  if (val) {
    v = __ldg(val);
    x |= kXAny;
  } else if (kind != kXDiag) {
    const int sp = kind == kXBeta ? 1 : 0;
    const uint64_t stored = __ldg(h.spres + sp * n + p);
    v = single_value(h, P, sp, p, r);
    if ((stored >> r) & 1ull) x |= kXAny | kXKeep;
  } else {
    x |= kXAny | kXKeep;
  }
  // The first excitation on (a, b), the second on the result of the first.
  a2 = P.a;
  b2 = P.b;
  unsigned neg = sign_one(kind == kXBeta || kind == kXBetaBeta, a2, b2, p, r);
  const uint64_t m1 = (1ull << p) ^ (1ull << r), m2 = (1ull << q) ^ (1ull << s);
  if (kind == kXBeta || kind == kXBetaBeta)
    b2 ^= m1;
  else
    a2 ^= m1;
  neg ^= sign_one(kind >= kXBetaBeta, a2, b2, q, s);
  if (kind >= kXBetaBeta)
    b2 ^= m2;
  else
    a2 ^= m2;
  if (neg) x |= kXNegative;
}

// |dz scale| > zt, the insertion rule (src/wavefunction.h:517-528): a double
// product decides unless it lies within 1e-14 of zt, where the
// double-double product does.
__device__ __forceinline__ bool above_threshold(dd scale, double dz, double zt) {
  const double sd = fabs(scale.hi * dz);
  if (sd > zt * (1.0 + 1e-14)) return true;
  if (sd < zt * (1.0 - 1e-14)) return false;
  return dd_gt(dd_abs(dd_mul_d(scale, dz)), dd{zt, 0.0});
}

// ---------------------------------------------------------------------------

// Per-entry record of a block's first phase: the slot (low word) where the
// determinant was found or the probe ended at an empty slot, and above it the
// packed excitation and these flags (neither: the column has no such entry).
constexpr unsigned kRecFound = 1u << 27;
constexpr unsigned kRecEmpty = 1u << 28;

struct alignas(16) ColumnShared {
  Prelude P;
  unsigned long long val[kRounds][kNT];  // the entries' matrix elements, then their candidate keys
  unsigned long long rec[kRounds][kNT];
  double x[kRounds][kNT];  // x of the entries found
  unsigned long long list_key[kMaxM];    // the CTA's candidates so far
  unsigned list_slot[kMaxM];
  SelectScratch sel;
  double newz[kNT], dot[kNT];  // the threads' sums and counts so far
  unsigned emit[kNT], upd[kNT], ins[kNT];
  double w_sum[kPartSum][kW];
  double dx, hdiag, zt;  // the column's scalars
  dd xss, scale;
  unsigned filter[64];  // of the picked slots
  unsigned out, n_tied, tied[kMaxM];
  const Slot* slots;          // the table, and
  const unsigned* part_slot;  // the slots of the keys that the merge selects from
  unsigned slot;        // the picked determinant's
  int last, some;
};

struct Selected {
  int n_list;
  unsigned long long bound;
};

// The determinant of a payload of cta_select's.
__device__ __forceinline__ void payload_key(const ColumnShared& S, unsigned base, unsigned payload, uint64_t& a,
                                            uint64_t& b) {
  load_key(S.slots + (base == kNoSlot ? payload : __ldcg(S.part_slot + payload)), a, b);
}

// cta_keep_tied for more keys than a warp ranks, n_listed of them from the list:
// the largest strings that `need` keys reach, bit by bit.
__device__ __noinline__ void cta_keep_tied_many(ColumnShared* s, int n, unsigned base, int n_listed,
                                                unsigned long long edge, int need, bool in_pool) {
  __builtin_assume(__isShared(s));
  ColumnShared& S = *s;
  const int tid = threadIdx.x;
  unsigned* counts = &S.sel.hist[0][0];
  counts[tid] = 0u;
  __syncthreads();
  const int norb = S.P.na + S.P.va, last = 2 * norb;
  uint64_t cut_a = 0, cut_b = 0;
  // A step for each bit of alpha and then of beta; the last keeps what reaches the cut.
#pragma unroll 1
  for (int step = 0;; ++step) {
    const bool alpha = step < norb;
    const uint64_t bit = step < last ? 1ull << (norb - 1 - (alpha ? step : step - norb)) : 0ull;
    const uint64_t try_a = alpha ? cut_a | bit : cut_a, try_b = alpha ? cut_b : cut_b | bit;
    unsigned c = 0;
#pragma unroll 1
    for (int i = tid - kNT; i < n; i += kNT) {
      const bool tied = i < 0 ? tid < n_listed : in_pool && (&S.val[0][0])[i] == edge;
      if (!tied) continue;
      const unsigned payload = i < 0            ? S.tied[tid]
                               : base == kNoSlot ? static_cast<unsigned>((&S.rec[0][0])[i])
                                                 : base + i;
      uint64_t a, b;
      payload_key(S, base, payload, a, b);
      if (a < try_a || (a == try_a && b < try_b)) continue;
      ++c;
      if (step == last) {
        const unsigned pos = atomicAdd(&S.out, 1u);
        S.list_key[pos] = edge;
        S.list_slot[pos] = payload;
      }
    }
    if (step == last) return;
    c = __reduce_add_sync(~0u, c);
    if ((tid & 31) == 0) atomicAdd(&counts[step], c);
    __syncthreads();
    const int reach = static_cast<int>(counts[step]);
    if (reach < need) continue;
    cut_a = try_a;
    cut_b = try_b;
    if (reach == need) step = last - 1;
  }
}

// Of cta_select's keys equal to `edge`, the payloads in S.tied (from the list)
// and those of the pool (with in_pool), the `need` whose determinants have the
// largest (alpha, beta) strings, added to S.list.  Out of line: few selections
// need it, and what the others run should stay small (the kernels' code takes
// turns in the instruction caches).  24 orbitals 6a6b, k = m = 32, where mirror
// pairs tie: 0.0747 ms an iteration, 0.0748 with any of the tied kept.
__device__ __noinline__ void cta_keep_tied(ColumnShared* s, int n, unsigned base, unsigned long long edge, int need,
                                           bool in_pool) {
  __builtin_assume(__isShared(s));
  ColumnShared& S = *s;
  const unsigned long long* pool = &S.val[0][0];
  const int tid = threadIdx.x;
  __syncthreads();
  const unsigned listed = S.n_tied;
  __syncthreads();
  if (in_pool)
#pragma unroll 1
    for (int i = tid; i < n; i += kNT)
      if (pool[i] == edge) {
        const unsigned pos = atomicAdd(&S.n_tied, 1u);
        if (pos < 32u) S.tied[pos] = base == kNoSlot ? static_cast<unsigned>((&S.rec[0][0])[i]) : base + i;
      }
  __syncthreads();
  const unsigned tied = S.n_tied;
  if (tied > 32u) {
    cta_keep_tied_many(s, n, base, static_cast<int>(listed), edge, need, in_pool);
    return;
  }
  if (tid >= 32) return;
  const bool mine = static_cast<unsigned>(tid) < tied;
  const unsigned payload = mine ? S.tied[tid] : 0u;
  uint64_t a = 0, b = 0;
  if (mine) payload_key(S, base, payload, a, b);
  unsigned rank = 0;
#pragma unroll 1
  for (unsigned j = 0; j < tied; ++j) {
    const uint64_t oa = __shfl_sync(~0u, a, j), ob = __shfl_sync(~0u, b, j);
    rank += oa > a || (oa == a && ob > b) ? 1u : 0u;
  }
  if (mine && static_cast<int>(rank) < need) {
    const unsigned pos = atomicAdd(&S.out, 1u);
    S.list_key[pos] = edge;
    S.list_slot[pos] = payload;
  }
}

// Reduces the CTA's candidates, S.list's n_list and the keys of n / kBlock
// whole blocks from S.val on (0 and those below `bound` left out), to the m largest in S.list, in no
// particular order; of equal keys at the m-th place the larger determinants
// stay, so that the set follows from the keys alone.  Their payloads: the slots in S.rec, or base + index when
// base is not kNoSlot (the slots then in S.part_slot).  Raises `bound` to the smallest value a kept key can
// have when some were left out.  Called by the whole CTA, each thread having
// written the keys tid + j kNT itself (0 beyond the last); ends with a barrier.  One copy of the
// code, out of line, serves a CTA's blocks and the merge of the lists: the
// rounds keep their registers, and a column's last CTA finds its instructions
// in the cache.
__device__ __noinline__ Selected cta_select(ColumnShared* s, int n, unsigned base, int n_list, int m,
                                            unsigned long long bound) {
  __builtin_assume(__isShared(s));
  ColumnShared& S = *s;
  const unsigned long long* pool = &S.val[0][0];
  const int tid = threadIdx.x;
  const unsigned long long floor = bound > 1ull ? bound : 1ull;
  bool any = false;
#pragma unroll 1
  for (int i = tid; i < n; i += kRounds * kNT)
#pragma unroll
    for (int j = 0; j < kRounds; ++j) any |= pool[i + j * kNT] >= floor;
  if (!__syncthreads_or(any)) return Selected{n_list, bound};  // nothing new above the bound
  const unsigned long long list_key = tid < n_list ? S.list_key[tid] : 0ull;
  const unsigned list_slot = tid < n_list ? S.list_slot[tid] : 0u;
  if (tid == 0) {
    S.out = 0u;
    S.n_tied = 0u;
  }
  const unsigned want = static_cast<unsigned>(m);
  const SelectEdge E = select_edge(S.sel, want, [&](auto f) {
    f(list_key);
#pragma unroll 1
    for (int i = tid; i < n; i += kRounds * kNT) {
      unsigned long long key[kRounds];
#pragma unroll
      for (int j = 0; j < kRounds; ++j) key[j] = pool[i + j * kNT];
#pragma unroll
      for (int j = 0; j < kRounds; ++j) f(key[j] >= floor ? key[j] : 0ull);
    }
  });
  const unsigned long long least = E.edge > floor ? E.edge : floor;
  const unsigned long long from = E.edge + (E.tied ? 1ull : 0ull), pool_from = from > floor ? from : floor;
  const auto keep = [&](unsigned long long key, unsigned slot) {
    const unsigned pos = atomicAdd(&S.out, 1u);
    S.list_key[pos] = key;
    S.list_slot[pos] = slot;
  };
  if (list_key >= from)
    keep(list_key, list_slot);
  else if (list_key == E.edge)
    S.tied[atomicAdd(&S.n_tied, 1u)] = list_slot;
#pragma unroll 1
  for (int i0 = tid; i0 < n; i0 += kRounds * kNT) {
    unsigned long long key[kRounds];
#pragma unroll
    for (int j = 0; j < kRounds; ++j) key[j] = pool[i0 + j * kNT];
#pragma unroll
    for (int j = 0; j < kRounds; ++j) {
      const int i = i0 + j * kNT;
      if (key[j] >= pool_from)
        keep(key[j], base == kNoSlot ? static_cast<unsigned>((&S.rec[0][0])[i]) : base + static_cast<unsigned>(i));
    }
  }
  const Selected r{static_cast<int>(min(E.total, want)), E.total > want ? least : bound};
  if (E.tied) cta_keep_tied(s, n, base, E.edge, static_cast<int>(E.need), E.edge >= floor);
  __syncthreads();
  return r;
}

// The m largest of the n keys of a column's lists, those below `bound` (which m
// keys reach) left out, into S.list with their indexes: up to 3,072 keys at a
// time in the shared memory of the rounds, where 1,024 at a time in registers
// took a selection for each (23 lists of 128: 200 iterations of 24 columns
// 10.9 ms, now 10.25; 96 lists of 128: 24.2 and 23.9 ms for 16 of 64 columns).
__device__ __forceinline__ int merge_lists(ColumnShared& S, const unsigned long long* keys, const unsigned* slots,
                                           int n, int m, unsigned long long bound) {
  constexpr int kKeys = 3 * kRounds * kNT;
  static_assert(offsetof(ColumnShared, rec) == offsetof(ColumnShared, val) + sizeof(S.val) &&
                    offsetof(ColumnShared, x) == offsetof(ColumnShared, rec) + sizeof(S.rec),
                "the rounds' arrays follow one another");
  unsigned long long* pool = &S.val[0][0];
  if (threadIdx.x == 0) S.part_slot = slots;
  Selected r{0, bound};
#pragma unroll 1
  for (int at = 0; at < n; at += kKeys) {
    const int some = min(n - at, kKeys);
#pragma unroll 1
    for (int i = threadIdx.x; i < some; i += kRounds * kNT) {
      unsigned long long key[kRounds];
#pragma unroll
      for (int j = 0; j < kRounds; ++j) key[j] = i + j * kNT < some ? __ldcg(keys + at + i + j * kNT) : 0ull;
#pragma unroll
      for (int j = 0; j < kRounds; ++j) pool[i + j * kNT] = key[j];
    }
    r = cta_select(&S, some, static_cast<unsigned>(at), r.n_list, m, r.bound);
  }
  return r.n_list;
}

// Continues a probe at slot i, which was empty when the first phase ended
// there: the determinant may have been inserted since (by another column), or
// i taken by another key.  Inserts it when `insert`; -1 when it stays absent.
// The occupancy is counted per CTA, not here.
__device__ __forceinline__ long long probe_again(const TableDev& t, uint64_t a, uint64_t b, uint64_t i, bool insert,
                                                 bool& inserted) {
  inserted = false;
#pragma unroll 1
  for (int q = 0; q < t.max_probe; ++q) {
    uint64_t ka, kb;
    if (insert)
      cas_key(t.slots + i, a, b, ka, kb);
    else
      load_key(t.slots + i, ka, kb);
    if (ka == kEmptyKey && kb == kEmptyKey) {
      inserted = insert;
      return insert ? static_cast<long long>(i) : -1;
    }
    if (ka == a && kb == b) return static_cast<long long>(i);
    i = (i + 1) & t.mask;
  }
  atomicOr(t.err, kErrProbe);
  return -1;
}

// A slot's bit in a 2048-bit filter.
__device__ __forceinline__ unsigned filter_bit(unsigned slot) { return (slot * 0x9E3779B1u) >> 21; }

// First phase of the block of entries [at, at + kBlock) of the column, below
// stop: their values (the diagonal's is filled in later), slots and x.
__device__ __forceinline__ void block_probe(const ColumnLaunch& L, ColumnShared& S, int at, int stop, bool timed) {
  const int tid = threadIdx.x;
  const int nr = min(kRounds, (stop - at + kNT - 1) / kNT);
  // The home slot and matrix element of a thread's next entry are requested before the last one's are
  // looked at, so that its decoding runs under their latency.
  const long long q0 = timed ? clock64() : 0;
  uint64_t na = 0, nb = 0;  // the requested slot's key and x, and the element
  double nx = 0.0, nv = 0.0;
#pragma unroll 1
  for (int r = 0; r <= nr; ++r) {
    uint64_t ka = na, kb = nb;
    double x = nx, v = nv;
    const int e = at + r * kNT + tid;
    if (r < nr) {
      unsigned info = 0u;
      uint64_t slot = 0;
      if (e < stop) {
        uint64_t a2, b2;
        gen_entry(L.ham, S.P, e, 0.0, info, a2, b2, nv);
        if (info & kXAny) {
          // (the diagonal entry's slot is the picked determinant's own)
          slot = e == 0 ? static_cast<uint64_t>(S.slot) : det_hash(a2, b2) & L.tab.mask;
          load_slot(L.tab.slots + slot, na, nb, nx);
        }
      }
      S.rec[r][tid] = slot | (static_cast<unsigned long long>(info) << 32);
    }
    if (r == 0) continue;
    const unsigned long long rec = S.rec[r - 1][tid];
    unsigned info = static_cast<unsigned>(rec >> 32);
    if (info & kXNegative) v = -v;
    if ((info & kXKeep) || ((info & kXAny) && v != 0.0)) {
      uint64_t slot = rec & 0xFFFFFFFFull, a2 = S.P.a, b2 = S.P.b;
      apply_x(info, a2, b2);
#pragma unroll 1
      for (int q = 1;; ++q) {
        whole_key(L.tab.slots + slot, ka, kb);
        if (ka == a2 && kb == b2) {
          info |= kRecFound;
          S.x[r - 1][tid] = x;
          break;
        }
        if (ka == kEmptyKey && kb == kEmptyKey) {
          info |= kRecEmpty;
          break;
        }
        if (q >= L.tab.max_probe) {
          atomicOr(L.tab.err, kErrProbe);
          break;
        }
        slot = (slot + 1) & L.tab.mask;
        load_slot(L.tab.slots + slot, ka, kb, x);
      }
      S.rec[r - 1][tid] = slot | (static_cast<unsigned long long>(info) << 32);
      S.val[r - 1][tid] = static_cast<unsigned long long>(__double_as_longlong(v));
    }
  }
  if (timed) atomicAdd(L.sect + 1, static_cast<unsigned long long>(clock64() - q0));
}

// Second phase: the z updates and the candidate keys, left in S.val with
// their slots in S.rec.  kOverlap, and `early`: the first phase may have run
// before the leader's update of x, so x is read again for the slots that
// S.filter holds.
template <bool kOverlap>
__device__ __forceinline__ void block_update(const ColumnLaunch& L, ColumnShared& S, int nr, bool early, bool timed) {
  const int tid = threadIdx.x;
  const double dxc = S.dx, zt = S.zt;
  const dd xss = S.xss, scale = S.scale;
  const long long q2 = timed ? clock64() : 0;
  double acc_newz = S.newz[tid], acc_dot = S.dot[tid];
  unsigned emit = S.emit[tid], upd = S.upd[tid], ins = S.ins[tid];
#pragma unroll 1
  for (int r = 0; r < nr; ++r) {
    const unsigned long long rec = S.rec[r][tid];
    const unsigned info = static_cast<unsigned>(rec >> 32);
    unsigned long long key = 0ull;
    if (info & (kRecFound | kRecEmpty)) {
      const bool diagonal = ((info >> 24) & 7u) == kXDiag;
      const double v = diagonal ? S.hdiag : __longlong_as_double(static_cast<long long>(S.val[r][tid]));
      ++emit;
      const double dz = v * dxc;
      long long slot = static_cast<long long>(rec & 0xFFFFFFFFull);
      double x = 0.0;
      if (info & kRecFound) {
        x = S.x[r][tid];
        if (kOverlap && early) {
          const unsigned h = filter_bit(static_cast<unsigned>(slot));
          if ((S.filter[h >> 5] >> (h & 31u)) & 1u) x = load_relaxed(&L.tab.slots[slot].x);
        }
      } else {
        bool inserted;
        uint64_t a2 = S.P.a, b2 = S.P.b;
        apply_x(info, a2, b2);
        slot = probe_again(L.tab, a2, b2, static_cast<uint64_t>(slot), above_threshold(scale, dz, zt), inserted);
        ins += inserted ? 1u : 0u;
        // Found after all: inserted by another column, with x = 0, since the first phase.
      }
      if (slot >= 0) {
        const double znew = atomicAdd(&L.tab.slots[slot].z, dz) + dz;
        ++upd;
        acc_newz += v * x;
        acc_dot += dz * x;
        key = score_key(score_of(x, znew, xss));
        S.rec[r][tid] = static_cast<unsigned long long>(slot);
      }
    }
    S.val[r][tid] = key;
  }
  S.newz[tid] = acc_newz;
  S.dot[tid] = acc_dot;
  S.emit[tid] = emit;
  S.upd[tid] = upd;
  S.ins[tid] = ins;
  if (timed) atomicAdd(L.sect + 2, static_cast<unsigned long long>(clock64() - q2));
}

// The column's picked determinant into S (prelude and slot); false, for the
// whole CTA, when the iteration has no such column.
__device__ __forceinline__ bool read_picked(const IterState* St, ColumnShared& S, int col, int norb) {
  if (threadIdx.x < 32) {
    const bool some = col < __ldcg(&St->k_cur);
    if (some) {
      const Det d{__ldcg(&St->det[col].a), __ldcg(&St->det[col].b)};
      const unsigned slot = static_cast<unsigned>(__ldcg(&St->slot[col]));
      build_prelude(S.P, d, norb);
      if (threadIdx.x == 0) S.slot = slot;
    }
    if (threadIdx.x == 0) S.some = some;
  }
  __syncthreads();
  return S.some;
}

// After the leader's end: whether what read_picked took before it still holds.
// 1 yes, 0 the iteration has no such column, 2 it was another determinant and
// has been read again.
__device__ __forceinline__ int confirm_picked(const IterState* St, ColumnShared& S, int col, int norb) {
  pdl_wait();
  if (col >= __ldcg(&St->k_cur)) return 0;
  if (__ldcg(&St->det[col].a) == S.P.a && __ldcg(&St->det[col].b) == S.P.b &&
      static_cast<unsigned>(__ldcg(&St->slot[col])) == S.slot)
    return 1;
  __syncthreads();
  read_picked(St, S, col, norb);
  return 2;
}

// One CTA's share of one column: CTA `blk` of the launch described by L
// (column blk / groups, slice blk % groups).  kOverlap: launched to start
// beside the leader; the first block is probed from the determinants as the
// leader publishes them when it has picked, while it solves for dx.  kSingle:
// groups is 1.
template <bool kOverlap, bool kSingle>
__device__ __forceinline__ void column_body(const ColumnLaunch& L, int blk) {
  const int G = kSingle ? 1 : L.groups;
  const int col = blk / G;
  const int g = blk - col * G;
  IterState* St = L.st;

  __shared__ __align__(16) ColumnShared S;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool timed = L.sect != nullptr && tid == 0;
  const long long c_start = timed ? clock64() : 0;
  bool early = false;  // probing before the leader has ended
  if (kOverlap) {
    if (tid == 0) pdl_trigger();
    if (tid < 64) S.filter[tid] = 0u;
    // (a determinant that the leader has not published yet may be of no sector:
    // the slice below holds for all determinants of the launch's own)
    early = read_picked(St, S, col, L.ham.norb) && S.P.na == L.na && S.P.nb == L.nb;
    if (!early) {
      pdl_wait();
      __syncthreads();  // every warp has S.some of the first reading before the second writes it
    }
  }
  if (!early && !read_picked(St, S, col, L.ham.norb)) return;
  const int total = S.P.total;
  // CTA g's slice: whole rounds of kNT entries, shared evenly.
  const int chunks = (total + kNT - 1) / kNT;
  const int beg = kNT * (g * chunks / G);
  const int end = min(total, kNT * ((g + 1) * chunks / G));

  S.newz[tid] = S.dot[tid] = 0.0;
  S.emit[tid] = S.upd[tid] = S.ins[tid] = 0u;
  int n_list = 0;
  unsigned long long bound = 0ull;  // a lower bound of the column's m-th largest key

  const long long c_rounds = timed ? clock64() : 0;
  const int M = L.list;
  int at = beg;
#pragma unroll 1
  while (at < end) {
    block_probe(L, S, at, end, timed);
    if (at == beg) {
      if (kOverlap && early) {
        const int state = confirm_picked(St, S, col, L.ham.norb);
        if (state == 0) return;
        if (state == 2) {  // read before the leader had published it: probe again
          early = false;
          continue;
        }
        if (tid < kMaxK && tid < __ldcg(&St->k_cur)) {
          const unsigned h = filter_bit(static_cast<unsigned>(__ldcg(&St->slot[tid])));
          atomicOr(&S.filter[h >> 5], 1u << (h & 31u));
        }
      }
      if (tid == 0) {
        S.dx = __ldcg(&St->dx[col]);
        S.hdiag = __ldcg(&St->hdiag[col]);
        S.zt = __ldcg(&St->zt);
        S.slots = L.tab.slots;
        S.xss = dd{__ldcg(&St->xss.hi), __ldcg(&St->xss.lo)};
        S.scale = dd{__ldcg(&St->scale.hi), __ldcg(&St->scale.lo)};
      }
      __syncthreads();
    }
    const int nr = min(kRounds, (end - at + kNT - 1) / kNT);
    block_update<kOverlap>(L, S, nr, early, timed);
    early = false;
    const unsigned long long shared_bound = __ldcg(L.bound + col);
    if (shared_bound > bound) bound = shared_bound;
    if (timed) atomicAdd(L.sect + 4, static_cast<unsigned long long>(nr));
    const long long q3 = timed ? clock64() : 0;
    for (int r = nr; r < kRounds; ++r) S.val[r][tid] = 0ull;
    const Selected sel = cta_select(&S, kBlock, kNoSlot, n_list, L.m, bound);
    n_list = sel.n_list;
    bound = sel.bound;
    if (timed) atomicAdd(L.sect + 3, static_cast<unsigned long long>(clock64() - q3));
    at += kBlock;
  }
  if (kOverlap && early) {  // an empty slice
    pdl_wait();
    if (col >= __ldcg(&St->k_cur)) return;
  }
  // This CTA's list and partial sums to global memory, then a ticket: the
  // last CTA of the column merges all of them.
  const size_t part = blk;  // column col's CTA g
  const long long c_post = timed ? clock64() : 0;
  if (timed) {
    atomicAdd(L.sect + 5, static_cast<unsigned long long>(c_rounds - c_start));
    atomicAdd(L.sect + 8, 1ull);
  }
  if (!kSingle && tid < M) {
    L.part_key[part * M + tid] = tid < n_list ? S.list_key[tid] : 0ull;
    L.part_slot[part * M + tid] = tid < n_list ? S.list_slot[tid] : 0u;
  }
  // The counters travel with the sums (exact in a double) and are added
  // once per column by its last CTA, not by every CTA into the same words.
  const double v[kPartSum] = {warp_sum(S.newz[tid]), warp_sum(S.dot[tid]),
                              static_cast<double>(__reduce_add_sync(~0u, S.emit[tid])),
                              static_cast<double>(__reduce_add_sync(~0u, S.upd[tid])),
                              static_cast<double>(__reduce_add_sync(~0u, S.ins[tid]))};
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < kPartSum; ++j) S.w_sum[j][warp] = v[j];
  }
  __syncthreads();
  if (warp == 0) {
    if (lane < kPartSum) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < kW; ++w) t += S.w_sum[lane][w];
      L.part_sum[kPartSum * part + lane] = t;
    }
    __syncwarp();
    // One fence for the whole CTA's list and sums (the barriers order
    // them before it), then the ticket.
    if (!kSingle && lane == 0) {
      if (bound != 0ull) atomicMax(L.bound + col, bound);
      __threadfence();
      S.last = (atomicAdd(L.done + col, 1u) == static_cast<unsigned>(G - 1));
    }
  }
  __syncthreads();
  const long long c_merge = timed ? clock64() : 0;
  if (timed) atomicAdd(L.sect + 6, static_cast<unsigned long long>(c_merge - c_post));
  if (!kSingle) {
    if (!S.last) return;
    __threadfence();
    const size_t lists = static_cast<size_t>(col) * G * M;
    n_list = merge_lists(S, L.part_key + lists, L.part_slot + lists, G * M, L.m, __ldcg(L.bound + col));
  }
  if (tid < L.m)
    L.cand_slot[static_cast<size_t>(col) * L.m + tid] =
        tid >= n_list ? kNoSlot
        : kSingle    ? S.list_slot[tid]
                     : __ldcg(L.part_slot + static_cast<size_t>(col) * G * M + S.list_slot[tid]);
  if (warp < kPartSum) {
    // Column sums in a fixed order, one per warp: lane-strided partials, then a fixed tree.
    double t = 0.0;
#pragma unroll 1
    for (int gg = lane; gg < G; gg += 32) t += __ldcg(L.part_sum + kPartSum * (static_cast<size_t>(col) * G + gg) + warp);
    t = warp_sum(t);
    if (lane == 0) S.w_sum[0][warp] = t;
  }
  __syncthreads();
  if (tid == 0) {
    const unsigned long long ce = static_cast<unsigned long long>(S.w_sum[0][2]);
    const unsigned long long cu = static_cast<unsigned long long>(S.w_sum[0][3]);
    const unsigned long long ci = static_cast<unsigned long long>(S.w_sum[0][4]);
    if (ce) {
      atomicAdd(&St->emitted, ce);
      atomicAdd(&St->emitted_total, ce);
    }
    if (cu) {
      atomicAdd(&St->updates, cu);
      atomicAdd(&St->updates_total, cu);
    }
    if (ci) {
      atomicAdd(&St->z_size, ci);
      atomicAdd(L.tab.n_occupied, ci);
    }
    St->newz[col] = S.w_sum[0][0];
    St->dot[col] = S.w_sum[0][1];
    St->cand_n[col] = n_list;
    L.done[col] = 0u;
    L.bound[col] = 0ull;
  }
  if (timed) {
    atomicAdd(L.sect + 7, static_cast<unsigned long long>(clock64() - c_merge));
    atomicAdd(L.sect + 9, 1ull);
  }
}

template <bool kOverlap, bool kSingle>
__global__ void __launch_bounds__(kNT, kColumnCtasPerSm) column_kernel(ColumnLaunch L) {
  column_body<kOverlap, kSingle>(L, blockIdx.x);
}

// Several instances in one grid: CTAs [cta_begin[i], cta_begin[i+1]) belong
// to instance i and keep the layout of its own launch.
__global__ void __launch_bounds__(kNT, kColumnCtasPerSm) column_kernel_batch(ColumnBatch B) {
  int lo = 0, hi = B.n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (B.cta_begin[mid] <= static_cast<int>(blockIdx.x))
      lo = mid;
    else
      hi = mid;
  }
  column_body<false, false>(B.L[lo], static_cast<int>(blockIdx.x) - B.cta_begin[lo]);
}

__global__ void __launch_bounds__(kNT) debug_column_kernel(HamDev h, Det d, double hd, uint64_t* ao,
                                                           uint64_t* bo, double* vo, int cap, int* nout) {
  __shared__ Prelude P;
  if ((threadIdx.x >> 5) == 0) build_prelude(P, d, h.norb);
  __syncthreads();
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < P.total; e += gridDim.x * blockDim.x) {
    unsigned x;
    uint64_t a2, b2;
    double v;
    gen_entry(h, P, e, hd, x, a2, b2, v);
    if (x & kXNegative) v = -v;
    if ((x & kXKeep) || ((x & kXAny) && v != 0.0)) {
      const int pos = atomicAdd(nout, 1);
      if (pos < cap) {
        ao[pos] = a2;
        bo[pos] = b2;
        vo[pos] = v;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Reduced density matrices of the wavefunction in the table (the adjoint of
// the energy with respect to the integrals): the sum over ordered pairs (D, D')
// of determinants with x != 0 that differ by at most two electrons, of
// x_D x_D' <D'|a+_r a_p|D> and <D'|a+_r a+_s a_q a_p|D>, with the phases of
// the column generation and no integral screening (the RDM is a property of
// the wavefunction).  Accumulated unnormalised, in spin blocks (see
// RdmLaunch), folded on the device.  The pairs are found in one of two ways:
// by comparing every two determinants (rdm_pairs_kernel) or by looking up
// every excitation of every determinant (rdm_lookup_kernel).  See launch_rdm.

__global__ void __launch_bounds__(256) collect_x_kernel(const Slot* slots, size_t n, Slot* list,
                                                        unsigned long long* count, unsigned long long cap) {
  scan_slots(slots, n, [&](const Slot& sl, size_t i) {
    if (slot_vacant(sl.a, sl.b) || sl.x == 0.0) return;
    const unsigned long long j = atomicAdd(count, 1ull);
    if (j < cap) list[j] = Slot{sl.a, sl.b, sl.x, static_cast<double>(i)};
  });
}

__device__ __forceinline__ size_t idx4(int n, int p, int q, int r, int s) {
  return ((static_cast<size_t>(p) * n + q) * n + r) * n + s;
}

// x of a determinant, 0 when it is absent; key and x in one load per slot, of a
// table that nothing writes meanwhile (so without whole_key).
__device__ __forceinline__ double find_x(const TableDev& t, uint64_t a, uint64_t b) {
  uint64_t i = det_hash(a, b) & t.mask;
#pragma unroll 1
  for (int p = 0; p < t.max_probe; ++p) {
    uint64_t ka, kb;
    double x;
    load_slot(t.slots + i, ka, kb, x);
    if (ka == a && kb == b) return x;
    if (ka == kEmptyKey && kb == kEmptyKey) return 0.0;
    i = (i + 1) & t.mask;
  }
  atomicOr(t.err, kErrProbe);
  return 0.0;
}

// Spatial RDMs from the spin blocks: rdm2 is the same-spin block from its
// canonical p < q, r < s elements, and the
// opposite spins (alpha, beta) + (beta, alpha) = ab[p][q][r][s] + ab[q][p][s][r].
__global__ void __launch_bounds__(256) rdm_fold_kernel(RdmLaunch R, double norm, double* rdm1, double* rdm2) {
  const int n = R.ham.norb;
  const size_t n2 = static_cast<size_t>(n) * n, n4 = n2 * n2;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    if (i < n2) rdm1[i] = R.g1[i] * norm;
    const unsigned pq = static_cast<unsigned>(i / n2), rs = static_cast<unsigned>(i - pq * n2);
    const int p = pq / n, q = pq - p * n, r = rs / n, s = rs - r * n;
    double same = 0.0;
    if (p != q && r != s) {
      const size_t c = idx4(n, min(p, q), max(p, q), min(r, s), max(r, s));
      same = ((p < q) == (r < s) ? 1.0 : -1.0) * R.g2ss[c];
    }
    rdm2[i] = (same + R.g2ab[i] + R.g2ab[idx4(n, q, p, s, r)]) * norm;
  }
}

// The diagonal terms of D: gamma_pp and Gamma_pqpq over its occupied pairs.
__device__ void rdm_diagonal(const RdmLaunch& R, uint64_t a, uint64_t b, double w) {
  const int n = R.ham.norb;
  for (uint64_t u = a; u; u &= u - 1) {
    const int p = __ffsll(static_cast<long long>(u)) - 1;
    atomicAdd(R.g1 + static_cast<size_t>(p) * n + p, w);
    for (uint64_t v = u & (u - 1); v; v &= v - 1) {
      const int q = __ffsll(static_cast<long long>(v)) - 1;
      atomicAdd(R.g2ss + idx4(n, p, q, p, q), w);
    }
    for (uint64_t v = b; v; v &= v - 1) {
      const int q = __ffsll(static_cast<long long>(v)) - 1;
      atomicAdd(R.g2ab + idx4(n, p, q, p, q), w);
    }
  }
  for (uint64_t u = b; u; u &= u - 1) {
    const int p = __ffsll(static_cast<long long>(u)) - 1;
    atomicAdd(R.g1 + static_cast<size_t>(p) * n + p, w);
    for (uint64_t v = u & (u - 1); v; v &= v - 1) {
      const int q = __ffsll(static_cast<long long>(v)) - 1;
      atomicAdd(R.g2ss + idx4(n, p, q, p, q), w);
    }
  }
}

// The terms of one connected pair D != D', w = x_D x_D'.  The orbitals that
// leave (p, q) and come (r, s), in increasing order, are the bits that differ.
__device__ void rdm_pair(const RdmLaunch& R, uint64_t a, uint64_t b, uint64_t a2, uint64_t b2, double w) {
  const int n = R.ham.norb;
  const auto low = [](uint64_t u) { return __ffsll(static_cast<long long>(u)) - 1; };
  const uint64_t ha = a & ~a2, pa = a2 & ~a, hb = b & ~b2, pb = b2 & ~b;
  if (ha && hb) {  // <a+_r(alpha) a+_s(beta) a_q(beta) a_p(alpha)>
    const int p = low(ha), r = low(pa), q = low(hb), s = low(pb);
    atomicAdd(R.g2ab + idx4(n, r, s, p, q), sign_ab(a, b, p, r, q, s) ? -w : w);
    return;
  }
  const bool beta = hb != 0;
  const uint64_t h = beta ? hb : ha, c = beta ? pb : pa;
  const int p = low(h), r = low(c);
  const uint64_t h2 = h & (h - 1), c2 = c & (c - 1);
  if (h2) {  // <a+_r a+_s a_q a_p>, p < q, r < s
    const int q = low(h2), s = low(c2);
    const int neg = beta ? sign_bb(a, b, p, q, r, s) : sign_aa(a, b, p, q, r, s);
    atomicAdd(R.g2ss + idx4(n, r, s, p, q), neg ? -w : w);
    return;
  }
  // <a+_r a_p> and the spectators k: <a+_r a+_k a_k a_p>
  if (beta ? sign_beta(a, b, p, r) : sign_alpha(a, b, p, r)) w = -w;
  atomicAdd(R.g1 + static_cast<size_t>(r) * n + p, w);
  for (uint64_t u = (beta ? b : a) & ~h; u; u &= u - 1) {
    const int k = low(u);
    const bool flip = (r < k) != (p < k);
    atomicAdd(R.g2ss + idx4(n, min(r, k), max(r, k), min(p, k), max(p, k)), flip ? -w : w);
  }
  for (uint64_t u = beta ? a : b; u; u &= u - 1) {
    const int k = low(u);
    atomicAdd(R.g2ab + (beta ? idx4(n, k, r, k, p) : idx4(n, r, k, p, k)), w);
  }
}

// Every two determinants of the list: a tile of kPairRows of them in shared
// memory against one per thread.  Bound by the additions of the pairs that
// connect (a warp runs them lane after lane).  8 rows a tile: 128 CTAs for the
// 509 determinants of a short solve, whose matrices then take 20 us instead of
// the 218 us of 7.4 million lookups.
constexpr int kPairRows = 8;
constexpr size_t kL2Bytes = static_cast<size_t>(126) << 20;
__global__ void __launch_bounds__(256) rdm_pairs_kernel(RdmLaunch R) {
  __shared__ Slot rows[kPairRows];
  const long long tj = (R.nlist + 255) / 256, ti = (R.nlist + kPairRows - 1) / kPairRows;
  for (long long tile = blockIdx.x; tile < ti * tj; tile += gridDim.x) {
    const long long i0 = tile / tj * kPairRows, j = tile % tj * 256 + threadIdx.x;
    const int rn = static_cast<int>(R.nlist - i0 < kPairRows ? R.nlist - i0 : kPairRows);
    __syncthreads();  // the rows of the previous tile are no longer read
    if (threadIdx.x < rn) rows[threadIdx.x] = R.list[i0 + threadIdx.x];
    __syncthreads();
    if (j >= R.nlist) continue;
    const Slot d = R.list[j];
    for (int i = 0; i < rn; ++i) {
      const Slot& e = rows[i];
      if (__popcll(d.a ^ e.a) + __popcll(d.b ^ e.b) > 4) continue;
      if (i0 + i == j)
        rdm_diagonal(R, d.a, d.b, d.x * d.x);
      else
        rdm_pair(R, d.a, d.b, e.a, e.b, d.x * e.x);
    }
  }
}

// One CTA per determinant of the list: every single and double excitation of
// it looked up in the table.  Bound by the scattered loads of the slots.
__global__ void __launch_bounds__(kNT) rdm_lookup_kernel(RdmLaunch R) {
  __shared__ Prelude P;
  const int n = R.ham.norb;
  const int warp = threadIdx.x >> 5;
  for (long long li = blockIdx.x; li < R.nlist; li += gridDim.x) {
    const Det D{R.list[li].a, R.list[li].b};
    const double xd = R.list[li].x;
    __syncthreads();  // P of the previous determinant is no longer read
    if (warp == 0) build_prelude(P, D, n);
    __syncthreads();
    if (threadIdx.x == 0) rdm_diagonal(R, D.a, D.b, xd * xd);
    for (int e = 1 + threadIdx.x; e < P.total; e += blockDim.x) {
      uint64_t a2 = D.a, b2 = D.b;
      if (e < P.off2) {
        const int t = e - 1;
        const int i = t / P.va;
        a2 ^= (1ull << P.occA[i]) ^ (1ull << P.virA[t - i * P.va]);
      } else if (e < P.off3) {
        const int t = e - P.off2;
        const int i = t / P.vb;
        b2 ^= (1ull << P.occB[i]) ^ (1ull << P.virB[t - i * P.vb]);
      } else if (e < P.off4) {
        const int t = e - P.off3;
        const int op = t / P.ca_vir, vp = t - op * P.ca_vir;
        int i, j, ri, sj;
        pair_decode(op, i, j);
        pair_decode(vp, ri, sj);
        a2 ^= (1ull << P.occA[i]) ^ (1ull << P.occA[j]) ^ (1ull << P.virA[ri]) ^ (1ull << P.virA[sj]);
      } else if (e < P.off5) {
        const int t = e - P.off4;
        const int op = t / P.cb_vir, vp = t - op * P.cb_vir;
        int i, j, ri, sj;
        pair_decode(op, i, j);
        pair_decode(vp, ri, sj);
        b2 ^= (1ull << P.occB[i]) ^ (1ull << P.occB[j]) ^ (1ull << P.virB[ri]) ^ (1ull << P.virB[sj]);
      } else {
        int t = e - P.off5;
        const int sbi = t % P.vb;
        t /= P.vb;
        const int rai = t % P.va;
        t /= P.va;
        const int pbi = t % P.nb;
        const int pai = t / P.nb;
        a2 ^= (1ull << P.occA[pai]) ^ (1ull << P.virA[rai]);
        b2 ^= (1ull << P.occB[pbi]) ^ (1ull << P.virB[sbi]);
      }
      const double x2 = find_x(R.tab, a2, b2);
      if (x2 != 0.0) rdm_pair(R, D.a, D.b, a2, b2, xd * x2);
    }
  }
}

}  // namespace

int column_entries(int norb, int na, int nb) {
  const long long va = norb - na, vb = norb - nb;
  const long long t = 1 + na * va + nb * vb + (long long)na * (na - 1) / 2 * (va * (va - 1) / 2) +
                      (long long)nb * (nb - 1) / 2 * (vb * (vb - 1) / 2) + (long long)na * nb * va * vb;
  return t > 0x7fffffffLL ? -1 : static_cast<int>(t);
}

int column_list_size(int m) { return m <= 32 ? 32 : (m <= 64 ? 64 : 128); }

int column_groups(int entries, int k, int resident) {
  // One block of kRounds rounds per CTA ...
  int g = (entries + kBlock - 1) / kBlock;
  // ... or, when k columns of such CTAs leave resident CTA slots empty, as
  // many CTAs as fill them, down to one round each.
  if (resident > 0 && k > 0) {
    const int fill = resident / k;
    const int one_round = (entries + kNT - 1) / kNT;
    g = std::max(g, std::min(fill, one_round));
  }
  // ... and at most 96: the last CTA of a column merges all of its CTAs'
  // lists at the end of the launch, so long columns take longer CTAs (the
  // 271,945-entry columns of 42 orbitals, 24 + 24 electrons, one sweep of
  // 64-column launches: 1074 us per launch with 355 CTAs each, 957 us with
  // the cap's 96, 932 us with 89).
  g = std::min(g, 96);
  return g < 1 ? 1 : g;
}

// Up to four waves of CTAs beside the leader's SM.  96 columns of 15 CTAs (64
// iterations of 24 orbitals): 14.4 ms started early, 14.9 ms after the
// leader.  64 columns of 96 CTAs (42 orbitals): 24.15 and 24.07 ms, the first
// wave being too small a part to pay for the second reading of x.
bool column_overlaps(int ctas, int sms) { return ctas <= 4 * kColumnCtasPerSm * (sms - 1); }

cudaError_t launch_column(const ColumnLaunch& a, cudaStream_t s) {
  const dim3 grid(a.k_grid * a.groups), block(kNT);
  // One CTA a column: no ticket, no lists in global memory, no merge.  600
  // iterations of 8 columns of 171 entries 14.3 ms, 16.4 ms with them.
  const bool single = a.groups == 1;
  if (a.overlap)
    return launch_overlapped(single ? column_kernel<true, true> : column_kernel<true, false>, grid, block, 0, s, a);
  (single ? column_kernel<false, true> : column_kernel<false, false>)<<<grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_column_batch(const ColumnBatch& b, cudaStream_t s) {
  if (b.n < 1 || b.n > kMaxBatch) return cudaErrorInvalidValue;
  column_kernel_batch<<<b.cta_begin[b.n], kNT, 0, s>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_collect_x(const TableDev& t, size_t capacity, Slot* list, unsigned long long* count,
                             unsigned long long cap, cudaStream_t s) {
  collect_x_kernel<<<148 * 8, 256, 0, s>>>(t.slots, capacity, list, count, cap);
  return cudaGetLastError();
}

cudaError_t launch_rdm_fold(const RdmLaunch& r, double norm, double* rdm1, double* rdm2, cudaStream_t s) {
  rdm_fold_kernel<<<148 * 8, 256, 0, s>>>(r, norm, rdm1, rdm2);
  return cudaGetLastError();
}

// N determinants with C excitations each take N^2 comparisons or N C lookups.
// A comparison with the additions it leads to costs 8 to 13 ps of the chip, a
// lookup 26 to 32 ps in a table in HBM, less in one the L2 holds.  Measured,
// comparisons against lookups: 24 orbitals (C 14,469, 4.3 GB) N 509 0.55 and
// 0.71 ms, N 9,700 1.7 and 4.9 ms, N 20,998 3.0 and 10.1 ms; 16 orbitals (C
// 3,690, 1.1 GB) N 3,582 0.39 and 0.48 ms, N 14,647 1.83 and 1.62 ms; 10
// orbitals (C 840, in L2) N 986 0.15 and 0.14 ms, N 5,740 0.53 and 0.29 ms.
// Hence up to 3 C determinants are compared, up to C where the L2 holds the
// table.
cudaError_t launch_rdm(const RdmLaunch& r, cudaStream_t s) {
  if (r.nlist <= 0) return cudaSuccess;
  const bool pairs = r.route ? r.route == 1 : r.nlist <= (r.tab.mask * sizeof(Slot) > kL2Bytes ? 3 : 1) * r.excitations;
  if (pairs) {
    const long long tiles = ((r.nlist + 255) / 256) * ((r.nlist + kPairRows - 1) / kPairRows);
    rdm_pairs_kernel<<<static_cast<unsigned>(tiles < 148LL * 8 ? tiles : 148LL * 8), 256, 0, s>>>(r);
  } else {
    const long long blocks = r.nlist < 148LL * 16 ? r.nlist : 148LL * 16;
    rdm_lookup_kernel<<<static_cast<unsigned>(blocks), kNT, 0, s>>>(r);
  }
  return cudaGetLastError();
}

// Scattered-access ceiling of the table, for the column kernel's roofline: a
// stream of pseudo-random slots, each touched the way a column entry touches
// its slot (the 16-byte key, then x and an FP64 atomic add on z that returns
// the old value; the add is of zero, so the table keeps its values).  ILP
// slots are in flight per thread; the grid fills every SM.
// MODE 0: the 16-byte key, x and an FP64 atomic add of zero with its return,
// as a column entry touches its slot; 1: key and x loads only; 2: the atomic
// with return only; 3: key load and an atomic add whose return is unused
// (a reduction, no round trip).
template <int ILP, int MODE>
__global__ void __launch_bounds__(256) scatter_probe_kernel(Slot* slots, uint64_t mask, long long entries,
                                                            uint64_t seed, double* sink) {
  double acc = 0.0;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x * ILP;
  for (long long e0 = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * ILP; e0 < entries;
       e0 += stride) {
    uint64_t sl[ILP], ka[ILP], kb[ILP];
#pragma unroll
    for (int q = 0; q < ILP; ++q) {
      sl[q] = fmix64(seed ^ static_cast<uint64_t>(e0 + q)) & mask;
      ka[q] = kb[q] = 0;
      if (MODE != 2 && e0 + q < entries) load_key(slots + sl[q], ka[q], kb[q]);
    }
#pragma unroll
    for (int q = 0; q < ILP; ++q) {
      if (e0 + q < entries && ka[q] != ~0ull - 1ull) {  // uses the key, as a probe does
        Slot* sp = slots + sl[q];
        if (MODE == 0) acc += sp->x + atomicAdd(&sp->z, 0.0) + static_cast<double>(kb[q] & 1ull);
        if (MODE == 1) acc += sp->x + static_cast<double>(kb[q] & 1ull);
        if (MODE == 2) acc += atomicAdd(&sp->z, 0.0);
        if (MODE == 3) {
          atomicAdd(&sp->z, 0.0);
          acc += static_cast<double>(kb[q] & 1ull);
        }
      }
    }
  }
  if (acc == 1234.5678) *sink = acc;  // keeps the loads
}

template <int MODE>
void scatter_probe_mode(const TableDev& t, long long entries, int ilp, int ctas, uint64_t seed, double* sink,
                        cudaStream_t s) {
  if (ilp >= 4)
    scatter_probe_kernel<4, MODE><<<ctas, 256, 0, s>>>(t.slots, t.mask, entries, seed, sink);
  else
    scatter_probe_kernel<1, MODE><<<ctas, 256, 0, s>>>(t.slots, t.mask, entries, seed, sink);
}

cudaError_t scatter_probe(const TableDev& t, long long entries, int ilp, int ctas, uint64_t seed, double* sink,
                          cudaStream_t s, int mode) {
  if (ctas < 1 || mode < 0 || mode > 3) return cudaErrorInvalidValue;
  if (mode == 0) scatter_probe_mode<0>(t, entries, ilp, ctas, seed, sink, s);
  if (mode == 1) scatter_probe_mode<1>(t, entries, ilp, ctas, seed, sink, s);
  if (mode == 2) scatter_probe_mode<2>(t, entries, ilp, ctas, seed, sink, s);
  if (mode == 3) scatter_probe_mode<3>(t, entries, ilp, ctas, seed, sink, s);
  return cudaGetLastError();
}

cudaError_t debug_column(const HamDev& h, Det d, double hdiag, uint64_t* a_out, uint64_t* b_out,
                         double* v_out, int cap, int* n_out, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(n_out, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  debug_column_kernel<<<64, kNT, 0, s>>>(h, d, hdiag, a_out, b_out, v_out, cap, n_out);
  return cudaGetLastError();
}

}  // namespace mcd
