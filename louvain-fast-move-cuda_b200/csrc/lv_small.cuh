// lv_small.cuh -- whole Louvain runs of small graphs, one launch for all levels.
//
// A graph of a few thousand vertices keeps the GPU busy for a microsecond or two per step, but the
// general path spends about 30 launches per pass and level on it (a 193-vertex run: 349 launches,
// 1.44 ms; a 10,000-vertex one: 649 launches, 2.7 ms -- about 4 us each, the work next to
// nothing). Here one thread-block cluster takes a graph through every pass and every level, with
// barriers between the steps: three per pass (commit + binning, gains, apply) and four per
// aggregation. The state stays in the run's global arrays (L2 holds all of it), tables in
// shared memory; the steps are those of lv_kernels.cuh, with the same sums, gains and tie rules.
// Every quantity that decides anything is an exact integer (integer weights) or a double sum
// whose order differs from the general path only as atomics' order does (fp32 weights).
//
// Which graphs (Run::plan_small): those whose tables always fit a block's shared memory (distinct
// keys <= n <= kSmallN) and whose entries one cluster works through faster than the launches cost.
// Class 0: little graphs (kPackN, kPackE), many at once (more than one per SM), run for throughput:
// a CTA of 256 threads each, four per SM, with rolled loops (unrolled, the kernel waited 9-11 stall
// cycles per instruction for instruction fetches: 6.0 -> 3.9 ms for 2,048 graphs of 200-2,000
// vertices). Class 1: the others, for latency: 512 threads with all registers, a cluster of up to 8
// CTAs per graph. (1,024 threads and rolled loops were slower for it: 13.2 against 11.5 ms on
// 1,024 graphs of 2,000-8,000 vertices; the general path takes 15.2.)
// Measured per call, general path -> here: 193 vertices 1.33 -> 0.28 ms, 7,548 vertices / 32 K entries
// 2.95 -> 0.86, 7,925 / 114 K entries 2.63 -> 1.17 (most of the limit), 2,048 graphs of 200-2,000
// vertices 7.7 -> 4.4, 1,024 graphs of 2,000-8,000 vertices 15.8 -> 11.4.
#pragma once

#include <cooperative_groups.h>

#include "lv_kernels.cuh"

namespace lv {

constexpr uint32_t kSmallN = 8192, kSmallE = 131072;  // what k_small takes at all
constexpr uint32_t kPackN = 2048, kPackE = 16384;     // class 0
constexpr int kSmallClasses = 2;
constexpr int kSmallNT[kSmallClasses] = {256, 512};
constexpr int kSmallMinB[kSmallClasses] = {4, 1};
constexpr int kSmallMaxCtas = 8;
// entries per lane in flight in the gain and apply steps, rolled loops: see above
template <int NT> constexpr bool kCompact = NT != 512;
template <int NT> constexpr int kSmallBatch = kCompact<NT> ? 2 : kBatch;
template <int NT> constexpr int kSmallApply = kCompact<NT> ? 2 : kApplyBatch;
constexpr int kSmallShare = 2048;  // entries that make a further CTA of the cluster worth its barriers
constexpr int kSmallLists = 4;  // rows of up to 8 and 32 entries, rows for a warp, rows for a CTA

struct SmallCfg {
  int mode, fast_first;
  uint32_t max_levels;
  uint32_t cap;   // table slots of a CTA (2 x the class's vertex limit)
};

// Counters of a cluster, in its first CTA's shared memory. Lists and movers alternate by pass parity.
struct SmallCnt {
  uint32_t list[2][kSmallLists];
  uint32_t movers[2], long_movers[2];  // movers with rows of up to 32 entries / longer
  uint32_t n2, n_cta;          // aggregation: next vertices; communities for a whole CTA
  uint32_t next;               // the graph being worked on
  unsigned long long I;        // internal weight: u64, or double bits
  unsigned long long S[2][kSmallMaxCtas];  // per CTA: sum of squared totals, by parity
};

// Everything the steps of one graph share (registers; uniform over the cluster).
template <bool WINT, int NT>
struct SmallRun {
  using Tr = WTraits<WINT>;
  using Acc = typename Tr::Acc;
  using Wt = typename Tr::W;
  const Dev& D;
  Dev L;             // the pointers of the current level that the shared steps read
  SmallCnt* cnt;
  uint32_t cta, ncta, gw, nw, tid, nt;  // this CTA, warp and thread in the cluster; their numbers
  int lane, wid;
  uint32_t cap, wcap;  // table slots per CTA / per warp
  uint32_t* keys;
  Acc* vals;
  unsigned long long* slots;
  uint16_t* list;
  uint32_t* lista;
  uint32_t vb, n;    // the graph's first vertex, its vertices at this level
  uint32_t *rs, *len;  // row start and length per vertex
  double *k;
  double m, two_m2, inv_m, inv_2m2;
  bool unit;
  uint32_t err;

  __device__ __forceinline__ void sync() const {
    if (ncta == 1) __syncthreads();
    else cooperative_groups::this_cluster().sync();
  }
  __device__ __forceinline__ VtxCtx vtx(uint32_t v) const {
    VtxCtx x;
    x.unit = unit;
    x.rs = rs[v];
    x.re = x.rs + len[v];
    x.cv = L.comm[v];
    x.kv = k[v];
    x.a_own = L.a[x.cv];
    x.m = m;
    x.two_m2 = two_m2;
    x.own_minus_k = __dsub_rn(x.a_own, x.kv);
    x.inv_m = inv_m;
    x.inv_2m2 = inv_2m2;
    x.ng = n;
    return x;
  }
  // a table of this warp (or, with w = 0 and the whole capacity, of this CTA)
  __device__ __forceinline__ ScratchTable<WINT> table(uint32_t at, uint32_t c) const {
    return ScratchTable<WINT>{keys + at, vals + at, slots + at, c - 1u, 32u - log2_pow2(c)};
  }
};

// Sum over the CTA into the cluster's per-CTA slot; fixed order, so repeatable.
template <bool WINT, int NT>
__device__ __forceinline__ void small_put_s(const SmallRun<WINT, NT>& R, unsigned long long su, double sf, int par,
                                            unsigned long long* red) {
  if (WINT) su = warp_sum(su);
  else su = (unsigned long long)__double_as_longlong(warp_sum(sf));
  if (R.lane == 0) red[R.wid] = su;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    double f = 0.0;
    for (int i = 0; i < (NT / 32); ++i) {
      if (WINT) t += red[i];
      else f = __dadd_rn(f, __longlong_as_double((long long)red[i]));
    }
    R.cnt->S[par][R.cta] = WINT ? t : (unsigned long long)__double_as_longlong(f);
  }
}

// Start of a level (init) or end of a pass: commits the pass's moves, packs the (total, community)
// words, sums the squared totals and lists the vertices active in pass `it`.
template <bool WINT, int NT>
__device__ __forceinline__ void small_commit(SmallRun<WINT, NT>& R, bool init, uint32_t it, int par,
                                             unsigned long long* red, unsigned long long& act_e,
                                             unsigned long long& act_v) {
  const Dev& D = R.D;
  unsigned long long su = 0;
  double sf = 0.0;
  act_e = act_v = 0;
  for (uint32_t base = R.gw * 32u; base < R.n; base += R.nw * 32u) {
    const uint32_t i = base + R.lane, v = R.vb + i;
    const bool live = i < R.n;
    int b = -1;
    if (live) {
      uint32_t c;
      double own;  // the total of community v
      if (init) {
        c = v;
        own = R.k[v];
        D.comm[v] = v;
        D.new_comm[v] = v;
        D.a[v] = own;
        D.cn[v] = ((unsigned long long)v << 32) | v;
        D.active_it[v] = 0;
        D.cd[v] = 0ull;
      } else {
        c = D.new_comm[v];
        own = D.a[v];
        if (D.comm[v] != c) {
          D.comm[v] = c;
          D.cn[v] = ((unsigned long long)c << 32) | c;
        }
      }
      if (WINT) {
        D.ca[v] = ((unsigned long long)(uint32_t)(init ? own : D.a[c]) << 32) | c;
        const unsigned long long x = (unsigned long long)own;
        su += x * x;
      } else {
        sf = __dadd_rn(sf, __dmul_rn(own, own));
      }
      if (init || D.active_it[v] == it) {
        const uint32_t d = R.len[v];
        if (d <= 32) b = d <= 8 ? 0 : 1;
        else b = table_cap(d, R.n) <= R.wcap ? 2 : 3;
        act_e += d;
        ++act_v;
      }
    }
    // lane q claims list q's space: the claims of all lists are one atomic latency
    uint32_t mine = 0, want = 0, before = 0;
#pragma unroll
    for (int q = 0; q < kSmallLists; ++q) {
      const unsigned mk = __ballot_sync(kFull, b == q);
      if (R.lane == q) want = __popc(mk);
      if (b == q) before = __popc(mk & lanemask_lt());
    }
    if (want) mine = atomicAdd(&R.cnt->list[par][R.lane], want);
    const uint32_t pos = __shfl_sync(kFull, mine, b < 0 ? 0 : b) + before;
    if (b >= 0) D.bins[b][R.vb + pos] = v;
  }
  small_put_s<WINT, NT>(R, su, sf, par, red);
}

// Gains of the listed vertices; movers appended to the list of this parity.
template <bool WINT, int NT>
__device__ __forceinline__ void small_gains(SmallRun<WINT, NT>& R, int par, bool fast, bool lowest,
                                            uint32_t (*s_mov)[64], unsigned long long* red,
                                            typename WTraits<WINT>::Acc* red_self, uint32_t* s_nl) {
  using Tr = WTraits<WINT>;
  using Acc = typename Tr::Acc;
  const Dev& D = R.D;
  const Dev& L = R.L;
  // (the list of movers with long rows lies in `members`, unused during passes)
  MoverStage mv{s_mov[R.wid], 0u, D.members + R.vb, &R.cnt->long_movers[par], nullptr, 0u};
  uint32_t nl_[kSmallLists];
#pragma unroll
  for (int q = 0; q < kSmallLists; ++q) nl_[q] = R.cnt->list[par][q];
  // rows whose tables need the whole CTA
  const uint32_t nc = nl_[3];
  for (uint32_t i = R.cta; i < nc; i += R.ncta) {
    const uint32_t v = D.bins[3][R.vb + i];
    const VtxCtx x = R.vtx(v);
    unsigned long long best = 0;
    if (fast) {
      best = fast_scan<WINT, kSmallBatch<NT>>(L, x, v, x.rs + threadIdx.x, NT);
    } else {
      const ScratchTable<WINT> tbl = R.table(0, table_cap(x.re - x.rs, x.ng));
      if (threadIdx.x == 0) *s_nl = 0;
      __syncthreads();
      Acc self_acc = Acc(0);
      insert_list<WINT, true, kSmallBatch<NT>>(L, x, v, threadIdx.x, NT, kFull, tbl, R.list, R.lista, s_nl, self_acc, R.err);
      self_acc = warp_sum(self_acc);
      if (R.lane == 0) red_self[R.wid] = self_acc;
      __syncthreads();
      Acc self_all = Acc(0);
#pragma unroll
      for (int j = 0; j < (NT / 32); ++j) self_all += red_self[j];
      best = list_scan<WINT, kSmallBatch<NT>>(L, x, tbl, R.list, R.lista, threadIdx.x, *s_nl, NT, Tr::to_float(self_all), lowest);
    }
    best = team_max<32>(best, kFull);
    if (R.lane == 0) red[R.wid] = best;
    __syncthreads();
    if (R.wid == 0) {
      best = team_max<32>(R.lane < (NT / 32) ? red[R.lane] : 0ull, kFull);
      const uint32_t c = key_comm(best, lowest);
      mv.add(D, R.lane == 0 && best && c != x.cv && (!fast || v <= c), v, x.cv, c, 0u);
    }
    __syncthreads();
  }
  // rows for a warp, then the short rows (teams of 8 lanes up to 32 entries, of 2 lanes up to 8): the
  // tiles of all lists are dealt to the warps in turn, so that the lists of a small graph run
  // side by side
  auto load = [&](uint32_t v) { return R.vtx(v); };
  uint32_t w0 = R.gw;  // this warp's first tile of the next list
  if (fast) {
    for (int b = 2; b >= 0; --b) {
      const uint32_t T = b == 2 ? 32u : b == 1 ? 8u : 2u, per = 32u / T;
      const uint32_t tiles = (nl_[b] + per - 1) / per;
      if (b == 1) mv.switch_to(D.movers + R.vb, &R.cnt->movers[par]);
      for (uint32_t t = w0; t < tiles; t += R.nw)
        fast_rows<WINT, kSmallBatch<NT>>(L, D.bins[b] + R.vb, t * per + R.lane / T, nl_[b], T, mv, load);
      w0 = (w0 + R.nw - tiles % R.nw) % R.nw;
    }
  } else {
    uint16_t* list = R.list + R.wid * (R.wcap / 2);
    uint32_t* lista = R.lista + R.wid * (R.wcap / 2);
    for (uint32_t i = w0; i < nl_[2]; i += R.nw) {
      const uint32_t v = D.bins[2][R.vb + i];
      const VtxCtx x = R.vtx(v);
      const ScratchTable<WINT> tbl = R.table(R.wid * R.wcap, table_cap(x.re - x.rs, x.ng));
      Acc self_acc = Acc(0);
      const uint32_t nl = insert_list<WINT, false, kSmallBatch<NT>>(L, x, v, R.lane, 32, kFull, tbl, list, lista, nullptr, self_acc, R.err);
      self_acc = warp_sum(self_acc);
      __syncwarp();
      unsigned long long best = list_scan<WINT, kSmallBatch<NT>>(L, x, tbl, list, lista, R.lane, nl, 32, Tr::to_float(self_acc), lowest);
      best = team_max<32>(best, kFull);
      __syncwarp();  // the listed slots are empty again before the next row inserts
      const uint32_t c = key_comm(best, lowest);
      mv.add(D, R.lane == 0 && best && c != x.cv, v, x.cv, c, 0u);
    }
    mv.switch_to(D.movers + R.vb, &R.cnt->movers[par]);
    w0 = (w0 + R.nw - nl_[2] % R.nw) % R.nw;
    for (uint32_t t = w0; t * 4u < nl_[1]; t += R.nw)
      short_rows<8, WINT, kCompact<NT>>(L, D.bins[1] + R.vb, t * 4u + (R.lane >> 3), nl_[1], lowest, R.unit, mv, load);
    w0 = (w0 + R.nw - (nl_[1] + 3u) / 4u % R.nw) % R.nw;
    for (uint32_t t = w0; t * 16u < nl_[0]; t += R.nw)
      short_rows<2, WINT, kCompact<NT>>(L, D.bins[0] + R.vb, t * 16u + (R.lane >> 1), nl_[0], lowest, R.unit, mv, load);
  }
  mv.finish();
}

// Totals, activity and the internal weight of the pass's moves (as k_apply): a warp takes one mover
// with a long row, or 32 others.
template <bool WINT, int NT>
__device__ __forceinline__ void small_apply(SmallRun<WINT, NT>& R, uint32_t count, uint32_t longs, uint32_t it) {
  const Dev& D = R.D;
  long long di = 0;
  double df = 0.0;
  const uint32_t steps = longs + (count + 31u) / 32u;
  for (uint32_t t = R.gw; t < steps; t += R.nw) {
    uint32_t rs = 0, len = 0, old = 0, nw = 0;
    const uint32_t idx = (t - longs) * 32u + R.lane;
    if (t < longs ? R.lane == 0 : idx < count) {
      const uint32_t v = t < longs ? D.members[R.vb + t] : D.movers[R.vb + idx];
      old = D.comm[v];
      nw = D.new_comm[v];
      rs = R.rs[v];
      len = R.len[v];
      const double kv = R.k[v];
      atomicAdd(&D.a[nw], kv);
      atomicAdd(&D.a[old], -kv);
    }
    apply_rows<WINT, kSmallApply<NT>>(R.L, rs, len, old, nw, it, R.unit, [&](int, int f, double wt, uint32_t wi) {
      if (WINT) di += (long long)f * (long long)wi;
      else df += (double)f * wt;
    });
  }
  if (WINT) {
    di = warp_sum(di);
    if (R.lane == 0 && di) atomicAdd(&R.cnt->I, (unsigned long long)di);
  } else {
    df = warp_sum(df);
    if (R.lane == 0 && df != 0.0) atomicAdd(reinterpret_cast<double*>(&R.cnt->I), df);
  }
}

// Whether a warp contracts a community of degree sum dsum: its table fits the warp's and it is not long.
__device__ __forceinline__ bool small_for_warp(uint32_t dsum, uint32_t n2, uint32_t wcap) {
  return table_cap(dsum, n2) <= wcap && dsum <= 2048u;
}

// New ids of the nonempty communities and where their members and entries go, by the cluster's
// first CTA: one scan over packed (degree sum, members, nonempty) words. `ids`: new id per old
// community; rs2: start of the new row's space; degree sums go to bins[4] (no list is live now).
template <bool WINT, int NT>
__device__ __forceinline__ void small_renumber(SmallRun<WINT, NT>& R, uint32_t e0, uint32_t* ids, uint32_t* rs2,
                                               unsigned long long* red) {
  const Dev& D = R.D;
  constexpr uint32_t PER = kSmallN / NT;
  const uint32_t per = (R.n + NT - 1) / NT;  // <= PER
  const uint32_t i0 = threadIdx.x * per;
  // degree sum < 2^32, members <= 8192
  auto word = [](unsigned long long x) { return x ? (x << 32) | ((x >> 32) << 16) | 1ull : 0ull; };
  unsigned long long own = 0, xs[PER];
#pragma unroll
  for (uint32_t j = 0; j < PER; ++j) {
    xs[j] = j < per && i0 + j < R.n ? D.cd[R.vb + i0 + j] : 0ull;
    own += word(xs[j]);
  }
  unsigned long long tot;
  unsigned long long at = block_excl_scan<unsigned long long, NT>(own, red, &tot);
  const uint32_t n2 = (uint32_t)tot & 0xFFFFu;
#pragma unroll
  for (uint32_t j = 0; j < PER; ++j) {
    const unsigned long long x = xs[j];
    if (!x) continue;
    const uint32_t s = R.vb + ((uint32_t)at & 0xFFFFu), dsum = (uint32_t)x;
    ids[R.vb + i0 + j] = s;
    D.rowB[s] = R.vb + ((uint32_t)(at >> 16) & 0xFFFFu);  // first member
    D.newdeg[s] = (uint32_t)(x >> 32);                    // members
    rs2[s] = e0 + (uint32_t)(at >> 32);
    D.bins[4][s] = dsum;
    if (!small_for_warp(dsum, n2, R.wcap)) D.bins[5][R.vb + atomicAdd(&R.cnt->n_cta, 1u)] = s;
    at += word(x);
  }
  if (threadIdx.x == 0) {
    R.cnt->n2 = n2;
    R.cnt->I = 0ull;  // the contraction adds the next level's self-loop weight
  }
  static_assert(PER * NT >= kSmallN && kSmallN < 65536, "16-bit fields of the scan");
}

// The contracted rows: emitted in list order into the row's space of the other entry buffers.
template <bool WINT, int NT>
__device__ __forceinline__ void small_contract(SmallRun<WINT, NT>& R, uint32_t* colN, typename WTraits<WINT>::W* wN,
                                               uint32_t* rs2, uint32_t* len2, double* k2, uint32_t* mrs,
                                               uint32_t* mex, uint32_t* shu, double* shd, uint32_t* s_nl) {
  using Tr = WTraits<WINT>;
  using Acc = typename Tr::Acc;
  using Wt = typename Tr::W;
  const Dev& D = R.D;
  const Wt* w = reinterpret_cast<const Wt*>(R.L.w);
  const uint32_t n2 = R.cnt->n2;
  const uint32_t lt = lanemask_lt();
  auto out_w = [](Acc x) { return contracted_weight<WINT>(x); };
  auto finish = [&](uint32_t s, uint32_t tb, uint32_t nl, Acc self, double ksum) {  // one thread
    const bool has = self != Acc(0);  // weights are positive
    if (has) {
      const Wt x = out_w(self);
      colN[tb + nl] = s;
      wN[tb + nl] = x;
      ksum += Tr::w_double(x);
      if (WINT) atomicAdd(&R.cnt->I, (unsigned long long)x);
      else atomicAdd(reinterpret_cast<double*>(&R.cnt->I), Tr::w_double(x));
    }
    len2[s] = nl + (has ? 1u : 0u);
    k2[s] = ksum;
  };
  // communities for the whole CTA: members NT at a time, entries spread over all threads
  const uint32_t nc = R.cnt->n_cta;
  for (uint32_t i = R.cta; i < nc; i += R.ncta) {
    const uint32_t s = D.bins[5][R.vb + i], mb = D.rowB[s], me = mb + D.newdeg[s], tb = rs2[s];
    const ScratchTable<WINT> tbl = R.table(0, table_cap(D.bins[4][s], n2));
    if (threadIdx.x == 0) *s_nl = 0;
    __syncthreads();
    Acc self = Acc(0);
    for (uint32_t b = mb; b < me; b += NT) {
      uint32_t rs = 0, len = 0;
      if (b + threadIdx.x < me) {
        const uint32_t v = D.members[b + threadIdx.x];
        rs = R.rs[v];
        len = R.len[v];
      }
      uint32_t total;
      const uint32_t ex = block_excl_scan<uint32_t, NT>(len, shu, &total);
      mrs[threadIdx.x] = rs;
      mex[threadIdx.x] = ex;
      __syncthreads();
      const uint32_t cnt = min((uint32_t)NT, me - b);
      for (uint32_t jb = 0; jb < total; jb += NT) {
        const uint32_t j = jb + threadIdx.x;
        bool made = false;
        uint32_t slot = 0;
        if (j < total) {
          uint32_t lo = 0, hi = cnt;
          while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (mex[mid] <= j) lo = mid; else hi = mid;
          }
          const uint32_t e = mrs[lo] + (j - mex[lo]);
          const uint32_t d = D.new_comm[R.L.col[e]];
          const Acc wv = R.unit ? Acc(1) : (Acc)w[e];
          if (d == s) {
            self += wv;
          } else {
            const int r = tbl.add_at(d, wv, slot);
            if (!r) R.err |= kErrTableFull;
            made = r == 2;
          }
        }
        const unsigned mk = __ballot_sync(kFull, made);
        if (mk) {
          uint32_t b0 = 0;
          if (R.lane == 0) b0 = atomicAdd(s_nl, (uint32_t)__popc(mk));
          b0 = __shfl_sync(kFull, b0, 0);
          if (made) R.list[b0 + __popc(mk & lt)] = (uint16_t)slot;
        }
      }
      __syncthreads();
    }
    self = block_sum<NT>(self, reinterpret_cast<Acc*>(shd));  // (its barriers order the list)
    const uint32_t nl = *s_nl;
    double ksum = 0.0;
    for (uint32_t q = threadIdx.x; q < nl; q += NT) {
      const uint32_t sl = R.list[q];
      uint32_t d;
      Acc sum;
      tbl.load(sl, d, sum);
      tbl.clear(sl);
      const Wt x = out_w(sum);
      colN[tb + q] = d;
      wN[tb + q] = x;
      ksum += Tr::w_double(x);
    }
    ksum = block_sum<NT>(ksum, shd);
    if (threadIdx.x == 0) finish(s, tb, nl, self, ksum);
    __syncthreads();
  }
  // small communities: 8 lanes each, four entries per lane, sums by comparing all pairs
  for (uint32_t base = R.gw * 4u; base < n2; base += R.nw * 4u) {
    const uint32_t i = base + ((uint32_t)R.lane >> 3), s = R.vb + i;
    const uint32_t tl = R.lane & 7;
    uint32_t mb = 0, mc = 0, tb = 0, dsum = 0;
    if (i < n2) {
      dsum = D.bins[4][s];
      if (dsum <= kPairMax) {
        mb = D.rowB[s];
        mc = D.newdeg[s];
        tb = rs2[s];
      } else {
        dsum = 0;
      }
    }
    if (!__any_sync(kFull, dsum > 0)) continue;
    contract_pairs<WINT, kCompact<NT>>(
        D.members, D.new_comm, R.L.col, w, R.unit, s, mb, mc, tb, dsum, colN, wN,
        [&](uint32_t v, uint32_t& rs, uint32_t& len) { rs = R.rs[v]; len = R.len[v]; }, finish);
  }
  // other communities for a warp: members 32 at a time, entries spread over the lanes
  uint16_t* list = R.list + R.wid * (R.wcap / 2);
  for (uint32_t i = R.gw; i < n2; i += R.nw) {
    const uint32_t s = R.vb + i, mb = D.rowB[s], me = mb + D.newdeg[s], tb = rs2[s], dsum = D.bins[4][s];
    if (dsum <= kPairMax || !small_for_warp(dsum, n2, R.wcap)) continue;
    const ScratchTable<WINT> tbl = R.table(R.wid * R.wcap, table_cap(dsum, n2));
    Acc self = Acc(0);
    uint32_t nl = 0;
    for (uint32_t b = mb; b < me; b += 32) {
      uint32_t rs = 0, len = 0;
      if (b + R.lane < me) {
        const uint32_t v = D.members[b + R.lane];
        rs = R.rs[v];
        len = R.len[v];
      }
      contract_rows<WINT, kCompact<NT> ? 1 : kContractBatch>(D.new_comm, R.L.col, w, R.unit, rs, len, s, tbl, list, nl, self, R.err);
    }
    self = warp_sum(self);
    __syncwarp();
    double ksum = 0.0;
    for (uint32_t q = R.lane; q < nl; q += 32) {
      const uint32_t sl = list[q];
      uint32_t d;
      Acc sum;
      tbl.load(sl, d, sum);
      tbl.clear(sl);
      const Wt x = out_w(sum);
      colN[tb + q] = d;
      wN[tb + q] = x;
      ksum += Tr::w_double(x);
    }
    ksum = warp_sum(ksum);
    if (R.lane == 0) finish(s, tb, nl, self, ksum);
    __syncwarp();
  }
}

// Graphs ids[0, count), largest first, taken from the counter *work by one cluster at a time. Runs
// from the level-0 input (k_prep*) to the final communities; ends at once when the input was
// found invalid. The pass and level loops end as those of the general path do (and at its guards).
template <bool WINT, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_small(int dslot, const uint32_t* ids, uint32_t count,
                                                          uint32_t* work, SmallCfg cfg) {
  using Tr = WTraits<WINT>;
  using Acc = typename Tr::Acc;
  using Wt = typename Tr::W;
  const Dev& D = c_dev[dslot];
  Ctrl* C = D.ctrl;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SmallCnt s_cnt;
  __shared__ uint32_t s_mov[(NT / 32)][64];
  __shared__ uint32_t mrs[NT], mex[NT], shu[33], s_nl;
  __shared__ unsigned long long red[33];
  __shared__ Acc red_self[(NT / 32)];
  __shared__ double shd[33];
  if (C->input_err) return;
  auto cluster = cooperative_groups::this_cluster();
  SmallRun<WINT, NT> R{D};
  R.ncta = cluster.num_blocks();
  R.cta = cluster.block_rank();
  R.cnt = R.cta == 0 ? &s_cnt : cluster.map_shared_rank(&s_cnt, 0);
  R.lane = threadIdx.x & 31;
  R.wid = threadIdx.x >> 5;
  R.gw = R.cta * (NT / 32) + R.wid;
  R.nw = R.ncta * (NT / 32);
  R.tid = R.cta * NT + threadIdx.x;
  R.nt = R.ncta * NT;
  R.cap = cfg.cap;
  R.wcap = cfg.cap / (NT / 32);
  constexpr size_t kSlotBytes = WINT ? 8 : 4 + sizeof(Acc);
  R.keys = reinterpret_cast<uint32_t*>(smem);
  R.vals = reinterpret_cast<Acc*>(smem + (size_t)R.cap * sizeof(uint32_t));
  R.slots = reinterpret_cast<unsigned long long*>(smem);
  R.list = reinterpret_cast<uint16_t*>(smem + (size_t)R.cap * kSlotBytes);
  R.lista = reinterpret_cast<uint32_t*>(smem + (size_t)R.cap * (kSlotBytes + 1));
  R.err = 0;
  {
    const ScratchTable<WINT> all = R.table(0, R.cap);
    for (uint32_t i = threadIdx.x; i < R.cap; i += NT) all.clear(i);
  }
  for (;;) {
    R.sync();  // the previous graph is done with the counters (and every CTA has started)
    if (R.tid == 0) R.cnt->next = atomicAdd(work, 1u);
    R.sync();
    const uint32_t gi = R.cnt->next;
    if (gi >= count) break;
    const uint32_t g = ids[gi];
    GraphState* st = &D.gs[g];
    const uint32_t vb = st->vb, ve = st->ve;
    R.vb = vb;
    R.n = ve - vb;
    R.m = st->m;
    R.two_m2 = st->two_m2;
    R.inv_m = st->inv_m;
    R.inv_2m2 = st->inv_2m2;
    R.unit = unit_weights<WINT>(C);
    const uint32_t e0 = D.row[vb];
    uint32_t *rs2 = D.bins[7], *len2 = D.bins[8];  // the next level's rows
    R.rs = D.hub_off;
    R.len = D.hubtab;
    double* k2 = D.kB;
    R.k = D.k;
    R.L.col = D.col;
    R.L.w = D.w;
    uint32_t* colN = D.colB;
    Wt* wN = reinterpret_cast<Wt*>(D.wB);
    R.L.comm = D.comm;
    R.L.new_comm = D.new_comm;
    R.L.a = D.a;
    R.L.ca = D.ca;
    R.L.cn = D.cn;
    R.L.active_it = D.active_it;
    for (uint32_t v = vb + R.tid; v < ve; v += R.nt) {
      const uint32_t r = D.row[v];
      R.rs[v] = r;
      R.len[v] = D.row[v + 1] - r;
    }
    if (R.tid == 0) {
      for (int p = 0; p < 2; ++p) {
        for (int q = 0; q < kSmallLists; ++q) R.cnt->list[p][q] = 0;
        R.cnt->movers[p] = R.cnt->long_movers[p] = 0;
      }
      R.cnt->I = st->I;
    }
    R.sync();
    uint32_t level = 0, total_iters = 0, moved = 0, it = 0;
    unsigned long long act_e = 0, act_v = 0, t_opt = 0, t_optk = 0, t_agg = 0;
    double Q = 0.0;
    unsigned long long i_end = 0;
    for (;;) {
      // ---- passes of a level
      const unsigned long long t0 = global_ns();
      double Q_level = 0.0;
      uint32_t iters = 0;
      int par = 0;
      bool init = true;
      it = 0;
      for (;;) {
        unsigned long long ne, nv;  // listed by this thread
        small_commit<WINT, NT>(R, init, it, par, red, ne, nv);
        R.sync();
        double S = 0.0;
        {
          unsigned long long su = 0;
          for (uint32_t c = 0; c < R.ncta; ++c) {
            const unsigned long long x = R.cnt->S[par][c];
            if (WINT) su += x;
            else S = __dadd_rn(S, __longlong_as_double((long long)x));
          }
          if (WINT) S = (double)su;
        }
        const unsigned long long ib = R.cnt->I;
        const double I = WINT ? (double)ib : __longlong_as_double((long long)ib);
        const double q = modularity_of(I, S, R.m);
        i_end = ib;
        if (init) {
          Q = Q_level = q;
        } else {
          const double dq = __dsub_rn(q, Q);
          Q = q;
          ++iters;
          ++total_iters;
          moved = R.cnt->movers[par ^ 1] + R.cnt->long_movers[par ^ 1];
          if (!(dq > C->threshold) || iters > C->max_iterations) break;
          if (total_iters > kGuardPasses) { R.err |= kErrLoop; break; }
        }
        init = false;
        act_e += ne;
        act_v += nv;
        const bool fast = cfg.fast_first && iters == 0;
        const bool lowest = fast || cfg.mode == 1 || (cfg.mode == 2 && iters <= 4);
        const unsigned long long t1 = global_ns();
        small_gains<WINT, NT>(R, par, fast, lowest, s_mov, red, red_self, &s_nl);
        R.sync();
        t_optk += global_ns() - t1;
        if (R.tid == 0) {  // the other parity's counters are free until the next commit
          for (int q = 0; q < kSmallLists; ++q) R.cnt->list[par ^ 1][q] = 0;
          R.cnt->movers[par ^ 1] = R.cnt->long_movers[par ^ 1] = 0;
        }
        small_apply<WINT, NT>(R, R.cnt->movers[par], R.cnt->long_movers[par], it);
        R.sync();
        par ^= 1;
        ++it;
      }
      const unsigned long long t2 = global_ns();
      t_opt += t2 - t0;
      // ---- aggregation
      uint32_t cont = __dsub_rn(Q, Q_level) > C->threshold ? 1u : 0u;
      if (cfg.max_levels > 0 && level + 1 >= cfg.max_levels) cont = 0;
      if (level >= kGuardLevels) { R.err |= kErrLoop; cont = 0; }
      if (R.tid == 0) R.cnt->n_cta = 0;
      for (uint32_t i = R.tid; i < R.n; i += R.nt) {
        const uint32_t v = vb + i;
        const unsigned long long old = atomicAdd(&D.cd[D.comm[v]], (1ull << 32) | R.len[v]);
        D.rank[v] = (uint32_t)(old >> 32);
      }
      R.sync();
      if (R.cta == 0) small_renumber<WINT, NT>(R, e0, D.bins[6], rs2, red);
      R.sync();
      const uint32_t n2 = R.cnt->n2;
      for (uint32_t i = R.tid; i < ve - vb; i += R.nt) {  // input vertices
        const uint32_t s = D.bins[6][D.comm[D.best[vb + i]]];
        if (cont) {
          D.best[vb + i] = s;
        } else {
          D.best[vb + i] = s - vb;
          D.out[vb + i] = (int32_t)(s - vb);
        }
      }
      if (!cont) {
        if (R.tid == 0) {
          st->Q = Q;
          st->Q_level = Q_level;
          st->I = i_end;
          st->iters = iters;
          st->total_iters = total_iters;
          st->level = level;
          st->moved = moved;
          st->n_best = n2;
          st->cont = 0;
          st->agg = 0;
          st->phase = kFinished;
          st->vb = st->ve = 0;
        }
        t_agg += global_ns() - t2;
        ++level;
        break;
      }
      for (uint32_t i = R.tid; i < R.n; i += R.nt) {
        const uint32_t v = vb + i, s = D.bins[6][D.comm[v]];
        D.new_comm[v] = s;
        D.members[D.rowB[s] + D.rank[v]] = v;
      }
      if (R.tid == 0) {
        for (int p = 0; p < 2; ++p) {
          for (int q = 0; q < kSmallLists; ++q) R.cnt->list[p][q] = 0;
          R.cnt->movers[p] = R.cnt->long_movers[p] = 0;
        }
      }
      R.sync();
      small_contract<WINT, NT>(R, colN, wN, rs2, len2, k2, mrs, mex, shu, shd, &s_nl);
      R.sync();
      // the new rows become the level's
      { uint32_t* t = R.rs; R.rs = rs2; rs2 = t; }
      { uint32_t* t = R.len; R.len = len2; len2 = t; }
      { double* t = R.k; R.k = k2; k2 = t; }
      { uint32_t* t = colN; colN = R.L.col; R.L.col = t; }
      { Wt* t = wN; wN = reinterpret_cast<Wt*>(R.L.w); R.L.w = t; }
      R.n = n2;
      R.unit = false;
      ++level;
      t_agg += global_ns() - t2;
    }
    act_e = warp_sum(act_e);
    act_v = warp_sum(act_v);
    if (R.lane == 0) {
      atomicAdd(&C->act_entries_total, act_e);
      atomicAdd(&C->act_vertices_total, act_v);
    }
    if (R.tid == 0) {
      atomicMax(&C->small_levels, level);
      if (gi == 0) {  // phase times of a run: the largest graph's
        C->t_opt_ns += t_opt;
        C->t_optk_ns += t_optk;
        C->t_agg_ns += t_agg;
      }
    }
  }
  R.sync();  // no CTA leaves while another still reads the counters in its shared memory
  if (R.err) report_err(C, R.err, 9);  // k_small
}

}  // namespace lv
