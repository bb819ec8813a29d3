// Host planner of the closed sigma (tps_ci_matvec, src/tpsci_outer.jl:462-527).
//
// The reference finds, for every bra, every ket of the sector fock_bra - trans
// and filters them with check_term (src/type_ClusteredTerm.jl:92-176): a ket
// couples through a term iff it equals the bra on every cluster the term does
// not touch.  Here that test is turned into a join: the rows of every
// (Fock sector, active-cluster set) are sorted by their spectator key (the
// local states on the untouched clusters), and for each (bra sector,
// transfer, active set) the bra and ket key lists are merge-joined.  Each
// matching key gives one work item = a dense block of (bra, ket, term)
// triples that all pass check_term.  Each bra row of a work item, with up to
// lane_kets of its kets, becomes one lane job of the sigma kernel; lane jobs are
// sorted so that a warp's 32 lanes do the same kind and amount of work.
#include <algorithm>
#include <array>
#include <cstring>
#include <unordered_map>

#include "fcg_internal.h"
#ifdef _OPENMP
#include <omp.h>
#endif

namespace fcg {
namespace {

inline int32_t TT(const std::vector<int32_t>& trm, int t, int col) { return trm[size_t(t) * kTrmCols + col]; }

// Fock sector key: 4 bits per (n_alpha, n_beta) entry; valid for <= 15 electrons/spin/cluster.
inline bool fock_key(const int16_t* f, int N, uint64_t* key) {
  uint64_t k = 0;
  for (int i = 0; i < 2 * N; ++i) {
    if (f[i] < 0 || f[i] > 15) return false;
    k |= uint64_t(f[i]) << (4 * i);
  }
  *key = k;
  return true;
}

struct Group {
  uint64_t key;
  int32_t start;  // relative to the (sector, set) permutation
  int32_t count;
};

// A lane job while planning: its term shape (nbody) and planner cost ride along for the sort.
struct PJob {
  LaneJob j;
  int32_t cost;
  int32_t nbody;
  bool block;  // of a block item: after the jobs of the other items
};

// What an item's lane jobs need besides the item.
struct ItemMeta {
  int64_t step_cost;  // planner cost of one ket of a lane job
  int32_t nbody;
  bool block;
};

}  // namespace

TermTables term_tables(const ProblemInfo& pi) {
  const Dressing& d = *pi.dressing;
  return TermTables{pi.trm->data(), pi.dress->data(), d.w_index.data(), d.w_mb.data(), d.rep.data(),
                    pi.blk_index->data(), pi.blocks->data(), pi.nmax + 1};
}

std::string term_lists(const ProblemInfo& pi, TermLists& L) {
  const std::vector<int32_t>& trm = *pi.trm;
  L = TermLists();
  std::unordered_map<uint32_t, int> mask_id;
  // (transfer, set, term) of every term; sets numbered in order of first appearance
  std::vector<std::array<int32_t, 3>> key(size_t(pi.n_terms));
  for (int t = 0; t < pi.n_terms; ++t) {
    const int nb = TT(trm, t, 0);
    uint32_t m = 0;
    for (int o = 0; o < nb; ++o) m |= 1u << TT(trm, t, 2 + o);
    auto it = mask_id.find(m);
    int s;
    if (it == mask_id.end()) {
      s = int(L.masks.size());
      mask_id[m] = s;
      L.masks.push_back(m);
    } else {
      s = it->second;
    }
    const int tr = TT(trm, t, 1);
    if (tr < 0 || tr >= pi.n_trans) return "term transfer id out of range";
    key[size_t(t)] = {tr, s, t};
  }
  std::stable_sort(key.begin(), key.end(), [](const std::array<int32_t, 3>& x, const std::array<int32_t, 3>& y) {
    return x[0] != y[0] ? x[0] < y[0] : x[1] < y[1];
  });
  L.first_of_tr.assign(size_t(pi.n_trans) + 1, 0);
  L.off.push_back(0);
  size_t q = 0;
  for (int tr = 0; tr < pi.n_trans; ++tr) {
    L.first_of_tr[tr] = int32_t(L.tr.size());
    while (q < key.size() && key[q][0] == tr) {
      const int s = key[q][1];
      L.tr.push_back(tr);
      L.set.push_back(s);
      for (; q < key.size() && key[q][0] == tr && key[q][1] == s; ++q) L.terms.push_back(key[q][2]);
      L.off.push_back(int32_t(L.terms.size()));
    }
  }
  L.first_of_tr[pi.n_trans] = int32_t(L.tr.size());
  // lists that may run as block jobs: three or four active clusters, and a W column short enough
  // once one index is contracted, whichever that is
  L.block.assign(L.tr.size(), 0);
  for (size_t j = 0; j < L.tr.size(); ++j) {
    bool ok = true;
    for (int q2 = L.off[j]; q2 < L.off[j + 1] && ok; ++q2) {
      const TermDress& d = (*pi.dress)[size_t(L.terms[size_t(q2)])];
      ok = d.nrem == 2 || d.nrem == 3;
      for (int q3 = 0; ok && q3 < d.nrem; ++q3) ok = d.rest_len / d.rem_dim[q3] <= kBlockU;
    }
    L.block[j] = ok ? 1 : 0;
  }
  return "";
}

std::vector<int32_t> zero_transfer_terms(const ProblemInfo& pi) {
  // 1-body terms of the zero transfer (compute_diagonal, src/tpsci_outer.jl:694-715)
  std::vector<int32_t> out;
  for (int tr = 0; tr < pi.n_trans; ++tr) {
    bool zero = true;
    for (int i = 0; i < 2 * pi.N; ++i) zero &= (*pi.trans)[size_t(tr) * 2 * pi.N + i] == 0;
    if (zero)
      for (int t = 0; t < pi.n_terms; ++t)
        if (TT(*pi.trm, t, 1) == tr) out.push_back(t);
  }
  return out;
}

std::string build_sectors(const ProblemInfo& pi, int64_t n_cfg, const int16_t* fock, const int16_t* cfg, Plan& P) {
  const int N = pi.N;
  const std::vector<int32_t>& trm = *pi.trm;
  const int n_terms = pi.n_terms;
  const std::vector<int16_t>& trans = *pi.trans;
  const int n_trans = pi.n_trans;
  const int nmax1 = pi.nmax + 1;
  P = Plan();
  P.N = N;
  P.n_cfg = n_cfg;
  if (N > kMaxClusters) return "more than 8 clusters";
  if (n_cfg >= (int64_t(1) << 31)) return "too many configurations";
  // ---- sectors -------------------------------------------------------------
  std::unordered_map<uint64_t, int32_t> sec_of;
  for (int64_t i = 0; i < n_cfg; ++i) {
    const int16_t* f = fock + i * 2 * N;
    bool same = !P.sec_start.empty() &&
                std::memcmp(fock + P.sec_start.back() * 2 * N, f, sizeof(int16_t) * 2 * N) == 0;
    if (same) {
      P.sec_count.back()++;
      continue;
    }
    uint64_t k;
    if (!fock_key(f, N, &k)) return "Fock sector entry outside [0, 15]";
    if (sec_of.count(k)) return "rows of a Fock sector are not contiguous";
    sec_of[k] = int32_t(P.sec_start.size());
    P.sec_start.push_back(i);
    P.sec_count.push_back(1);
    P.sec_fock.insert(P.sec_fock.end(), f, f + 2 * N);
  }
  for (int64_t i = 0; i < n_cfg * N; ++i)
    if (cfg[i] < 0 || cfg[i] > 255) return "local state index outside [0, 255]";
  for (int64_t i = 0; i < n_cfg; ++i)
    for (int c = 0; c < N; ++c) {
      int fa = fock[(i * N + c) * 2], fbb = fock[(i * N + c) * 2 + 1];
      if (fa > pi.norb[c] || fbb > pi.norb[c]) return "Fock sector exceeds cluster size";
      int bl = (*pi.blk_index)[dense_block_index(nmax1, c, kOpH, fa, fbb, fa, fbb)];
      if (bl < 0) return "a row uses a Fock sector with no local basis";
      if (cfg[i * N + c] >= (*pi.blocks)[bl].mb) return "local state index beyond the sector's basis";
    }
  P.zero_terms = zero_transfer_terms(pi);
  return "";
}

std::string build_join(const ProblemInfo& pi, const int16_t* fock, const int16_t* cfg, Plan& P) {
  P.n_triples = P.flops_ref = P.flops_dressed = 0;
  (void)fock;
  const int N = pi.N;
  const std::vector<int32_t>& trm = *pi.trm;
  const int n_terms = pi.n_terms;
  const std::vector<int16_t>& trans = *pi.trans;
  const int n_trans = pi.n_trans;
  const int64_t n_sec = int64_t(P.sec_start.size());
  std::unordered_map<uint64_t, int32_t> sec_of;
  for (int64_t sct = 0; sct < n_sec; ++sct) {
    uint64_t k;
    fock_key(&P.sec_fock[size_t(sct) * 2 * N], N, &k);
    sec_of[k] = int32_t(sct);
  }

  TermLists L;
  {
    const std::string m = term_lists(pi, L);
    if (!m.empty()) return m;
  }
  const std::vector<uint32_t>& masks = L.masks;
  const int n_sets = int(masks.size());

  // ---- groups of every (sector, set) -----------------------------------------
  std::vector<int64_t> fs_perm_off(n_sec * n_sets + 1, 0);
  for (int64_t s = 0; s < n_sec; ++s)
    for (int k = 0; k < n_sets; ++k) fs_perm_off[s * n_sets + k + 1] = P.sec_count[s];
  for (int64_t i = 0; i < n_sec * n_sets; ++i) fs_perm_off[i + 1] += fs_perm_off[i];
  if (fs_perm_off.back() >= (int64_t(1) << 31)) return "grouping pool exceeds 2^31 rows";
  P.perm_pool.assign(fs_perm_off.back(), 0);
  std::vector<std::vector<Group>> groups(n_sec * n_sets);
#pragma omp parallel
  {
    std::vector<std::pair<uint64_t, int32_t>> kv;
#pragma omp for schedule(dynamic, 4)
    for (int64_t fs = 0; fs < n_sec * n_sets; ++fs) {
      int64_t s = fs / n_sets;
      uint32_t m = masks[fs % n_sets];
      int64_t st = P.sec_start[s], n = P.sec_count[s];
      kv.resize(n);
      for (int64_t i = 0; i < n; ++i) {
        const int16_t* c = cfg + (st + i) * N;
        uint64_t key = 0;
        for (int ci = 0; ci < N; ++ci)
          if (!((m >> ci) & 1)) key |= uint64_t(uint16_t(c[ci]) & 0xFF) << (8 * ci);
        kv[i] = {key, int32_t(st + i)};
      }
      std::sort(kv.begin(), kv.end());
      int32_t* perm = &P.perm_pool[fs_perm_off[fs]];
      auto& g = groups[fs];
      g.clear();
      for (int64_t i = 0; i < n; ++i) {
        perm[i] = kv[i].second;
        if (i == 0 || kv[i].first != kv[i - 1].first)
          g.push_back({kv[i].first, int32_t(i), 1});
        else
          g.back().count++;
      }
    }
  }

  // ---- work items: merge-join per (bra sector, transfer, set) --------------
  // items and term-sector records are collected per bra sector and concatenated in
  // sector order, so the plan (and the kernel's summation order) does not depend on
  // thread timing
  std::vector<std::vector<WorkItem>> tItems(n_sec);
  std::vector<std::vector<TermSector>> tTS(n_sec);
  std::vector<std::vector<ItemMeta>> tMeta(n_sec);
  std::vector<std::vector<PJob>> tJobs(n_sec);
  std::vector<int64_t> tTri(n_sec, 0), tFlop(n_sec, 0), tFlopD(n_sec, 0);
  const TermTables tt = term_tables(pi);
#pragma omp parallel
  {
    std::vector<int16_t> fk(2 * N);
    std::vector<TermSector> tsl;
#pragma omp for schedule(dynamic, 1)
    for (int64_t sb = 0; sb < n_sec; ++sb) {
      const int16_t* fb = &P.sec_fock[sb * 2 * N];
      for (int tr = 0; tr < n_trans; ++tr) {
        if (L.first_of_tr[tr] == L.first_of_tr[tr + 1]) continue;
        for (int i = 0; i < 2 * N; ++i) fk[i] = int16_t(fb[i] - trans[size_t(tr) * 2 * N + i]);
        uint64_t key;
        if (!fock_key(fk.data(), N, &key)) continue;
        auto it = sec_of.find(key);
        if (it == sec_of.end()) continue;
        int64_t sk = it->second;
        for (int j = L.first_of_tr[tr]; j < L.first_of_tr[tr + 1]; ++j) {
          // term-sector records of this (bra sector, ket sector, term list)
          tsl.clear();
          int64_t flop = 0, flopd = 0, tri = 0;
          for (int q = L.off[j]; q < L.off[j + 1]; ++q) {
            const int t = L.terms[q];
            if (term_exists(tt, t, fb, fk.data())) {  // a missing TDM block contributes nothing
              flop += term_ref_flops(trm.data(), t);
              ++tri;
            }
            TermSector ts;
            int64_t fma;
            if (tt.rep[t] != t || !term_sector_of(tt, t, fb, fk.data(), ts, &fma)) continue;
            flopd += 2 * fma;
            tsl.push_back(ts);
          }
          if (tsl.empty()) continue;
          const int32_t ts_off = int32_t(tTS[sb].size());  // relative; rebased at concatenation
          tTS[sb].insert(tTS[sb].end(), tsl.begin(), tsl.end());
          // one lane step (one ket): every term's multiply-adds, about 8 loads and index steps
          // per term, and the coefficient update
          const int64_t step_cost = flopd / 2 + 8 * int64_t(tsl.size()) + 4;
          const int nbody_tl = TT(trm, L.terms[L.off[j]], 0);
          const int set = L.set[j];
          const auto& gb = groups[sb * n_sets + set];
          const auto& gk = groups[sk * n_sets + set];
          int64_t pb = fs_perm_off[sb * n_sets + set], pk = fs_perm_off[sk * n_sets + set];
          size_t a = 0, b = 0;
          while (a < gb.size() && b < gk.size()) {
            if (gb[a].key < gk[b].key) {
              ++a;
            } else if (gk[b].key < gb[a].key) {
              ++b;
            } else {
              WorkItem w;
              w.bra_off = int32_t(pb + gb[a].start);
              w.ket_off = int32_t(pk + gk[b].start);
              w.nb = gb[a].count;
              w.nk = gk[b].count;
              w.ts_off = ts_off;
              w.nt = int32_t(tsl.size());
              tItems[sb].push_back(w);
              tMeta[sb].push_back(ItemMeta{step_cost, nbody_tl, block_item(L.block[j] != 0, w.nb, w.nk)});
              tTri[sb] += int64_t(w.nb) * w.nk * tri;
              tFlop[sb] += int64_t(w.nb) * w.nk * flop;
              tFlopD[sb] += int64_t(w.nb) * w.nk * flopd;
              ++a;
              ++b;
            }
          }
        }
      }
    }
  }
  size_t tot = 0, tots = 0;
  for (int64_t sb = 0; sb < n_sec; ++sb) {
    tot += tItems[sb].size();
    tots += tTS[sb].size();
  }
  if (tots >= (size_t(1) << 31)) return "term-sector pool exceeds 2^31 records";
  if (tot >= (size_t(1) << 31)) return "work items exceed 2^31";
  // lane jobs of every item, as long as the state's size allows
  int64_t flopd_all = 0, n_lane[4] = {0, 0, 0, 0};
  for (int64_t sb = 0; sb < n_sec; ++sb) {
    flopd_all += tFlopD[sb];
    for (const WorkItem& w : tItems[sb])
      for (int i = 0; i < 4; ++i) n_lane[i] += int64_t(w.nb) * ((w.nk + kLaneKets[i] - 1) / kLaneKets[i]);
  }
  const int max_kets = kLaneKets[lane_kets(n_lane)];
  const bool with_blocks = flopd_all / 2 >= kBlockMinFma;
  P.lane_kets = max_kets;
#pragma omp parallel for schedule(dynamic, 8)
  for (int64_t sb = 0; sb < n_sec; ++sb)
    for (size_t i = 0; i < tItems[sb].size(); ++i) {
      const WorkItem& w = tItems[sb][i];
      const ItemMeta& m = tMeta[sb][i];
      for (int bj = 0; bj < w.nb; ++bj)
        for (int k0 = 0; k0 < w.nk; k0 += max_kets) {
          PJob pj;
          pj.j.b = P.perm_pool[size_t(w.bra_off) + bj];
          pj.j.kp = w.ket_off + k0;
          pj.j.ts_off = w.ts_off;  // relative; rebased at concatenation
          pj.j.len = uint16_t(std::min(max_kets, w.nk - k0));
          pj.j.nt = uint16_t(w.nt);
          pj.cost = int32_t(std::min<int64_t>(m.step_cost * pj.j.len, int64_t(1) << 30));
          pj.nbody = m.nbody;
          pj.block = m.block && with_blocks;
          tJobs[sb].push_back(pj);
        }
    }
  // concatenation in sector order, each sector's part copied by one thread
  std::vector<int64_t> item_off(n_sec + 1, 0), tsp_off(n_sec + 1, 0), job_off(n_sec + 1, 0);
  for (int64_t sb = 0; sb < n_sec; ++sb) {
    item_off[sb + 1] = item_off[sb] + int64_t(tItems[sb].size());
    tsp_off[sb + 1] = tsp_off[sb] + int64_t(tTS[sb].size());
    job_off[sb + 1] = job_off[sb] + int64_t(tJobs[sb].size());
    P.n_triples += tTri[sb];
    P.flops_ref += tFlop[sb];
    P.flops_dressed += tFlopD[sb];
  }
  P.items.resize(tot);
  P.ts_pool.resize(tots);
#pragma omp parallel for schedule(dynamic, 8)
  for (int64_t sb = 0; sb < n_sec; ++sb) {
    const int32_t base = int32_t(tsp_off[sb]);
    WorkItem* di = P.items.data() + item_off[sb];
    for (const WorkItem& w : tItems[sb]) {
      *di = w;
      di->ts_off += base;
      ++di;
    }
    std::copy(tTS[sb].begin(), tTS[sb].end(), P.ts_pool.begin() + tsp_off[sb]);
    for (PJob& q : tJobs[sb]) q.j.ts_off += base;
    std::vector<WorkItem>().swap(tItems[sb]);
    std::vector<TermSector>().swap(tTS[sb]);
  }
  // The lane jobs of block items come last.  Before and after that line, the lane jobs of windows
  // of kSortWindow bra sectors are sorted by term shape, then by decreasing cost (ties in planning
  // order: the rows of one work item stay together and share their kets), so that the 32 lanes of
  // a warp run the same code on about the same number of kets.  The last warp task is padded with
  // idle lanes (len 0).
  const int64_t n_jobs = job_off[n_sec];
  const int64_t n_wt = (n_jobs + 31) / 32;  // warp tasks
  P.jobs.resize(size_t(n_wt) * 32);
  for (int64_t i = n_jobs; i < n_wt * 32; ++i) P.jobs[size_t(i)] = LaneJob{0, 0, 0, 0, 0};
  std::vector<int32_t> job_cost(static_cast<size_t>(n_jobs));
  {
    constexpr int64_t kSortWindow = 8;
    const int64_t n_win = (n_sec + kSortWindow - 1) / kSortWindow;
    // first position of each window's jobs, of the other items and of the block items
    std::vector<int64_t> at[2] = {std::vector<int64_t>(size_t(n_win) + 1, 0), std::vector<int64_t>(size_t(n_win) + 1, 0)};
    for (int64_t sb = 0; sb < n_sec; ++sb)
      for (const PJob& q : tJobs[sb]) ++at[q.block ? 1 : 0][size_t(sb / kSortWindow) + 1];
    for (auto& a : at)
      for (int64_t w = 0; w < n_win; ++w) a[size_t(w) + 1] += a[size_t(w)];
    P.n_direct = at[0][size_t(n_win)];
    for (int64_t& x : at[1]) x += P.n_direct;
#pragma omp parallel
    {
      std::vector<uint64_t> keys;  // (nbody, decreasing cost, position in the window): one sort key
      std::vector<const PJob*> src;
#pragma omp for schedule(dynamic, 1)
      for (int64_t wdx = 0; wdx < n_win; ++wdx) {
        const int64_t s0 = wdx * kSortWindow, s1 = std::min(n_sec, (wdx + 1) * kSortWindow);
        keys.clear();
        src.clear();
        for (int64_t sb = s0; sb < s1; ++sb)
          for (const PJob& q : tJobs[sb]) {
            const uint64_t c = uint64_t(std::min<int32_t>(q.cost, (1 << 26) - 1));
            keys.push_back((uint64_t(q.block) << 63) | (uint64_t(q.nbody) << 58) | (((uint64_t(1) << 26) - 1 - c) << 32) | uint64_t(src.size()));
            src.push_back(&q);
          }
        std::sort(keys.begin(), keys.end());
        const int64_t n0 = at[0][size_t(wdx) + 1] - at[0][size_t(wdx)];
        for (size_t i = 0; i < keys.size(); ++i) {
          const PJob& q = *src[size_t(keys[i] & 0xFFFFFFFFu)];
          const int64_t o = int64_t(i) < n0 ? at[0][size_t(wdx)] + int64_t(i) : at[1][size_t(wdx)] + int64_t(i) - n0;
          P.jobs[size_t(o)] = q.j;
          job_cost[size_t(o)] = q.cost;
        }
        for (int64_t sb = s0; sb < s1; ++sb) std::vector<PJob>().swap(tJobs[sb]);
      }
    }
  }
  P.wt_cost.assign(size_t(n_wt), 0);
  P.wt_len.assign(size_t(n_wt), 0);
#pragma omp parallel for schedule(static)
  for (int64_t w = 0; w < n_wt; ++w) {
    int32_t c = 0, l = 0;
    for (int64_t i = w * 32; i < std::min(n_jobs, w * 32 + 32); ++i) {
      c = std::max(c, job_cost[size_t(i)]);
      l = std::max<int32_t>(l, P.jobs[size_t(i)].len);
    }
    P.wt_cost[size_t(w)] = c;
    P.wt_len[size_t(w)] = l;
  }
  P.task_values = 0;
  for (int32_t l : P.wt_len) P.task_values += 32 * int64_t(l);
  make_chunks(P, kTargetChunks, P.chunk_lo, P.chunk_val);
  return "";
}

std::string build_plan(const ProblemInfo& pi, int64_t n_cfg, const int16_t* fock, const int16_t* cfg, Plan& P) {
  std::string m = build_sectors(pi, n_cfg, fock, cfg, P);
  return m.empty() ? build_join(pi, fock, cfg, P) : m;
}

void make_chunks(const Plan& P, int64_t target, std::vector<int64_t>& lo, std::vector<int64_t>& val) {
  // chunk c starts at the first warp task whose cost prefix reaches c times the chunk cost;
  // each chunk holds about 1 / target of the work, within [kMinChunkCost, kChunkCost]
  const int64_t n_wt = int64_t(P.wt_cost.size());
  int64_t total = 0;
  for (int32_t c : P.wt_cost) total += c;
  const int64_t chunk_cost =
      std::max<int64_t>(kMinChunkCost, std::min<int64_t>(kChunkCost, total / std::max<int64_t>(target, 1)));
  const int64_t n_chunks = (total + chunk_cost - 1) / chunk_cost;
  lo.assign(size_t(n_chunks) + 1, n_wt);
  val.assign(size_t(n_chunks) + 1, 0);
  int64_t cum = 0, vals = 0, c = 0;
  for (int64_t i = 0; i < n_wt; ++i) {
    while (c < n_chunks && cum >= c * chunk_cost) {
      lo[size_t(c)] = i;
      val[size_t(c)] = vals;
      ++c;
    }
    cum += P.wt_cost[size_t(i)];
    vals += 32 * int64_t(P.wt_len[size_t(i)]);
  }
  for (; c <= n_chunks; ++c) val[size_t(c)] = vals;
}

std::string term_dress(const std::vector<int32_t>& trm, int n_terms, std::vector<TermDress>& dress) {
  dress.assign(size_t(n_terms), TermDress{});
  for (int t = 0; t < n_terms; ++t) {
    const int32_t* r = &trm[int64_t(t) * kTrmCols];
    TermDress& d = dress[size_t(t)];
    const int nb = r[0];
    if (nb == 1) {
      d.pos = -1;
      d.rest_len = 1;
      d.nrem = 0;
      continue;
    }
    // contract the ints with the cluster of the longest orbital multi-index
    d.pos = 0;
    for (int o = 1; o < nb; ++o)
      if (r[22 + o] > r[22 + d.pos]) d.pos = o;
    d.nrem = nb - 1;
    d.rest_len = 1;
    for (int o = 0, q = 0; o < nb; ++o) {
      if (o == d.pos) continue;
      d.rem_pos[q] = o;
      d.rem_dim[q] = r[22 + o];
      d.rest_len *= r[22 + o];
      ++q;
    }
    if (d.rest_len > 32767) return "dressed index too long";
  }
  return "";
}

OpCells op_cells(const std::vector<int>& norb, int nmax, const std::vector<int64_t>& opb,
                 const std::vector<int32_t>& blk_index, const std::vector<BlockInfo>& blocks) {
  const int s = nmax + 1, ss = s * s;
  struct At {
    int64_t key;  // dense block index: cluster, operator, bra sector, ket sector
    int32_t block;
  };
  std::vector<At> at;
  at.reserve(blocks.size());
  for (size_t b = 0; b < blocks.size(); ++b) {
    const int64_t* r = &opb[b * kOpbCols];
    const int64_t key = dense_block_index(s, int(r[0]), int(r[1]), int(r[2]), int(r[3]), int(r[4]), int(r[5]));
    if (blk_index[size_t(key)] == int32_t(b)) at.push_back(At{key, int32_t(b)});  // (the last of equal entries)
  }
  const auto before = [](const At& x, const At& y) { return x.key < y.key; };
  if (!std::is_sorted(at.begin(), at.end(), before)) std::sort(at.begin(), at.end(), before);
  OpCells C;
  C.cells.reserve(at.size());
  C.first_run.assign(norb.size() * kNumOps + 1, 0);
  std::vector<int32_t> mb(norb.size() * size_t(ss), 0), mk(norb.size() * size_t(ss), 0);
  const auto row = [&](size_t q) { return &opb[size_t(at[q].block) * kOpbCols]; };
  size_t i = 0;
  for (size_t op = 0; op < norb.size() * kNumOps; ++op) {
    C.first_run[op] = int32_t(C.runs.size());
    const size_t i0 = i;
    while (i < at.size() && size_t(row(i)[0]) * kNumOps + size_t(row(i)[1]) == op) ++i;
    // one run per change of sector (an operator has one)
    for (size_t q = i0; q < i; ++q) {
      const int64_t* r = row(q);
      const int32_t da = int32_t(r[2] - r[4]), db = int32_t(r[3] - r[5]);
      const BlockInfo& B = blocks[size_t(at[q].block)];
      int32_t &b = mb[size_t(r[0] * ss + r[2] * s + r[3])], &k = mk[size_t(r[0] * ss + r[4] * s + r[5])];
      C.uniform = C.uniform && (b == 0 || b == B.mb) && (k == 0 || k == B.mk);
      b = B.mb, k = B.mk;
      bool known = false;
      for (size_t z = size_t(C.first_run[op]); z < C.runs.size(); ++z) known = known || (C.runs[z].da == da && C.runs[z].db == db);
      if (known) continue;
      OpCells::Run R{da, db, int32_t(C.cells.size()), 0};
      for (size_t z = q; z < i; ++z) {
        const int64_t* rz = row(z);
        if (rz[2] - rz[4] == da && rz[3] - rz[5] == db) C.cells.push_back(OpCells::Cell{int32_t(rz[2] * s + rz[3]), at[z].block});
      }
      R.last = int32_t(C.cells.size());
      C.runs.push_back(R);
    }
  }
  C.first_run.back() = int32_t(C.runs.size());
  return C;
}

std::string build_dress(int nmax, const std::vector<int32_t>& trm, int n_terms, const OpCells& cells,
                        const std::vector<BlockInfo>& blocks, const std::vector<TermInfo>& terms,
                        const std::vector<TermDress>& dress, bool merge, Dressing& out) {
  const int s = nmax + 1, ss = s * s;
  out.rep.resize(size_t(n_terms));  // (the vectors keep their memory for the next term set)
  out.w_index.assign(size_t(n_terms) * ss, -1);
  out.w_mb.assign(size_t(n_terms) * ss, 0);
  // the blocks of a term's dressed cluster and operator, in order of the bra sector
  struct List {
    const OpCells::Cell *p = nullptr, *end = nullptr;
  };
  auto blocks_of = [&](int t) {
    const int32_t* r = &trm[int64_t(t) * kTrmCols];
    const int pos = dress[size_t(t)].pos < 0 ? 0 : dress[size_t(t)].pos;
    const size_t op = size_t(r[2 + pos]) * kNumOps + r[6 + pos];
    for (int32_t i = cells.first_run[op]; i < cells.first_run[op + 1]; ++i) {
      const OpCells::Run& R = cells.runs[size_t(i)];
      if (R.da == r[10 + pos] && R.db == r[14 + pos]) return List{&cells.cells[0] + R.first, &cells.cells[0] + R.last};
    }
    return List{};
  };
  // sets of terms that share a W: term by term, next[t] the next one of t's set (or -1)
  std::vector<int32_t> next(size_t(n_terms), -1);
  if (!merge) {
    for (int t = 0; t < n_terms; ++t) out.rep[size_t(t)] = t;
  } else {
    // by a hash of everything but the dressed operator: transfer, clusters, changes of Fock sector,
    // fermionic parities, and the other clusters' operators and index lengths
    auto hash_of = [&](int t) {
      const int32_t* r = &trm[int64_t(t) * kTrmCols];
      const int pos = dress[size_t(t)].pos;
      uint64_t h = 1469598103934665603ull;
      auto f = [&](int32_t v) { h = (h ^ uint64_t(uint32_t(v))) * 1099511628211ull; };
      f(r[1]), f(r[0]), f(pos);
      for (int o = 0; o < r[0]; ++o) {
        f(r[2 + o]), f(r[10 + o]), f(r[14 + o]), f(r[18 + o]);
        if (o != pos) f(r[6 + o]), f(r[22 + o]);
      }
      return h ^ (h >> 29);
    };
    auto same = [&](int t, int t2) {
      const int32_t *r = &trm[int64_t(t) * kTrmCols], *r2 = &trm[int64_t(t2) * kTrmCols];
      const int pos = dress[size_t(t)].pos;
      if (r[1] != r2[1] || r[0] != r2[0] || pos != dress[size_t(t2)].pos) return false;
      for (int o = 0; o < r[0]; ++o) {
        if (r[2 + o] != r2[2 + o] || r[10 + o] != r2[10 + o] || r[14 + o] != r2[14 + o] || r[18 + o] != r2[18 + o])
          return false;
        if (o != pos && (r[6 + o] != r2[6 + o] || r[22 + o] != r2[22 + o])) return false;
      }
      return true;
    };
    // the operators' blocks must have the same local dimensions wherever several exist
    auto fits = [&](int t, int t0) {
      if (cells.uniform) return true;
      for (int m = t0; m >= 0 && m != t; m = next[size_t(m)])
        for (List x = blocks_of(t), y = blocks_of(m); x.p != x.end && y.p != y.end;) {
          if (x.p->fb != y.p->fb) {
            ++(x.p->fb < y.p->fb ? x : y).p;
            continue;
          }
          const BlockInfo &B = blocks[size_t(x.p++->block)], &B2 = blocks[size_t(y.p++->block)];
          if (B.mb != B2.mb || B.mk != B2.mk) return false;
        }
      return true;
    };
    size_t cap = 64;
    while (cap < 2 * size_t(n_terms)) cap <<= 1;
    std::vector<int32_t> table(cap, -1);           // open addressing: the first term of a set
    std::vector<int32_t> last(size_t(n_terms), -1);  // by first term: the set's last term so far
    for (int t = 0; t < n_terms; ++t) {
      out.rep[size_t(t)] = t;
      if (dress[size_t(t)].pos < 0) continue;
      size_t at = size_t(hash_of(t)) & (cap - 1);
      while (table[at] >= 0 && !same(t, table[at])) at = (at + 1) & (cap - 1);
      const int t0 = table[at] >= 0 ? table[at] : t;
      if (!fits(t, t0)) continue;
      table[at] = t0;
      if (t0 != t) {
        out.rep[size_t(t)] = t0;
        next[size_t(last[size_t(t0)])] = t;
      }
      last[size_t(t0)] = t;
    }
  }
  // the jobs of a set, bra sector by bra sector: its terms' lists merged, the terms of a sector in order
  struct Member {
    List list;
    DressSrc src;
    int nidx;  // index length of the dressed operator
  };
  std::vector<Member> set;
  std::vector<DressJob>& jobs = out.jobs;
  std::vector<DressSrc>& src = out.src;
  size_t n_src = 0, n_jobs = 0;
  for (int t = 0; t < n_terms; ++t) n_src += size_t(blocks_of(t).end - blocks_of(t).p);
  jobs.resize(n_src);
  src.resize(n_src);
  n_src = 0;
  int64_t n_w = 0;
  for (int t0 = 0; t0 < n_terms; ++t0) {
    if (out.rep[size_t(t0)] != t0) continue;
    const TermDress& d = dress[size_t(t0)];
    const int nb = trm[int64_t(t0) * kTrmCols], pos = d.pos < 0 ? 0 : d.pos;
    set.clear();
    for (int t = t0; t >= 0; t = next[size_t(t)]) {
      const int32_t* r = &trm[int64_t(t) * kTrmCols];
      int stride[4];
      stride[0] = 1;
      for (int o = 1; o < 4; ++o) stride[o] = stride[o - 1] * r[22 + o - 1];
      Member M{blocks_of(t), DressSrc{}, r[22 + pos]};
      M.src.ints_off = terms[size_t(t)].ints_off;
      M.src.nq = nb == 1 ? 1 : r[22 + pos];
      M.src.stride_q = stride[pos];
      for (int q = 0; q < d.nrem; ++q) M.src.rem_stride[q] = stride[d.rem_pos[q]];
      if (M.list.p != M.list.end) set.push_back(M);
    }
    DressJob J{};
    J.rest_len = d.rest_len;
    J.nrem = d.nrem;
    for (int q = 0; q < d.nrem; ++q) J.rem_dim[q] = d.rem_dim[q];
    J.one_body = nb == 1;
    int64_t* w_index = &out.w_index[size_t(t0) * ss];
    int32_t* w_mb = &out.w_mb[size_t(t0) * ss];
    for (;;) {
      int cell = ss;
      for (const Member& M : set)
        if (M.list.p != M.list.end) cell = std::min(cell, M.list.p->fb);
      if (cell == ss) break;
      J.src0 = int32_t(n_src);
      for (Member& M : set) {
        if (M.list.p == M.list.end || M.list.p->fb != cell) continue;
        const BlockInfo& B = blocks[size_t(M.list.p++->block)];
        if (nb > 1 && B.nidx != M.nidx) return "term dims do not match the TDM block";
        M.src.g_off = B.off;
        src[n_src++] = M.src;
        J.mb = B.mb;
        J.mk = B.mk;
      }
      J.n_src = int32_t(n_src) - J.src0;
      n_w = (n_w + kAlign - 1) / kAlign * kAlign;  // vector-load alignment of W blocks
      J.w_off = n_w;
      jobs[n_jobs++] = J;
      w_index[cell] = n_w;
      w_mb[cell] = J.mb;
      n_w += int64_t(d.rest_len) * J.mb * J.mk;
    }
  }
  jobs.resize(n_jobs);
  out.n_w = n_w;
  return "";
}

}  // namespace fcg
