// C entry point over the dressing tables of fermicg_gb300/csrc/plan.cpp (term_dress, op_cells,
// build_dress), so that they can be checked against a plain restatement without a GPU.
#include "../fermicg_gb300/csrc/fcg_internal.h"

#include <algorithm>
#include <cstring>

using namespace fcg;

// rows: the caller's block table (kOpbCols each); trm: term rows (kTrmCols each).  Out: rep [n_terms],
// w_index and w_mb [n_terms][(nmax + 1)^2], jobs as (w_off, mb, mk, src0, n_src, one_body) and sources as
// (block offset, ints offset, nq, stride_q), up to `cap` of each.  Returns the number of jobs, or -1.
extern "C" int64_t ds_build(int n_clusters, const int32_t* norb_in, int64_t n_blocks, const int64_t* rows, int n_terms,
                            const int32_t* trm_in, int merge, int64_t cap, int32_t* rep, int64_t* w_index, int32_t* w_mb,
                            int64_t* jobs, int64_t* src, int64_t* n_src) {
  const std::vector<int> norb(norb_in, norb_in + n_clusters);
  const int nmax = *std::max_element(norb.begin(), norb.end()), s = nmax + 1;
  const std::vector<int64_t> opb(rows, rows + n_blocks * kOpbCols);
  const std::vector<int32_t> trm(trm_in, trm_in + int64_t(n_terms) * kTrmCols);
  std::vector<int32_t> index(size_t(n_clusters) * kNumOps * s * s * s * s, -1);
  std::vector<BlockInfo> blocks;
  for (int64_t b = 0; b < n_blocks; ++b) {
    const int64_t* r = rows + b * kOpbCols;
    index[size_t(dense_block_index(s, int(r[0]), int(r[1]), int(r[2]), int(r[3]), int(r[4]), int(r[5])))] = int32_t(b);
    blocks.push_back(BlockInfo{r[9], int32_t(r[6]), int32_t(r[7]), int32_t(r[8]), 0});
  }
  std::vector<TermInfo> terms{size_t(n_terms)};
  for (int t = 0; t < n_terms; ++t) terms[size_t(t)].ints_off = int64_t(t);
  std::vector<TermDress> dress;
  Dressing D;
  if (!term_dress(trm, n_terms, dress).empty()) return -1;
  if (!build_dress(nmax, trm, n_terms, op_cells(norb, nmax, opb, index, blocks), blocks, terms, dress, merge != 0, D).empty())
    return -1;
  if (int64_t(D.jobs.size()) > cap || int64_t(D.src.size()) > cap) return -1;
  std::copy(D.rep.begin(), D.rep.end(), rep);
  std::copy(D.w_index.begin(), D.w_index.end(), w_index);
  std::copy(D.w_mb.begin(), D.w_mb.end(), w_mb);
  for (size_t i = 0; i < D.jobs.size(); ++i) {
    const DressJob& J = D.jobs[i];
    const int64_t v[6] = {J.w_off, J.mb, J.mk, J.src0, J.n_src, J.one_body};
    std::memcpy(jobs + 6 * i, v, sizeof(v));
  }
  for (size_t i = 0; i < D.src.size(); ++i) {
    const DressSrc& S = D.src[i];
    const int64_t v[4] = {S.g_off, S.ints_off, S.nq, S.stride_q};
    std::memcpy(src + 4 * i, v, sizeof(v));
  }
  *n_src = int64_t(D.src.size());
  return int64_t(D.jobs.size());
}
