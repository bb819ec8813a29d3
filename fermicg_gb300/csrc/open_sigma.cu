// Open (first-order interacting space) sigma on the GPU: open_matvec_thread
// (src/tpsci_matvec_thread.jl:11-885) behind fcg_sigma_open / fcg_sigma_open_fetch.
//
// For every ket row of the state and every term whose target sector passes the job
// filter (:26-56), every bra local-state tuple of the term's active clusters gets
//     x = sign * sum W[(rest), b_w, k_w] prod_c G_c[i_c, b_c, k_c]
// and contributes x * c_ket to sigma[bra config] when |x| > thresh / max_r |c_ket[r]|,
// the per-contribution test of _collect_significant_thread! (:830-885).
//
// Pipeline (one stream):
//   screen_kernel   one thread per (ket row, term) job: a rigorous max-norm bound
//                   sum_rest Wmax * prod Gmax skips jobs whose every contribution would
//                   fail the threshold (the role of upper_bound_thread, :897-1023; skipping
//                   changes no result), the survivors are compacted;
//   expand_jobs_kernel  persistent warps take the surviving (ket, term) jobs from a counter,
//                   stage the job's W block and TDM columns in shared memory, screen every
//                   bra tuple in float with a rigorous margin, evaluate the few that can pass
//                   exactly (threshold per contribution, as the reference), and insert into
//                   an open-addressed table keyed by (bra sector, mixed-radix local-state
//                   index) with atomic accumulation of the R values;
//   compact_kernel  occupied slots -> (key, values).
// A table that overflows its probe limit sets a flag and the call is repeated with a
// table twice as large.
#include <cmath>
#include <cstring>
#include <unordered_map>
#include <unordered_set>

#include "fcg_ctx.cuh"

using namespace fcg;

namespace {

constexpr unsigned long long kEmpty = ~0ull;
constexpr int kMaxProbe = 1 << 16;
constexpr int kKeyIdxBits = 40;

// counters: [0] kept jobs, [1] elements of kept jobs, [2] table overflow, [3] output rows,
// [4] next job of the expand warps
struct OpenParams {
  const OpenTerm* ot;
  const OpenItem* items;
  const int64_t* prefix;  // job prefix over items
  int64_t n_items;
  int64_t n_jobs;
  const int16_t* cfg;
  const double* c;  // row-major [n_cfg][R]
  const int64_t* strides;  // [n_bra_sectors][N]
  int N;
  int R;
  double thresh;
};

__device__ __forceinline__ int64_t find_item(const int64_t* prefix, int64_t lo, int64_t hi, int64_t x) {
  while (lo < hi) {
    int64_t mid = (lo + hi + 1) >> 1;
    if (__ldg(prefix + mid) <= x)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ double row_maxabs(const double* c, int R) {
  double m = 0.0;
  for (int r = 0; r < R; ++r) m = fmax(m, fabs(c[r]));
  return m;
}

// rigorous bound on max over bra tuples of |x| for one (ket, term) job
__device__ double job_bound(const OpenTerm& o, const double* __restrict__ wmax, const double* __restrict__ gmax,
                            const int16_t* ck) {
  const TermSector& ts = o.ts;
  const double* wm = wmax + o.wmax_off + int64_t(ts.rest_len) * ck[ts.cw];
  if (ts.nrem == 0) return wm[0];
  const double* g0 = gmax + o.gmax_off[0] + int64_t(ts.g_dim[0]) * ck[ts.cr[0]];
  const int d0 = ts.g_dim[0];
  double bnd = 0.0;
  if (ts.nrem == 1) {
    for (int i = 0; i < d0; ++i) bnd += wm[i] * g0[i];
    return bnd;
  }
  const double* g1 = gmax + o.gmax_off[1] + int64_t(ts.g_dim[1]) * ck[ts.cr[1]];
  const int d1 = ts.g_dim[1];
  if (ts.nrem == 2) {
    for (int j = 0; j < d1; ++j) {
      double a = 0.0;
      for (int i = 0; i < d0; ++i) a += wm[i + d0 * j] * g0[i];
      bnd += a * g1[j];
    }
    return bnd;
  }
  const double* g2 = gmax + o.gmax_off[2] + int64_t(ts.g_dim[2]) * ck[ts.cr[2]];
  const int d2 = ts.g_dim[2];
  for (int l = 0; l < d2; ++l) {
    double al = 0.0;
    for (int j = 0; j < d1; ++j) {
      double a = 0.0;
      for (int i = 0; i < d0; ++i) a += wm[i + d0 * (j + d1 * l)] * g0[i];
      al += a * g1[j];
    }
    bnd += al * g2[l];
  }
  return bnd;
}

__global__ void screen_kernel(OpenParams p, const double* __restrict__ wmax, const double* __restrict__ gmax,
                              int2* __restrict__ kept, unsigned long long* __restrict__ counters) {
  const int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= p.n_jobs) return;
  const int64_t it = find_item(p.prefix, 0, p.n_items - 1, j);
  const OpenItem I = p.items[it];
  const int64_t local = j - p.prefix[it];
  const int ti = int(local % I.nt);
  const int row = I.row0 + int(local / I.nt);
  const OpenTerm& o = p.ot[I.ot_off + ti];
  const double maxc = row_maxabs(p.c + int64_t(row) * p.R, p.R);
  if (!(maxc > 0.0)) return;
  const double bnd = job_bound(o, wmax, gmax, p.cfg + int64_t(row) * kCfgStride);
  // keep unless every |x| <= bnd < thresh / maxc (a 1e-9 margin covers the bound's rounding)
  if (!(bnd * (1.0 + 1e-9) > p.thresh / maxc)) return;
  const unsigned long long pos = atomicAdd(counters + 0, 1ull);
  kept[pos] = make_int2(row, I.ot_off + ti);
  atomicAdd(counters + 1, (unsigned long long)o.out_count);
}

__device__ __forceinline__ void table_add(unsigned long long* keys, double* vals, unsigned long long cap_mask,
                                          unsigned long long key, double x, const double* crow, int R,
                                          unsigned long long* overflow) {
  unsigned long long h = key * 0x9E3779B97F4A7C15ull;
  h ^= h >> 29;
  unsigned long long slot = h & cap_mask;
  for (int probe = 0; probe < kMaxProbe; ++probe) {
    unsigned long long cur = keys[slot];
    if (cur == kEmpty) {
      unsigned long long prev = atomicCAS(keys + slot, kEmpty, key);
      if (prev == kEmpty || prev == key) cur = key;
      else cur = prev;
    }
    if (cur == key) {
      for (int r = 0; r < R; ++r) atomicAdd(vals + slot * R + r, x * crow[r]);
      return;
    }
    slot = (slot + 1) & cap_mask;
  }
  atomicExch(overflow, 1ull);
}

constexpr int kExpWarps = 8;      // warps of an expand CTA at most
constexpr int kOpenMaxR = 16;     // roots of one open sigma at most (checked on the host)
constexpr int kExpSlice = 36 * 1024;      // largest float tiles of one job a warp keeps in shared memory
constexpr int kExpCtaBytes = 104 * 1024;  // shared-memory budget of one expand CTA (two per SM)
constexpr int kQueue = 64;        // candidates a warp holds: flushed 32 at a time, so 31 + 32 always fit
// The float pre-filter keeps a contribution for the exact double evaluation unless
// |x32| + kFilterMargin * s32 <= thresh / max|c|, where s32 = sum of |products| of the same
// sum.  The float evaluation differs from the exact value by at most about
// (number of factors + summed terms) * 2^-24 * s (below 1e-5 s for every shape here), so
// the margin of 1e-4 s never drops a contribution the double evaluation would keep.
constexpr float kFilterMargin = 1e-4f;
// Whole tiles and units are skipped on an upper bound of s32 (the column maxima in place of the
// columns not looked at yet); this factor covers the bound's own float rounding and the margin.
constexpr float kBoundSlack = 1.002f;

// Shared memory of one warp, in floats: the W block of the ket's dressed-cluster state
// [rest][mb0 | 1] (bra states fastest, so that a warp's lanes read consecutive words; an odd
// stride, so that it is written without bank conflicts too), the TDM
// columns of the remaining clusters [mb_{r+1}][d_r], and for clusters of more than
// kExpMaxD orbital indices (D = 0) the per-lane sums T1, T1a [JL][32] and u, ua [d2][32].
struct ExpandTiles {
  int w, g[3], t1, t1a, u, ua;
  int bytes;
};

__host__ __device__ inline ExpandTiles expand_tiles(int nrem, int rest, const int16_t* g_dim, const int16_t* mb,
                                                    bool lane_sums) {
  ExpandTiles t{};
  int f = 0;
  t.w = f;
  f += rest * (mb[0] | 1);
  for (int r = 0; r < 3; ++r) {
    f = (f + 3) & ~3;
    t.g[r] = f;
    if (r < nrem) f += g_dim[r] * mb[r + 1];
  }
  const int jl = lane_sums && nrem >= 2 ? rest / g_dim[0] : 0;
  const int d2 = lane_sums && nrem >= 3 ? g_dim[2] : 0;
  t.t1 = f;
  f += 32 * jl;
  t.t1a = f;
  f += 32 * jl;
  t.u = f;
  f += 32 * d2;
  t.ua = f;
  f += 32 * d2;
  t.bytes = 4 * ((f + 3) & ~3);
  return t;
}

// The exact contribution of one bra tuple (columns already selected): the sums of the
// per-element formula, in its order, with its fused multiply-adds.
__device__ __forceinline__ double exact_x(int nrem, int d0, int d1, int d2, const double* wc, const double* g0,
                                          const double* g1, const double* g2) {
  if (nrem == 0) return wc[0];
  double x = 0.0;
  if (nrem == 1) {
    for (int i = 0; i < d0; ++i) x = fma(wc[i], g0[i], x);
  } else if (nrem == 2) {
    for (int jj = 0; jj < d1; ++jj) {
      double acc = 0.0;
      for (int i = 0; i < d0; ++i) acc = fma(wc[i + d0 * jj], g0[i], acc);
      x = fma(acc, g1[jj], x);
    }
  } else {
    for (int l = 0; l < d2; ++l) {
      double al = 0.0;
      for (int jj = 0; jj < d1; ++jj) {
        double acc = 0.0;
        for (int i = 0; i < d0; ++i) acc = fma(wc[i + d0 * (jj + d1 * l)], g0[i], acc);
        al = fma(acc, g1[jj], al);
      }
      x = fma(al, g2[l], x);
    }
  }
  return x;
}

// What a warp needs of its current job to evaluate and store one contribution.
struct ExpandJob {
  int nrem, rest, d0, d1, d2;
  int mb[4];
  int64_t sa[4];  // key stride of each active cluster's bra state
  int64_t base;   // key of the ket's other clusters
  unsigned long long keybase;
  double tc;      // contributions of |x| <= tc are dropped
  const double* w;
  const double* g[3];
  const double* crow;  // the ket's coefficients times the term's sign (shared memory)
};

struct ExpandTable {
  unsigned long long* keys;
  double* vals;
  unsigned long long cap_mask;
  unsigned long long* counters;
};

// exact value, threshold, accumulation of x * c_ket of the bra tuple (b0, b1, b2, b3)
__device__ __forceinline__ void expand_exact(const ExpandJob& J, const ExpandTable& H, int R, int b0, int b1, int b2,
                                             int b3) {
  const double x = exact_x(J.nrem, J.d0, J.d1, J.d2, J.w + int64_t(J.rest) * b0, J.g[0] + int64_t(J.d0) * b1,
                           J.g[1] + int64_t(J.d1) * b2, J.g[2] + int64_t(J.d2) * b3);
  if (!(fabs(x) > J.tc)) return;
  const int64_t idx = J.base + b0 * J.sa[0] + b1 * J.sa[1] + b2 * J.sa[2] + b3 * J.sa[3];
  table_add(H.keys, H.vals, H.cap_mask, J.keybase | (unsigned long long)idx, x, J.crow, R, H.counters + 2);
}

// A warp's candidates: those of one step are appended, and every 32 are evaluated by the whole
// warp, one per lane (few lanes pass the screen at a time, and an FP64 instruction costs the
// same for one lane as for 32).  Entry: b3 | b2 << 8 | (b0 + mb0 * b1) << 16.
struct ExpandQueue {
  unsigned* q;
  int n;
};

__device__ __forceinline__ void queue_run(const ExpandQueue& Q, int at, const ExpandJob& J, const ExpandTable& H, int R) {
  const unsigned e = Q.q[at];
  const int pr = int(e >> 16), b1 = pr / J.mb[0];
  expand_exact(J, H, R, pr - b1 * J.mb[0], b1, int((e >> 8) & 255u), int(e & 255u));
}

__device__ __forceinline__ void queue_push(ExpandQueue& Q, bool keep, unsigned entry, const ExpandJob& J,
                                           const ExpandTable& H, int R) {
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  if (m == 0) return;
  const int lane = threadIdx.x & 31;
  if (keep) Q.q[Q.n + __popc(m & ((1u << lane) - 1u))] = entry;
  Q.n += __popc(m);
  __syncwarp();
  if (Q.n >= 32) {
    Q.n -= 32;
    queue_run(Q, Q.n + lane, J, H, R);
    __syncwarp();  // the entries are read before the next push overwrites them
  }
}

constexpr int kExpMaxD = 6;  // longest orbital index of the register sums

// One warp per kept (ket, term) job, taken from a counter.  The job's W block and TDM columns
// are staged in the warp's shared-memory slice (the float copies the library keeps of both);
// each lane owns one (b0, b1) pair at a time and keeps
//   T1[j, l] = sum_i W[i, j, l, b0] G0[i, b1]
// and its absolute-value twin in registers (D: bound of the two index lengths; 0: in shared
// memory), from which every (b2, b3) is screened in float.  Pairs and (pair, b2) units that no
// lane's bound can lift over the threshold are skipped whole.  What passes the screen is
// queued and evaluated exactly, 32 at a time, with the per-element double formula, and
// thresholded as the reference does.  Jobs whose tiles exceed a slice are evaluated per
// element, exactly, from global memory.
//
// What bounds it: the screen's instructions (about 10 per surviving contribution) and the
// latency of a job's first loads, which 16 or more warps per SM cover; contributions over the
// threshold are rare (0.4 % at 1e-3), so neither the FP64 pipe nor the table's atomics are.
// A CTA per job (two resident per SM, five barriers per job) and a divergent exact evaluation
// took 57 ms longer on 3 001 configurations of the 24-orbital problem at 1e-3, 4 roots (1.09e6
// kept jobs, 9.7e9 contributions): whole call 126.8 -> 69.4 ms.
template <int D>
__global__ void __launch_bounds__(32 * kExpWarps, D == 3 || D == 4 ? 2 : 1) expand_jobs_kernel(
    OpenParams p, const int2* __restrict__ kept, int64_t n_kept, const double* __restrict__ w,
    const double* __restrict__ op, const float* __restrict__ w32, const float* __restrict__ op32,
    const double* __restrict__ gmax, ExpandTable H, int slice) {
  extern __shared__ __align__(16) unsigned char xsm[];
  __shared__ double s_cs[kExpWarps][kOpenMaxR];
  __shared__ unsigned s_queue[kExpWarps][kQueue];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float* xf = reinterpret_cast<float*>(xsm + size_t(wid) * slice);
  ExpandQueue Q{s_queue[wid], 0};
  const int R = p.R;
  for (;;) {
    unsigned long long jn = 0;
    if (lane == 0) jn = atomicAdd(H.counters + 4, 1ull);
    jn = __shfl_sync(0xffffffffu, jn, 0);
    if (int64_t(jn) >= n_kept) break;
    const int2 job = kept[jn];
    const OpenTerm& o = p.ot[job.y];
    const TermSector& ts = o.ts;
    const int16_t* ck = p.cfg + int64_t(job.x) * kCfgStride;
    const double* c_ket = p.c + int64_t(job.x) * R;
    ExpandJob J{};
    J.tc = p.thresh / row_maxabs(c_ket, R);
    const float tcf = float(J.tc * (1.0 - 1e-6));
    const int nrem = ts.nrem, rest = ts.rest_len;
    const int d0 = nrem >= 1 ? ts.g_dim[0] : 1, d1 = nrem >= 2 ? ts.g_dim[1] : 1, d2 = nrem >= 3 ? ts.g_dim[2] : 1;
    J.nrem = nrem, J.rest = rest, J.d0 = d0, J.d1 = d1, J.d2 = d2;
    // bra key of (b0, .., b3) = keybase | (base + sum_a b_a * st[c_a])
    const int64_t* st = p.strides + int64_t(o.bsec) * p.N;
    for (int c = 0; c < p.N; ++c) J.base += int64_t(ck[c]) * st[c];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      J.mb[a] = 1;
      if (a < o.n_act) {
        J.mb[a] = o.mb_act[a];
        J.sa[a] = st[o.c_act[a]];
        J.base -= int64_t(ck[o.c_act[a]]) * J.sa[a];
      }
    }
    J.keybase = (unsigned long long)(o.bsec) << kKeyIdxBits;
    // a kept value x contributes x * (sg * c) = (sg * x) * c to every root
    const double sg = ts.sign < 0 ? -1.0 : 1.0;
    if (lane < R) s_cs[wid][lane] = sg * c_ket[lane];
    J.crow = s_cs[wid];
    const int64_t w_at = ts.w_off + int64_t(rest) * ts.w_mb * ck[ts.cw];  // [rest][mb0] for the ket state
    J.w = w + w_at;
    int64_t g_at[3] = {0, 0, 0};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      J.g[r] = op;
      if (r < nrem) {
        g_at[r] = ts.g_off[r] + int64_t(ts.g_dim[r]) * ts.g_mb[r] * ck[ts.cr[r]];
        J.g[r] = op + g_at[r];
      }
    }
    const int mb0 = J.mb[0], mbp = mb0 | 1, P = mb0 * J.mb[1];
    const ExpandTiles t = expand_tiles(nrem, rest, ts.g_dim, o.mb_act, D == 0);
    if (nrem == 0) {
      __syncwarp();
      for (int b0 = lane; b0 < mb0; b0 += 32) expand_exact(J, H, R, b0, 0, 0, 0);
    } else if (t.bytes <= slice) {
      for (int i = lane; i < rest * mb0; i += 32) {
        const int b0 = i / rest;
        xf[t.w + (i - b0 * rest) * mbp + b0] = __ldg(w32 + w_at + i);
      }
#pragma unroll
      for (int r = 0; r < 3; ++r)
        if (r < nrem) {
          const int n = ts.g_dim[r] * J.mb[r + 1];
          for (int i = lane; i < n; i += 32) xf[t.g[r] + i] = __ldg(op32 + g_at[r] + i);
        }
      __syncwarp();
      const float* W = xf + t.w;
      const float* G0 = xf + t.g[0];
      if (nrem == 1) {
        for (int p0 = 0; p0 < P; p0 += 32) {
          const int pr = p0 + lane;
          bool keep = false;
          if (pr < P) {
            const int b1 = pr / mb0, b0 = pr - b1 * mb0;
            float x32 = 0.f, s32 = 0.f;
            for (int i = 0; i < d0; ++i) {
              const float wv = W[i * mbp + b0], gv = G0[i + d0 * b1];
              x32 = fmaf(wv, gv, x32);
              s32 = fmaf(fabsf(wv), fabsf(gv), s32);
            }
            keep = fabsf(x32) + kFilterMargin * s32 > tcf;
          }
          queue_push(Q, keep, unsigned(pr) << 16, J, H, R);
        }
      } else {
        constexpr int E = D > 0 ? D : 1;
        // column maxima of the second and third remaining clusters for the ket's states
        const double* gm1 = gmax + o.gmax_off[1] + int64_t(d1) * ck[ts.cr[1]];
        const double* gm2 = nrem == 3 ? gmax + o.gmax_off[2] + int64_t(d2) * ck[ts.cr[2]] : nullptr;
        float m1[E], m2[E];
        if (D > 0) {
#pragma unroll
          for (int j = 0; j < E; ++j) {
            m1[j] = j < d1 ? __double2float_ru(gm1[j]) : 0.f;
            m2[j] = nrem == 3 ? (j < d2 ? __double2float_ru(gm2[j]) : 0.f) : (j == 0 ? 1.f : 0.f);
          }
        }
        const float* G1 = xf + t.g[1];
        const float* G2 = xf + t.g[2];
        for (int p0 = 0; p0 < P; p0 += 32) {
          const int pr = p0 + lane;
          const bool live = pr < P;
          const int b1 = live ? pr / mb0 : 0, b0 = live ? pr - b1 * mb0 : 0;
          const float* g0 = G0 + d0 * b1;
          if constexpr (D > 0) {
            float t1[E * E], ta[E * E];  // [j + E * l]
#pragma unroll
            for (int e = 0; e < E * E; ++e) t1[e] = ta[e] = 0.f;
            for (int i = 0; i < d0; ++i) {
              const float gv = live ? g0[i] : 0.f, ga = fabsf(gv);
              const float* wi = W + i * mbp + b0;
#pragma unroll
              for (int l = 0; l < E; ++l) {
                if (l < d2) {
#pragma unroll
                  for (int j = 0; j < E; ++j)
                    if (j < d1) {
                      const float wv = wi[d0 * (j + d1 * l) * mbp];
                      t1[j + E * l] = fmaf(wv, gv, t1[j + E * l]);
                      ta[j + E * l] = fmaf(fabsf(wv), ga, ta[j + E * l]);
                    }
                }
              }
            }
            float top = 0.f;  // bound of s32 over every (b2, b3) of this pair
#pragma unroll
            for (int l = 0; l < E; ++l) {
              float a = 0.f;
#pragma unroll
              for (int j = 0; j < E; ++j) a = fmaf(ta[j + E * l], m1[j], a);
              top = fmaf(a, m2[l], top);
            }
            if (!__any_sync(0xffffffffu, top * kBoundSlack > tcf)) continue;
            for (int b2 = 0; b2 < J.mb[2]; ++b2) {
              const float* g1 = G1 + d1 * b2;
              float g1v[E];
#pragma unroll
              for (int j = 0; j < E; ++j) g1v[j] = j < d1 ? g1[j] : 0.f;
              float ul[E], ua[E];
#pragma unroll
              for (int l = 0; l < E; ++l) {
                ul[l] = ua[l] = 0.f;
#pragma unroll
                for (int j = 0; j < E; ++j) {
                  ul[l] = fmaf(t1[j + E * l], g1v[j], ul[l]);
                  ua[l] = fmaf(ta[j + E * l], fabsf(g1v[j]), ua[l]);
                }
                if (nrem == 2) break;
              }
              if (nrem == 2) {
                queue_push(Q, fabsf(ul[0]) + kFilterMargin * ua[0] > tcf, unsigned(pr) << 16 | unsigned(b2) << 8, J, H, R);
                continue;
              }
              float bnd = 0.f;
#pragma unroll
              for (int l = 0; l < E; ++l) bnd = fmaf(ua[l], m2[l], bnd);
              if (!__any_sync(0xffffffffu, bnd * kBoundSlack > tcf)) continue;
              for (int b3 = 0; b3 < J.mb[3]; ++b3) {
                const float* g2 = G2 + d2 * b3;
                float x32 = 0.f, s32 = 0.f;
#pragma unroll
                for (int l = 0; l < E; ++l) {
                  const float gv = l < d2 ? g2[l] : 0.f;
                  x32 = fmaf(ul[l], gv, x32);
                  s32 = fmaf(ua[l], fabsf(gv), s32);
                }
                queue_push(Q, fabsf(x32) + kFilterMargin * s32 > tcf,
                           unsigned(pr) << 16 | unsigned(b2) << 8 | unsigned(b3), J, H, R);
              }
            }
          } else {
            // index lengths over kExpMaxD: the lane's sums in its column of shared memory
            const int JL = d1 * d2;
            float* t1 = xf + t.t1 + lane;
            float* ta = xf + t.t1a + lane;
            float* us = xf + t.u + lane;
            float* ua = xf + t.ua + lane;
            for (int jl = 0; jl < JL; ++jl) {
              float a = 0.f, b = 0.f;
              for (int i = 0; i < d0; ++i) {
                const float gv = live ? g0[i] : 0.f, wv = W[(i + d0 * jl) * mbp + b0];
                a = fmaf(wv, gv, a);
                b = fmaf(fabsf(wv), fabsf(gv), b);
              }
              t1[32 * jl] = a;
              ta[32 * jl] = b;
            }
            for (int b2 = 0; b2 < J.mb[2]; ++b2) {
              const float* g1 = G1 + d1 * b2;
              float x0 = 0.f, s0 = 0.f;
              for (int l = 0; l < d2; ++l) {
                float a = 0.f, b = 0.f;
                for (int j = 0; j < d1; ++j) {
                  a = fmaf(t1[32 * (j + d1 * l)], g1[j], a);
                  b = fmaf(ta[32 * (j + d1 * l)], fabsf(g1[j]), b);
                }
                if (nrem == 2) {
                  x0 = a, s0 = b;
                } else {
                  us[32 * l] = a;
                  ua[32 * l] = b;
                }
              }
              if (nrem == 2) {
                queue_push(Q, fabsf(x0) + kFilterMargin * s0 > tcf, unsigned(pr) << 16 | unsigned(b2) << 8, J, H, R);
                continue;
              }
              for (int b3 = 0; b3 < J.mb[3]; ++b3) {
                const float* g2 = G2 + d2 * b3;
                float x32 = 0.f, s32 = 0.f;
                for (int l = 0; l < d2; ++l) {
                  x32 = fmaf(us[32 * l], g2[l], x32);
                  s32 = fmaf(ua[32 * l], fabsf(g2[l]), s32);
                }
                queue_push(Q, fabsf(x32) + kFilterMargin * s32 > tcf,
                           unsigned(pr) << 16 | unsigned(b2) << 8 | unsigned(b3), J, H, R);
              }
            }
          }
        }
      }
      if (lane < Q.n) queue_run(Q, lane, J, H, R);  // the job's last candidates
      Q.n = 0;
    } else {
      // tiles too large: every element exactly, from global memory
      __syncwarp();
      for (int64_t e = lane; e < o.out_count; e += 32) {
        int64_t loc = e;
        int b[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          b[a] = int(loc % J.mb[a]);
          loc /= J.mb[a];
        }
        expand_exact(J, H, R, b[0], b[1], b[2], b[3]);
      }
    }
    __syncwarp();  // tiles, coefficients and queue are rewritten for the next job
  }
}

__global__ void compact_kernel(const unsigned long long* __restrict__ keys, const double* __restrict__ vals,
                               unsigned long long cap, int R, unsigned long long* __restrict__ okeys,
                               double* __restrict__ ovals, unsigned long long* __restrict__ counters) {
  const unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= cap) return;
  const unsigned long long k = keys[s];
  if (k == kEmpty) return;
  const unsigned long long pos = atomicAdd(counters + 3, 1ull);
  okeys[pos] = k;
  for (int r = 0; r < R; ++r) ovals[pos * R + r] = vals[s * R + r];
}

__global__ void pack_rows_kernel(const double* __restrict__ c, double* __restrict__ out, int64_t n, int R) {
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n * R) return;
  int64_t row = i / R;
  int r = int(i - row * R);
  out[i] = c[row + n * r];
}

inline bool fock_key(const int16_t* f, int N, uint64_t* key) {
  uint64_t k = 0;
  for (int i = 0; i < 2 * N; ++i) {
    if (f[i] < 0 || f[i] > 15) return false;
    k |= uint64_t(f[i]) << (4 * i);
  }
  *key = k;
  return true;
}

}  // namespace

#define FCG_CUDA(call)                                                               \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess) {                                                         \
      ctx->err = std::string(#call) + ": " + cudaGetErrorString(e_);                 \
      return e_ == cudaErrorMemoryAllocation ? FCG_ENOMEM : FCG_ECUDA;               \
    }                                                                                \
  } while (0)

#define FCG_REQUIRE(cond, code, msg) \
  do {                               \
    if (!(cond)) {                   \
      ctx->err = (msg);              \
      return (code);                 \
    }                                \
  } while (0)

extern "C" {

int fcg_sigma_open(fcg_ctx* ctx, int R, const double* c, double thresh, int nbody, int64_t* n_out) {
  if (!ctx) return FCG_EINVAL;
  FCG_REQUIRE(ctx->have_state, FCG_ESTATE, "fcg_state_set must come first");
  FCG_REQUIRE(c && n_out, FCG_EINVAL, "null pointer");
  FCG_REQUIRE(R >= 1 && R <= kOpenMaxR, FCG_ELIMIT, "R must be in [1, 16]");
  FCG_REQUIRE(thresh >= 0.0, FCG_EINVAL, "thresh must be >= 0");
  FCG_CUDA(cudaSetDevice(ctx->device));
  {
    const int rc = ensure_open_dressed(ctx);
    if (rc) return rc;
  }
  *n_out = 0;
  const int N = ctx->N;
  const int nmax1 = ctx->nmax + 1;
  const Plan& P = ctx->plan;
  // ---- host plan: bra sectors and open term records per (ket sector, transfer) -------
  ProblemInfo pi;
  pi.N = N;
  pi.norb = ctx->norb;
  pi.nmax = ctx->nmax;
  pi.trm = &ctx->trm;
  pi.n_terms = ctx->n_terms;
  pi.trans = &ctx->trans;
  pi.n_trans = ctx->n_trans;
  pi.blk_index = &ctx->h_blk_index;
  pi.blocks = &ctx->h_blocks;
  pi.dress = &ctx->dress;
  pi.dressing = &ctx->open_dressing;
  std::vector<std::vector<int>> terms_of(ctx->n_trans);
  for (int t = 0; t < ctx->n_terms; ++t) terms_of[ctx->trm[int64_t(t) * kTrmCols + 1]].push_back(t);
  std::unordered_map<uint64_t, int32_t> bsec_of;
  ctx->open_bra_fock.clear();
  ctx->open_strides.clear();
  ctx->open_dims.clear();
  std::vector<OpenTerm> ots;
  std::vector<OpenItem> items;
  std::vector<int16_t> fb(2 * N);
  int64_t flops_ref = 0;
  std::unordered_set<int32_t> tdm_used;  // TDM blocks the jobs read
  for (size_t sk = 0; sk < P.sec_start.size(); ++sk) {
    const int16_t* fk = &P.sec_fock[sk * 2 * N];
    for (int tr = 0; tr < ctx->n_trans; ++tr) {
      if (terms_of[tr].empty()) continue;
      bool ok = true;
      for (int i = 0; i < 2 * N; ++i) {
        fb[i] = int16_t(fk[i] + ctx->trans[size_t(tr) * 2 * N + i]);
        if (fb[i] < 0 || fb[i] > ctx->norb[i / 2]) ok = false;
      }
      if (!ok) continue;
      // every cluster must have a local basis in its bra sector (:39-46)
      int64_t dims[kMaxClusters];
      for (int ci = 0; ci < N && ok; ++ci) {
        int bl = ctx->h_blk_index[dense_block_index(nmax1, ci, kOpH, fb[2 * ci], fb[2 * ci + 1], fb[2 * ci],
                                                    fb[2 * ci + 1])];
        if (bl < 0)
          ok = false;
        else
          dims[ci] = ctx->h_blocks[bl].mb;
      }
      if (!ok) continue;
      uint64_t key;
      fock_key(fb.data(), N, &key);
      int32_t bs;
      auto it = bsec_of.find(key);
      if (it == bsec_of.end()) {
        bs = int32_t(ctx->open_bra_fock.size() / (2 * N));
        FCG_REQUIRE(bs < (1 << 23), FCG_ELIMIT, "too many bra sectors for the open sigma key");
        bsec_of[key] = bs;
        ctx->open_bra_fock.insert(ctx->open_bra_fock.end(), fb.begin(), fb.end());
        int64_t stride = 1;
        for (int ci = 0; ci < N; ++ci) {
          ctx->open_strides.push_back(stride);
          ctx->open_dims.push_back(dims[ci]);
          stride *= dims[ci];
        }
        FCG_REQUIRE(stride < (int64_t(1) << kKeyIdxBits), FCG_ELIMIT, "bra sector product space exceeds 2^40");
      } else {
        bs = it->second;
      }
      const int32_t ot_off = int32_t(ots.size());
      for (int t : terms_of[tr]) {
        const int32_t* r = &ctx->trm[int64_t(t) * kTrmCols];
        if (r[0] > nbody) continue;
        OpenTerm o{};
        if (!make_term_sector(pi, t, fb.data(), fk, o.ts)) continue;
        const int pos = ctx->dress[t].pos < 0 ? 0 : ctx->dress[t].pos;
        const int cw = r[2 + pos];
        o.wmax_off = ctx->wmax_index[(int64_t(t) * nmax1 + fb[2 * cw]) * nmax1 + fb[2 * cw + 1]];
        o.bsec = bs;
        o.n_act = int8_t(1 + o.ts.nrem);
        o.c_act[0] = int8_t(cw);
        o.mb_act[0] = int16_t(o.ts.w_mb);
        int64_t cnt = o.ts.w_mb;
        for (int q = 0; q < o.ts.nrem; ++q) {
          const int cq = o.ts.cr[q];
          const int op = r[6 + ctx->dress[t].rem_pos[q]];
          const int bl = ctx->h_blk_index[dense_block_index(nmax1, cq, op, fb[2 * cq], fb[2 * cq + 1], fk[2 * cq],
                                                            fk[2 * cq + 1])];
          o.gmax_off[q] = ctx->gmax_off[bl];
          o.c_act[1 + q] = int8_t(cq);
          o.mb_act[1 + q] = int16_t(o.ts.g_mb[q]);
          cnt *= o.ts.g_mb[q];
        }
        FCG_REQUIRE(cnt < (int64_t(1) << 31), FCG_ELIMIT, "bra tuples of one term exceed 2^31");
        o.out_count = int32_t(cnt);
        // the reference's GEMM flops of this (ket, term) job (contract_matvec_thread,
        // src/tpsci_matvec_thread.jl:279-818, no prescreen): bra dims M and orbital index
        // lengths n in term order
        {
          const int nbd = r[0];
          int64_t M[4] = {1, 1, 1, 1}, nn[4] = {1, 1, 1, 1};
          for (int o2 = 0; o2 < nbd; ++o2) {
            const int cq = r[2 + o2];
            const int bl = ctx->h_blk_index[dense_block_index(nmax1, cq, r[6 + o2], fb[2 * cq], fb[2 * cq + 1],
                                                              fk[2 * cq], fk[2 * cq + 1])];
            M[o2] = ctx->h_blocks[bl].mb;
            nn[o2] = r[22 + o2];
            tdm_used.insert(bl);
          }
          int64_t f = 0;
          if (nbd == 2) f = nn[0] * nn[1] * M[0] + nn[1] * M[0] * M[1];
          if (nbd == 3) f = M[2] * (nn[0] * nn[1] * nn[2] + nn[0] * nn[1] * M[1] + nn[0] * M[0] * M[1]);
          if (nbd == 4)
            f = M[3] * (nn[0] * nn[1] * nn[2] * nn[3] +
                        M[2] * (nn[0] * nn[1] * nn[2] + nn[0] * nn[1] * M[1] + nn[0] * M[0] * M[1]));
          flops_ref += 2 * f * int64_t(P.sec_count[sk]);
        }
        ots.push_back(o);
      }
      const int32_t nt = int32_t(ots.size()) - ot_off;
      if (nt > 0) items.push_back(OpenItem{int32_t(P.sec_start[sk]), int32_t(P.sec_count[sk]), ot_off, nt});
    }
  }
  ctx->open_R = R;
  ctx->open_rows = 0;
  if (items.empty()) return FCG_OK;
  std::vector<int64_t> prefix(items.size() + 1, 0);
  for (size_t i = 0; i < items.size(); ++i) prefix[i + 1] = prefix[i] + int64_t(items[i].nrow) * items[i].nt;
  const int64_t n_jobs = prefix.back();
  // ---- device ---------------------------------------------------------------------------
  cudaStream_t s = ctx->stream;
  const int64_t n = ctx->n_cfg;
  FCG_CUDA(ctx->d_oterms.upload(ots.data(), ots.size(), s));
  FCG_CUDA(ctx->d_oitems.upload(items.data(), items.size(), s));
  FCG_CUDA(ctx->d_oprefix.upload(prefix.data(), prefix.size(), s));
  FCG_CUDA(ctx->d_ostrides.upload(ctx->open_strides.data(), ctx->open_strides.size(), s));
  FCG_CUDA(ctx->d_in64.alloc(size_t(n) * R));
  FCG_CUDA(ctx->d_c64.alloc(size_t(n) * R));
  FCG_CUDA(cudaMemcpyAsync(ctx->d_in64.p, c, sizeof(double) * n * R, cudaMemcpyHostToDevice, s));
  pack_rows_kernel<<<unsigned((n * R + 255) / 256), 256, 0, s>>>(ctx->d_in64.p, ctx->d_c64.p, n, R);
  FCG_CUDA(cudaGetLastError());
  FCG_CUDA(ctx->d_counters.alloc(5));
  FCG_CUDA(cudaMemsetAsync(ctx->d_counters.p, 0, 4 * sizeof(unsigned long long), s));
  FCG_CUDA(ctx->d_ojobs.alloc(size_t(n_jobs)));
  OpenParams p{};
  p.ot = ctx->d_oterms.p;
  p.items = ctx->d_oitems.p;
  p.prefix = ctx->d_oprefix.p;
  p.n_items = int64_t(items.size());
  p.n_jobs = n_jobs;
  p.cfg = ctx->d_cfg.p;
  p.c = ctx->d_c64.p;
  p.strides = ctx->d_ostrides.p;
  p.N = N;
  p.R = R;
  p.thresh = thresh;
  FCG_CUDA(cudaEventRecord(ctx->ev0, s));
  screen_kernel<<<unsigned((n_jobs + 255) / 256), 256, 0, s>>>(p, ctx->d_wmax.p, ctx->d_gmax.p, ctx->d_ojobs.p,
                                                              ctx->d_counters.p);
  FCG_CUDA(cudaGetLastError());
  unsigned long long cnt[4];
  FCG_CUDA(cudaMemcpyAsync(cnt, ctx->d_counters.p, sizeof(cnt), cudaMemcpyDeviceToHost, s));
  FCG_CUDA(cudaStreamSynchronize(s));
  const int64_t n_kept = int64_t(cnt[0]);
  const int64_t n_elem = int64_t(cnt[1]);
  int launches = 2;
  if (n_kept > 0) {
    // a warp's slice: the largest job tiles, up to kExpSlice; as many warps to a CTA as fit.
    // The register sums serve index lengths up to kExpMaxD (the second and third remaining
    // clusters of the longest term), the shared-memory sums anything longer.
    int d_max = 1, slice = 16;
    for (const OpenTerm& o : ots)
      for (int r = 1; r < o.ts.nrem; ++r) d_max = std::max<int>(d_max, o.ts.g_dim[r]);
    for (const OpenTerm& o : ots)
      slice = std::max(slice, expand_tiles(o.ts.nrem, o.ts.rest_len, o.ts.g_dim, o.mb_act, d_max > kExpMaxD).bytes);
    slice = std::min(slice, kExpSlice);
    const int warps = std::min(kExpWarps, kExpCtaBytes / slice), threads = 32 * warps;
    const size_t smem = size_t(warps) * size_t(slice);
    auto kernel = d_max <= 3 ? expand_jobs_kernel<3>
                  : d_max == 4 ? expand_jobs_kernel<4>
                  : d_max <= kExpMaxD ? expand_jobs_kernel<kExpMaxD> : expand_jobs_kernel<0>;
    FCG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kExpCtaBytes));
    int per_sm = 0, n_sm = 0;
    FCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    FCG_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, ctx->device));
    const int64_t grid =
        std::max<int64_t>(1, std::min<int64_t>(int64_t(std::max(per_sm, 1)) * n_sm, (n_kept + warps - 1) / warps));
    // table: twice the contributions, power of two, at least 4096 slots; doubled on overflow
    unsigned long long cap = 4096;
    while (cap < 2ull * (unsigned long long)n_elem && cap < (1ull << 28)) cap <<= 1;
    for (int attempt = 0;; ++attempt) {
      FCG_CUDA(ctx->d_hkeys.alloc(cap));
      FCG_CUDA(ctx->d_hvals.alloc(cap * R));
      FCG_CUDA(cudaMemsetAsync(ctx->d_hkeys.p, 0xFF, cap * sizeof(unsigned long long), s));
      FCG_CUDA(cudaMemsetAsync(ctx->d_hvals.p, 0, cap * R * sizeof(double), s));
      FCG_CUDA(cudaMemsetAsync(ctx->d_counters.p + 2, 0, 3 * sizeof(unsigned long long), s));
      FCG_CUDA(cudaEventRecord(ctx->ev2, s));
      kernel<<<unsigned(grid), threads, smem, s>>>(
          p, ctx->d_ojobs.p, n_kept, ctx->d_ow64.p, ctx->d_op64.p, ctx->d_ow32.p, ctx->d_op32.p, ctx->d_gmax.p,
          ExpandTable{ctx->d_hkeys.p, ctx->d_hvals.p, cap - 1, ctx->d_counters.p}, slice);
      FCG_CUDA(cudaGetLastError());
      FCG_CUDA(cudaEventRecord(ctx->ev3, s));
      FCG_CUDA(cudaMemcpyAsync(cnt, ctx->d_counters.p, sizeof(cnt), cudaMemcpyDeviceToHost, s));
      FCG_CUDA(cudaStreamSynchronize(s));
      launches += 2;
      if (cnt[2] == 0) break;
      FCG_REQUIRE(attempt < 3 && cap < (1ull << 31), FCG_ENOMEM, "open sigma hash table overflow");
      cap <<= 1;
    }
    FCG_CUDA(ctx->d_okeys.alloc(cap));
    FCG_CUDA(ctx->d_ovals.alloc(cap * R));
    compact_kernel<<<unsigned((cap + 255) / 256), 256, 0, s>>>(ctx->d_hkeys.p, ctx->d_hvals.p, cap, R,
                                                               ctx->d_okeys.p, ctx->d_ovals.p, ctx->d_counters.p);
    FCG_CUDA(cudaGetLastError());
    FCG_CUDA(cudaEventRecord(ctx->ev1, s));
    FCG_CUDA(cudaMemcpyAsync(cnt, ctx->d_counters.p, sizeof(cnt), cudaMemcpyDeviceToHost, s));
    FCG_CUDA(cudaStreamSynchronize(s));
    launches += 1;
    const int64_t n_rows = int64_t(cnt[3]);
    FCG_CUDA(ctx->open_keys.alloc(size_t(n_rows)));
    FCG_CUDA(ctx->open_vals.alloc(size_t(n_rows) * R));
    ctx->open_rows = n_rows;
    FCG_CUDA(cudaMemcpyAsync(ctx->open_keys.p, ctx->d_okeys.p, n_rows * sizeof(unsigned long long),
                             cudaMemcpyDeviceToHost, s));
    FCG_CUDA(cudaMemcpyAsync(ctx->open_vals.p, ctx->d_ovals.p, n_rows * R * sizeof(double),
                             cudaMemcpyDeviceToHost, s));
    FCG_CUDA(cudaStreamSynchronize(s));
    float ms = 0.f;
    FCG_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    ctx->stats.last_kernel_ms = ms;
    FCG_CUDA(cudaEventElapsedTime(&ms, ctx->ev2, ctx->ev3));
    ctx->stats.open_expand_ms = ms;
  }
  // compulsory bytes: the TDM blocks the jobs touch, C, and one key + row per output
  int64_t tdm_bytes = 0;
  for (int32_t bl : tdm_used) {
    const BlockInfo& B = ctx->h_blocks[bl];
    tdm_bytes += int64_t(B.nidx) * B.mb * B.mk * 8;
  }
  ctx->stats.open_flops_reference = flops_ref;
  ctx->stats.open_bytes = tdm_bytes + 8 * n * R + ctx->open_rows * (6 * int64_t(N) + 8 * int64_t(R));
  ctx->stats.kernel_launches = launches;
  ctx->stats.open_jobs = n_jobs;
  ctx->stats.open_jobs_kept = n_kept;
  ctx->stats.open_contractions = n_elem;
  *n_out = ctx->open_rows;
  return FCG_OK;
}

int fcg_sigma_open_fetch(fcg_ctx* ctx, int16_t* fock, int16_t* cfg, double* coeff) {
  if (!ctx) return FCG_EINVAL;
  FCG_REQUIRE(fock && cfg && coeff, FCG_EINVAL, "null pointer");
  const int N = ctx->N;
  const int R = ctx->open_R;
  const int64_t m = ctx->open_rows;
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < m; ++i) {
    const unsigned long long key = ctx->open_keys.p[i];
    const int64_t bs = int64_t(key >> kKeyIdxBits);
    int64_t idx = int64_t(key & ((1ull << kKeyIdxBits) - 1));
    std::memcpy(fock + i * 2 * N, &ctx->open_bra_fock[bs * 2 * N], sizeof(int16_t) * 2 * N);
    for (int c = 0; c < N; ++c) {
      const int64_t d = ctx->open_dims[bs * N + c];
      cfg[i * N + c] = int16_t(idx % d);
      idx /= d;
    }
    for (int r = 0; r < R; ++r) coeff[i + m * r] = ctx->open_vals.p[size_t(i) * R + r];
  }
  return FCG_OK;
}

}  // extern "C"
