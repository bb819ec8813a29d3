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
//   plan kernels    bra sectors and one OpenTerm record per (ket sector, term) whose target exists
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
//   compact_kernel  occupied slots -> (key, values); the slots are emptied for the next call.
// A table that overflows its probe limit sets a flag and the call is repeated with a
// table twice as large.
#include <cmath>
#include <cstring>

#include "dprim.cuh"
#include "fcg_ctx.cuh"

using namespace fcg;

namespace {

constexpr unsigned long long kEmpty = ~0ull;
constexpr int kMaxProbe = 1 << 16;
constexpr int kKeyIdxBits = 40;

// counters: [0] kept jobs, [1] elements of kept jobs, [2] table overflow, [3] output rows,
// [4] next job of the expand warps; of the plan: [5] bra sectors, [6] records, [7] items, [8] jobs,
// [9] reference flops, [10] error, [11] longest index of the register sums, [12] largest tiles with
// register sums, [13] with shared-memory sums, [14] bytes of the TDM blocks in use
constexpr int kCounters = 15;
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
// threshold are rare (0.4 % at 1e-3), so the table's atomics are not.  24 orbitals, 300 configurations, 1e-3:
// issue slots 32 %, FP64 pipe 54 % (the exact values), 16 warps an SM by the 128 registers of a thread.
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

// A block per kCompactSlots table slots: the occupied ones to the output (one place reserved per
// block), each emptied as it is read, so that the next call finds the table as new and a call
// fills (10.7 GB, 1.6 ms at 2^28 slots of 4 roots) only what it adds.  Bound: the read of the keys:
// 1.26 ms for 2^28 slots and 4.9e6 rows (a thread and an atomic per slot: 3.3 ms).
constexpr int kCompactThreads = 256, kCompactKeys = 16, kCompactSlots = kCompactThreads * kCompactKeys;
__global__ void __launch_bounds__(kCompactThreads) compact_kernel(unsigned long long* __restrict__ keys,
                                                                  double* __restrict__ vals, int R,
                                                                  unsigned long long* __restrict__ okeys,
                                                                  double* __restrict__ ovals,
                                                                  unsigned long long* __restrict__ counters) {
  __shared__ unsigned warp_n[kCompactThreads / 32];
  __shared__ unsigned long long first;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned long long base = (unsigned long long)blockIdx.x * kCompactSlots + 2 * threadIdx.x;
  ulonglong2 k[kCompactKeys / 2];
  int n = 0;
#pragma unroll
  for (int i = 0; i < kCompactKeys / 2; ++i) {
    k[i] = *reinterpret_cast<const ulonglong2*>(keys + base + 2 * kCompactThreads * i);
    n += (k[i].x != kEmpty) + (k[i].y != kEmpty);
  }
  int before = n;  // inclusive, then exclusive, over the warp
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, before, d);
    if (lane >= d) before += y;
  }
  if (lane == 31) warp_n[wid] = unsigned(before);
  before -= n;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned sum = 0;
    for (int w = 0; w < kCompactThreads / 32; ++w) {
      const unsigned c = warp_n[w];
      warp_n[w] = sum;
      sum += c;
    }
    first = sum ? atomicAdd(counters + 3, (unsigned long long)sum) : 0ull;
  }
  __syncthreads();
  unsigned long long pos = first + warp_n[wid] + (unsigned long long)before;
  auto take = [&](unsigned long long key, unsigned long long slot) {
    if (key == kEmpty) return;
    okeys[pos] = key;
    keys[slot] = kEmpty;
    for (int r = 0; r < R; ++r) {
      ovals[pos * R + r] = vals[slot * R + r];
      vals[slot * R + r] = 0.0;
    }
    ++pos;
  };
#pragma unroll
  for (int i = 0; i < kCompactKeys / 2; ++i) {
    const unsigned long long slot = base + 2 * kCompactThreads * i;
    take(k[i].x, slot);
    take(k[i].y, slot + 1);
  }
}

constexpr int64_t kOpenWarps = 152 * 32;

// ---- plan ------------------------------------------------------------------------------------
// Over the pairs (ket sector, transfer), ket sector major: count, number the bra sectors and scan,
// write.  Bound: the table reads of term_sector_of, a serial chain per term.  Host loops with
// hash maps took 29 ms for 193 sectors x 1441 transfers (194,496 records) and their upload 1 ms;
// the kernels take under 1 ms, and the call 28 ms instead of 69 with the emptied table below.
struct OpenPlan {
  TermTables tt;  // the open dressing's
  const int16_t* sec_fock;
  const int32_t* sec_start;  // rows of the ket sectors
  const int32_t* sec_count;
  const int16_t* trans;
  const int32_t* first_of_tr;  // terms of each transfer
  const int32_t* tr_terms;
  const int32_t* norb;
  const int64_t* wmax_index;
  const int64_t* gmax_off;
  int64_t n_pairs;
  int n_trans, N, nbody;
  int warp_pairs;  // pairs of a warp of the count and records kernels
  uint64_t* key;    // bra sector of each pair (4 bits per entry)
  int32_t* nt;      // its terms with at most nbody clusters whose TDM blocks exist; -1: no target
  int64_t* ot;      // the same for the scan (0 without a target)
  int64_t* has;     // 1: an item (some terms)
  int64_t* jobs;    // (row, term) jobs
};

// the bra sector of pair i (4 bits per entry), false: none
__device__ __forceinline__ bool open_target(const OpenPlan& p, int64_t i, uint64_t* key) {
  const int64_t sk = i / p.n_trans;
  const int tr = int(i - sk * p.n_trans);
  if (p.first_of_tr[tr] == p.first_of_tr[tr + 1]) return false;
  const int16_t* fk = p.sec_fock + sk * 2 * p.N;
  uint64_t k = 0;
  for (int c = 0; c < p.N; ++c) {
    const int fa = fk[2 * c] + p.trans[(int64_t(tr) * p.N + c) * 2], fb = fk[2 * c + 1] + p.trans[(int64_t(tr) * p.N + c) * 2 + 1];
    if (fa < 0 || fa > p.norb[c] || fb < 0 || fb > p.norb[c]) return false;
    // every cluster must have a local basis in its bra sector (:39-46)
    if (p.tt.blk[dense_block_index(p.tt.nmax1, c, kOpH, fa, fb, fa, fb)] < 0) return false;
    k |= uint64_t(fa | fb << 4) << (8 * c);
  }
  *key = k;
  return true;
}

// The (pair, term) combinations of a warp's pairs, side by side over its lanes.  A warp has p.warp_pairs
// pairs, lane l the l-th; the terms of a pair are checked in order, 32 combinations a step.  Bound: the
// chain of table reads of one term (about 7 us with its record), so few pairs are spread over many warps:
// 12 orbitals, one row, count and records 96 us with a thread for every pair's list, 19 so.
struct OpenLanes {
  uint64_t key = 0;        // of this lane's pair: bra sector,
  int first = 0;           // first term,
  int begin = 0, end = 0;  // and its combinations [begin, end)
  int total = 0;           // of the warp
};
__device__ __forceinline__ int64_t open_pair_of(const OpenPlan& p) {  // this thread's pair (n_pairs: past the last)
  const int64_t thread = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  return lane < p.warp_pairs ? min((thread >> 5) * p.warp_pairs + lane, p.n_pairs + 1) : p.n_pairs + 1;
}
__device__ __forceinline__ OpenLanes open_lanes(const OpenPlan& p, bool target, int64_t i, uint64_t key) {
  OpenLanes L;
  int n = 0;
  if (target) {
    const int tr = int(i % p.n_trans);
    L.key = key;
    L.first = p.first_of_tr[tr];
    n = p.first_of_tr[tr + 1] - L.first;
  }
  L.end = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, L.end, d);
    if (int(threadIdx.x & 31) >= d) L.end += y;
  }
  L.begin = L.end - n;
  L.total = __shfl_sync(0xffffffffu, L.end, 31);
  return L;
}

// one combination: ket sector, term, bra sector
struct OpenPair {
  int64_t i;  // pair
  int lane;   // whose pair
  int t;
  const int16_t* fk;
  int64_t rows;
  int16_t fb[2 * kMaxClusters];
};
// combination x of the warp (all lanes take part; x >= total: none, t < 0)
__device__ __forceinline__ OpenPair open_pair(const OpenPlan& p, const OpenLanes& L, int x) {
  int lane = 0;  // pairs that end at or before x
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
    if (__shfl_sync(0xffffffffu, L.end, lane + d - 1) <= x) lane += d;
  OpenPair P;
  P.lane = lane;
  const uint64_t key = __shfl_sync(0xffffffffu, L.key, lane);
  const int q = __shfl_sync(0xffffffffu, L.first, lane) + x - __shfl_sync(0xffffffffu, L.begin, lane);
  P.i = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * p.warp_pairs + lane;
  P.t = -1;
  if (x >= L.total) return P;
  const int64_t sk = P.i / p.n_trans;
  P.t = p.tr_terms[q];
  P.fk = p.sec_fock + sk * 2 * p.N;
  P.rows = p.sec_count[sk];
#pragma unroll
  for (int c = 0; c < 2 * kMaxClusters; ++c) P.fb[c] = int16_t((key >> (4 * c)) & 15);
  return P;
}

__global__ void open_count_kernel(OpenPlan p) {
  const int64_t i = open_pair_of(p);
  const int lane = threadIdx.x & 31;
  uint64_t key = 0;
  const bool target = i < p.n_pairs && open_target(p, i, &key);
  const OpenLanes L = open_lanes(p, target, i, key);
  int nt = 0;
  for (int x0 = 0; x0 < L.total; x0 += 32) {
    const OpenPair P = open_pair(p, L, x0 + lane);
    bool exists, record = false;
    int64_t fma;
    if (P.t >= 0 && p.tt.trm[int64_t(P.t) * kTrmCols] <= p.nbody)
      term_count(p.tt, P.t, P.fb, P.fk, &exists, &record, &fma);
    const unsigned has = __ballot_sync(0xffffffffu, record);
    const int lo = max(L.begin - x0, 0), hi = min(L.end - x0, 32);  // this lane's pair in the step
    if (lo < hi) nt += __popc(has & ((hi < 32 ? 1u << hi : 0u) - 1u) & ~((1u << lo) - 1u));
  }
  if (i > p.n_pairs) return;
  if (i < p.n_pairs) p.nt[i] = target ? nt : -1;
  if (target) p.key[i] = key;
  p.ot[i] = nt;
  p.has[i] = nt > 0 ? 1 : 0;
  p.jobs[i] = nt > 0 ? int64_t(nt) * p.sec_count[i / p.n_trans] : 0;
}

// bra sectors numbered by their first pair: an open-addressed table of pairs (kEmpty: none)
__global__ void open_sectors_kernel(OpenPlan p, unsigned long long* __restrict__ table, int64_t mask,
                                    int64_t* __restrict__ slot_of) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= p.n_pairs || p.nt[i] < 0) return;
  const uint64_t key = p.key[i];
  uint64_t h = key * 0x9E3779B97F4A7C15ull;
  h ^= h >> 29;
  for (int64_t at = int64_t(h & uint64_t(mask));; at = (at + 1) & mask) {  // at most half full
    const unsigned long long cur = atomicCAS(table + at, kEmpty, (unsigned long long)i);
    if (cur == kEmpty || p.key[cur] == key) {
      if (cur > (unsigned long long)i) atomicMin(table + at, (unsigned long long)i);
      slot_of[i] = at;
      return;
    }
  }
}

__global__ void open_first_kernel(OpenPlan p, const unsigned long long* __restrict__ table,
                                  const int64_t* __restrict__ slot_of, int64_t* __restrict__ rep,
                                  int64_t* __restrict__ flag) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i > p.n_pairs) return;
  const int64_t r = i < p.n_pairs && p.nt[i] >= 0 ? int64_t(table[slot_of[i]]) : -1;
  if (i < p.n_pairs) rep[i] = r;
  flag[i] = r == i ? 1 : 0;
}

// the last elements of four scanned arrays of n behind one another, for the host
__global__ void open_sizes_kernel(const int64_t* __restrict__ a, int64_t n, unsigned long long* __restrict__ out) {
  out[threadIdx.x] = (unsigned long long)a[(threadIdx.x + 1) * n - 1];
}

// The same with the scans, a CTA (1024 threads) per array: spaces of few sectors, whose call is some
// twenty launches of a few microseconds (12 orbitals, one row: 3 us for five kernels' 9).
constexpr int64_t kOpenScan = 8192;
__global__ void __launch_bounds__(1024) open_scan_kernel(int64_t* __restrict__ a, int64_t n, unsigned long long* __restrict__ out) {
  __shared__ int64_t sums[32];
  int64_t* v = a + blockIdx.x * n;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t before = 0;  // of the earlier rounds
  for (int64_t i0 = 0; i0 < n; i0 += 1024) {
    const int64_t i = i0 + threadIdx.x;
    const int64_t own = i < n ? v[i] : 0;
    int64_t x = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) sums[wid] = x;
    __syncthreads();
    int64_t all = 0, below = 0;
    for (int w = 0; w < 32; ++w) {
      const int64_t y = sums[w];
      all += y;
      if (w < wid) below += y;
    }
    if (i < n) v[i] = before + below + x - own;
    before += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = (unsigned long long)v[n - 1];
}

// what the records of a thread add to the counters
struct OpenSums {
  unsigned long long flops = 0, d_max = 1, reg = 0, shared = 0, err = 0;
};

// the record of a combination (false: none); used[block] = 1 for every TDM block read
__device__ __forceinline__ bool open_record(const OpenPlan& p, const OpenPair& P, int32_t bs, OpenTerm& o,
                                            int32_t* __restrict__ used, OpenSums& S) {
  const int t = P.t;
  const int32_t* r = p.tt.trm + int64_t(t) * kTrmCols;
  int64_t fma;
  o = OpenTerm{};
  if (r[0] > p.nbody || !term_sector_of(p.tt, t, P.fb, P.fk, o.ts, &fma)) return false;
  const int nmax1 = p.tt.nmax1;
  auto block_of = [&](int c, int op) {
    return p.tt.blk[dense_block_index(nmax1, c, op, P.fb[2 * c], P.fb[2 * c + 1], P.fk[2 * c], P.fk[2 * c + 1])];
  };
  const TermDress& dr = p.tt.dress[t];
  const int cw = r[2 + (dr.pos < 0 ? 0 : dr.pos)];
  o.wmax_off = p.wmax_index[(int64_t(t) * nmax1 + P.fb[2 * cw]) * nmax1 + P.fb[2 * cw + 1]];
  o.bsec = bs;
  o.n_act = int8_t(1 + o.ts.nrem);
  o.c_act[0] = int8_t(cw);
  o.mb_act[0] = int16_t(o.ts.w_mb);
  int64_t cnt = o.ts.w_mb;
  for (int a = 0; a < o.ts.nrem; ++a) {
    o.gmax_off[a] = p.gmax_off[block_of(o.ts.cr[a], r[6 + dr.rem_pos[a]])];
    o.c_act[1 + a] = o.ts.cr[a];
    o.mb_act[1 + a] = int16_t(o.ts.g_mb[a]);
    cnt *= o.ts.g_mb[a];
    if (a > 0) S.d_max = max(S.d_max, (unsigned long long)o.ts.g_dim[a]);
  }
  if (cnt >= (int64_t(1) << 31)) S.err = 2;
  o.out_count = int32_t(cnt);
  S.reg = max(S.reg, (unsigned long long)expand_tiles(o.ts.nrem, o.ts.rest_len, o.ts.g_dim, o.mb_act, false).bytes);
  S.shared = max(S.shared, (unsigned long long)expand_tiles(o.ts.nrem, o.ts.rest_len, o.ts.g_dim, o.mb_act, true).bytes);
  // the reference's GEMM flops of this (ket, term) job (contract_matvec_thread,
  // src/tpsci_matvec_thread.jl:279-818, no prescreen): bra dims M and orbital index
  // lengths n in term order
  int64_t M[4] = {1, 1, 1, 1}, n[4] = {1, 1, 1, 1};
#pragma unroll
  for (int a = 0; a < 4; ++a)
    if (a < r[0]) {
      const int bl = block_of(r[2 + a], r[6 + a]);
      M[a] = p.tt.blocks[bl].mb;
      n[a] = r[22 + a];
      used[bl] = 1;
    }
  int64_t f = 0;
  if (r[0] == 2) f = n[0] * n[1] * M[0] + n[1] * M[0] * M[1];
  if (r[0] == 3) f = M[2] * (n[0] * n[1] * n[2] + n[0] * n[1] * M[1] + n[0] * M[0] * M[1]);
  if (r[0] == 4)
    f = M[3] * (n[0] * n[1] * n[2] * n[3] + M[2] * (n[0] * n[1] * n[2] + n[0] * n[1] * M[1] + n[0] * M[0] * M[1]));
  S.flops += (unsigned long long)(2 * f * P.rows);
  return true;
}

// the records, items and bra sectors; counters [9] .. [13].  Scanned: flag (bra sector ids), ot, has, jobs.
__global__ void open_records_kernel(OpenPlan p, const int64_t* __restrict__ rep, const int64_t* __restrict__ id,
                                    OpenTerm* __restrict__ ots, OpenItem* __restrict__ items,
                                    int64_t* __restrict__ prefix, int16_t* __restrict__ bra_fock,
                                    int64_t* __restrict__ strides, int64_t* __restrict__ bra_dims,
                                    int32_t* __restrict__ used, unsigned long long* __restrict__ counters) {
  const int64_t i = open_pair_of(p);
  const int lane = threadIdx.x & 31;
  if (i == 0) prefix[p.has[p.n_pairs]] = p.jobs[p.n_pairs];
  const bool target = i < p.n_pairs && rep[i] >= 0;
  const uint64_t key = target ? p.key[i] : 0;
  const int32_t bs = target ? int32_t(id[rep[i]]) : 0;
  OpenSums S;
  if (target && rep[i] == i) {
    int64_t stride = 1;
    for (int c = 0; c < p.N; ++c) {
      const int fa = int((key >> (8 * c)) & 15), fb = int((key >> (8 * c + 4)) & 15);
      const int64_t dim = p.tt.blocks[p.tt.blk[dense_block_index(p.tt.nmax1, c, kOpH, fa, fb, fa, fb)]].mb;
      bra_fock[(int64_t(bs) * p.N + c) * 2] = int16_t(fa);
      bra_fock[(int64_t(bs) * p.N + c) * 2 + 1] = int16_t(fb);
      strides[int64_t(bs) * p.N + c] = stride;
      bra_dims[int64_t(bs) * p.N + c] = dim;
      stride = min(stride * dim, int64_t(1) << kKeyIdxBits);
    }
    if (stride >= (int64_t(1) << kKeyIdxBits)) S.err = 1;
  }
  if (target && p.has[i] != p.has[i + 1]) {
    const int64_t it = p.has[i];
    prefix[it] = p.jobs[i];
    items[it] = OpenItem{p.sec_start[i / p.n_trans], p.sec_count[i / p.n_trans], int32_t(p.ot[i]),
                         int32_t(p.ot[i + 1] - p.ot[i])};
  }
  // the warp's records follow one another from its first pair's
  const OpenLanes L = open_lanes(p, target, i, target ? p.key[i] : 0);
  int64_t at = __shfl_sync(0xffffffffu, p.ot[min(i, p.n_pairs)], 0);
  OpenTerm o;
  for (int x0 = 0; x0 < L.total; x0 += 32) {
    const OpenPair P = open_pair(p, L, x0 + lane);
    const int32_t b = __shfl_sync(0xffffffffu, bs, P.lane & 31);
    const bool has = P.t >= 0 && open_record(p, P, b, o, used, S);
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (has) ots[at + __popc(m & ((1u << lane) - 1u))] = o;
    at += __popc(m);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    S.flops += __shfl_xor_sync(0xffffffffu, S.flops, d);
    S.d_max = max(S.d_max, __shfl_xor_sync(0xffffffffu, S.d_max, d));
    S.reg = max(S.reg, __shfl_xor_sync(0xffffffffu, S.reg, d));
    S.shared = max(S.shared, __shfl_xor_sync(0xffffffffu, S.shared, d));
    S.err = max(S.err, __shfl_xor_sync(0xffffffffu, S.err, d));
  }
  if (lane != 0) return;
  if (S.flops) atomicAdd(counters + 9, S.flops);
  auto raise = [&](int k, unsigned long long v) {  // a stale read only costs an atomic
    if (*reinterpret_cast<volatile unsigned long long*>(counters + k) < v) atomicMax(counters + k, v);
  };
  raise(10, S.err);
  raise(11, S.d_max);
  raise(12, S.reg);
  raise(13, S.shared);
}

__global__ void open_bytes_kernel(int64_t n_blocks, const int32_t* __restrict__ used, const BlockInfo* __restrict__ blocks,
                                  unsigned long long* __restrict__ counters) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n_blocks && used[i])
    atomicAdd(counters + 14, (unsigned long long)(int64_t(blocks[i].nidx) * blocks[i].mb * blocks[i].mk * 8));
}

__global__ void pack_rows_kernel(const double* __restrict__ c, double* __restrict__ out, int64_t n, int R) {
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n * R) return;
  int64_t row = i / R;
  int r = int(i - row * R);
  out[i] = c[row + n * r];
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
  const Plan& P = ctx->plan;
  cudaStream_t s = ctx->stream;
  auto& O = ctx->oplan;
  constexpr int kT = 256;
  auto grid_of = [](int64_t n) { return unsigned(std::max<int64_t>((n + kT - 1) / kT, 1)); };
  // ---- plan: bra sectors and open term records per (ket sector, transfer) -----------------
  const int64_t n_sec = int64_t(P.sec_start.size()), n_pairs = n_sec * ctx->n_trans;
  int64_t cap_tab = 64;
  while (cap_tab < 2 * n_pairs) cap_tab <<= 1;
  std::vector<int32_t> rows(size_t(2 * n_sec));  // first rows, then row counts
  for (int64_t i = 0; i < n_sec; ++i) {
    rows[size_t(i)] = int32_t(P.sec_start[size_t(i)]);
    rows[size_t(n_sec + i)] = int32_t(P.sec_count[size_t(i)]);
  }
  FCG_CUDA(O.d_rows.upload(rows.data(), rows.size(), s));
  // table, flag, ot, has, jobs, slot, rep, keys, counts, scratch of the scans
  const int64_t n1 = n_pairs + 1, scr = dprim::scan_scratch(n1) + 1;
  FCG_CUDA(O.d_i64.alloc(size_t(cap_tab + 8 * n1 + scr)));
  FCG_CUDA(O.d_used.alloc(ctx->h_blocks.size()));
  FCG_CUDA(ctx->d_counters.alloc(kCounters));
  FCG_CUDA(cudaMemsetAsync(ctx->d_counters.p, 0, kCounters * sizeof(unsigned long long), s));
  FCG_CUDA(cudaMemsetAsync(O.d_used.p, 0, ctx->h_blocks.size() * sizeof(int32_t), s));
  OpenPlan op{};
  op.tt = TermTables{O.trm, O.dress, O.w_index, O.w_mb, O.rep, ctx->d_blk_index.p, ctx->d_blocks.p, ctx->nmax + 1};
  op.sec_fock = ctx->d_sec_fock.p;
  op.sec_start = O.d_rows.p;
  op.sec_count = O.d_rows.p + n_sec;
  op.trans = O.trans;
  op.first_of_tr = O.first_of_tr;
  op.tr_terms = O.tr_terms;
  op.norb = ctx->d_norb.p;
  op.wmax_index = O.wmax_index;
  op.gmax_off = O.gmax_off;
  op.n_pairs = n_pairs;
  op.n_trans = ctx->n_trans;
  op.N = N;
  op.nbody = nbody;
  // as few pairs to a warp as keep the chip's warps (32 an SM) busy
  op.warp_pairs = 1;
  while (op.warp_pairs < 32 && n_pairs > int64_t(op.warp_pairs) * kOpenWarps) op.warp_pairs *= 2;
  const unsigned warp_grid = unsigned(((n_pairs + op.warp_pairs) / op.warp_pairs * 32 + kT - 1) / kT);
  auto* table = reinterpret_cast<unsigned long long*>(O.d_i64.p);
  int64_t* flag = O.d_i64.p + cap_tab;
  op.ot = flag + n1;
  op.has = op.ot + n1;
  op.jobs = op.has + n1;
  int64_t *slot = op.jobs + n1, *rep = slot + n1;
  op.key = reinterpret_cast<uint64_t*>(rep + n1);
  op.nt = reinterpret_cast<int32_t*>(op.key + n1);
  int64_t* scratch = O.d_i64.p + cap_tab + 8 * n1;
  FCG_CUDA(cudaMemsetAsync(table, 0xFF, size_t(cap_tab) * sizeof(int64_t), s));
  open_count_kernel<<<warp_grid, kT, 0, s>>>(op);
  FCG_CUDA(cudaGetLastError());
  open_sectors_kernel<<<grid_of(n_pairs), kT, 0, s>>>(op, table, cap_tab - 1, slot);
  FCG_CUDA(cudaGetLastError());
  open_first_kernel<<<grid_of(n1), kT, 0, s>>>(op, table, slot, rep, flag);
  FCG_CUDA(cudaGetLastError());
  if (n1 <= kOpenScan) {
    open_scan_kernel<<<4, 1024, 0, s>>>(flag, n1, ctx->d_counters.p + 5);
  } else {
    for (int k = 0; k < 4; ++k) FCG_CUDA(dprim::exclusive_scan<int64_t>(flag + k * n1, n1, scratch, s));
    open_sizes_kernel<<<1, 4, 0, s>>>(flag, n1, ctx->d_counters.p + 5);
  }
  FCG_CUDA(cudaGetLastError());
  FCG_CUDA(O.h_cnt.alloc(kCounters));
  const unsigned long long* cnt = O.h_cnt.p;  // page-locked: three or four waits of a call end with this copy
  constexpr size_t kCntBytes = kCounters * sizeof(unsigned long long);
  FCG_CUDA(cudaMemcpyAsync(O.h_cnt.p, ctx->d_counters.p, kCntBytes, cudaMemcpyDeviceToHost, s));
  FCG_CUDA(cudaStreamSynchronize(s));
  const int64_t n_bra = int64_t(cnt[5]), n_ots = int64_t(cnt[6]), n_items = int64_t(cnt[7]), n_jobs = int64_t(cnt[8]);
  FCG_REQUIRE(n_bra < (1 << 23), FCG_ELIMIT, "too many bra sectors for the open sigma key");
  FCG_REQUIRE(n_ots < (int64_t(1) << 31), FCG_ELIMIT, "too many term records for the open sigma");
  ctx->open_R = R;
  ctx->open_rows = 0;
  FCG_CUDA(ctx->d_oterms.alloc(size_t(n_ots)));
  FCG_CUDA(ctx->d_oitems.alloc(size_t(n_items)));
  FCG_CUDA(ctx->d_oprefix.alloc(size_t(n_items + 1)));
  FCG_CUDA(ctx->d_ostrides.alloc(size_t(n_bra * N)));
  // local dimensions of the bra sectors, then their Fock sectors
  const size_t bra_bytes = size_t(n_bra * N) * (sizeof(int64_t) + 2 * sizeof(int16_t));
  FCG_CUDA(O.d_bra.alloc(bra_bytes));
  int64_t* d_dims = reinterpret_cast<int64_t*>(O.d_bra.p);
  int16_t* d_fock = reinterpret_cast<int16_t*>(d_dims + n_bra * N);
  open_records_kernel<<<warp_grid, kT, 0, s>>>(op, rep, flag, ctx->d_oterms.p, ctx->d_oitems.p, ctx->d_oprefix.p, d_fock,
                                               ctx->d_ostrides.p, d_dims, O.d_used.p, ctx->d_counters.p);
  FCG_CUDA(cudaGetLastError());
  open_bytes_kernel<<<grid_of(int64_t(ctx->h_blocks.size())), kT, 0, s>>>(int64_t(ctx->h_blocks.size()), O.d_used.p,
                                                                         ctx->d_blocks.p, ctx->d_counters.p);
  FCG_CUDA(cudaGetLastError());
  ctx->open_bra.resize(bra_bytes);
  ctx->open_sectors = n_bra;
  if (n_bra > 0) FCG_CUDA(cudaMemcpyAsync(ctx->open_bra.data(), O.d_bra.p, bra_bytes, cudaMemcpyDeviceToHost, s));
  const int64_t n = ctx->n_cfg;
  if (n_items == 0) {  // no term reaches a sector with a basis
    FCG_CUDA(cudaMemcpyAsync(O.h_cnt.p, ctx->d_counters.p, kCntBytes, cudaMemcpyDeviceToHost, s));
    FCG_CUDA(cudaStreamSynchronize(s));
    FCG_REQUIRE(cnt[10] == 0, FCG_ELIMIT, "bra sector product space exceeds 2^40");
    return FCG_OK;
  }
  // ---- device ---------------------------------------------------------------------------
  FCG_CUDA(ctx->d_in64.alloc(size_t(n) * R));
  FCG_CUDA(ctx->d_c64.alloc(size_t(n) * R));
  FCG_CUDA(cudaMemcpyAsync(ctx->d_in64.p, c, sizeof(double) * n * R, cudaMemcpyHostToDevice, s));
  pack_rows_kernel<<<unsigned((n * R + 255) / 256), 256, 0, s>>>(ctx->d_in64.p, ctx->d_c64.p, n, R);
  FCG_CUDA(cudaGetLastError());
  FCG_CUDA(ctx->d_ojobs.alloc(size_t(n_jobs)));
  OpenParams p{};
  p.ot = ctx->d_oterms.p;
  p.items = ctx->d_oitems.p;
  p.prefix = ctx->d_oprefix.p;
  p.n_items = n_items;
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
  FCG_CUDA(cudaMemcpyAsync(O.h_cnt.p, ctx->d_counters.p, kCntBytes, cudaMemcpyDeviceToHost, s));
  FCG_CUDA(cudaStreamSynchronize(s));
  FCG_REQUIRE(cnt[10] == 0, FCG_ELIMIT, cnt[10] == 1 ? "bra sector product space exceeds 2^40"
                                                        : "bra tuples of one term exceed 2^31");
  const int64_t n_kept = int64_t(cnt[0]);
  const int64_t n_elem = int64_t(cnt[1]);
  const int64_t flops_ref = int64_t(cnt[9]), tdm_bytes = int64_t(cnt[14]);
  int launches = 8;  // (the scans of a large plan not counted)
  if (n_kept > 0) {
    // a warp's slice: the largest job tiles, up to kExpSlice; as many warps to a CTA as fit.
    // The register sums serve index lengths up to kExpMaxD (the second and third remaining
    // clusters of the longest term), the shared-memory sums anything longer.
    const int d_max = int(cnt[11]);
    const int slice = std::min(kExpSlice, std::max(16, int(d_max > kExpMaxD ? cnt[13] : cnt[12])));
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
    size_t keys_after = 0, vals_after = 0;
    for (int attempt = 0;; ++attempt) {
      // the table is empty up to clean_keys / clean_vals: every call empties the slots it used
      if (cap > ctx->d_hkeys.n) O.clean_keys = 0;
      if (cap * R > ctx->d_hvals.n) O.clean_vals = 0;
      FCG_CUDA(ctx->d_hkeys.alloc(cap));
      FCG_CUDA(ctx->d_hvals.alloc(cap * R));
      if (O.clean_keys < cap)
        FCG_CUDA(cudaMemsetAsync(ctx->d_hkeys.p + O.clean_keys, 0xFF, (cap - O.clean_keys) * sizeof(unsigned long long), s));
      if (O.clean_vals < cap * R)
        FCG_CUDA(cudaMemsetAsync(ctx->d_hvals.p + O.clean_vals, 0, (cap * R - O.clean_vals) * sizeof(double), s));
      const size_t clean_keys = std::max<size_t>(O.clean_keys, cap), clean_vals = std::max<size_t>(O.clean_vals, cap * R);
      O.clean_keys = O.clean_vals = 0;  // until this call's slots are emptied
      FCG_CUDA(cudaMemsetAsync(ctx->d_counters.p + 2, 0, 3 * sizeof(unsigned long long), s));
      FCG_CUDA(cudaEventRecord(ctx->ev2, s));
      kernel<<<unsigned(grid), threads, smem, s>>>(
          p, ctx->d_ojobs.p, n_kept, ctx->d_ow64.p, ctx->d_op64.p, ctx->d_ow32.p, ctx->d_op32.p, ctx->d_gmax.p,
          ExpandTable{ctx->d_hkeys.p, ctx->d_hvals.p, cap - 1, ctx->d_counters.p}, slice);
      FCG_CUDA(cudaGetLastError());
      FCG_CUDA(cudaEventRecord(ctx->ev3, s));
      FCG_CUDA(cudaMemcpyAsync(O.h_cnt.p, ctx->d_counters.p, kCntBytes, cudaMemcpyDeviceToHost, s));
      FCG_CUDA(cudaStreamSynchronize(s));
      launches += 2;
      if (cnt[2] == 0) {
        keys_after = clean_keys;
        vals_after = clean_vals;
        break;
      }
      FCG_REQUIRE(attempt < 3 && cap < (1ull << 31), FCG_ENOMEM, "open sigma hash table overflow");
      cap <<= 1;
    }
    FCG_CUDA(ctx->d_okeys.alloc(cap));
    FCG_CUDA(ctx->d_ovals.alloc(cap * R));
    compact_kernel<<<unsigned(cap / kCompactSlots), kCompactThreads, 0, s>>>(ctx->d_hkeys.p, ctx->d_hvals.p, R,
                                                                           ctx->d_okeys.p, ctx->d_ovals.p,
                                                                           ctx->d_counters.p);
    FCG_CUDA(cudaGetLastError());
    FCG_CUDA(cudaEventRecord(ctx->ev1, s));
    FCG_CUDA(cudaMemcpyAsync(O.h_cnt.p, ctx->d_counters.p, kCntBytes, cudaMemcpyDeviceToHost, s));
    FCG_CUDA(cudaStreamSynchronize(s));
    launches += 1;
    O.clean_keys = keys_after;
    O.clean_vals = vals_after;
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
  const int64_t* dims = reinterpret_cast<const int64_t*>(ctx->open_bra.data());
  const int16_t* bra_fock = reinterpret_cast<const int16_t*>(dims + ctx->open_sectors * N);
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < m; ++i) {
    const unsigned long long key = ctx->open_keys.p[i];
    const int64_t bs = int64_t(key >> kKeyIdxBits);
    int64_t idx = int64_t(key & ((1ull << kKeyIdxBits) - 1));
    std::memcpy(fock + i * 2 * N, bra_fock + bs * 2 * N, sizeof(int16_t) * 2 * N);
    for (int c = 0; c < N; ++c) {
      const int64_t d = dims[bs * N + c];
      cfg[i * N + c] = int16_t(idx % d);
      idx /= d;
    }
    for (int r = 0; r < R; ++r) coeff[i + m * r] = ctx->open_vals.p[size_t(i) * R + r];
  }
  return FCG_OK;
}

}  // extern "C"
