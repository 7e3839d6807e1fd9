// Persistent Lonestar-style graph traversals on the grid barrier: BFS (push
// worklist, pull, topology push; direction chosen per level by a fixed
// heuristic or by the learned policy), SSSP (near-far buckets with atomicMin)
// and pull PageRank (FP32 state, FP64 per-vertex accumulation, fixed
// iteration count).  One grid kernel per traversal, one grid barrier per level /
// bucket step / iteration; without a launch configuration of the caller's, thin
// BFS levels and thin graphs' SSSP rounds run on one cluster instead
// (bfs_cluster_kernel, sssp_cluster_kernel).
//
// Reference: the GGC "outlined iterate" kernels gg_main_pipe_1_gpu_gb of
// LONESTAR/apps/bfs/kernel_gsrb.cu:591-626 (BFS), apps/sssp/kernel_gsrb.cu:637-687
// (SSSP, DELTA default 10000, apps/sssp/support.cu:10), apps/pr/kernel_gsrb.cu:543-587
// (push-residual PR), all launched as one persistent kernel that hits
// kernelAtomicTreeBarrierUniqSRB once per level.  Level and distance
// conventions: source 0, unreachable INT_MAX, BFS level L for vertices first
// reached in round L (bfs/kernel_gsrb.cu:299-311, :473-479, :724).
#include "internal.h"
#include "graph_common.cuh"
#include "cluster_link.cuh"

#include <algorithm>
#include <string.h>
#include <utility>
#include <vector>

using namespace gsrbrt;
using namespace gsrbg;

namespace {

enum BfsDir : uint32_t { DIR_PUSH = 0, DIR_PULL = 1, DIR_TOPO = 2 };

struct BfsArgs {
  DevCSR g;
  uint32_t src;
  int32_t* level;
  uint32_t* q[2];
  uint32_t* hq[2];
  LevelCounters* cnt;  // [3]
  uint32_t* overflow;
  LevelTrace* trace;
  uint32_t trace_cap;
  const MLPWeights* mlp;
  int32_t mode;        // GSRB_BFS_* (include/gsrb.h)
  float alpha, beta;   // direction-optimizing thresholds (Beamer, Asanovic, Patterson, SC'12)
  uint32_t* out;       // [0] levels, [1] fallback level (0 = none), [2] policy decisions, [3] overflow
  unsigned long long* out_edges;
  uint32_t* solo;      // [0] last level, [1] nu, [2] prev_nf, [3] solo levels, [4..5] mu, [6..7] edges
  bool symmetric;      // rows are also in-edge lists: pull levels allowed
  bool lb;             // load-balanced expansion of large push levels (GSRB_BFS_FLAG_LB)
  uint32_t* lb_pre;    // [n] edge offset of each regular-queue entry
  uint32_t* lb_own;    // [m / kLbChunk + 2] entry owning each chunk's first edge
  uint32_t* lb_part;   // [kLbMaxCtas] per-CTA edge totals
  uint32_t* phase;     // [0] PHASE_*, [1] policy decisions, [2] fallback level so far
  bool staged;         // init kernel, then cluster and grid kernels in turn (a.phase says whose turn it is)
  bool stage;          // the launch has the CTAs' stages
};

// Whose turn it is in a traversal that alternates between one cluster (thin
// levels) and the whole grid (fat ones).
enum : uint32_t { PHASE_GRID = 1, PHASE_DONE = 2, PHASE_CLUSTER = 3 };

constexpr uint32_t kThinDegree = 8;           // graphs below this mean degree start and usually end on the cluster
constexpr uint32_t kClQueue = 4096;           // entries per CTA and parity
constexpr uint32_t kClMaxFrontier = 16384;    // larger levels go to the grid: past this 16 SMs' gathers
constexpr uint32_t kClMaxEdges = 65536;       // (one a cycle and SM) cost more than a grid level
constexpr uint32_t kClEnterFrontier = 3840;   // and come back below these (what one CTA's queue could hold,
constexpr unsigned long long kClEnterEdges = 16384;  // fat entries in pieces)
constexpr uint32_t kClPiece = 64;             // edges of a piece

// Single-CTA phase: when a push level's frontier fits one pass of one CTA
// (<= blockDim.x vertices and <= 4 blockDim.x out-edges) the heuristic and
// learned schedules hand the following levels to the team's first CTA, which
// runs them with __syncthreads and shared-memory queue counters while the
// other CTAs wait at one grid barrier; it hands back when the frontier grows
// past 2x the entry limits, after kSoloMaxLevels levels, or when the traversal
// ends.  Small-frontier levels of high-diameter graphs (meshes, road
// networks) then cost no grid barrier.
constexpr uint32_t kSoloMaxLevels = 16384;
// The policy's topology-push output must exceed this logit (probability 0.88).
constexpr float kTopoLogit = 2.f;

// The single-CTA phase, run by every thread of the team's first CTA from level
// L (whose frontier, nreg + nbig vertices of level L-1, is in the global
// queues; the caller has already done level L's accounting).  Leaves the
// frontier of the last level it ran in the global queues and counters, and
// that level, nu, mu, edges and prev_nf (accounting not yet applied for the
// last level's discoveries, as the level loop expects) in a.solo.
__device__ __noinline__ void bfs_solo(const BfsArgs& a, uint32_t L, uint32_t nreg, uint32_t nbig, uint32_t nu,
                                      unsigned long long mu, unsigned long long edges, uint32_t prev_nf) {
  __shared__ LevelCounters s_c;
  const DevCSR& g = a.g;
  const Team one{0u, 1u};
  uint32_t levels = 0;
  for (;;) {
    const uint2* qin = reinterpret_cast<const uint2*>(a.q[(L - 1) & 1]);
    const uint2* hin = reinterpret_cast<const uint2*>(a.hq[(L - 1) & 1]);
    uint2* qout = reinterpret_cast<uint2*>(a.q[L & 1]);
    uint2* hout = reinterpret_cast<uint2*>(a.hq[L & 1]);
    if (threadIdx.x == 0) {
      s_c.n_reg = 0;
      s_c.n_big = 0;
      s_c.m_next = 0;
    }
    __syncthreads();
    unsigned long long m_acc = 0;
    const int32_t Li = (int32_t)L;
    auto push_edge = [&](uint32_t, uint32_t j, bool active) {
      uint2 r = make_uint2(0u, 0u);
      bool disc = false;
      if (active) {
        const uint32_t v = __ldg(g.dst + j);
        if (__ldcg(a.level + v) == kInf) disc = atomicCAS(a.level + v, kInf, Li) == kInf;
        if (disc) r = make_uint2(__ldg(g.row + v), __ldg(g.row + v + 1));
      }
      const uint32_t d = r.y - r.x;
      warp_append(disc && d <= kBigDegree, r, qout, &s_c.n_reg, g.n, a.overflow);
      warp_append(disc && d > kBigDegree, r, hout, &s_c.n_big, g.n, a.overflow);
      m_acc += d;
    };
    expand_hub_ranges(one, hin, nbig, push_edge);
    const PushSink sink{qout, hout, &s_c.n_reg, &s_c.n_big, g.n, a.overflow, nullptr, nullptr, 0u};
    auto lanes = [&](uint32_t b, uint32_t mine, uint32_t kmax) {
      bfs_push_lanes(g, a.level, Li, b, mine, kmax, false, sink, m_acc);
    };
    expand_range_queue(one, qin, nreg, push_edge, lanes);
    const unsigned long long ws = warp_sum_u64(m_acc);
    if (lane_id() == 0 && ws) atomicAdd(&s_c.m_next, ws);
    __syncthreads();
    ++levels;
    const uint32_t nr = (uint32_t)s_c.n_reg, nb = (uint32_t)s_c.n_big;
    const uint32_t nf = nr + nb;
    const unsigned long long mf = s_c.m_next;
    const bool stop = nf == 0 || nf > 2u * blockDim.x || mf > 8ull * blockDim.x || levels >= kSoloMaxLevels;
    if (stop) {
      if (threadIdx.x == 0) {
        a.cnt[L % 3].n_reg = nr;
        a.cnt[L % 3].n_real = nr;
        a.cnt[L % 3].n_big = nb;
        a.cnt[L % 3].m_next = mf;
        a.cnt[(L + 1) % 3].n_reg = 0;
        a.cnt[(L + 1) % 3].n_real = 0;
        a.cnt[(L + 1) % 3].n_big = 0;
        a.cnt[(L + 1) % 3].m_next = 0;
        a.solo[0] = L;
        a.solo[1] = nu;
        a.solo[2] = prev_nf;
        a.solo[3] += levels;
        *reinterpret_cast<unsigned long long*>(a.solo + 4) = mu;
        *reinterpret_cast<unsigned long long*>(a.solo + 6) = edges;
      }
      return;  // the caller's grid barrier publishes all of it
    }
    // next level (the level loop's accounting, done here)
    ++L;
    nu -= nf;
    mu -= mf;
    edges += mf;
    if (threadIdx.x == 0 && L - 1 < a.trace_cap) {
      LevelTrace t;
      t.level = L;
      t.dir = 3u;  // single-CTA push
      t.nf = nf;
      t.nu = nu;
      t.mf = mf;
      t.mu = mu;
      t.t_ns = gsrb::ptx::globaltimer_ns();
      t.pred = __int_as_float(0x7fc00000);
      t.fallback = 0u;
      a.trace[L - 1] = t;
    }
    prev_nf = nf;
    nreg = nr;
    nbig = nb;
  }
}

// Block-wide exclusive prefix sum of x (blockDim.x a multiple of 32, <= 1024);
// *total receives the block's sum.  `s` holds 32 words of shared memory.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t x, uint32_t* s, uint32_t* total) {
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += y;
  }
  if (lane == 31) s[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint32_t v = lane < nw ? s[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= (uint32_t)o) v += y;
    }
    s[lane] = v;
  }
  __syncthreads();
  const uint32_t before = wid ? s[wid - 1] : 0u;
  *total = s[nw - 1];
  __syncthreads();
  return before + inc - x;
}

// Load-balanced expansion of a push level's regular queue (the reference's
// thread-block load balancer, apps/bfs/kernel_gsrb.cu:312-399, inspector
// :360-383, with its prefix sum and binary-search edge assignment): every warp
// gets the same number of edges whatever the degrees.
//   1. each CTA sums the degrees of its slice of the queue;      (team barrier)
//   2. each CTA offsets its slice by the totals of the CTAs before it, writes
//      every entry's first-edge offset (lb_pre) and, for every kLbChunk-edge
//      chunk that starts inside an entry's edges, the entry (lb_own);  (barrier)
//   3. warps take chunks grid-stride; a warp walks its chunk 32 edges at a
//      time with a window of 32 queue entries, each lane finding its edge's
//      entry by a binary search over the window's offsets in registers.
// Returns false if a team barrier failed.
template <int V, class F>
__device__ __forceinline__ bool bfs_lb_expand(gsrb::GridSync<V>& bar, const BfsArgs& a, const Team& team,
                                              const uint2* __restrict__ qin, uint32_t nq, F& push_edge) {
  uint32_t* s_scan = list_smem().scan;
  __shared__ uint32_t s_off, s_tot;
  const uint32_t G = team.ncta, c = team.cta;
  const uint32_t s0 = (uint32_t)((uint64_t)nq * c / G), s1 = (uint32_t)((uint64_t)nq * (c + 1) / G);
  // 1. slice totals
  uint32_t local = 0;
  for (uint32_t i = s0 + threadIdx.x; i < s1; i += blockDim.x) {
    const uint2 r = __ldcg(qin + i);
    local += r.y - r.x;
  }
  uint32_t tsum = 0;
  (void)block_exclusive_scan(local, s_scan, &tsum);
  if (threadIdx.x == 0) a.lb_part[c] = tsum;
  if (!bar.sync()) return false;
  // 2. offsets, owners of chunk starts
  uint32_t off = 0, tot = 0;
  for (uint32_t k = threadIdx.x; k < G; k += blockDim.x) {
    const uint32_t v = __ldcg(a.lb_part + k);
    tot += v;
    if (k < c) off += v;
  }
  uint32_t t1 = 0, t2 = 0;
  (void)block_exclusive_scan(off, s_scan, &t1);
  (void)block_exclusive_scan(tot, s_scan, &t2);
  if (threadIdx.x == 0) {
    s_off = t1;
    s_tot = t2;
  }
  __syncthreads();
  uint32_t carry = s_off;
  const uint32_t W = s_tot;
  for (uint32_t base = s0; base < s1; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    uint32_t d = 0;
    if (i < s1) {
      const uint2 r = __ldcg(qin + i);
      d = r.y - r.x;
    }
    uint32_t tile = 0;
    const uint32_t ex = block_exclusive_scan(d, s_scan, &tile);
    if (i < s1) {
      const uint32_t P = carry + ex;
      a.lb_pre[i] = P;
      for (uint32_t k = (P + kLbChunk - 1) / kLbChunk; k * kLbChunk < P + d; ++k) a.lb_own[k] = i;
    }
    carry += tile;
  }
  if (!bar.sync()) return false;
  // 3. edge-balanced walk
  const uint32_t lane = lane_id();
  const uint32_t nchunks = (W + kLbChunk - 1) / kLbChunk;
  for (uint32_t chunk = team.warp(); chunk < nchunks; chunk += team.nwarps()) {
    uint32_t o = __ldcg(a.lb_own + chunk);
    uint32_t t0 = chunk * kLbChunk;
    const uint32_t t_end = min(t0 + kLbChunk, W);
    for (;;) {
      const uint32_t wi = o + lane;
      uint32_t p = W, b = 0;
      if (wi < nq) {
        p = __ldcg(a.lb_pre + wi);
        b = __ldcg(&qin[wi].x);
      }
      const uint32_t p_next = o + 32 < nq ? __ldcg(a.lb_pre + o + 32) : W;
      const uint32_t t_lim = min(t_end, p_next);
      const uint32_t t = t0 + lane;
      // largest window slot j with p_j <= t (offsets are non-decreasing)
      uint32_t j = 0;
#pragma unroll
      for (uint32_t st = 16; st > 0; st >>= 1) {
        const uint32_t pc = __shfl_sync(0xffffffffu, p, j + st);
        if (pc <= t) j += st;
      }
      const uint32_t pj = __shfl_sync(0xffffffffu, p, j), bj = __shfl_sync(0xffffffffu, b, j);
      push_edge(0u, bj + (t - pj), t < t_lim);
      if (t0 + 32 <= t_lim) {
        o += __shfl_sync(0xffffffffu, j, 31);
        t0 += 32;
        if (t0 == t_end) break;
      } else if (t_lim == t_end) {
        break;
      } else {
        o += 32;  // the window's entries end before the chunk does
        t0 = t_lim;
      }
    }
  }
  return true;
}

// A push level's hub queue (2..kHubList ranges) expanded edge-balanced over the
// team: every CTA builds the ranges' edge prefix in shared memory (the same in
// every CTA, so no barrier is needed) and its threads take edges grid-stride.
__device__ __forceinline__ void bfs_push_hubs(const BfsArgs& a, const Team& team, const uint2* __restrict__ hin,
                                           uint32_t nbig, int32_t Li, const PushSink sink,
                                           unsigned long long& m_acc) {
  ListSmem& L_ = list_smem();
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nbig; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    uint32_t d = 0;
    if (i < nbig) {
      const uint2 r = __ldcg(hin + i);
      L_.b[i] = r.x;
      d = r.y - r.x;
    }
    uint32_t tile = 0;
    const uint32_t ex = block_exclusive_scan(d, L_.scan, &tile);
    if (i < nbig) L_.p[i] = carry + ex;
    carry += tile;
  }
  if (threadIdx.x == 0) L_.p[nbig] = carry;
  __syncthreads();
  bfs_push_list(a.g, a.level, Li, L_.p, L_.b, nbig, team.tid(), team.nthreads(), sink, m_acc);
  __syncthreads();
}

// The traversal body, relative to a team (the whole grid, or one instance's
// CTA range in a batch, synchronised by `bar`).  a_shared: the arguments in
// shared memory, for the single-CTA phase (a call that takes their address; of
// the kernel's parameters that is a local copy, whose reads miss L1 after every
// barrier, and the whole level loop would use it).
template <int V>
__device__ __forceinline__ void bfs_run(gsrb::GridSync<V>& bar, bool ok, const BfsArgs& a, const BfsArgs& a_shared,
                                        const Team team) {
  __shared__ uint32_t s_dir;
  __shared__ float s_pred;
  __shared__ MLPShared s_mlp;
  const DevCSR& g = a.g;
  const uint32_t tid = team.tid(), nthreads = team.nthreads();
  BfsStage* const stage = cta_stage<BfsStage>(a.stage);
  if (a.mode == GSRB_BFS_LEARNED) mlp_stage(a.mlp, &s_mlp);  // visible after the barrier below

  uint32_t nu, prev_nf = 1, L = 1, decisions = 0;
  uint32_t fb_level = 0;  // level at which the policy fell back (0 = never)
  unsigned long long mu, edges;
  if (a.staged) {
    // the state is where the init kernel or the cluster left it
    if (__ldcg(a.phase) != PHASE_GRID) return;
    __syncthreads();  // the staged policy weights
    L = __ldcg(a.solo + 0) + 1u;
    nu = __ldcg(a.solo + 1);
    prev_nf = __ldcg(a.solo + 2);
    mu = __ldcg(reinterpret_cast<const unsigned long long*>(a.solo + 4));
    edges = __ldcg(reinterpret_cast<const unsigned long long*>(a.solo + 6));
    decisions = __ldcg(a.phase + 1);
    fb_level = __ldcg(a.phase + 2);
  } else {
    // init (bfs_init, bfs/kernel_gsrb.cu:299-311) fused into the persistent kernel
    for (uint32_t v = tid; v < g.n; v += nthreads) a.level[v] = (v == a.src) ? 0 : kInf;
    const uint32_t dsrc = g.row[a.src + 1] - g.row[a.src];
    if (tid == 0) {
      const bool hub = dsrc > kBigDegree;
      reinterpret_cast<uint2*>(hub ? a.hq[0] : a.q[0])[0] = make_uint2(g.row[a.src], g.row[a.src + 1]);
      a.cnt[0].n_reg = a.cnt[0].n_real = hub ? 0 : 1;
      a.cnt[0].n_big = hub ? 1 : 0;
      a.cnt[0].m_next = dsrc;
      a.cnt[1].n_reg = a.cnt[1].n_real = a.cnt[1].n_big = a.cnt[1].m_next = 0;
      a.cnt[2].n_reg = a.cnt[2].n_real = a.cnt[2].n_big = a.cnt[2].m_next = 0;
    }
    ok = bar.sync() && ok;
    nu = g.n - 1;
    mu = (unsigned long long)g.m - dsrc;
    edges = dsrc;
  }
  uint32_t dir = DIR_PUSH;
  bool fallback = a.mode != GSRB_BFS_LEARNED || fb_level != 0;
  float pred = __int_as_float(0x7fc00000);
  const uint32_t L0 = L;
  bool to_cluster = false;
  uint32_t last_dir = DIR_PUSH, last_nf = 0;  // the policy's last decision and the frontier it saw
  unsigned long long last_mf = 0;
  for (; ok; ++L) {
    const LevelCounters cur = {__ldcg(&a.cnt[(L - 1) % 3].n_reg), __ldcg(&a.cnt[(L - 1) % 3].n_big),
                               __ldcg(&a.cnt[(L - 1) % 3].m_next), __ldcg(&a.cnt[(L - 1) % 3].n_real)};
    // nreg counts queue slots (the expansion's bound), n_real the entries
    const uint32_t nreg = (uint32_t)cur.n_reg, nbig = (uint32_t)cur.n_big;
    const uint32_t nf = (uint32_t)cur.n_real + nbig;
    if (nf == 0) break;
    const unsigned long long mf = cur.m_next;
    // ---- choose the level's direction (identical in every CTA)
    if (!fallback && L > 1 && pred == pred) {
      const float actual = log2f(1.f + (float)nf);
      if (fabsf(actual - pred) > 1.f) {  // missed by more than 2x
        fallback = true;
        fb_level = L;
      }
    }
    if (a.staged && L > L0 && nbig == 0 && nf <= kClEnterFrontier && mf <= kClEnterEdges) {
      // a thin frontier goes to the cluster (after at least one level here)
      if (tid == 0) {
        a.solo[0] = L - 1;
        a.solo[1] = nu;
        a.solo[2] = prev_nf;
        *reinterpret_cast<unsigned long long*>(a.solo + 4) = mu;
        *reinterpret_cast<unsigned long long*>(a.solo + 6) = edges;
        a.phase[0] = PHASE_CLUSTER;
        a.phase[1] = decisions;
        a.phase[2] = fb_level;
      }
      to_cluster = true;
      break;
    }
    if (L > 1) {
      nu -= nf;
      mu -= mf;
      edges += mf;
    }
    uint32_t nd = DIR_PUSH;
    if (a.mode == GSRB_BFS_PULL) {
      nd = L == 1 ? DIR_PUSH : DIR_PULL;
    } else if (a.mode == GSRB_BFS_TOPO) {
      nd = DIR_TOPO;
    } else if (a.mode == GSRB_BFS_HEURISTIC || (a.mode == GSRB_BFS_LEARNED && fallback)) {
      nd = dir;
      if (dir != DIR_PULL && (double)mf > (double)mu / a.alpha) nd = DIR_PULL;
      else if (dir == DIR_PULL && (double)nf < (double)g.n / a.beta) nd = DIR_PUSH;
    } else if (a.mode == GSRB_BFS_LEARNED) {
      // the network is evaluated again only when the frontier's size or edge
      // count has moved by more than 2x since its last decision (on meshes and
      // road networks that skips most levels); a reused decision carries no
      // prediction, so it cannot trigger the fallback
      const bool reuse = decisions > 0 && nf <= 2u * last_nf && 2u * nf >= last_nf && mf <= 2ull * last_mf &&
                         2ull * mf >= last_mf;
      if (reuse) {
        nd = last_dir;
        pred = __int_as_float(0x7fc00000);
      } else {
        if (threadIdx.x < 32) {
          float feat[kFeat], out[kOut];
          level_features(feat, g.n, g.m, L, nf, mf, nu, mu, prev_nf, dir);
          mlp_forward_smem(&s_mlp, feat, out);
          if (threadIdx.x == 0) {
            // the topology push scans all n vertices: taken only on a confident
            // output; the first level always pushes (its frontier is the source,
            // and the training labels hold no pull decision for it)
            s_dir = (out[0] > 0.f && L > 1) ? DIR_PULL : (out[1] > kTopoLogit ? DIR_TOPO : DIR_PUSH);
            s_pred = out[2];
          }
        }
        __syncthreads();
        nd = s_dir;
        pred = s_pred;
        last_dir = nd;
        last_nf = nf;
        last_mf = mf;
        ++decisions;
      }
    }
    // a pull level reads rows as in-edges: only on symmetric graphs
    if (nd == DIR_PULL && !a.symmetric) nd = DIR_PUSH;
    dir = nd;
    if (team.cta == 0 && threadIdx.x == 0) {
      // the counter set of level L + 1 was last read before barrier L - 1
      a.cnt[(L + 1) % 3].n_reg = 0;
      a.cnt[(L + 1) % 3].n_real = 0;
      a.cnt[(L + 1) % 3].n_big = 0;
      a.cnt[(L + 1) % 3].m_next = 0;
      if (L - 1 < a.trace_cap) {
        LevelTrace t;
        t.level = L;
        t.dir = dir;
        t.nf = nf;
        t.nu = nu;
        t.mf = mf;
        t.mu = mu;
        t.t_ns = gsrb::ptx::globaltimer_ns();
        t.pred = (a.mode == GSRB_BFS_LEARNED && !fallback) ? pred : __int_as_float(0x7fc00000);
        t.fallback = fallback ? 1u : 0u;
        a.trace[L - 1] = t;
      }
    }
    prev_nf = nf;

    if (!a.staged && team.ncta > 1 && dir == DIR_PUSH && nf <= blockDim.x && mf <= 4ull * blockDim.x &&
        (a.mode == GSRB_BFS_HEURISTIC || a.mode == GSRB_BFS_LEARNED)) {
      if (team.cta == 0) bfs_solo(a_shared, L, nreg, nbig, nu, mu, edges, prev_nf);
      ok = bar.sync();
      if (!ok) break;
      L = __ldcg(a.solo + 0);
      nu = __ldcg(a.solo + 1);
      prev_nf = __ldcg(a.solo + 2);
      mu = __ldcg(reinterpret_cast<const unsigned long long*>(a.solo + 4));
      edges = __ldcg(reinterpret_cast<const unsigned long long*>(a.solo + 6));
      dir = DIR_PUSH;
      pred = __int_as_float(0x7fc00000);  // no prediction for the level after the phase
      continue;
    }

    const uint2* qin = reinterpret_cast<const uint2*>(a.q[(L - 1) & 1]);
    const uint2* hin = reinterpret_cast<const uint2*>(a.hq[(L - 1) & 1]);
    uint2* qout = reinterpret_cast<uint2*>(a.q[L & 1]);
    uint2* hout = reinterpret_cast<uint2*>(a.hq[L & 1]);
    LevelCounters* c = &a.cnt[L % 3];
    unsigned long long m_acc = 0;
    const int32_t Li = (int32_t)L;
    // regular-queue slots reserved per warp in chunks of 64 (one counter atomic
    // per chunk) when the queue's 2n slots can hold every warp's holes
    WarpRes res{0ull, 0u, 63ull * team.nwarps() <= g.n ? 64u : 0u};
    // The CTA's stage takes the entries of levels in which a warp appends a few
    // times at most, where a reservation per warp would be an atomic each on one
    // line: pull levels, and the walk of a hub where the next level may pull (a
    // push level is slower on the packed queue: R-MAT-18's second 600 -> 718 us).
    const bool hub_stage = dir == DIR_PUSH && nbig == 1 && a.symmetric && a.mode != GSRB_BFS_PUSH;
    const bool staged = a.stage && mf >= kStageMinEdges &&
                        (dir == DIR_PULL ? g.n / (32u * kStageMaxAppends) <= team.nwarps()
                                         : hub_stage && mf / (32u * kStageMaxAppends) <= team.nwarps());
    uint32_t real_w = 0;  // regular entries this warp appended past the stage (warp-uniform)
    const PushSink sink{qout, hout, &c->n_reg, &c->n_big, g.n, a.overflow, &res, &real_w, 2u * g.n};

    auto append = [&](bool disc, uint2 r, bool may_stage) {
      const uint32_t d = r.y - r.x;
      const bool reg1[1] = {disc && d <= kBigDegree};
      if (may_stage && staged)
        real_w += stage_append<1>(reg1, &r, stage, qout, &c->n_reg, g.n, 2u * g.n, a.overflow, res, make_uint2(0u, 0u));
      else
        push_append_reg<1>(reg1, &r, sink);
      warp_append(disc && d > kBigDegree, r, hout, &c->n_big, g.n, a.overflow);
      m_acc += d;
    };
    auto claim = [&](uint32_t j, bool active, bool may_stage) {
      uint2 r = make_uint2(0u, 0u);
      bool disc = false;
      if (active) {
        const uint32_t v = __ldg(g.dst + j);
        if (__ldcg(a.level + v) == kInf) disc = atomicCAS(a.level + v, kInf, Li) == kInf;
        if (disc) r = make_uint2(__ldg(g.row + v), __ldg(g.row + v + 1));
      }
      append(disc, r, may_stage);
    };
    auto push_edge = [&](uint32_t, uint32_t j, bool active) { claim(j, active, false); };

    if (dir == DIR_PUSH) {
      if (nbig > 1 && nbig <= kHubList) {
        // hubs edge-balanced over the team: every CTA builds the same prefix
        bfs_push_hubs(a, team, hin, nbig, Li, sink, m_acc);
      } else {
        auto hub_edge = [&](uint32_t, uint32_t j, bool active) { claim(j, active, true); };
        expand_hub_ranges(team, hin, nbig, hub_edge);
      }
      if (a.lb && team.ncta > 1 && mf >= kLbMinEdges) {
        // uniform across the team: every CTA takes the two extra barriers
        if (!bfs_lb_expand(bar, a, team, qin, nreg, push_edge)) {
          ok = false;
          break;
        }
      } else {
        const bool precheck = nf > kPushPrecheckFrontier;
        auto lanes = [&](uint32_t b, uint32_t mine, uint32_t kmax) {
          bfs_push_lanes(g, a.level, Li, b, mine, kmax, precheck, sink, m_acc);
        };
        expand_range_queue(team, qin, nreg, push_edge, lanes);
      }
    } else if (dir == DIR_TOPO) {
      // topology-driven push: scan every vertex, expand those at level L - 1
      expand_hub_ranges(team, hin, nbig, push_edge);
      const uint32_t lane = lane_id();
      const uint32_t gw = tid >> 5, nw = nthreads >> 5;
      for (uint32_t base = gw * 32u; base < g.n; base += nw * 32u) {
        const uint32_t u = base + lane;
        uint32_t b = 0, e = 0;
        if (u < g.n && __ldcg(a.level + u) == Li - 1) {
          b = __ldg(g.row + u);
          e = __ldg(g.row + u + 1);
          if (e - b > kBigDegree) e = b;  // hubs were expanded above
        }
        const uint32_t deg = e - b;
        uint32_t coop = __ballot_sync(0xffffffffu, deg > kWarpDegree);
        while (coop) {
          const int s = __ffs(coop) - 1;
          coop &= coop - 1;
          const uint32_t bb = __shfl_sync(0xffffffffu, b, s), ee = __shfl_sync(0xffffffffu, e, s);
          for (uint32_t j0 = bb; j0 < ee; j0 += 32) push_edge(0, j0 + lane, j0 + lane < ee);
        }
        const uint32_t mine = deg <= kWarpDegree ? deg : 0u;
        const uint32_t kmax = warp_max_u32(mine);
        for (uint32_t k = 0; k < kmax; ++k) push_edge(u, b + k, k < mine);
      }
    } else {
      // pull: every unvisited vertex looks for a neighbour at level L - 1, four
      // edges per lane in flight; vertices of more than kWarpDegree edges look
      // at their first four (in R-MAT rows the hubs) before the warp walks the
      // rest together.  Levels are read through L1: a line cached before a
      // vertex got level L still says INF, and neither is L - 1 (what was
      // written before the level's barrier is not stale after it).
      const uint32_t lane = lane_id();
      const uint32_t gw = tid >> 5, nw = nthreads >> 5;
      for (uint32_t base = gw * 32u; base < g.n; base += nw * 32u) {
        const uint32_t v = base + lane;
        bool unv = false;
        uint32_t b = 0, e = 0;
        if (v < g.n && __ldcg(a.level + v) == kInf) {
          b = __ldg(g.row + v);
          e = __ldg(g.row + v + 1);
          unv = b < e;
        }
        const uint32_t deg = e - b;
        bool found = false;
        const uint32_t lim = deg <= kWarpDegree ? e : b + 4u;
        bool more = unv;
        for (uint32_t k = b; __any_sync(0xffffffffu, more); k += 4) {
          uint32_t u[4];
          int32_t l[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) u[r] = more && k + r < lim ? __ldg(g.dst + k + r) : kHole;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            l[r] = kInf;
            if (u[r] != kHole) l[r] = __ldca(a.level + u[r]);
          }
          const bool hit = l[0] == Li - 1 || l[1] == Li - 1 || l[2] == Li - 1 || l[3] == Li - 1;
          found = found || hit;
          more = more && !hit && k + 4 < lim;
        }
        uint32_t coop = __ballot_sync(0xffffffffu, unv && !found && deg > kWarpDegree);
        while (coop) {
          const int s = __ffs(coop) - 1;
          coop &= coop - 1;
          const uint32_t bb = __shfl_sync(0xffffffffu, b, s), ee = __shfl_sync(0xffffffffu, e, s);
          bool hit = false;
          for (uint32_t j0 = bb + 4; j0 < ee && !hit; j0 += 128) {
            uint32_t u[4];
            int32_t l[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const uint32_t j = j0 + 32u * r + lane;
              u[r] = j < ee ? __ldg(g.dst + j) : kHole;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              l[r] = kInf;
              if (u[r] != kHole) l[r] = __ldca(a.level + u[r]);
            }
            hit = __any_sync(0xffffffffu, l[0] == Li - 1 || l[1] == Li - 1 || l[2] == Li - 1 || l[3] == Li - 1);
          }
          if ((int)lane == s) found = hit;
        }
        if (found) gsrb::ptx::st_relaxed_gpu_s32(a.level + v, Li);
        // the new frontier's entries: the row range is known
        append(found, found ? make_uint2(b, e) : make_uint2(0u, 0u), true);
      }
    }
    // edge sums and entry counts of the new frontier; in a staged level one
    // update per CTA (one per warp made 4736 atomics on one line of the L2:
    // R-MAT-22's first level 27.7 -> 16.3 us)
    warp_res_close(qout, 2u * g.n, res, make_uint2(0u, 0u));
    const unsigned long long ws = warp_sum_u64(m_acc);
    if (lane_id() == 0 && ws) {
      if (staged) atomicAdd(&stage->msum, ws);
      else atomicAdd(&c->m_next, ws);
    }
    if (lane_id() == 0 && real_w) atomicAdd(&c->n_real, (unsigned long long)real_w);
    if (staged) stage_flush(*stage, qout, &c->n_reg, 2u * g.n, a.overflow, &c->n_real, &c->m_next);
    ok = bar.sync();
  }
  if (to_cluster) return;
  if (team.cta == 0 && threadIdx.x == 0) {
    if (a.staged) a.phase[0] = PHASE_DONE;
    a.out[0] = L - 1;  // levels with a non-empty frontier beyond the source
    a.out[2] = decisions;
    a.out[3] = ok ? 0u : 1u;
    *a.out_edges = edges;
  }
  // first level at which the policy fell back (0 = never), kept in a
  // register: scanning the trace for it here cost one thread a dependent load
  // per level (about 1 ms on a 4095-level mesh)
  if (team.cta == 0 && threadIdx.x == 0 && a.mode == GSRB_BFS_LEARNED) a.out[1] = fb_level;
}

// ---- thin levels on one cluster ---------------------------------------------
// A 2048^2 grid has 4073 levels of at most 2051 vertices: on the grid a level
// cost 11.4 us at 2 x 512 threads per SM, of which the barrier is two and the
// rest the chain of trips to L2.  Here a level is: entry (shared memory) ->
// destinations -> claims with the candidates' row ranges -> shared-memory
// append -> records exchanged, 2.1 us (about 4200 cycles).
static_assert(kClEnterFrontier + kClEnterEdges / kClPiece <= kClQueue, "entries and pieces fit one CTA's queue");
struct BfsClShared {
  uint2 q[2][kClQueue];  // edge ranges of the frontier's vertices, by parity of the level
  ClusterLink link;
  uint32_t n[2];      // entries asked for in the level being built, by parity
  uint32_t extra[2];  // entries that went to the global queues
  uint32_t empty[2];  // slots they left empty here
  uint32_t m[2];      // their out-edges
  uint32_t fat[2];    // bit 0: an entry of more than 4 edges, bit 1: of more than 8
};

// Bulk prefetches of an array into L2, 4 KiB each (whole 16-byte units inside it).
__device__ __forceinline__ void prefetch_l2(const void* array, uint64_t bytes, uint32_t tid, uint32_t nt) {
  const uint64_t a0 = (uint64_t)array, b = (a0 + 15) & ~15ull, e = (a0 + bytes) & ~15ull;
  for (uint64_t at = b + (uint64_t)tid * 4096; at < e; at += (uint64_t)nt * 4096) {
    const uint32_t len = (uint32_t)min((uint64_t)4096, e - at);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(len) : "memory");
  }
}

// Level, queue and counter set-up of a traversal that starts on the cluster
// or (hub sources) on the grid; the CSR of a thin graph is brought into L2, so
// that a level's misses do not wait for DRAM in turn (prefetch != 0).
__global__ void __launch_bounds__(512) bfs_init_kernel(BfsArgs a, uint32_t* flags, uint32_t prefetch) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const DevCSR& g = a.g;
  for (uint32_t v = tid; v < g.n; v += nt) a.level[v] = v == a.src ? 0 : kInf;
  if (tid == 0) {
    for (int k = 0; k < 32; ++k) flags[k] = 0;
    const uint32_t b = g.row[a.src], e = g.row[a.src + 1];
    const bool hub = e - b > kBigDegree;
    reinterpret_cast<uint2*>(hub ? a.hq[0] : a.q[0])[0] = make_uint2(b, e);
    for (int k = 0; k < 3; ++k) a.cnt[k].n_reg = a.cnt[k].n_real = a.cnt[k].n_big = a.cnt[k].m_next = 0;
    a.cnt[0].n_reg = a.cnt[0].n_real = hub ? 0 : 1;
    a.cnt[0].n_big = hub ? 1 : 0;
    a.cnt[0].m_next = e - b;
    a.solo[1] = g.n - 1;
    a.solo[2] = 1;
    *reinterpret_cast<unsigned long long*>(a.solo + 4) = (unsigned long long)g.m - (e - b);
    *reinterpret_cast<unsigned long long*>(a.solo + 6) = e - b;
    // (the policy decides a traversal's first level: that one runs on the grid)
    a.phase[0] = hub || a.mode == GSRB_BFS_LEARNED ? PHASE_GRID : PHASE_CLUSTER;
  }
  if (prefetch) {
    prefetch_l2(g.row, (uint64_t)(g.n + 1) * 4, tid, nt);
    prefetch_l2(g.dst, (uint64_t)g.m * 4, tid, nt);
  }
}

// K edges per lane (bit r of `act`: edge j[r]): destinations, claims
// (compare-and-swap INF -> L, with the row ranges of the candidates), append.
// Warp-synchronous.
template <int K>
__device__ __forceinline__ void bfs_cl_push(const BfsArgs& a, BfsClShared& s, uint32_t L, const uint32_t* j,
                                            uint32_t act) {
  const DevCSR& g = a.g;
  const uint32_t p = L & 1u;
  uint32_t v[K];
  int32_t old[K];
  uint2 rg[K];
#pragma unroll
  for (int r = 0; r < K; ++r) v[r] = ((act >> r) & 1u) ? __ldg(g.dst + j[r]) : 0u;
#pragma unroll
  for (int r = 0; r < K; ++r) {
    old[r] = 0;
    if ((act >> r) & 1u) old[r] = atomicCAS(a.level + v[r], kInf, (int32_t)L);
  }
#pragma unroll
  for (int r = 0; r < K; ++r) {
    rg[r] = make_uint2(0u, 0u);
    if ((act >> r) & 1u) rg[r] = make_uint2(__ldg(g.row + v[r]), __ldg(g.row + v[r] + 1));
  }
  uint32_t mask[K], tot = 0, m_acc = 0, dmax = 0;
#pragma unroll
  for (int r = 0; r < K; ++r) {
    const bool disc = ((act >> r) & 1u) && old[r] == kInf;
    if (!disc) rg[r] = make_uint2(0u, 0u);
    const uint32_t d = rg[r].y - rg[r].x;
    // the first edges are on their way to the SM while the level ends
    if (d) asm volatile("prefetch.global.L1 [%0];" ::"l"(g.dst + rg[r].x));
    dmax = max(dmax, d);
    m_acc += d;
    mask[r] = __ballot_sync(0xffffffffu, disc);
    tot += __popc(mask[r]);
  }
  if (!tot) return;
  const uint32_t lane = lane_id();
  uint32_t pos = 0;
  if (lane == 0) pos = atomicAdd(&s.n[p], tot);
  m_acc = __reduce_add_sync(0xffffffffu, m_acc);
  const bool fat = __any_sync(0xffffffffu, dmax > 4u);
  if (lane == 0) atomicAdd(&s.m[p], m_acc);
  pos = __shfl_sync(0xffffffffu, pos, 0);
  bool hub = false;
  if (fat) {
    hub = __any_sync(0xffffffffu, dmax > kBigDegree);
    const bool fat8 = __any_sync(0xffffffffu, dmax > 8u);
    if (lane == 0) atomicOr(&s.fat[p], fat8 ? 3u : 1u);
  }
  const uint32_t lt = lanemask_lt();
  if (pos + tot <= kClQueue && !hub) {
#pragma unroll
    for (int r = 0; r < K; ++r) {
      if ((mask[r] >> lane) & 1u) s.q[p][pos + __popc(mask[r] & lt)] = rg[r];
      pos += __popc(mask[r]);
    }
    return;
  }
  // no room left, or a hub: these go to the global queues and the level that
  // follows to the grid.  The slots reserved above stay empty ranges.
  const uint32_t left = pos < kClQueue ? min(tot, kClQueue - pos) : 0u;
  for (uint32_t k = lane; k < left; k += 32) s.q[p][pos + k] = make_uint2(0u, 0u);
  LevelCounters* c = &a.cnt[L % 3];
#pragma unroll
  for (int r = 0; r < K; ++r) {
    const bool disc = (mask[r] >> lane) & 1u, big = rg[r].y - rg[r].x > kBigDegree;
    warp_append(disc && !big, rg[r], reinterpret_cast<uint2*>(a.q[p]), &c->n_reg, 2u * a.g.n, a.overflow);
    warp_append(disc && big, rg[r], reinterpret_cast<uint2*>(a.hq[p]), &c->n_big, a.g.n, a.overflow);
  }
  if (lane == 0) {
    atomicAdd(&s.extra[p], tot);
    atomicAdd(&s.empty[p], left);
  }
}

// A level over the CTA's own entries, all of at most 1 << SH edges: K edges per
// lane, (1 << SH) / K lanes per entry.  A level is a chain of dependent
// instructions as much as of trips to L2, so one edge per lane (fewer
// instructions per warp on more warps) wins while one pass takes them all, then
// two per lane over two passes of one (2048^2 grid 9.6 -> 8.7 ms; four measured
// the same as two).
template <int SH, int K>
__device__ __forceinline__ void bfs_cl_thin(const BfsArgs& a, BfsClShared& s, uint32_t L, uint32_t own) {
  constexpr int kSh = SH - (K - 1);  // log2 of the lanes per entry
  const uint32_t p = (L - 1) & 1u;
  for (uint32_t i = threadIdx.x; ((i - lane_id()) >> kSh) < own; i += blockDim.x) {
    uint2 r = make_uint2(0u, 0u);
    if ((i >> kSh) < own) r = s.q[p][i >> kSh];
    uint32_t j[K], act = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      j[k] = r.x + (i & ((1u << kSh) - 1u)) * K + k;
      if (j[k] < r.y) act |= 1u << k;
    }
    bfs_cl_push<K>(a, s, L, j, act);
  }
}

__global__ void __launch_bounds__(kClThreads, 1) bfs_cluster_kernel(BfsArgs a, unsigned long long timeout_ns) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  BfsClShared& s = *reinterpret_cast<BfsClShared*>(cl_smem);
  if (__ldcg(a.phase) != PHASE_CLUSTER) return;  // the same in every CTA
  const uint32_t rank = gsrb::ptx::cluster_ctarank(), ncta = gsrb::ptx::cluster_nctarank();
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t L = __ldcg(a.solo + 0) + 1u, nu = __ldcg(a.solo + 1), prev_nf = __ldcg(a.solo + 2);
  unsigned long long mu = __ldcg(reinterpret_cast<const unsigned long long*>(a.solo + 4));
  unsigned long long edges = __ldcg(reinterpret_cast<const unsigned long long*>(a.solo + 6));
  uint32_t nf = (uint32_t)__ldcg(&a.cnt[(L - 1) % 3].n_real);
  unsigned long long mf = __ldcg(&a.cnt[(L - 1) % 3].m_next);
  const uint32_t slots = (uint32_t)__ldcg(&a.cnt[(L - 1) % 3].n_reg);
  if (threadIdx.x == 0) {
    link_init(s.link, ncta);
    s.n[0] = s.n[1] = s.extra[0] = s.extra[1] = s.empty[0] = s.empty[1] = s.m[0] = s.m[1] = 0;
    s.fat[0] = s.fat[1] = 3u;  // of the entries read below nothing is known
  }
  gsrb::ptx::cluster_sync();  // also: every CTA has read the counters
  if (rank == 0 && threadIdx.x < 3)
    a.cnt[threadIdx.x].n_reg = a.cnt[threadIdx.x].n_real = a.cnt[threadIdx.x].n_big = a.cnt[threadIdx.x].m_next = 0;
  // this CTA's part of the frontier (holes and isolated vertices dropped; at
  // most kClEnterFrontier entries in all)
  uint32_t p = (L - 1) & 1u;
  {
    const uint2* qg = reinterpret_cast<const uint2*>(a.q[p]);
    const uint32_t s0 = (uint32_t)((uint64_t)slots * rank / ncta), s1 = (uint32_t)((uint64_t)slots * (rank + 1) / ncta);
    for (uint32_t i = s0 + threadIdx.x; i < s1; i += blockDim.x) {
      // fat entries in pieces (a source of 3644 edges on one warp took 86 us)
      const uint2 r = __ldcg(qg + i);
      const uint32_t pieces = (r.y - r.x + kClPiece - 1) / kClPiece;
      uint32_t at = pieces ? atomicAdd(&s.n[p], pieces) : 0u;
      for (uint32_t b = r.x; b < r.y; b += kClPiece) s.q[p][at++] = make_uint2(b, min(b + kClPiece, r.y));
    }
  }
  uint32_t phases = 0, fl = 0, own;
  bool ok, first = true, agreed = false;
  // the last warp of CTA 0 (idle in thin levels) keeps the traversal's account
  const bool books = rank == 0 && wid == nw - 1;
  if (threadIdx.x == 0) link_expect(s.link, p, ncta);
  __syncthreads();
  if (wid == 0) link_publish(s.link, p, make_uint4(s.n[p], 0u, 0u, 0u), rank, ncta);
  for (;;) {
    // the frontier of level L - 1 is in q[p], its records in tab[p]
    ok = link_wait(s.link, p, phases, timeout_ns);
    const LinkSum t = link_sum<false>(s.link, p, rank, ncta);
    own = t.own;
    if (!first) {
      nf = t.x + t.y;
      mf = t.z;
      fl = t.w ? 1u : 0u;
    }
    if (!ok || nf == 0 || fl || nf > kClMaxFrontier || (uint32_t)mf > kClMaxEdges) break;
    first = false;
    const uint32_t o = L & 1u;  // the level being built
    const uint32_t fat = s.fat[p];  // (cleared for level L + 1 in level L's tail)
    if (threadIdx.x == 0) {
      // published; next used in level L + 1, after this level's barrier
      s.n[p] = s.extra[p] = s.empty[p] = s.m[p] = 0;
      link_expect(s.link, o, ncta);
    }
    if (books) {
      if (L > 1) {
        nu -= nf;
        mu -= mf;
        edges += mf;
      }
      prev_nf = nf;
      if (lane == 0 && L - 1 < a.trace_cap) {
        LevelTrace r;
        r.level = L;
        r.dir = 3u;  // push outside the grid's level loop
        r.nf = nf;
        r.nu = nu;
        r.mf = mf;
        r.mu = mu;
        r.t_ns = gsrb::ptx::globaltimer_ns();
        r.pred = __int_as_float(0x7fc00000);
        r.fallback = 0u;
        a.trace[L - 1] = r;
      }
    }
    auto step = [&](const uint32_t* j, const uint32_t*, uint32_t act) { bfs_cl_push<4>(a, s, L, j, act); };
    const bool uneven = link_uneven(t);
    if (uneven) ok = link_meet(s.link, phases, ncta, timeout_ns);
    if (!ok) {
      // gave up: on to the end of the step
    } else if (uneven) {
      // redistribute: an equal slice of all entries, read from their CTAs
      const uint32_t i0 = (uint32_t)((uint64_t)t.x * rank / ncta), i1 = (uint32_t)((uint64_t)t.x * (rank + 1) / ncta);
      const uint32_t gsz = cl_group(i1 - i0);
      for (uint32_t base = i0 + wid * gsz; base < i1; base += nw * gsz) {
        const bool in = lane < gsz && base + lane < i1;
        const uint32_t at = link_locate(s.link, p, ncta, in ? base + lane : 0u);
        uint2 r = make_uint2(0u, 0u);
        if (in)
          r = ld_cluster_v2(gsrb::ptx::mapa_shared(gsrb::ptx::smem_u32(&s.q[p][at & 0xffffu]), at >> 16));
        walk_group(r.x, r.y - r.x, step);
      }
    } else if (fat == 0u) {
      if (own <= kClThreads / 4) bfs_cl_thin<2, 1>(a, s, L, own);
      else bfs_cl_thin<2, 2>(a, s, L, own);
    } else if (fat == 1u) {
      bfs_cl_thin<3, 2>(a, s, L, own);
    } else {
      const uint32_t gsz = cl_group(own);
      for (uint32_t base = wid * gsz; base < own; base += nw * gsz) {
        uint2 r = make_uint2(0u, 0u);
        if (lane < gsz && base + lane < own) r = s.q[p][base + lane];
        walk_group(r.x, r.y - r.x, step);
      }
    }
    agreed = true;
    if (!(ok = link_agree(ok))) break;
    agreed = false;
    if (wid == 0) {
      // slots (past the queue's end the entries went to the global queue), the
      // entries beyond them (less the empty slots), edges, any in the global queue
      if (lane == 0) s.fat[p] = 0;  // every thread has read it; next set in level L + 1
      const uint32_t k = min(s.n[o], kClQueue);
      link_publish(s.link, o, make_uint4(k, s.extra[o] - s.empty[o], s.m[o], s.extra[o]), rank, ncta);
    }
    p = o;
    ++L;
  }
  if (!agreed) ok = link_agree(ok);
  if (!ok && threadIdx.x == 0) atomicExch(a.overflow + 1, 1u);
  if (nf == 0 || !ok) {
    if (books && lane == 0) {
      a.out[0] = L - 1;
      a.out[1] = __ldcg(a.phase + 2);
      a.out[2] = __ldcg(a.phase + 1);
      a.out[3] = ok ? 0u : 1u;
      *a.out_edges = edges;
      a.phase[0] = PHASE_DONE;
    }
  } else {
    // hand the frontier of level L - 1 to the grid
    LevelCounters* c = &a.cnt[(L - 1) % 3];
    __shared__ unsigned long long s_base;
    if (threadIdx.x == 0) s_base = atomicAdd(&c->n_reg, (unsigned long long)own);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < own; i += blockDim.x) {
      const unsigned long long at = s_base + i;
      if (at < 2ull * a.g.n) reinterpret_cast<uint2*>(a.q[p])[at] = s.q[p][i];
      else atomicExch(a.overflow, 1u);
    }
    if (books && lane == 0) {
      c->n_real = nf - (uint32_t)__ldcg(&c->n_big);
      c->m_next = mf;
      a.solo[0] = L - 1;
      a.solo[1] = nu;
      a.solo[2] = prev_nf;
      *reinterpret_cast<unsigned long long*>(a.solo + 4) = mu;
      *reinterpret_cast<unsigned long long*>(a.solo + 6) = edges;
      a.phase[0] = PHASE_GRID;
    }
  }
  gsrb::ptx::cluster_sync();  // no CTA leaves while a record to it may be in flight
}

constexpr int kGraphMaxThreads = 1024;

template <int V>
__global__ void __launch_bounds__(kGraphMaxThreads)
bfs_kernel(const __grid_constant__ gsrb::GridBarrier gb, const __grid_constant__ BfsArgs a) {
  __shared__ gsrb::BarrierShared bsh;
  __shared__ BfsArgs s_args;
  if (threadIdx.x == 0) s_args = a;  // read after the first level's barrier
  gsrb::GridSync<V> bar;
  const bool ok = bar.init(gb, &bsh);
  bfs_run<V>(bar, ok, a, s_args, Team{blockIdx.x, gridDim.x});
  bar.finish();
}

// ------------------------------------------------------------------- SSSP ---
struct SsspArgs {
  DevCSR g;
  uint32_t src;
  int32_t* dist;
  uint32_t* q[2];
  uint32_t* hq[2];
  uint32_t* far[2];
  uint32_t* mark;       // near-queue stamps
  uint32_t* fmark;      // far-pile stamps
  LevelCounters* cnt;   // [3] near counters
  unsigned long long* fcnt;  // [2] far counters
  uint32_t* overflow;
  LevelTrace* trace;
  uint32_t trace_cap;
  int32_t delta;
  uint32_t* out;        // [0] relax rounds, [1] buckets, [3] failure
  unsigned long long* out_edges;
  uint32_t* phase;      // [0] PHASE_*
  uint32_t* state;      // where the cluster left off: [0] rounds, [1] buckets, [2..3] near threshold
  bool staged;          // init and cluster kernels before the grid kernel (a.phase says whether it has work)
  bool stage;           // the launch has the CTAs' stages
};

// Vertices of more edges than this go to the near hub queue and are relaxed
// edge-balanced over the whole team, kHubList at a time (with 4096 and a list
// per CTA above 256, R-MAT-17's second round waited for the CTAs whose share of
// the frontier held the most edges: 93 -> 66 us).
constexpr uint32_t kSsspBig = 256;
constexpr uint32_t kSsspStep = 2;         // the grid's first step after the cluster (queue parity, counter set, stamp)
constexpr uint32_t kProbeMeanDegree = 8;  // graphs of this mean degree probe before claiming in every round
// Larger rounds probe on other graphs too: what they relax may be one vertex's
// in-edges, whose claims take turns (a round of 14,500 vertices with a common
// neighbour 14.0 us for 6.6; at 4096, which rounds of a 2048^2 grid reach, that
// grid takes 41.3 ms for 40.0).
constexpr uint32_t kRelaxPrecheckFrontier = 8192;

// Where an SSSP relax step puts the vertices whose distance it lowered.
struct RelaxSink {
  uint32_t* qout;               // near queue of the next round
  uint32_t* hout;               // near hub queue
  unsigned long long* n_reg;
  unsigned long long* n_big;
  uint32_t* fout;               // far pile
  unsigned long long* fc;
  uint32_t stamp;               // near-queue stamp of this round
  uint32_t fgen;                // far-pile generation
  int32_t T;                    // near threshold (at most kInf, which no queued distance reaches)
  IdStage* stage;               // the CTA's near-queue entries (null: none)
  WarpRes* res;                 // the warp's near-queue reservation (past the stage)
  uint32_t near_cap;            // near-queue capacity in slots (holes included)
  bool precheck;                // read a distance before claiming it (large rounds)
};

// A path length at kInf or beyond is no path: the sum saturates there.
__device__ __forceinline__ int32_t add_sat(int32_t a, int32_t b) {
  int32_t r;
  asm("add.sat.s32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// Relax four edges per lane at once: edge r of the lane is j[r] (where bit r of
// `act` is set), leaving a vertex at distance du[r].  Every dependent step is
// issued for all four before the next (destinations and weights, distance
// probes, the atomicMin claims, the stamps), and the warp reserves queue space
// once per step.  The row range of a destination (its degree, for the queue
// it enters) is loaded alongside its stamp exchange; in small rounds
// (!s.precheck) the distance probe is skipped -- the atomicMin itself tells
// whether the edge improves -- and the row range goes out with the claim.
// The same claims land either way, so distances are the same.
// Warp-synchronous.
__device__ __forceinline__ void sssp_relax4e(const SsspArgs& a, const int32_t* du, const uint32_t* j, uint32_t act,
                                             const RelaxSink& s, uint32_t& my_edges) {
  const DevCSR& g = a.g;
  uint32_t v[4];
  int32_t nd[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const bool on = (act >> r) & 1u;
    v[r] = on ? __ldg(g.dst + j[r]) : 0u;
    nd[r] = on ? add_sat(du[r], __ldg(g.w + j[r])) : kInf;
  }
  my_edges += __popc(act);
  // (Results of loads and atomics are only looked at in a loop of their own:
  // a comparison inside the branch that issues an atomic would make the warp
  // wait for each of the four in turn.)
  bool imp[4];
  uint32_t rb[4], re[4];
  int32_t old[4];
  if (s.precheck) {
    int32_t cur[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      cur[r] = kInf;
      if (nd[r] < kInf) cur[r] = __ldcg(a.dist + v[r]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) imp[r] = nd[r] < cur[r];
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r) imp[r] = nd[r] < kInf;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    old[r] = 0;
    if (imp[r]) old[r] = atomicMin(a.dist + v[r], nd[r]);
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    rb[r] = re[r] = 0;
    if (imp[r] && nd[r] < s.T) {
      rb[r] = __ldg(g.row + v[r]);
      re[r] = __ldg(g.row + v[r] + 1);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) imp[r] = imp[r] && nd[r] < old[r];
  uint32_t st[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const bool near = nd[r] < s.T;
    st[r] = 0;
    if (imp[r]) st[r] = atomicExch((near ? a.mark : a.fmark) + v[r], near ? s.stamp : s.fgen);
  }
  bool to_near[4], to_far[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    to_near[r] = imp[r] && nd[r] < s.T && st[r] != s.stamp;
    to_far[r] = imp[r] && nd[r] >= s.T && st[r] != s.fgen;
  }
  uint32_t d[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) d[r] = to_near[r] ? re[r] - rb[r] : 0u;
  bool reg[4], big[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    reg[r] = to_near[r] && d[r] <= kSsspBig;
    big[r] = to_near[r] && d[r] > kSsspBig;
  }
  stage_append<4>(reg, v, s.stage, s.qout, s.n_reg, g.n, s.near_cap, a.overflow, *s.res, kHole);
  warp_append_k<4>(big, v, s.hout, s.n_big, g.n, a.overflow);
  warp_append_k<4>(to_far, v, s.fout, s.fc, g.n, a.overflow);
}

// A list of vertices relaxed edge-balanced: their edge counts' prefix p[0..cnt]
// (p[cnt] = total), first edges b[] and distances d[] in shared memory.  Thread
// x of nthr takes edges (x & ~31) + lane + k * nthr, four per step, each
// finding its vertex by binary search over p.  Warp-synchronous loops.
__device__ __forceinline__ void sssp_relax_list(const SsspArgs& a, const uint32_t* p, const uint32_t* b,
                                                const int32_t* d, uint32_t cnt, uint32_t x, uint32_t nthr,
                                                const RelaxSink& s, uint32_t& my_edges) {
  const uint32_t total = p[cnt];
  for (uint32_t t0 = (x & ~31u) + lane_id(); t0 - lane_id() < total; t0 += 4u * nthr) {
    int32_t du[4];
    uint32_t j[4];
    uint32_t act = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t t = t0 + (uint32_t)r * nthr;
      du[r] = 0;
      j[r] = 0;
      if (t < total) {
        const uint32_t o = list_owner(p, cnt, t);
        j[r] = b[o] + (t - p[o]);
        du[r] = d[o];
        act |= 1u << r;
      }
    }
    sssp_relax4e(a, du, j, act, s, my_edges);
  }
}

template <int V>
__device__ __forceinline__ void sssp_run(gsrb::GridSync<V>& bar, bool ok, const SsspArgs& a, const Team team) {
  const DevCSR& g = a.g;
  const uint32_t tid = team.tid(), nthreads = team.nthreads();
  IdStage* const stage = cta_stage<IdStage>(a.stage);
  uint32_t step = 1;       // index of the near counter set in use (rotating by 3)
  uint32_t rounds = 0, buckets = 1;
  // near threshold: vertices with dist < T are relaxed in the current bucket
  long long T = a.delta;
  if (a.staged) {
    if (__ldcg(a.phase) != PHASE_GRID) return;
    __syncthreads();  // the stage is empty
    step = kSsspStep;
    rounds = __ldcg(a.state + 0);
    buckets = __ldcg(a.state + 1);
    T = __ldcg(reinterpret_cast<const long long*>(a.state + 2));
  } else {
    for (uint32_t v = tid; v < g.n; v += nthreads) {
      a.dist[v] = (v == a.src) ? 0 : kInf;
      a.mark[v] = 0;
      a.fmark[v] = 0;
    }
    const uint32_t dsrc = g.row[a.src + 1] - g.row[a.src];
    if (tid == 0) {
      const bool hub = dsrc > kSsspBig;
      if (hub) a.hq[0][0] = a.src;
      else a.q[0][0] = a.src;
      for (int k = 0; k < 3; ++k) a.cnt[k].n_reg = a.cnt[k].n_big = a.cnt[k].m_next = 0;
      a.cnt[0].n_reg = hub ? 0 : 1;
      a.cnt[0].n_big = hub ? 1 : 0;
      a.fcnt[0] = a.fcnt[1] = 0;
    }
    ok = bar.sync() && ok;
  }

  // graphs with fat rows probe a distance before every claim: most edges of a
  // round improve nothing, and their hubs' atomics serialise on one address
  // (R-MAT-17, a round of 15,640 vertices and 2.8 M edges)
  const bool probe = g.m / kProbeMeanDegree >= g.n;
  uint32_t fpar = 0;       // far pile parity
  uint32_t fgen = 1;       // generation of the current far pile (fmark stamps: a vertex enters a pile once)
  unsigned long long relaxed_edges = 0;
  while (ok) {
    const LevelCounters cur = {__ldcg(&a.cnt[(step - 1) % 3].n_reg), __ldcg(&a.cnt[(step - 1) % 3].n_big), 0, 0};
    const uint32_t nreg = (uint32_t)cur.n_reg, nbig = (uint32_t)cur.n_big;
    const uint32_t nf = nreg + nbig;
    if (team.cta == 0 && threadIdx.x == 0) {
      a.cnt[(step + 1) % 3].n_reg = 0;
      a.cnt[(step + 1) % 3].n_big = 0;
      a.cnt[(step + 1) % 3].m_next = 0;
    }
    if (nf == 0) {
      // ---- near bucket empty: advance the threshold and refill from the far pile
      const uint32_t nfar = (uint32_t)__ldcg(&a.fcnt[fpar]);
      if (nfar == 0) break;
      T += a.delta;
      ++buckets;
      const uint32_t* fin = a.far[fpar];
      uint32_t* fout = a.far[fpar ^ 1];
      unsigned long long* fc_out = &a.fcnt[fpar ^ 1];
      uint32_t* qout = a.q[step & 1];
      uint32_t* hout = a.hq[step & 1];
      LevelCounters* c = &a.cnt[step % 3];
      const uint32_t stamp = step;
      const uint32_t next_gen = fgen + 1;
      if (team.cta == 0 && threadIdx.x == 0) *fc_out = 0;  // last read before the previous barrier
      // fc_out must be zero before anyone appends: appends happen below, after
      // this CTA's store, so publish it through the barrier first
      ok = bar.sync();
      if (!ok) break;
      const uint32_t lane = lane_id();
      const uint32_t gw = tid >> 5, nw = nthreads >> 5;
      for (uint32_t base = gw * 32u; base < nfar; base += nw * 32u) {
        const uint32_t i = base + lane;
        uint32_t v = 0;
        bool near = false, keep = false;
        if (i < nfar) {
          v = __ldcg(fin + i);
          const int32_t dv = __ldcg(a.dist + v);
          if ((long long)dv < T) near = atomicExch(a.mark + v, stamp) != stamp;
          else keep = atomicExch(a.fmark + v, next_gen) != next_gen;
        }
        uint32_t d = 0;
        if (near) d = __ldg(g.row + v + 1) - __ldg(g.row + v);
        warp_append(near && d <= kSsspBig, v, qout, &c->n_reg, g.n, a.overflow);
        warp_append(near && d > kSsspBig, v, hout, &c->n_big, g.n, a.overflow);
        warp_append(keep, v, fout, fc_out, g.n, a.overflow);
      }
      fpar ^= 1;
      fgen = next_gen;
      ++step;
      ok = bar.sync();
      continue;
    }
    // ---- relax the near frontier
    ++rounds;
    if (team.cta == 0 && threadIdx.x == 0 && rounds - 1 < a.trace_cap) {
      LevelTrace t;
      t.level = rounds;
      t.dir = 0;
      t.nf = nf;
      t.nu = buckets;
      t.mf = 0;
      t.mu = (unsigned long long)T;
      t.t_ns = gsrb::ptx::globaltimer_ns();
      t.pred = __int_as_float(0x7fc00000);
      t.fallback = 0;
      a.trace[rounds - 1] = t;
    }
    const uint32_t* qin = a.q[(step - 1) & 1];
    const uint32_t* hin = a.hq[(step - 1) & 1];
    uint32_t* qout = a.q[step & 1];
    uint32_t* hout = a.hq[step & 1];
    LevelCounters* c = &a.cnt[step % 3];
    uint32_t* fout = a.far[fpar];
    unsigned long long* fc = &a.fcnt[fpar];
    const uint32_t stamp = step + 1;  // stamps of vertices queued for the next round
    uint32_t my_edges = 0;
    // near-queue reservations in chunks of 64 slots when the queue (2n slots)
    // can hold the holes of every warp
    WarpRes res{0ull, 0u, 63ull * team.nwarps() <= g.n ? 64u : 0u};
    const RelaxSink sink{qout, hout, &c->n_reg, &c->n_big, fout, fc, stamp, fgen, (int32_t)min(T, (long long)kInf), stage, &res, 2u * g.n,
                         probe || nf > kRelaxPrecheckFrontier};
    // vertex lists relaxed edge-balanced: edge prefix, first edge, distance
    ListSmem& L_ = list_smem();
    uint32_t* s_lp = L_.p;
    uint32_t* s_lb = L_.b;
    int32_t* s_ld = L_.d;
    uint32_t* s_scan = L_.scan;
    // builds the list's arrays from vertex ids (CTA-wide)
    auto build_list = [&](auto id_of, uint32_t cnt) {
      uint32_t carry = 0;
      for (uint32_t base = 0; base < cnt; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        uint32_t d = 0;
        if (i < cnt) {
          const uint32_t u = id_of(i);
          const uint32_t b = __ldg(g.row + u);
          d = __ldg(g.row + u + 1) - b;
          s_lb[i] = b;
          s_ld[i] = __ldcg(a.dist + u);
        }
        uint32_t tile = 0;
        const uint32_t ex = block_exclusive_scan(d, s_scan, &tile);
        if (i < cnt) s_lp[i] = carry + ex;
        carry += tile;
      }
      if (threadIdx.x == 0) s_lp[cnt] = carry;
      __syncthreads();
    };
    for (uint32_t h0 = 0; h0 < nbig; h0 += kHubList) {
      // big vertices, kHubList at a time: every CTA builds the same list; the
      // team's threads share its edges
      const uint32_t cnt = min(nbig - h0, kHubList);
      build_list([&](uint32_t i) { return __ldcg(hin + h0 + i); }, cnt);
      sssp_relax_list(a, s_lp, s_lb, s_ld, cnt, team.tid(), team.nthreads(), sink, my_edges);
      __syncthreads();
    }
    {
      // regular queue, edge-balanced over each warp's group, four edges per
      // lane in flight
      const uint32_t lane = lane_id();
      const uint32_t nwarps = team.nwarps(), gsz = group_size_of(nreg, nwarps);
      for (uint32_t base = spread_warp(team) * gsz; base < nreg; base += nwarps * gsz) {
        const uint32_t i = base + lane;
        uint32_t u = 0, b = 0, e = 0;
        int32_t du0 = 0;
        if (lane < gsz && i < nreg) {
          u = __ldcg(qin + i);
          if (u != kHole) {
            // the distance is read alongside the row range (one round trip):
            // a later decrease in this round re-queues the vertex anyway
            b = __ldg(g.row + u);
            e = __ldg(g.row + u + 1);
            du0 = __ldcg(a.dist + u);
          }
        }
        auto step = [&](const uint32_t* j, const uint32_t* own, uint32_t act) {
          int32_t du[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) du[r] = __shfl_sync(0xffffffffu, du0, own[r]);
          sssp_relax4e(a, du, j, act, sink, my_edges);
        };
        walk_group(b, e - b, step);
      }
    }
    warp_res_close(qout, 2u * g.n, res, kHole);
    if (stage) stage_flush(*stage, qout, &c->n_reg, 2u * g.n, a.overflow, nullptr, nullptr);
    relaxed_edges += my_edges;
    ++step;
    ok = bar.sync();
  }
  // per-thread relaxed-edge counts -> one total
  const unsigned long long ws = warp_sum_u64(relaxed_edges);
  if (lane_id() == 0 && ws) atomicAdd(a.out_edges, ws);
  if (team.cta == 0 && threadIdx.x == 0) {
    a.out[0] = rounds;
    a.out[1] = buckets;
    a.out[3] = ok ? 0u : 1u;
  }
}

// ---- thin graphs on one cluster ------------------------------------------------
// The rounds of a mesh's SSSP relax a few thousand edges: as in
// bfs_cluster_kernel the near queue stays in shared memory and the step's
// records are its barrier, and so do the far piles.  An entry carries the
// distance it was queued with: one that no longer equals the vertex's distance
// is skipped (whoever lowered it queued another entry), so no stamps are
// exchanged.  When a round outgrows the cluster the rest of the traversal runs
// on the grid (2048^2 grid, 5000 rounds: at most 10,000 entries).
constexpr uint32_t kSsspClQueue = 3072;   // near entries per CTA and parity
constexpr uint32_t kSsspClFar = 4096;     // far entries per CTA and parity
constexpr uint32_t kSsspClDegree = 1024;  // vertices of more edges go to the grid's team-wide lists

struct SsspClShared {
  uint4 q[2][kSsspClQueue];  // {vertex, first edge, end, distance} by parity of the step
  uint2 far[2][kSsspClFar];  // {vertex, distance}
  ClusterLink link;
  uint32_t n[2];     // near slots asked for, by parity of the step being built
  uint32_t m[2];     // their edges
  uint32_t fat[2];   // bit 0: an entry of more than 4 edges, bit 1: of more than 8
  uint32_t leave[2]; // an entry went to the global queues
  uint32_t farn[2];  // far slots asked for, by far parity
};

__global__ void __launch_bounds__(512) sssp_init_kernel(SsspArgs a, uint32_t* flags, uint32_t prefetch) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const DevCSR& g = a.g;
  for (uint32_t v = tid; v < g.n; v += nt) {
    a.dist[v] = v == a.src ? 0 : kInf;
    a.mark[v] = 0;
    a.fmark[v] = 0;
  }
  if (tid == 0) {
    for (int k = 0; k < 32; ++k) flags[k] = 0;
    for (int k = 0; k < 3; ++k) a.cnt[k].n_reg = a.cnt[k].n_big = a.cnt[k].m_next = 0;
    a.fcnt[0] = a.fcnt[1] = 0;
    const uint32_t d = g.row[a.src + 1] - g.row[a.src];
    if (d > kSsspClDegree) {  // the grid's queues of its first step
      a.hq[(kSsspStep - 1) & 1][0] = a.src;
      a.cnt[(kSsspStep - 1) % 3].n_big = 1;
    }
    a.state[1] = 1;
    *reinterpret_cast<long long*>(a.state + 2) = a.delta;
    a.phase[0] = d > kSsspClDegree ? PHASE_GRID : PHASE_CLUSTER;
  }
  if (prefetch) {
    prefetch_l2(g.row, (uint64_t)(g.n + 1) * 4, tid, nt);
    prefetch_l2(g.dst, (uint64_t)g.m * 4, tid, nt);
    prefetch_l2(g.w, (uint64_t)g.m * 4, tid, nt);
  }
}

// To the grid's queues of step kSsspStep, each vertex once.  Warp-synchronous.
__device__ __forceinline__ void sssp_to_grid_near(const SsspArgs& a, bool pred, uint32_t v, uint32_t deg) {
  constexpr uint32_t p = (kSsspStep - 1) & 1u;
  LevelCounters* c = &a.cnt[(kSsspStep - 1) % 3];
  if (pred) pred = atomicExch(a.mark + v, kSsspStep) != kSsspStep;
  warp_append(pred && deg <= kSsspBig, v, a.q[p], &c->n_reg, 2u * a.g.n, a.overflow);
  warp_append(pred && deg > kSsspBig, v, a.hq[p], &c->n_big, a.g.n, a.overflow);
}
__device__ __forceinline__ void sssp_to_grid_far(const SsspArgs& a, bool pred, uint32_t v) {
  if (pred) pred = atomicExch(a.fmark + v, 1u) != 1u;  // the grid's first far generation
  warp_append(pred, v, a.far[0], &a.fcnt[0], a.g.n, a.overflow);
}

// Appends lane entries to the near queue being built (parity o) / the far pile f.
__device__ __forceinline__ void sssp_cl_near(const SsspArgs& a, SsspClShared& s, uint32_t o, bool pred, uint4 e) {
  const uint32_t mask = __ballot_sync(0xffffffffu, pred);
  if (!mask) return;
  const uint32_t lane = lane_id(), tot = __popc(mask), d = pred ? e.z - e.y : 0u;
  uint32_t pos = 0;
  if (lane == 0) pos = atomicAdd(&s.n[o], tot);
  const uint32_t m = __reduce_add_sync(0xffffffffu, d);
  if (lane == 0) atomicAdd(&s.m[o], m);
  const bool fat = __any_sync(0xffffffffu, d > 4u);
  pos = __shfl_sync(0xffffffffu, pos, 0);
  bool hub = false;
  if (fat) {
    hub = __any_sync(0xffffffffu, d > kSsspClDegree);
    const bool fat8 = __any_sync(0xffffffffu, d > 8u);
    if (lane == 0) atomicOr(&s.fat[o], fat8 ? 3u : 1u);
  }
  const uint32_t at = pos + __popc(mask & lanemask_lt());
  if (pos + tot <= kSsspClQueue && !hub) {
    if (pred) s.q[o][at] = e;
    return;
  }
  // no room, or a vertex for the grid: the slots reserved here stay empty
  if (pred && at < kSsspClQueue) s.q[o][at] = make_uint4(0u, 0u, 0u, 0u);
  sssp_to_grid_near(a, pred, e.x, d);
  if (lane == 0) atomicOr(&s.leave[o], 1u);
}
__device__ __forceinline__ void sssp_cl_far(const SsspArgs& a, SsspClShared& s, uint32_t o, uint32_t f, bool pred,
                                            uint32_t v, int32_t d) {
  const uint32_t mask = __ballot_sync(0xffffffffu, pred);
  if (!mask) return;
  const uint32_t tot = __popc(mask);
  uint32_t pos = 0;
  if (lane_id() == 0) pos = atomicAdd(&s.farn[f], tot);
  pos = __shfl_sync(0xffffffffu, pos, 0);
  const uint32_t at = pos + __popc(mask & lanemask_lt());
  if (pred && at < kSsspClFar) s.far[f][at] = make_uint2(v, (uint32_t)d);
  if (pos + tot <= kSsspClFar) return;
  sssp_to_grid_far(a, pred && at >= kSsspClFar, v);
  if (lane_id() == 0) atomicOr(&s.leave[o], 1u);
}

// K edges per lane (bit r of `act`: edge j[r]) of entries at distance du[r],
// current when cur[r] still equals it.  Warp-synchronous.
template <int K>
__device__ __forceinline__ void sssp_cl_push(const SsspArgs& a, SsspClShared& s, uint32_t o, uint32_t f, int32_t T,
                                             const uint32_t* j, const int32_t* du, const int32_t* cur, uint32_t act,
                                             uint32_t& relaxed) {
  const DevCSR& g = a.g;
  uint32_t v[K];
  int32_t nd[K], old[K];
  uint2 rg[K];
#pragma unroll
  for (int r = 0; r < K; ++r) {
    v[r] = 0;
    nd[r] = 0;
    if ((act >> r) & 1u) {
      v[r] = __ldg(g.dst + j[r]);
      nd[r] = __ldg(g.w + j[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < K; ++r) {
    nd[r] = add_sat(du[r], nd[r]);
    const bool on = ((act >> r) & 1u) && cur[r] == du[r];
    relaxed += on;
    if (!on || nd[r] == kInf) act &= ~(1u << r);
    old[r] = 0;
    if ((act >> r) & 1u) old[r] = atomicMin(a.dist + v[r], nd[r]);
  }
#pragma unroll
  for (int r = 0; r < K; ++r) {
    rg[r] = make_uint2(0u, 0u);
    if (((act >> r) & 1u) && nd[r] < T) rg[r] = make_uint2(__ldg(g.row + v[r]), __ldg(g.row + v[r] + 1));
  }
#pragma unroll
  for (int r = 0; r < K; ++r) {
    const bool imp = ((act >> r) & 1u) && nd[r] < old[r], near = imp && nd[r] < T;
    if (near) {
      // the first edges are on their way to the SM while the round ends (a row
      // without edges may begin at the arrays' end; a test for that in place of
      // the clamp took 2.5 % of a 2048^2 grid)
      const uint32_t j0 = min(rg[r].x, g.m - 1u);
      asm volatile("prefetch.global.L1 [%0];" ::"l"(g.dst + j0));
      asm volatile("prefetch.global.L1 [%0];" ::"l"(g.w + j0));
    }
    sssp_cl_near(a, s, o, near, make_uint4(v[r], rg[r].x, rg[r].y, (uint32_t)nd[r]));
    sssp_cl_far(a, s, o, f, imp && !near, v[r], nd[r]);
  }
}

// A round over the CTA's own entries, all of at most 1 << SH edges (see bfs_cl_thin).
template <int SH, int K>
__device__ __forceinline__ void sssp_cl_thin(const SsspArgs& a, SsspClShared& s, uint32_t p, uint32_t f, int32_t T,
                                             uint32_t own, uint32_t& relaxed) {
  constexpr int kSh = SH - (K - 1);
  for (uint32_t i = threadIdx.x; ((i - lane_id()) >> kSh) < own; i += blockDim.x) {
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    if ((i >> kSh) < own) e = s.q[p][i >> kSh];
    uint32_t j[K], act = 0;
    int32_t du[K], cur[K];
    int32_t c = -1;
    if (e.y < e.z) c = __ldcg(a.dist + e.x);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      j[k] = e.y + (i & ((1u << kSh) - 1u)) * K + k;
      if (j[k] < e.z) act |= 1u << k;
      du[k] = (int32_t)e.w;
      cur[k] = c;
    }
    sssp_cl_push<K>(a, s, p ^ 1u, f, T, j, du, cur, act, relaxed);
  }
}

__global__ void __launch_bounds__(kClThreads, 1) sssp_cluster_kernel(SsspArgs a, unsigned long long timeout_ns) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  SsspClShared& s = *reinterpret_cast<SsspClShared*>(cl_smem);
  if (__ldcg(a.phase) != PHASE_CLUSTER) return;  // the same in every CTA
  const DevCSR& g = a.g;
  const uint32_t rank = gsrb::ptx::cluster_ctarank(), ncta = gsrb::ptx::cluster_nctarank();
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) {
    link_init(s.link, ncta);
    s.n[0] = s.n[1] = s.m[0] = s.m[1] = s.leave[0] = s.leave[1] = s.farn[0] = s.farn[1] = 0;
    s.fat[0] = s.fat[1] = 3u;  // nothing is known of the source
    if (rank == 0) {
      s.q[0][0] = make_uint4(a.src, g.row[a.src], g.row[a.src + 1], 0u);
      s.n[0] = 1;
    }
    link_expect(s.link, 0u, ncta);
  }
  gsrb::ptx::cluster_sync();
  if (wid == 0) link_publish(s.link, 0u, make_uint4(s.n[0], 0u, 0u, 0u), rank, ncta);
  uint32_t phases = 0, p = 0, f = 0, rounds = 0, buckets = 1, own, relaxed = 0;
  unsigned long long edges = 0;
  long long T = a.delta;
  const bool books = rank == 0 && wid == nw - 1;
  bool ok, done = false, agreed = false;
  for (;;) {
    // this step's near entries are in q[p], the far pile in far[f]
    ok = link_wait(s.link, p, phases, timeout_ns);
    const LinkSum t = link_sum<true>(s.link, p, rank, ncta);
    own = t.own;
    if (!ok || t.w || t.x > kClMaxFrontier || t.z > kClMaxEdges) break;
    if (t.x == 0 && t.y == 0) {
      done = true;
      break;
    }
    const uint32_t o = p ^ 1u;
    const uint32_t fat = s.fat[p];
    if (threadIdx.x == 0) {
      s.n[p] = s.m[p] = s.leave[p] = 0;  // published; next used in the step after this one
      link_expect(s.link, o, ncta);
    }
    if (t.x == 0) {
      // near bucket empty: advance the threshold and refill from the far piles
      T += a.delta;
      ++buckets;
      const int32_t T32 = (int32_t)min(T, (long long)kInf);
      const uint32_t nfar = min(s.farn[f], kSsspClFar);
      for (uint32_t base = wid * 32u; base < nfar; base += nw * 32u) {
        uint2 e = make_uint2(0u, 0u);
        bool live = base + lane < nfar;
        if (live) {
          e = s.far[f][base + lane];
          live = __ldcg(a.dist + e.x) == (int32_t)e.y;  // else lowered since: queued elsewhere
        }
        const bool near = live && (int32_t)e.y < T32;
        uint2 rg = make_uint2(0u, 0u);
        if (near) rg = make_uint2(__ldg(g.row + e.x), __ldg(g.row + e.x + 1));
        sssp_cl_near(a, s, o, near, make_uint4(e.x, rg.x, rg.y, e.y));
        sssp_cl_far(a, s, o, f ^ 1u, live && !near, e.x, (int32_t)e.y);
      }
      f ^= 1u;
    } else {
      ++rounds;
      if (books && lane == 0 && rounds - 1 < a.trace_cap) {
        LevelTrace r;
        r.level = rounds;
        r.dir = 3u;
        r.nf = t.x;
        r.nu = buckets;
        r.mf = 0;
        r.mu = (unsigned long long)T;
        r.t_ns = gsrb::ptx::globaltimer_ns();
        r.pred = __int_as_float(0x7fc00000);
        r.fallback = 0;
        a.trace[rounds - 1] = r;
      }
      const int32_t T32 = (int32_t)min(T, (long long)kInf);
      auto group = [&](uint4 e) {
        int32_t c = -1;
        if (e.y < e.z) c = __ldcg(a.dist + e.x);
        auto step = [&](const uint32_t* j, const uint32_t* from, uint32_t act) {
          int32_t du[4], cur[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            du[r] = __shfl_sync(0xffffffffu, (int32_t)e.w, from[r]);
            cur[r] = __shfl_sync(0xffffffffu, c, from[r]);
          }
          sssp_cl_push<4>(a, s, o, f, T32, j, du, cur, act, relaxed);
        };
        walk_group(e.y, e.z - e.y, step);
      };
      const bool uneven = link_uneven(t);
      if (uneven) ok = link_meet(s.link, phases, ncta, timeout_ns);
      if (!ok) {
        // gave up: on to the end of the step
      } else if (uneven) {
        // redistribute: an equal slice of all entries, read from their CTAs
        const uint32_t i0 = (uint32_t)((uint64_t)t.x * rank / ncta);
        const uint32_t i1 = (uint32_t)((uint64_t)t.x * (rank + 1) / ncta);
        const uint32_t gsz = cl_group(i1 - i0);
        for (uint32_t base = i0 + wid * gsz; base < i1; base += nw * gsz) {
          const bool in = lane < gsz && base + lane < i1;
          const uint32_t at = link_locate(s.link, p, ncta, in ? base + lane : 0u);
          uint4 e = make_uint4(0u, 0u, 0u, 0u);
          if (in)
            e = ld_cluster_v4(gsrb::ptx::mapa_shared(gsrb::ptx::smem_u32(&s.q[p][at & 0xffffu]), at >> 16));
          group(e);
        }
      } else if (fat == 0u) {
        if (own <= kClThreads / 4) sssp_cl_thin<2, 1>(a, s, p, f, T32, own, relaxed);
        else sssp_cl_thin<2, 2>(a, s, p, f, T32, own, relaxed);
      } else {
        const uint32_t gsz = cl_group(own);
        for (uint32_t base = wid * gsz; base < own; base += nw * gsz) {
          uint4 e = make_uint4(0u, 0u, 0u, 0u);
          if (lane < gsz && base + lane < own) e = s.q[p][base + lane];
          group(e);
        }
      }
      if (relaxed >= 1u << 30) {
        edges += relaxed;
        relaxed = 0;
      }
    }
    agreed = true;
    if (!(ok = link_agree(ok))) break;
    agreed = false;
    if (wid == 0) {
      if (lane == 0) {
        s.fat[p] = 0;  // every thread has read it
        if (t.x == 0) s.farn[f ^ 1u] = 0;  // the pile just read
      }
      link_publish(s.link, o, make_uint4(min(s.n[o], kSsspClQueue), min(s.farn[f], kSsspClFar), s.m[o], s.leave[o]),
                   rank, ncta);
    }
    p = o;
  }
  if (!agreed) ok = link_agree(ok);
  if (!ok && threadIdx.x == 0) atomicExch(a.overflow + 1, 1u);
  edges = warp_sum_u64(edges + relaxed);
  if (lane == 0 && edges) atomicAdd(a.out_edges, edges);
  if (!done && ok) {
    // the grid takes over: this step's entries and the far piles, each vertex once
    for (uint32_t base = wid * 32u; base < own; base += nw * 32u) {
      uint4 e = make_uint4(0u, 0u, 0u, 0u);
      if (base + lane < own) e = s.q[p][base + lane];
      sssp_to_grid_near(a, e.y < e.z, e.x, e.z - e.y);
    }
    const uint32_t nfar = min(s.farn[f], kSsspClFar);
    for (uint32_t base = wid * 32u; base < nfar; base += nw * 32u) {
      uint2 e = make_uint2(0u, 0u);
      if (base + lane < nfar) e = s.far[f][base + lane];
      sssp_to_grid_far(a, base + lane < nfar, e.x);
    }
  }
  if (books && lane == 0) {
    if (done || !ok) {
      a.out[0] = rounds;
      a.out[1] = buckets;
      a.out[3] = ok ? 0u : 1u;
    } else {
      a.state[0] = rounds;
      a.state[1] = buckets;
      *reinterpret_cast<long long*>(a.state + 2) = T;
    }
    a.phase[0] = done || !ok ? PHASE_DONE : PHASE_GRID;
  }
  gsrb::ptx::cluster_sync();  // no CTA leaves while a record to it may be in flight
}

template <int V>
__global__ void __launch_bounds__(1024)
sssp_kernel(gsrb::GridBarrier gb, SsspArgs a) {
  __shared__ gsrb::BarrierShared bsh;
  gsrb::GridSync<V> bar;
  const bool ok = bar.init(gb, &bsh);
  sssp_run<V>(bar, ok, a, Team{blockIdx.x, gridDim.x});
  bar.finish();
}

// ------------------------------------------------------------------ batches ---
// Many traversals in one persistent launch: instance i owns CTAs
// [first_i, first_i + count_i) and a barrier slot of its own (sub-grid
// barriers carved from the same state block).  A CTA finds its instance in a
// table, copies the instance's descriptor and runs the same traversal body as
// the single-instance kernels.  Only barrier variants whose verdict does not
// involve hardware cluster barriers are used (instances of one CTA are allowed).
struct BatchDesc {
  gsrb::GridBarrier gb;
  uint32_t first;
  uint32_t count;
  uint32_t kind;  // 0 BFS, 1 SSSP
  uint32_t pad;
  BfsArgs bfs;
  SsspArgs sssp;
};

// One kernel per kind: a kernel holding both bodies spilled 1.4 KB a thread,
// more than the L1 holds for a CTA (16 R-MAT SSSPs: 1.8 ms).  The descriptor is
// copied to shared memory, so the body's reads of it cost no L2 trip.
template <int V, int KIND>
__global__ void __launch_bounds__(kGraphMaxThreads)
batch_kernel(const BatchDesc* __restrict__ descs, const uint16_t* __restrict__ cta_inst) {
  __shared__ gsrb::BarrierShared bsh;
  __shared__ uint4 s_desc[(sizeof(BatchDesc) + 15) / 16];
  static_assert(sizeof(BatchDesc) % 4 == 0, "copied word by word");
  const uint32_t* src = reinterpret_cast<const uint32_t*>(descs + cta_inst[blockIdx.x]);
  for (uint32_t i = threadIdx.x; i < sizeof(BatchDesc) / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(s_desc)[i] = src[i];
  __syncthreads();
  const BatchDesc& d = *reinterpret_cast<const BatchDesc*>(s_desc);
  const Team team{blockIdx.x - d.first, d.count};
  gsrb::GridSync<V> bar;
  const bool ok = bar.init(d.gb, &bsh);
  if (KIND == 0) bfs_run<V>(bar, ok, d.bfs, d.bfs, team);
  else sssp_run<V>(bar, ok, d.sssp, team);
  bar.finish();
}

// --------------------------------------------------------------- PageRank ---
// What a pull pass over a symmetric graph reads besides its input values.
struct PullArgs {
  const uint32_t* hubs;   // vertices of degree > kPrHubDegree, ascending
  const uint32_t* hub_c0; // [nhubs + 1] first chunk of each hub
  const uint32_t* chunk_hub;  // [nchunks] hub index of each chunk
  uint32_t nhubs, nchunks;
  double* part;           // [nchunks] chunk sums
  uint32_t* hub_done;     // [nhubs] finished chunks (monotonic over passes)
  unsigned long long* ticket;  // block tickets (monotonic over passes)
  int32_t gather_l1;      // 1: x/deg gathers through L1 (ld.ca), 0: L2 only (ld.cg)
};
struct PrArgs {
  DevCSR g;
  float alpha;
  int32_t iters;
  float* rank;            // output x (FP32)
  float* contrib[2];      // x / deg, double-buffered by iteration parity
  PullArgs pull;
  uint32_t* out;
};

// One x/deg gather.  Through L1 the hubs' entries (read by many rows of a
// power-law graph) hit in the SM: an edge-parallel pass over RMAT-22 with
// nothing but these gathers runs at 340 G edges/s through L1 against 224
// through L2 only.  The buffer a gather reads was last written two iterations
// earlier, before the grid barrier whose acquire orders those writes before
// every later load of the CTA (the acquire invalidates the SM's L1).
__device__ __forceinline__ float pr_gather(const float* cin, uint32_t d, int l1) {
  return l1 ? __ldca(cin + d) : __ldcg(cin + d);
}

// Sum of cin[dst[j]] over j in [j0, j1) by one warp: lanes stride the range,
// 4 independent gathers in flight per lane, FP64 per lane, fixed-order
// butterfly at the end (the same bits on every run).  The destinations of the
// next 128 edges are loaded while this step's gathers are in flight, so a
// step costs one dependent round trip (the gather), not two.
__device__ __forceinline__ double warp_gather_sum(const uint32_t* __restrict__ dst, const float* cin, uint32_t j0,
                                                  uint32_t j1, uint32_t lane, int l1) {
  double s = 0.0;
  uint32_t j = j0 + lane;
  uint32_t d0 = 0, d1 = 0, d2 = 0, d3 = 0;
  if (j + 96 < j1) {
    d0 = __ldg(dst + j);
    d1 = __ldg(dst + j + 32);
    d2 = __ldg(dst + j + 64);
    d3 = __ldg(dst + j + 96);
  }
  for (; j + 96 < j1; j += 128) {
    const float c0 = pr_gather(cin, d0, l1), c1 = pr_gather(cin, d1, l1), c2 = pr_gather(cin, d2, l1),
                c3 = pr_gather(cin, d3, l1);
    if (j + 224 < j1) {
      d0 = __ldg(dst + j + 128);
      d1 = __ldg(dst + j + 160);
      d2 = __ldg(dst + j + 192);
      d3 = __ldg(dst + j + 224);
    }
    s += (double)c0;
    s += (double)c1;
    s += (double)c2;
    s += (double)c3;
  }
  for (; j < j1; j += 32) s += (double)pr_gather(cin, __ldg(dst + j), l1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// One pull pass: done(v, degree, sum of cin over v's row) once for every vertex,
// by one lane; pass number `it` of the launch, warp gw of nw.
//  * Hubs (degree > kPrHubDegree) are cut into chunks of kPrChunk edges; a warp
//    sums a chunk, stores it, and bumps the hub's counter (acq_rel); the warp
//    that finishes a hub's last chunk adds the chunk sums in chunk order.
//  * Every other vertex: a warp takes 32 consecutive vertices and walks their
//    concatenated edge lists 32 edges per round (coalesced dst loads); each
//    lane finds the owner of its edge by a binary search over the lanes'
//    exclusive degree prefix, and a segmented shuffle scan hands each owner its
//    segment's sum.  Per-vertex FP64 sums in a fixed order.
template <class F>
__device__ __forceinline__ void pull_pass(const DevCSR& g, const PullArgs& a, const float* cin, uint32_t it, uint32_t gw,
                                          uint32_t nw, F& done) {
  const uint32_t lane = lane_id();
  // ---- hub chunks
  for (uint32_t c = gw; c < a.nchunks; c += nw) {
    const uint32_t k = __ldg(a.chunk_hub + c);
    const uint32_t u = __ldg(a.hubs + k);
    const uint32_t c0 = __ldg(a.hub_c0 + k), c1 = __ldg(a.hub_c0 + k + 1);
    const uint32_t ub = __ldg(g.row + u), ue = __ldg(g.row + u + 1);
    const uint32_t j0 = ub + (c - c0) * kPrChunk;
    const uint32_t j1 = min(ue, j0 + kPrChunk);
    const double t = warp_gather_sum(g.dst, cin, j0, j1, lane, a.gather_l1);
    uint32_t last = 0;
    if (lane == 0) {
      a.part[c] = t;
      const uint32_t target = (c1 - c0) * (it + 1u);
      last = gsrb::ptx::atom_add_acq_rel_gpu(a.hub_done + k, 1u) + 1u == target;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (last) {
      // fixed order: lane-strided chunk sums, then the same butterfly
      double s = 0.0;
      for (uint32_t i = c0 + lane; i < c1; i += 32) s += __ldcg(a.part + i);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) done(u, ue - ub, s);
    }
  }
  // ---- everything else: blocks of 32 consecutive vertices, taken by warps
  // from a ticket counter (block sizes vary by orders of magnitude)
  const uint32_t nblocks = (g.n + 31u) >> 5;
  const unsigned long long tbase = (unsigned long long)it * (nblocks + nw);
  for (;;) {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(a.ticket, 1ull);
    t = __shfl_sync(0xffffffffu, t, 0);
    const unsigned long long blk = t - tbase;
    if (blk >= nblocks) break;  // every warp draws exactly one ticket past the end
    const uint32_t v = (uint32_t)blk * 32u + lane;
    uint32_t b = 0, d = 0;
    bool mine = false;
    if (v < g.n) {
      b = __ldg(g.row + v);
      const uint32_t dd = __ldg(g.row + v + 1) - b;
      mine = dd <= kPrHubDegree;
      d = mine ? dd : 0u;
    }
    uint32_t inc = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if ((int)lane >= o) inc += y;
    }
    const uint32_t excl = inc - d;
    const uint32_t E = __shfl_sync(0xffffffffu, inc, 31);
    double acc = 0.0;
    // kRounds rounds of 32 edges per step: all gathers of a step in flight together
    constexpr int kRounds = 4;
    for (uint32_t f0 = 0; f0 < E; f0 += 32u * kRounds) {
      uint32_t own[kRounds], nbr[kRounds];
      double val[kRounds];
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const uint32_t f = f0 + 32u * r + lane;
        // owner = the last lane whose exclusive prefix is <= f; the search
        // carries that prefix along (lane 0's is 0), so it costs no shuffle
        uint32_t lo = 0, oe = 0;
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1) {
          const uint32_t x = __shfl_sync(0xffffffffu, excl, lo + step);
          if (x <= f) {
            lo += step;
            oe = x;
          }
        }
        // the lane (of this round) where the owner's segment begins: the
        // segmented scan below compares lanes against it instead of
        // shuffling owners
        own[r] = oe > f0 + 32u * r ? oe - (f0 + 32u * r) : 0u;
        const uint32_t ob = __shfl_sync(0xffffffffu, b, lo);
        nbr[r] = f < E ? __ldg(g.dst + ob + (f - oe)) : 0u;
      }
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const uint32_t f = f0 + 32u * r + lane;
        val[r] = f < E ? (double)pr_gather(cin, nbr[r], a.gather_l1) : 0.0;
      }
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const uint32_t rb = f0 + 32u * r;
        if (rb >= E) break;  // warp-uniform
        // segmented inclusive scan: lane l - o belongs to the same owner
        // as lane l exactly when l - o is not before the owner's first lane
        double x = val[r];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(0xffffffffu, x, o);
          if ((int)lane - o >= (int)own[r]) x += y;
        }
        // this lane's vertex: its segment in this round ends at flat index
        // min(excl + d, rb + 32, E) - 1
        const uint32_t seg_b = excl > rb ? excl : rb;
        const uint32_t seg_e = min(min(excl + d, rb + 32u), E);
        const uint32_t endl = seg_e > seg_b ? seg_e - 1u - rb : 0u;
        const double t2 = __shfl_sync(0xffffffffu, x, endl);
        if (seg_e > seg_b) acc += t2;
      }
    }
    if (mine) done(v, d, acc);
  }
}

// Pull PageRank, one grid barrier per iteration (see pull_pass).
template <int V>
__global__ void __launch_bounds__(1024)
pagerank_kernel(gsrb::GridBarrier gb, PrArgs a) {
  __shared__ gsrb::BarrierShared bsh;
  gsrb::GridSync<V> bar;
  bool ok = bar.init(gb, &bsh);
  const DevCSR& g = a.g;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  const float base = 1.f - a.alpha;
  // x0 = 1 - alpha (apps/pr/kernel_gsrb.cu:311)
  for (uint32_t v = tid; v < g.n; v += nthreads) {
    const uint32_t d = __ldg(g.row + v + 1) - __ldg(g.row + v);
    a.rank[v] = base;
    a.contrib[0][v] = d ? base / (float)d : 0.f;
  }
  ok = bar.sync() && ok;
  const uint32_t gw = tid >> 5, nw = nthreads >> 5;
  int32_t it = 0;
  for (; ok && it < a.iters; ++it) {
    const float* cin = a.contrib[it & 1];
    float* cout = a.contrib[(it + 1) & 1];
    auto done = [&](uint32_t v, uint32_t d, double sum) {
      const float x = (float)((double)base + (double)a.alpha * sum);
      a.rank[v] = x;
      cout[v] = d ? x / (float)d : 0.f;
    };
    pull_pass(g, a.pull, cin, (uint32_t)it, gw, nw, done);
    ok = bar.sync();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out[0] = (uint32_t)it;
    a.out[3] = ok ? 0u : 1u;
  }
  bar.finish();
}

// ------------------------------------------------------ push-residual PR ---
// The reference's PageRank (apps/pr/kernel_gsrb.cu:298-508, restated):
//   init_1  p[v] = 1 - alpha; r[w] += 1 / outdeg(u) over every edge u -> w
//   init_2  r[v] *= (1 - alpha) * alpha; every vertex enters the worklist
//   round   for every u in the worklist: res = exchange(r[u], 0); p[u] += res;
//           for every edge u -> w: prev = r[w] += alpha * res / outdeg(u), and
//           w enters the next worklist when r[w] crosses epsilon from below
// until the worklist is empty or max_iters rounds ran; one grid barrier per
// round (+1 when hub vertices, degree > kBigDegree, are in the worklist: their
// residual is taken first and their edges are split across the grid).  FP32
// atomics in an order that changes from run to run, as in the reference;
// p[u] is updated atomically (the reference's plain += races when a vertex is
// in a worklist twice).
struct PrrArgs {
  DevCSR g;
  float alpha, eps;
  int32_t max_iters;
  float* p;             // output ranks
  float* r;             // residuals
  float* hub_upd;       // alpha * res / outdeg of the hubs of the current round, by vertex
  float* share[2];      // pulled rounds: alpha * res / outdeg by vertex, in turn ([0] is hub_upd)
  uint32_t* mark;       // round stamps: a vertex enters a worklist at most once
  uint32_t* q[2];
  uint32_t* hq[2];
  LevelCounters* cnt;   // [3]
  uint32_t* overflow;
  uint32_t* out;        // [0] rounds, [1] worklist pushes (low 32 bits), [3] failure
  unsigned long long* out_edges;
  PullArgs pull;
  bool symmetric;       // rows are also in-edge lists: rounds with many edges may pull
  bool stage;           // the launch has the CTAs' stages
};

// A round whose worklist holds at least 1 / kPrrDense of the edges is pulled on
// a symmetric graph: the same round (every vertex of the list takes its
// residual, every neighbour receives its shares) without an atomic per edge.
// R-MAT-20: a pull round takes 0.15 ms whatever the list, a push round about
// 1 ms for all the edges.
constexpr unsigned long long kPrrDense = 8;

// Vertices of the regular queue with more edges than this are pushed by their
// whole CTA (after the CTA's warps have walked their queue groups), so that one
// warp does not walk thousands of edges while the rest of the grid waits at
// the round's barrier (the thread-block tier of the reference's nested
// parallelism, LONESTAR/rt/include/internal.h.prehip:99-158).
constexpr uint32_t kCtaDegree = 256;
constexpr uint32_t kCtaListCap = 256;

// Where a residual push step puts the vertices whose residual crossed epsilon.
struct PrrSink {
  uint32_t* qout;
  uint32_t* hout;
  unsigned long long* n_reg;
  unsigned long long* n_big;
  uint32_t stamp;  // a vertex enters the next worklist at most once per round
  IdStage* stage;  // the CTA's worklist entries (null: none)
  WarpRes* res;    // the warp's worklist reservation (past the stage)
};

// Push residual along four edges per lane at once: edge r of the lane is j[r]
// (bit r of `act`), carrying upd[r].  The four destinations, then the four
// residual additions, then the four worklist stamps are issued together, and
// the warp reserves queue space once per step (apps/pr/kernel_gsrb.cu:430-470:
// r[dst] += alpha * res / outdeg, pushed when it crosses epsilon).
// Warp-synchronous.
__device__ __forceinline__ void prr_push4e(const PrrArgs& a, const float* upd, const uint32_t* j, uint32_t act,
                                           const PrrSink& s, unsigned long long& pushes,
                                           unsigned long long& medges) {
  const DevCSR& g = a.g;
  uint32_t w[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) w[r] = ((act >> r) & 1u) ? __ldg(g.dst + j[r]) : 0u;
  float prev[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    prev[r] = a.eps;
    if ((act >> r) & 1u) prev[r] = atomicAdd(a.r + w[r], upd[r]);
  }
  bool cross[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) cross[r] = ((act >> r) & 1u) && prev[r] + upd[r] > a.eps && prev[r] < a.eps;
  // the row range of a candidate goes out with its stamp exchange (one round
  // trip instead of two; unused when the exchange finds it already queued)
  uint32_t rb[4], re[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    rb[r] = cross[r] ? __ldg(g.row + w[r]) : 0u;
    re[r] = cross[r] ? __ldg(g.row + w[r] + 1) : 0u;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    uint32_t st = s.stamp;
    if (cross[r]) st = atomicExch(a.mark + w[r], s.stamp);
    cross[r] = st != s.stamp;
  }
  bool reg[4], big[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t d = cross[r] ? re[r] - rb[r] : 0u;
    reg[r] = cross[r] && d <= kBigDegree;
    big[r] = cross[r] && d > kBigDegree;
    pushes += cross[r] ? 1u : 0u;
    medges += d;
  }
  stage_append<4>(reg, w, s.stage, s.qout, s.n_reg, g.n, 2u * g.n, a.overflow, *s.res, kHole);
  warp_append_k<4>(big, w, s.hout, s.n_big, g.n, a.overflow);
}

// A list of vertices pushed edge-balanced: edge prefix p[0..cnt], first edges
// b[], updates (float bits) d[] in shared memory; thread x of nthr takes edges
// (x & ~31) + lane + k * nthr, four per step.  Warp-synchronous loops.
__device__ __forceinline__ void prr_push_list(const PrrArgs& a, const uint32_t* p, const uint32_t* b,
                                              const int32_t* d, uint32_t cnt, uint32_t x, uint32_t nthr,
                                              const PrrSink& s, unsigned long long& pushes,
                                              unsigned long long& medges) {
  const uint32_t total = p[cnt];
  for (uint32_t t0 = (x & ~31u) + lane_id(); t0 - lane_id() < total; t0 += 4u * nthr) {
    float upd[4];
    uint32_t j[4];
    uint32_t act = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t t = t0 + (uint32_t)r * nthr;
      upd[r] = 0.f;
      j[r] = 0;
      if (t < total) {
        const uint32_t o = list_owner(p, cnt, t);
        j[r] = b[o] + (t - p[o]);
        upd[r] = __int_as_float(d[o]);
        act |= 1u << r;
      }
    }
    prr_push4e(a, upd, j, act, s, pushes, medges);
  }
}

template <int V>
__global__ void __launch_bounds__(1024)
pr_residual_kernel(gsrb::GridBarrier gb, PrrArgs a) {
  __shared__ gsrb::BarrierShared bsh;
  gsrb::GridSync<V> bar;
  bool ok = bar.init(gb, &bsh);
  const DevCSR& g = a.g;
  const Team team{blockIdx.x, gridDim.x};
  const uint32_t tid = team.tid(), nthreads = team.nthreads();
  const uint32_t lane = lane_id();
  IdStage* const stage = cta_stage<IdStage>(a.stage);
  // init_1
  for (uint32_t v = tid; v < g.n; v += nthreads) {
    a.p[v] = 1.f - a.alpha;
    a.r[v] = 0.f;
    a.mark[v] = 0;
  }
  if (tid == 0)
    for (int k = 0; k < 3; ++k) a.cnt[k].n_reg = a.cnt[k].n_real = a.cnt[k].n_big = a.cnt[k].m_next = 0;
  ok = bar.sync() && ok;
  bool dense = a.symmetric;
  uint32_t pulls = 0;
  if (dense) {
    // the neighbours' 1 / outdeg, pulled (an atomic per edge took about 1 ms on R-MAT-20)
    for (uint32_t v = tid; v < g.n; v += nthreads) {
      const uint32_t d = __ldg(g.row + v + 1) - __ldg(g.row + v);
      a.hub_upd[v] = d ? 1.f / (float)d : 0.f;
    }
    ok = bar.sync() && ok;
    auto done = [&](uint32_t v, uint32_t, double sum) { a.r[v] = (float)sum; };
    if (ok) pull_pass(g, a.pull, a.hub_upd, pulls, tid >> 5, nthreads >> 5, done);
    ++pulls;
  } else {
    for (uint32_t gwarp = tid >> 5; gwarp * 32u < g.n; gwarp += nthreads >> 5) {
      const uint32_t u = gwarp * 32u + lane;
      uint32_t b = 0, e = 0;
      if (u < g.n) {
        b = __ldg(g.row + u);
        e = __ldg(g.row + u + 1);
      }
      const float upd = e > b ? 1.f / (float)(e - b) : 0.f;
      // warp-strided edges of the 32 vertices, one vertex at a time
      for (int src = 0; src < 32; ++src) {
        const uint32_t bb = __shfl_sync(0xffffffffu, b, src), ee = __shfl_sync(0xffffffffu, e, src);
        const float uu = __shfl_sync(0xffffffffu, upd, src);
        for (uint32_t j = bb + lane; j < ee; j += 32) atomicAdd(a.r + __ldg(g.dst + j), uu);
      }
    }
  }
  ok = bar.sync() && ok;
  // init_2: scale, every vertex enters the worklist (hubs to the hub queue; a
  // pulled first round needs no list)
  for (uint32_t base = (tid >> 5) * 32u; base < g.n; base += nthreads) {
    const uint32_t v = base + lane;
    bool reg = false, big = false;
    if (v < g.n) {
      const float res = a.r[v] * ((1.f - a.alpha) * a.alpha);
      a.r[v] = res;
      const uint32_t d = __ldg(g.row + v + 1) - __ldg(g.row + v);
      if (dense) a.share[0][v] = d ? res * a.alpha / (float)d : 0.f;
      big = d > kBigDegree;
      reg = !big;
    }
    if (!dense) {
      warp_append(reg, v, a.q[0], &a.cnt[0].n_reg, g.n, a.overflow);
      warp_append(big, v, a.hq[0], &a.cnt[0].n_big, g.n, a.overflow);
    }
  }
  __shared__ unsigned long long s_edges, s_active;  // empty at the start of every round
  if (threadIdx.x == 0) s_edges = s_active = 0;
  ok = bar.sync() && ok;
  bool shares = dense;  // the shares of the residuals are there, in share[pulls_from]
  uint32_t pulls_from = 0;
  uint32_t round = 0;
  unsigned long long pushes = 0;
  for (; ok && round < (uint32_t)a.max_iters; ++round) {
    LevelCounters* c = &a.cnt[(round + 1) % 3];
    uint32_t* qout = a.q[(round + 1) & 1];
    uint32_t* hout = a.hq[(round + 1) & 1];
    if (dense) {
      // the list is the vertices above epsilon (in the first round all of
      // them); a pull costs the same with the rest's residuals, so those are
      // taken along and less is left over at the end.  The pass that sums a
      // vertex's new residual also adds the old one to its rank and leaves the
      // new one's share for the next pass, so a round is one pass and one
      // barrier (with the shares in a pass of their own, behind another barrier, a
      // 100 x 100 grid took 0.95 ms, now 0.65; pushed, 0.90)
      if (!shares) {
        for (uint32_t v = tid; v < g.n; v += nthreads) {
          const uint32_t d = __ldg(g.row + v + 1) - __ldg(g.row + v);
          a.share[0][v] = d ? a.r[v] * a.alpha / (float)d : 0.f;
        }
        pulls_from = 0;
        shares = true;
        ok = bar.sync();
        if (!ok) break;
      }
      const float* share = a.share[pulls_from];
      float* share_out = a.share[pulls_from ^ 1u];
      pulls_from ^= 1u;
      if (tid == 0) {
        // counters of the round after next, last read ahead of the barrier that ended the round before
        LevelCounters* z = &a.cnt[(round + 2) % 3];
        z->n_reg = z->n_big = z->n_real = z->m_next = 0;
      }
      unsigned long long medges = 0;
      uint32_t nact = 0;
      auto done = [&](uint32_t v, uint32_t d, double sum) {
        const float r = (float)sum;
        a.p[v] += a.r[v];
        a.r[v] = r;
        share_out[v] = d ? r * a.alpha / (float)d : 0.f;
        if (r > a.eps) {
          ++nact;
          medges += d;
        }
      };
      pull_pass(g, a.pull, share, pulls, tid >> 5, nthreads >> 5, done);
      ++pulls;
      medges = warp_sum_u64(medges);
      const uint32_t wact = __reduce_add_sync(0xffffffffu, nact);
      if (lane == 0 && wact) {
        atomicAdd(&s_edges, medges);
        atomicAdd(&s_active, (unsigned long long)wact);
      }
      __syncthreads();
      if (threadIdx.x == 0 && s_active) {
        atomicAdd(&c->m_next, s_edges);
        atomicAdd(&c->n_real, s_active);
        s_edges = s_active = 0;
      }
      ok = bar.sync();
      if (!ok) break;
      const unsigned long long act = __ldcg(&c->n_real), me = __ldcg(&c->m_next);
      if (tid == 0) pushes += act;
      if (act == 0) {
        ++round;
        break;
      }
      dense = me * kPrrDense >= g.m;
      if (!dense) {
        shares = false;
        // the rounds that follow push: make the list
        for (uint32_t base = (tid >> 5) * 32u; base < g.n; base += nthreads) {
          const uint32_t v = base + lane;
          bool in = v < g.n && a.r[v] > a.eps;
          uint32_t d = 0;
          if (in) d = __ldg(g.row + v + 1) - __ldg(g.row + v);
          const bool reg[1] = {in && d <= kBigDegree};
          const uint32_t vv[1] = {v};
          WarpRes none{0ull, 0u, 0u};
          stage_append<1>(reg, vv, stage, qout, &c->n_reg, g.n, 2u * g.n, a.overflow, none, kHole);
          warp_append(in && d > kBigDegree, v, hout, &c->n_big, g.n, a.overflow);
        }
        if (stage) stage_flush(*stage, qout, &c->n_reg, 2u * g.n, a.overflow, nullptr, nullptr);
        ok = bar.sync();
        if (!ok) break;
      }
      continue;
    }
    const uint32_t nreg = (uint32_t)__ldcg(&a.cnt[round % 3].n_reg);
    const uint32_t nbig = (uint32_t)__ldcg(&a.cnt[round % 3].n_big);
    if (nreg + nbig == 0) break;
    if (tid == 0) {
      LevelCounters* z = &a.cnt[(round + 2) % 3];
      z->n_reg = z->n_big = z->n_real = z->m_next = 0;
    }
    const uint32_t* qin = a.q[round & 1];
    const uint32_t* hin = a.hq[round & 1];
    unsigned long long medges = 0;  // edges of the vertices this thread queues
    // a vertex whose residual crosses epsilon twice in one round (its own
    // exchange in this round restarted it from 0) enters the next list once
    const uint32_t stamp = round + 2u;
    auto push = [&](bool cross, uint32_t w) {
      uint32_t d = 0;
      if (cross) cross = atomicExch(a.mark + w, stamp) != stamp;
      if (cross) d = __ldg(g.row + w + 1) - __ldg(g.row + w);
      // (the worklist's slots may include reservation holes: 2n of them)
      warp_append(cross && d <= kBigDegree, w, qout, &c->n_reg, 2u * g.n, a.overflow);
      warp_append(cross && d > kBigDegree, w, hout, &c->n_big, g.n, a.overflow);
      pushes += cross ? 1u : 0u;
      medges += d;
    };
    // worklist reservations in chunks of 64 slots when the queue (2n slots)
    // can hold the holes of every warp (see WarpRes)
    WarpRes wres{0ull, 0u, 63ull * (nthreads >> 5) <= g.n ? 64u : 0u};
    const PrrSink sink{qout, hout, &c->n_reg, &c->n_big, stamp, stage, &wres};
    ListSmem& L_ = list_smem();
    // builds an edge-balanced list from vertex ids and their updates (CTA-wide)
    auto build_list = [&](auto id_of, auto upd_of, uint32_t cnt) {
      uint32_t carry = 0;
      for (uint32_t base = 0; base < cnt; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        uint32_t d = 0;
        if (i < cnt) {
          const uint32_t u = id_of(i);
          const uint32_t b = __ldg(g.row + u);
          d = __ldg(g.row + u + 1) - b;
          L_.b[i] = b;
          L_.d[i] = __float_as_int(upd_of(i, u));
        }
        uint32_t tile = 0;
        const uint32_t ex = block_exclusive_scan(d, L_.scan, &tile);
        if (i < cnt) L_.p[i] = carry + ex;
        carry += tile;
      }
      if (threadIdx.x == 0) L_.p[cnt] = carry;
      __syncthreads();
    };
    if (nbig) {
      // hubs: take the residual once, then share the edges across the grid
      for (uint32_t k = tid; k < nbig; k += nthreads) {
        const uint32_t u = __ldcg(hin + k);
        const float res = atomicExch(a.r + u, 0.f);
        atomicAdd(a.p + u, res);
        a.hub_upd[u] = res * a.alpha / (float)(__ldg(g.row + u + 1) - __ldg(g.row + u));
      }
      ok = bar.sync();
      if (!ok) break;
      if (nbig <= kHubList) {
        build_list([&](uint32_t i) { return __ldcg(hin + i); },
                   [&](uint32_t, uint32_t u) { return __ldcg(a.hub_upd + u); }, nbig);
        prr_push_list(a, L_.p, L_.b, L_.d, nbig, tid, nthreads, sink, pushes, medges);
        __syncthreads();
      } else {
        auto hub_edge = [&](uint32_t u, uint32_t j, bool active) {
          bool cross = false;
          uint32_t w = 0;
          if (active) {
            w = __ldg(g.dst + j);
            const float upd = __ldcg(a.hub_upd + u);
            const float prev = atomicAdd(a.r + w, upd);
            cross = prev + upd > a.eps && prev < a.eps;
          }
          push(cross, w);
        };
        expand_hubs(team, g, hin, nbig, hub_edge);
      }
    }
    // regular worklist: a lane per vertex exchanges its residual once; edges
    // of degree > kCtaDegree vertices go to the CTA's edge-balanced list, the
    // rest edge-balanced over the warp, four edges per lane in flight
    __shared__ uint32_t s_cta_u[kCtaListCap];
    __shared__ float s_cta_upd[kCtaListCap];
    __shared__ uint32_t s_ncta;
    if (threadIdx.x == 0) s_ncta = 0;
    __syncthreads();
    const uint32_t nwarps = nthreads >> 5, gsz = group_size_of(nreg, nwarps);
    for (uint32_t base = spread_warp(team) * gsz; base < nreg; base += nwarps * gsz) {
      const uint32_t i = base + lane;
      const bool in = lane < gsz && i < nreg;
      uint32_t u = 0, b = 0, e = 0;
      float upd = 0.f;
      if (in) u = __ldcg(qin + i);
      if (in && u != kHole) {
        b = __ldg(g.row + u);
        e = __ldg(g.row + u + 1);
        const float res = atomicExch(a.r + u, 0.f);
        atomicAdd(a.p + u, res);
        upd = e > b ? res * a.alpha / (float)(e - b) : 0.f;
      }
      uint32_t deg = e - b;
      if (deg > kCtaDegree) {
        const uint32_t slot = atomicAdd(&s_ncta, 1u);
        if (slot < kCtaListCap) {
          s_cta_u[slot] = u;
          s_cta_upd[slot] = upd;
          deg = 0;
        }
      }
      auto step = [&](const uint32_t* j, const uint32_t* own, uint32_t act) {
        float u4[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) u4[r] = __shfl_sync(0xffffffffu, upd, own[r]);
        prr_push4e(a, u4, j, act, sink, pushes, medges);
      };
      walk_group(b, deg, step);
    }
    __syncthreads();
    const uint32_t ncta = min(s_ncta, kCtaListCap);
    if (ncta) {
      build_list([&](uint32_t i) { return s_cta_u[i]; }, [&](uint32_t i, uint32_t) { return s_cta_upd[i]; }, ncta);
      prr_push_list(a, L_.p, L_.b, L_.d, ncta, threadIdx.x, blockDim.x, sink, pushes, medges);
    }
    warp_res_close(qout, 2u * g.n, wres, kHole);
    medges = warp_sum_u64(medges);
    if (lane == 0 && medges) atomicAdd(&s_edges, medges);
    if (stage) stage_flush(*stage, qout, &c->n_reg, 2u * g.n, a.overflow, nullptr, nullptr);
    else __syncthreads();
    if (threadIdx.x == 0 && s_edges) {
      atomicAdd(&c->m_next, s_edges);
      s_edges = 0;
    }
    ok = bar.sync();
    if (!ok) break;
    dense = a.symmetric && __ldcg(&c->m_next) * kPrrDense >= g.m;
  }
  const unsigned long long ws = warp_sum_u64(pushes);
  if (lane == 0 && ws) atomicAdd(a.out_edges, ws);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out[0] = round;
    a.out[3] = ok ? 0u : 1u;
  }
  bar.finish();
}

template <template <int> class K>
struct Dummy {};

#define GSRB_GRAPH_FN(KERNEL)                                                    \
  [](int variant) -> const void* {                                              \
    switch (variant) {                                                          \
      case gsrb::V_CLUSTER: return (const void*)KERNEL<gsrb::V_CLUSTER>;         \
      case gsrb::V_DSMEM: return (const void*)KERNEL<gsrb::V_DSMEM>;             \
      case gsrb::V_SOFT2: return (const void*)KERNEL<gsrb::V_SOFT2>;             \
      case gsrb::V_FLAT: return (const void*)KERNEL<gsrb::V_FLAT>;               \
      case gsrb::V_TREE: return (const void*)KERNEL<gsrb::V_TREE>;               \
      case gsrb::V_CCG: return (const void*)KERNEL<gsrb::V_CCG>;                 \
      case gsrb::V_CLUSTER_RED: return (const void*)KERNEL<gsrb::V_CLUSTER_RED>; \
      case gsrb::V_FLIP: return (const void*)KERNEL<gsrb::V_FLIP>;               \
      case gsrb::V_FANOUT: return (const void*)KERNEL<gsrb::V_FANOUT>;           \
      case gsrb::V_HIER: return (const void*)KERNEL<gsrb::V_HIER>;               \
      default: return nullptr;                                                  \
    }                                                                           \
  }

const void* bfs_fn(int v) { return GSRB_GRAPH_FN(bfs_kernel)(v); }
const void* sssp_fn(int v) { return GSRB_GRAPH_FN(sssp_kernel)(v); }
const void* pr_fn(int v) { return GSRB_GRAPH_FN(pagerank_kernel)(v); }
const void* prr_fn(int v) { return GSRB_GRAPH_FN(pr_residual_kernel)(v); }
template <int KIND>
const void* batch_fn_k(int v) {
  switch (v) {  // variants without hardware cluster barriers (teams may be single CTAs)
    case gsrb::V_SOFT2: return (const void*)batch_kernel<gsrb::V_SOFT2, KIND>;
    case gsrb::V_FLAT: return (const void*)batch_kernel<gsrb::V_FLAT, KIND>;
    case gsrb::V_TREE: return (const void*)batch_kernel<gsrb::V_TREE, KIND>;
    case gsrb::V_FLIP: return (const void*)batch_kernel<gsrb::V_FLIP, KIND>;
    case gsrb::V_FANOUT: return (const void*)batch_kernel<gsrb::V_FANOUT, KIND>;
    case gsrb::V_HIER: return (const void*)batch_kernel<gsrb::V_HIER, KIND>;
    default: return nullptr;
  }
}
const void* batch_fn(int v, int kind) { return kind == 0 ? batch_fn_k<0>(v) : batch_fn_k<1>(v); }

}  // namespace

const void* gsrb_graph_kernel_for(int variant) { return bfs_fn(variant); }

// ------------------------------------------------------------ host side ----
struct gsrb_graph {
  gsrb_ctx* ctx = nullptr;
  uint32_t n = 0;
  uint32_t m = 0;
  bool owns = false;
  uint32_t* row = nullptr;
  uint32_t* dst = nullptr;
  int32_t* w = nullptr;
  // scratch
  uint32_t* q[2] = {};
  uint32_t* hq[2] = {};
  uint32_t* far[2] = {};
  uint32_t* mark = nullptr;
  uint32_t* fmark = nullptr;
  LevelCounters* cnt = nullptr;
  unsigned long long* fcnt = nullptr;
  uint32_t* flags = nullptr;  // [0] overflow, [1] a cluster's wait ran out, [4..8) out, [8..16) BFS single-CTA state, edges at byte 64, PageRank tickets at byte 96
  LevelTrace* trace = nullptr;
  uint32_t trace_cap = 0;
  float* contrib[2] = {};
  uint32_t* hubs = nullptr;       // PageRank hubs (degree > kPrHubDegree)
  uint32_t nhubs = 0;
  uint32_t* hub_c0 = nullptr;     // [nhubs + 1] first chunk of each hub
  uint32_t* chunk_hub = nullptr;  // [nchunks] hub of each chunk
  uint32_t nchunks = 0;
  double* hub_part = nullptr;     // [nchunks] chunk sums
  uint32_t* hub_done = nullptr;   // [nhubs] chunk counters
  MLPWeights* mlp = nullptr;
  bool mlp_set = false;
  MLPWeights mlp_host{};        // host copy of the policy weights (the launch choice runs on the host)
  gsrb_cfg_t launch[2]{};       // the two launch configurations head 3 chooses between
  bool launch_set = false;
  uint32_t* lb_pre = nullptr;   // [n] load-balanced BFS: edge offset of each queue entry
  uint32_t* lb_own = nullptr;   // [m / kLbChunk + 2] queue entry owning each chunk's first edge
  uint32_t* lb_part = nullptr;  // [kLbMaxCtas] per-CTA edge totals
  bool symmetric = false;       // every edge (u, v) has its reverse (v, u)
  // graph statistics of the SSSP policy's features (taken when the graph is created)
  uint32_t max_degree = 0;
  std::vector<uint32_t> h_row;  // host copy of row_start (source degrees for the host-side policy heads)
  int32_t w_min = 0, w_max = 0;
  double w_mean = 0.0;
  MLPWeights sssp_host{};       // SSSP policy weights (evaluated on the host, once per traversal)
  bool sssp_set = false;
  int32_t last_delta = 0;       // bucket width of the last SSSP launched on this graph (0: none)
};

namespace {

template <class T>
cudaError_t dalloc(T** p, size_t count) {
  return cudaMalloc((void**)p, sizeof(T) * (count ? count : 1));
}

DevCSR dev_csr(const gsrb_graph* G) {
  DevCSR d;
  d.n = G->n;
  d.m = G->m;
  d.row = G->row;
  d.dst = G->dst;
  d.w = G->w;
  return d;
}

// splitmix64's output mix (Steele, Lea, Flood, OOPSLA'14), as a hash of an edge.
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// Symmetry test of a CSR: sums (mod 2^64) of two hashes of every edge (u, v)
// and of its reverse (v, u).  The edge multiset equals its reverse exactly
// when the graph is symmetric; then both pairs of sums agree, and otherwise
// they differ except with probability about 2^-128.  One warp per row.
__global__ void __launch_bounds__(256) edge_hash_kernel(DevCSR g, unsigned long long* sums) {
  const uint32_t lane = lane_id();
  const uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  unsigned long long f1 = 0, r1 = 0, f2 = 0, r2 = 0;
  for (uint32_t u = w0; u < g.n; u += nw) {
    const uint32_t b = g.row[u], e = g.row[u + 1];
    for (uint32_t j = b + lane; j < e; j += 32) {
      const uint32_t v = g.dst[j];
      const unsigned long long fw = ((unsigned long long)u << 32) | v, rv = ((unsigned long long)v << 32) | u;
      f1 += mix64(fw);
      r1 += mix64(rv);
      f2 += mix64(fw ^ 0x5851f42d4c957f2dull);
      r2 += mix64(rv ^ 0x5851f42d4c957f2dull);
    }
  }
  f1 = warp_sum_u64(f1);
  r1 = warp_sum_u64(r1);
  f2 = warp_sum_u64(f2);
  r2 = warp_sum_u64(r2);
  if (lane == 0) {
    atomicAdd(sums + 0, f1);
    atomicAdd(sums + 1, r1);
    atomicAdd(sums + 2, f2);
    atomicAdd(sums + 3, r2);
  }
}

// Edge-weight statistics: minimum, maximum (as order-preserving unsigned keys)
// and the int64 sum.  Grid-stride over the weights.
__global__ void __launch_bounds__(256) edge_weight_stats_kernel(const int32_t* __restrict__ w, uint64_t m,
                                                                unsigned long long* out) {
  uint32_t lo = 0xffffffffu, hi = 0;
  long long sum = 0;
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < m; j += (uint64_t)gridDim.x * blockDim.x) {
    const int32_t x = w[j];
    const uint32_t key = (uint32_t)x ^ 0x80000000u;  // signed order as unsigned order
    lo = min(lo, key);
    hi = max(hi, key);
    sum += x;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if (lane_id() == 0) {
    atomicMin(out + 0, (unsigned long long)lo);
    atomicMax(out + 1, (unsigned long long)hi);
    atomicAdd(out + 2, (unsigned long long)sum);
  }
}

// The gather floor of a pull pass: every edge's x/deg[dst[j]] gathered
// edge-parallel (grid-stride, eight loads in flight per thread, no per-vertex
// bookkeeping), through L1 (L1 != 0) or L2 only.  Measures what the random
// gathers alone cost on this graph (gsrb_probe_gather).
template <int L1>
__global__ void __launch_bounds__(512) gather_probe_kernel(const uint32_t* __restrict__ dst, uint64_t m,
                                                           const float* cin, double* sink) {
  double s = 0.0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  for (; j + 7 * stride < m; j += 8 * stride) {
    uint32_t d[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) d[k] = __ldg(dst + j + k * stride);
    float c[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k] = L1 ? __ldca(cin + d[k]) : __ldcg(cin + d[k]);
#pragma unroll
    for (int k = 0; k < 8; ++k) s += (double)c[k];
  }
  for (; j < m; j += stride) s += (double)(L1 ? __ldca(cin + dst[j]) : __ldcg(cin + dst[j]));
  if (s == -1.0) *sink = s;  // keeps the loads; never true for non-negative inputs
}

gsrb_status_t graph_scratch(gsrb_graph* G) {
  const size_t n = G->n;
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 2 && !e; ++k) {
    // 4n words: BFS keeps an edge range (two words) per queue slot, and up to
    // 2n slots (entries plus reservation holes)
    e = dalloc(&G->q[k], 4 * n);
    if (!e) e = dalloc(&G->hq[k], 2 * n);
    if (!e) e = dalloc(&G->far[k], n);
    if (!e) e = dalloc(&G->contrib[k], n);
  }
  if (!e) e = dalloc(&G->mark, n);
  if (!e) e = dalloc(&G->fmark, n);
  if (!e) e = dalloc(&G->cnt, 3);
  if (!e) e = dalloc(&G->fcnt, 2);
  if (!e) e = dalloc(&G->flags, 32);
  G->trace_cap = 1u << 16;
  if (!e) e = dalloc(&G->trace, G->trace_cap);
  if (!e) e = dalloc(&G->mlp, 1);
  if (!e) e = cudaMemset(G->mlp, 0, sizeof(MLPWeights));
  if (!e) e = dalloc(&G->lb_pre, 2 * n);  // one per queue slot (holes included)
  if (!e) e = dalloc(&G->lb_own, (size_t)G->m / kLbChunk + 2);
  if (!e) e = dalloc(&G->lb_part, kLbMaxCtas);
  // PageRank hub chunks (degree > kPrHubDegree), built on the host from row_start
  if (!e) {
    std::vector<uint32_t>& hrow = G->h_row;
    hrow.assign(n + 1, 0u);
    e = cudaMemcpy(hrow.data(), G->row, sizeof(uint32_t) * (n + 1), cudaMemcpyDeviceToHost);
    std::vector<uint32_t> hl, c0, ch;
    for (size_t v = 0; !e && v < n; ++v) {
      const uint32_t d = hrow[v + 1] - hrow[v];
      if (d > G->max_degree) G->max_degree = d;
      if (d <= kPrHubDegree) continue;
      c0.push_back((uint32_t)ch.size());
      for (uint32_t j = 0; j < d; j += kPrChunk) ch.push_back((uint32_t)hl.size());
      hl.push_back((uint32_t)v);
    }
    c0.push_back((uint32_t)ch.size());
    G->nhubs = (uint32_t)hl.size();
    G->nchunks = (uint32_t)ch.size();
    if (!e) e = dalloc(&G->hubs, hl.size());
    if (!e) e = dalloc(&G->hub_c0, c0.size());
    if (!e) e = dalloc(&G->chunk_hub, ch.size());
    if (!e) e = dalloc(&G->hub_part, ch.size());
    if (!e) e = dalloc(&G->hub_done, hl.size());
    if (!e && !hl.empty()) e = cudaMemcpy(G->hubs, hl.data(), sizeof(uint32_t) * hl.size(), cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(G->hub_c0, c0.data(), sizeof(uint32_t) * c0.size(), cudaMemcpyHostToDevice);
    if (!e && !ch.empty())
      e = cudaMemcpy(G->chunk_hub, ch.data(), sizeof(uint32_t) * ch.size(), cudaMemcpyHostToDevice);
  }
  // symmetric? (pull directions and pull PageRank read a row as in-edges)
  if (!e) {
    unsigned long long* sums = reinterpret_cast<unsigned long long*>(G->lb_part);
    e = cudaMemset(sums, 0, 4 * sizeof(unsigned long long));
    if (!e) {
      edge_hash_kernel<<<1184, 256>>>(dev_csr(G), sums);
      e = cudaGetLastError();
    }
    unsigned long long h[4] = {0, 0, 0, 0};
    if (!e) e = cudaMemcpy(h, sums, sizeof h, cudaMemcpyDeviceToHost);
    G->symmetric = h[0] == h[1] && h[2] == h[3];
  }
  // edge weights: minimum, maximum, mean
  if (!e && G->w && G->m) {
    unsigned long long* st = reinterpret_cast<unsigned long long*>(G->lb_part);
    const unsigned long long init[3] = {0xffffffffull, 0ull, 0ull};
    e = cudaMemcpy(st, init, sizeof init, cudaMemcpyHostToDevice);
    if (!e) {
      edge_weight_stats_kernel<<<1184, 256>>>(G->w, G->m, st);
      e = cudaGetLastError();
    }
    unsigned long long h[3] = {0, 0, 0};
    if (!e) e = cudaMemcpy(h, st, sizeof h, cudaMemcpyDeviceToHost);
    G->w_min = (int32_t)((uint32_t)h[0] ^ 0x80000000u);
    G->w_max = (int32_t)((uint32_t)h[1] ^ 0x80000000u);
    G->w_mean = (double)(long long)h[2] / (double)G->m;
  }
  if (!e) e = cudaDeviceSynchronize();
  if (e) return cuda_err(e, "graph scratch");
  return GSRB_OK;
}

void graph_free(gsrb_graph* G) {
  if (G->owns) {
    cudaFree(G->row);
    cudaFree(G->dst);
    cudaFree(G->w);
  }
  for (int k = 0; k < 2; ++k) {
    cudaFree(G->q[k]);
    cudaFree(G->hq[k]);
    cudaFree(G->far[k]);
    cudaFree(G->contrib[k]);
  }
  cudaFree(G->mark);
  cudaFree(G->fmark);
  cudaFree(G->cnt);
  cudaFree(G->fcnt);
  cudaFree(G->flags);
  cudaFree(G->trace);
  cudaFree(G->hubs);
  cudaFree(G->hub_c0);
  cudaFree(G->chunk_hub);
  cudaFree(G->hub_part);
  cudaFree(G->hub_done);
  cudaFree(G->mlp);
  cudaFree(G->lb_pre);
  cudaFree(G->lb_own);
  cudaFree(G->lb_part);
}


gsrb_cfg_t graph_cfg(gsrb_ctx* ctx, const gsrb_cfg_t* in) {
  gsrb_cfg_t c = resolve_cfg(ctx, in);
  if (!in) {
    c.ctas_per_sm = 2;
    c.threads = 512;
    c.cluster = 2;
  }
  return c;
}

PullArgs pull_args(const gsrb_graph* G, const gsrb_cfg_t& c) {
  PullArgs a;
  a.hubs = G->hubs;
  a.hub_c0 = G->hub_c0;
  a.chunk_hub = G->chunk_hub;
  a.nhubs = G->nhubs;
  a.nchunks = G->nchunks;
  a.part = G->hub_part;
  a.hub_done = G->hub_done;
  a.ticket = reinterpret_cast<unsigned long long*>(G->flags + 24);
  a.gather_l1 = c.form == GSRB_FORM_L2 ? 0 : 1;
  return a;
}

// Dynamic shared memory of a launch: the CTAs' stages where the grid is co-resident
// with them, else none (8 x 128 threads per SM fit without; the kernel then
// appends through the warps' reservations).
template <class S>
size_t with_stage(gsrb_ctx* ctx, const void* fn, int grid, const gsrb_cfg_t& c, int cluster) {
  int cap = 0;
  return coresident_ctas(ctx, fn, c.threads, sizeof(S), cluster < 1 ? 1 : cluster, &cap) == GSRB_OK && cap >= grid
             ? sizeof(S)
             : 0;
}

// CTAs of the cluster that runs thin steps: 0 where it cannot be placed (the grid
// then runs every step).
int cluster_ctas(gsrb_ctx* ctx, const void* fn, size_t smem) {
  int cap = 0;
  const int k = (int)kClCtas;
  return coresident_ctas(ctx, fn, (int)kClThreads, smem, k, &cap) == GSRB_OK && cap >= k ? k : 0;
}

// Statistics from a copy of the graph's 32 status words.
gsrb_status_t stats_of(const gsrb_graph* G, const uint32_t* h, gsrb_traversal_stats_t* st, float ms) {
  if (st) {
    unsigned long long edges = 0;
    memcpy(&edges, h + 16, sizeof(edges));
    st->levels = h[4];
    st->aux = h[5];
    st->decisions = h[6];
    st->edges = edges;
    st->kernel_ms = ms;
    st->trace_records = h[4] < G->trace_cap ? h[4] : G->trace_cap;
    st->launch = 0;
    st->delta = G->last_delta;
  }
  if (h[0]) return GSRB_ERR_OVERFLOW;
  if (h[7] || h[1]) return GSRB_ERR_TIMEOUT;
  return GSRB_OK;
}

// Enqueues the copy of the status words into the pinned block (slot k of kSlots,
// 32 words each) of the context that runs the traversal, on its stream; valid
// after that stream has been waited for.  (A graph may be used from another
// context than the one it was made on.)
cudaError_t copy_status(gsrb_ctx* ctx, const gsrb_graph* G, int k) {
  return cudaMemcpyAsync(ctx->h_status + 32 * k, G->flags, 128, cudaMemcpyDeviceToHost, ctx->stream);
}

// End of a traversal (the context's events 62 and 63 around it): one wait for the stream.
gsrb_status_t finish_stats(gsrb_ctx* ctx, const gsrb_graph* G, gsrb_traversal_stats_t* st) {
  GSRB_CUDA(copy_status(ctx, G, 0));
  GSRB_CUDA(cudaStreamSynchronize(ctx->stream));
  float ms = 0;
  GSRB_CUDA(cudaEventElapsedTime(&ms, ctx->events[62], ctx->events[63]));
  return stats_of(G, ctx->h_status, st, ms);
}

}  // namespace

extern "C" {

gsrb_status_t gsrb_graph_upload(gsrb_ctx_t ctx, const gsrb_host_csr_t* h, gsrb_graph_t* out) {
  if (!ctx || !h || !out || !h->row_start || (h->nedges && !h->edge_dst) || h->nedges >= (1ull << 32))
    return GSRB_ERR_ARG;
  gsrb_graph* G = new gsrb_graph();
  G->ctx = ctx;
  G->n = h->nnodes;
  G->m = (uint32_t)h->nedges;
  G->owns = true;
  cudaError_t e = dalloc(&G->row, (size_t)G->n + 1);
  if (!e) e = dalloc(&G->dst, G->m);
  if (!e) e = dalloc(&G->w, G->m);
  if (!e) e = cudaMemcpy(G->row, h->row_start, sizeof(uint32_t) * ((size_t)G->n + 1), cudaMemcpyHostToDevice);
  if (!e && G->m) e = cudaMemcpy(G->dst, h->edge_dst, sizeof(uint32_t) * G->m, cudaMemcpyHostToDevice);
  if (!e && G->m && h->edge_data) e = cudaMemcpy(G->w, h->edge_data, sizeof(int32_t) * G->m, cudaMemcpyHostToDevice);
  gsrb_status_t st = e ? cuda_err(e, "graph upload") : graph_scratch(G);
  if (st) {
    graph_free(G);
    delete G;
    return st;
  }
  *out = G;
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_wrap(gsrb_ctx_t ctx, uint32_t n, uint64_t m, const uint32_t* d_row, const uint32_t* d_dst,
                              const int32_t* d_w, gsrb_graph_t* out) {
  if (!ctx || !out || !d_row || (m && !d_dst) || m >= (1ull << 32)) return GSRB_ERR_ARG;
  gsrb_graph* G = new gsrb_graph();
  G->ctx = ctx;
  G->n = n;
  G->m = (uint32_t)m;
  G->owns = false;
  G->row = const_cast<uint32_t*>(d_row);
  G->dst = const_cast<uint32_t*>(d_dst);
  G->w = const_cast<int32_t*>(d_w);
  gsrb_status_t st = graph_scratch(G);
  if (st) {
    graph_free(G);
    delete G;
    return st;
  }
  *out = G;
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_free(gsrb_graph_t G) {
  if (!G) return GSRB_ERR_ARG;
  cudaStreamSynchronize(G->ctx->stream);
  graph_free(G);
  delete G;
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_info(gsrb_graph_t G, uint32_t* n, uint64_t* m, uint32_t* nhubs) {
  if (!G) return GSRB_ERR_ARG;
  if (n) *n = G->n;
  if (m) *m = G->m;
  if (nhubs) *nhubs = G->nhubs;
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_is_symmetric(gsrb_graph_t G, int32_t* symmetric) {
  if (!G || !symmetric) return GSRB_ERR_ARG;
  *symmetric = G->symmetric ? 1 : 0;
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_set_policy(gsrb_graph_t G, const float* h_weights, size_t count) {
  if (!G || !h_weights || count != sizeof(MLPWeights) / sizeof(float)) return GSRB_ERR_ARG;
  GSRB_CUDA(cudaMemcpy(G->mlp, h_weights, sizeof(MLPWeights), cudaMemcpyHostToDevice));
  memcpy(&G->mlp_host, h_weights, sizeof(MLPWeights));
  G->mlp_set = true;
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_set_launch_choices(gsrb_graph_t G, const gsrb_cfg_t* cfg0, const gsrb_cfg_t* cfg1) {
  if (!G) return GSRB_ERR_ARG;
  if (!cfg0 && !cfg1) {
    G->launch_set = false;
    return GSRB_OK;
  }
  if (!cfg0 || !cfg1) return GSRB_ERR_ARG;
  const gsrb_cfg_t* in[2] = {cfg0, cfg1};
  for (int k = 0; k < 2; ++k) {
    const gsrb_cfg_t c = graph_cfg(G->ctx, in[k]);
    if (!bfs_fn(c.variant)) return GSRB_ERR_UNSUPPORTED;
    const int grid = grid_of(G->ctx, c);
    if (grid <= 0 || grid % c.cluster || c.threads % 32 || c.threads > kGraphMaxThreads) return GSRB_ERR_ARG;
    G->launch[k] = c;
  }
  G->launch_set = true;
  return GSRB_OK;
}

namespace {

// Host forward pass of the policy network (the layout of MLPWeights; ReLU on
// the two hidden layers).  Used for the per-traversal launch choice, which is
// taken before the launch.
void mlp_forward_host(const MLPWeights& W, const float* x, float* out) {
  float h1[kHid], h2[kHid];
  for (int j = 0; j < kHid; ++j) {
    float z = W.b1[j];
    for (int i = 0; i < kFeat; ++i) z += W.w1[j][i] * x[i];
    h1[j] = z > 0.f ? z : 0.f;
  }
  for (int j = 0; j < kHid; ++j) {
    float z = W.b2[j];
    for (int k = 0; k < kHid; ++k) z += W.w2[j][k] * h1[k];
    h2[j] = z > 0.f ? z : 0.f;
  }
  for (int o = 0; o < kOut; ++o) {
    float z = W.b3[o];
    for (int k = 0; k < kHid; ++k) z += W.w3[o][k] * h2[k];
    out[o] = z;
  }
}

}  // namespace

gsrb_status_t gsrb_graph_policy_launch(gsrb_graph_t G, uint32_t src, int32_t* choice, float* score) {
  if (!G || !choice || src >= G->n) return GSRB_ERR_ARG;
  if (!G->mlp_set) return GSRB_ERR_STATE;
  // the first level's features, as the traversal computes them: the frontier
  // is the source, every other vertex and edge is unvisited
  const uint32_t dsrc = G->h_row[src + 1] - G->h_row[src];
  float feat[kFeat], out[kOut];
  level_features(feat, G->n, G->m, 1, 1, dsrc, G->n - 1, (unsigned long long)G->m - dsrc, 1, DIR_PUSH);
  mlp_forward_host(G->mlp_host, feat, out);
  *choice = out[3] > 0.f ? 1 : 0;
  if (score) *score = out[3];
  return GSRB_OK;
}

// The SSSP policy's 12 features of a traversal from a source: graph size,
// degree distribution, edge-weight range and the source's degree (log-scaled).
static void sssp_features_of(uint32_t n, uint64_t m, uint32_t max_degree, uint32_t src_degree, double w_mean,
                             int32_t w_min, int32_t w_max, int32_t symmetric, float* f) {
  const double nn = n ? (double)n : 1.0;
  const double md = (double)m / nn;
  f[0] = (float)log2(nn);
  f[1] = (float)log2(1.0 + (double)m);
  f[2] = (float)log2(1.0 + md);
  f[3] = (float)log2(1.0 + (double)max_degree);
  f[4] = (float)log2(1.0 + (double)src_degree);
  f[5] = (float)log2(1.0 + (w_mean > 0 ? w_mean : 0.0));
  f[6] = (float)log2(1.0 + (w_max > 0 ? (double)w_max : 0.0));
  f[7] = (float)log2(1.0 + (w_min > 0 ? (double)w_min : 0.0));
  f[8] = symmetric ? 1.f : 0.f;
  f[9] = f[3] - f[2];            // degree skew
  f[10] = f[6] - f[5];           // weight spread
  f[11] = f[0] - 2.f * f[2];     // size against mean degree (high for meshes)
}

void gsrb_sssp_features(uint32_t n, uint64_t m, uint32_t max_degree, uint32_t src_degree, double w_mean,
                        int32_t w_min, int32_t w_max, int32_t symmetric, float* h_out12) {
  sssp_features_of(n, m, max_degree, src_degree, w_mean, w_min, w_max, symmetric, h_out12);
}

gsrb_status_t gsrb_graph_sssp_features(gsrb_graph_t G, uint32_t src, float* h_out12) {
  if (!G || !h_out12 || src >= G->n) return GSRB_ERR_ARG;
  sssp_features_of(G->n, G->m, G->max_degree, G->h_row[src + 1] - G->h_row[src], G->w_mean, G->w_min, G->w_max,
                   G->symmetric ? 1 : 0, h_out12);
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_set_sssp_policy(gsrb_graph_t G, const float* h_weights, size_t count) {
  if (!G) return GSRB_ERR_ARG;
  if (!h_weights) {
    G->sssp_set = false;
    return GSRB_OK;
  }
  if (count != sizeof(MLPWeights) / sizeof(float)) return GSRB_ERR_ARG;
  memcpy(&G->sssp_host, h_weights, sizeof(MLPWeights));
  G->sssp_set = true;
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_sssp_plan(gsrb_graph_t G, uint32_t src, int32_t* delta, int32_t* choice, float* scores) {
  if (!G || src >= G->n) return GSRB_ERR_ARG;
  if (!G->sssp_set) return GSRB_ERR_STATE;
  float feat[kFeat], out[kOut];
  gsrb_status_t st = gsrb_graph_sssp_features(G, src, feat);
  if (st) return st;
  mlp_forward_host(G->sssp_host, feat, out);
  // head 2: log2(bucket width / mean edge weight)
  const double wm = G->w_mean >= 1.0 ? G->w_mean : 1.0;
  double d = exp2((double)(out[2] < -30.f ? -30.f : (out[2] > 30.f ? 30.f : out[2]))) * wm;
  if (!(d >= 1.0)) d = 1.0;
  if (d > 1073741824.0) d = 1073741824.0;
  if (delta) *delta = (int32_t)llround(d);
  if (choice) *choice = out[3] > 0.f ? 1 : 0;
  if (scores) {
    scores[0] = out[2];
    scores[1] = out[3];
  }
  return GSRB_OK;
}

gsrb_status_t gsrb_probe_gather(gsrb_ctx_t ctx, gsrb_graph_t G, int32_t l1, float* ms) {
  if (!ctx || !G || !ms) return GSRB_ERR_ARG;
  if (!G->m) {
    *ms = 0.f;
    return GSRB_OK;
  }
  std::lock_guard<std::mutex> g(ctx->mu);
  // x/deg of the first PageRank buffer (any FP32 values do; zeroed here)
  GSRB_CUDA(cudaMemsetAsync(G->contrib[0], 0, sizeof(float) * G->n, ctx->stream));
  double* sink = reinterpret_cast<double*>((char*)G->flags + 64);
  const dim3 grid((unsigned)ctx->num_sms * 2u), block(512);
  auto launch = [&]() -> cudaError_t {
    if (l1) gather_probe_kernel<1><<<grid, block, 0, ctx->stream>>>(G->dst, G->m, G->contrib[0], sink);
    else gather_probe_kernel<0><<<grid, block, 0, ctx->stream>>>(G->dst, G->m, G->contrib[0], sink);
    return cudaGetLastError();
  };
  if (!ctx->events[62]) GSRB_CUDA(cudaEventCreate(&ctx->events[62]));
  if (!ctx->events[63]) GSRB_CUDA(cudaEventCreate(&ctx->events[63]));
  for (int i = 0; i < 3; ++i) GSRB_CUDA(launch());
  constexpr int kReps = 10;
  GSRB_CUDA(cudaEventRecord(ctx->events[62], ctx->stream));
  for (int i = 0; i < kReps; ++i) GSRB_CUDA(launch());
  GSRB_CUDA(cudaEventRecord(ctx->events[63], ctx->stream));
  GSRB_CUDA(cudaEventSynchronize(ctx->events[63]));
  float t = 0;
  GSRB_CUDA(cudaEventElapsedTime(&t, ctx->events[62], ctx->events[63]));
  *ms = t / kReps;
  gsrbrt::g_launches.fetch_add(3 + kReps, std::memory_order_relaxed);
  return GSRB_OK;
}

gsrb_status_t gsrb_graph_trace(gsrb_graph_t G, void* h_out, uint32_t max_records, uint32_t* records) {
  if (!G || !h_out) return GSRB_ERR_ARG;
  uint32_t h[32];
  GSRB_CUDA(cudaStreamSynchronize(G->ctx->stream));
  GSRB_CUDA(cudaMemcpy(h, G->flags, sizeof(h), cudaMemcpyDeviceToHost));
  uint32_t r = h[4] < G->trace_cap ? h[4] : G->trace_cap;
  if (r > max_records) r = max_records;
  if (r) GSRB_CUDA(cudaMemcpy(h_out, G->trace, sizeof(LevelTrace) * r, cudaMemcpyDeviceToHost));
  if (records) *records = r;
  return GSRB_OK;
}

gsrb_status_t gsrb_bfs(gsrb_ctx_t ctx, gsrb_graph_t G, uint32_t src, int32_t* d_level, int32_t mode,
                       const gsrb_cfg_t* cfgin, gsrb_traversal_stats_t* stats) {
  const bool lb = (mode & GSRB_BFS_FLAG_LB) != 0;
  mode &= ~GSRB_BFS_FLAG_LB;
  if (!ctx || !G || !d_level || src >= G->n || mode < 0 || mode > GSRB_BFS_TOPO) return GSRB_ERR_ARG;
  if (mode == GSRB_BFS_LEARNED && !G->mlp_set) return GSRB_ERR_STATE;
  if (mode == GSRB_BFS_PULL && !G->symmetric) return GSRB_ERR_UNSUPPORTED;
  gsrb_cfg_t c = graph_cfg(ctx, cfgin);
  uint32_t launch = 0;
  if (mode == GSRB_BFS_LEARNED && !cfgin && G->launch_set) {
    // the policy's head 3 picks the launch configuration (barrier variant and
    // CTA shape) from the first level's features
    int32_t k = 0;
    gsrb_status_t st = gsrb_graph_policy_launch(G, src, &k, nullptr);
    if (st) return st;
    c = G->launch[k];
    launch = 1u + (uint32_t)k;
  }
  const void* fn = bfs_fn(c.variant);
  if (!fn) return GSRB_ERR_UNSUPPORTED;
  const int grid = grid_of(ctx, c);
  if (grid % c.cluster || c.threads % 32 || c.threads > kGraphMaxThreads) return GSRB_ERR_ARG;
  if (lb && grid > (int)kLbMaxCtas) return GSRB_ERR_ARG;
  BfsArgs a;
  a.symmetric = G->symmetric;
  a.lb = lb;
  a.lb_pre = G->lb_pre;
  a.lb_own = G->lb_own;
  a.lb_part = G->lb_part;
  a.g = dev_csr(G);
  a.src = src;
  a.level = d_level;
  a.q[0] = G->q[0];
  a.q[1] = G->q[1];
  a.hq[0] = G->hq[0];
  a.hq[1] = G->hq[1];
  a.cnt = G->cnt;
  a.overflow = G->flags;
  a.trace = G->trace;
  a.trace_cap = G->trace_cap;
  a.mlp = G->mlp;
  a.mode = mode;
  a.alpha = 15.f;
  a.beta = 18.f;
  a.out = G->flags + 4;
  a.out_edges = (unsigned long long*)((char*)G->flags + 64);
  a.solo = G->flags + 8;
  a.phase = G->flags + 20;
  G->last_delta = 0;
  std::lock_guard<std::mutex> g(ctx->mu);
  gsrb::GridBarrier gb = make_barrier(ctx, c, 0, (uint32_t)grid, 0, 0);
  void* args[] = {&gb, &a};
  if (!ctx->events[62]) GSRB_CUDA(cudaEventCreate(&ctx->events[62]));
  if (!ctx->events[63]) GSRB_CUDA(cudaEventCreate(&ctx->events[63]));
  // The schedules that choose per level run thin levels on one cluster, unless
  // the caller chose the launch: then every level runs under that.
  const int ncl = !cfgin && (mode == GSRB_BFS_HEURISTIC || mode == GSRB_BFS_LEARNED)
                      ? cluster_ctas(ctx, (const void*)bfs_cluster_kernel, sizeof(BfsClShared))
                      : 0;
  a.staged = ncl > 0;
  // refused before anything is enqueued that writes the caller's array
  gsrb_status_t st = require_coresident(ctx, fn, grid, c.threads, 0, c.cluster);
  if (st) return st;
  const size_t smem = with_stage<BfsStage>(ctx, fn, grid, c, c.cluster);
  a.stage = smem != 0;
  GSRB_CUDA(cudaEventRecord(ctx->events[62], ctx->stream));
  if (!a.staged) {
    GSRB_CUDA(cudaMemsetAsync(G->flags, 0, 128, ctx->stream));
    st = launch_persistent(ctx, fn, grid, c.threads, smem, c.cluster, coop_of(c), args);
    if (st) return st;
    GSRB_CUDA(cudaEventRecord(ctx->events[63], ctx->stream));
  } else {
    uint32_t* flags = G->flags;
    // mean degree < kThinDegree and a CSR that leaves L2 room for the levels:
    // bring it in
    const bool thin = G->m / kThinDegree < G->n;
    uint32_t prefetch = thin && ((uint64_t)G->m + G->n) * 4 <= (uint64_t)ctx->l2_bytes / 4 * 3 ? 1u : 0u;
    void* iargs[] = {&a, &flags, &prefetch};
    st = launch_plain(ctx, (const void*)bfs_init_kernel, dim3(ctx->num_sms * 2), dim3(512), 0, iargs);
    if (st) return st;
    unsigned long long timeout_ns = gb.timeout_ns;
    void* cargs[] = {&a, &timeout_ns};
    auto cluster = [&] {
      return launch_persistent(ctx, (const void*)bfs_cluster_kernel, ncl, kClThreads, sizeof(BfsClShared), ncl, 0,
                               cargs);
    };
    auto whole = [&] { return launch_persistent(ctx, fn, grid, c.threads, smem, c.cluster, coop_of(c), args); };
    // A kernel whose turn it is not returns at once, so the usual order is
    // queued without a look at the device: the cluster for the whole of a thin
    // graph; cluster, grid and the thin last levels on the cluster again
    // otherwise (no cluster first for a hub as the source, or
    // when the policy decides the first level).
    const bool cluster_first = mode != GSRB_BFS_LEARNED && G->h_row[src + 1] - G->h_row[src] <= kBigDegree;
    if (cluster_first) st = cluster();
    for (uint32_t turn = thin && cluster_first ? 0u : 1u;; ++turn) {
      if (!st && turn) st = whole();
      if (!st && turn) st = cluster();
      if (st) {
        cudaStreamSynchronize(ctx->stream);  // nothing writes the caller's array after the return
        return st;
      }
      GSRB_CUDA(cudaEventRecord(ctx->events[63], ctx->stream));
      GSRB_CUDA(copy_status(ctx, G, 0));
      GSRB_CUDA(cudaStreamSynchronize(ctx->stream));
      const uint32_t phase = ctx->h_status[a.phase - G->flags];
      if (phase == PHASE_DONE) break;
      // (every turn runs at least one level; n levels are the most there are)
      if ((phase != PHASE_GRID && phase != PHASE_CLUSTER) || turn > G->n) return GSRB_ERR_STATE;
    }
  }
  if (a.staged) {  // the status is here
    float ms = 0;
    GSRB_CUDA(cudaEventElapsedTime(&ms, ctx->events[62], ctx->events[63]));
    st = stats_of(G, ctx->h_status, stats, ms);
  } else {
    st = finish_stats(ctx, G, stats);
  }
  if (stats) stats->launch = launch;
  return st;
}

gsrb_status_t gsrb_sssp(gsrb_ctx_t ctx, gsrb_graph_t G, uint32_t src, int32_t* d_dist, int32_t delta,
                        const gsrb_cfg_t* cfgin, gsrb_traversal_stats_t* stats) {
  if (!ctx || !G || !d_dist || src >= G->n || delta < 0) return GSRB_ERR_ARG;
  gsrb_cfg_t c = graph_cfg(ctx, cfgin);
  uint32_t launch = 0;
  if (delta == GSRB_SSSP_DELTA_LEARNED) {
    // the SSSP policy picks the bucket width and, without a cfg, the launch
    // configuration; both change the schedule, never the distances
    int32_t k = 0;
    gsrb_status_t st = gsrb_graph_sssp_plan(G, src, &delta, &k, nullptr);
    if (st) return st;
    if (!cfgin && G->launch_set) {
      c = G->launch[k];
      launch = 1u + (uint32_t)k;
    }
  }
  const void* fn = sssp_fn(c.variant);
  if (!fn) return GSRB_ERR_UNSUPPORTED;
  const int grid = grid_of(ctx, c);
  if (grid % c.cluster || c.threads % 32) return GSRB_ERR_ARG;
  SsspArgs a;
  a.g = dev_csr(G);
  a.src = src;
  a.dist = d_dist;
  for (int k = 0; k < 2; ++k) {
    a.q[k] = G->q[k];
    a.hq[k] = G->hq[k];
    a.far[k] = G->far[k];
  }
  a.mark = G->mark;
  a.fmark = G->fmark;
  a.cnt = G->cnt;
  a.fcnt = G->fcnt;
  a.overflow = G->flags;
  a.trace = G->trace;
  a.trace_cap = G->trace_cap;
  a.delta = delta;
  a.out = G->flags + 4;
  a.out_edges = (unsigned long long*)((char*)G->flags + 64);
  a.phase = G->flags + 20;
  a.state = G->flags + 8;
  G->last_delta = delta;
  std::lock_guard<std::mutex> g(ctx->mu);
  // thin graphs (mean degree < kThinDegree) start on one cluster, unless the
  // caller chose the launch; the grid kernel queued behind it returns at once
  // unless the traversal outgrew the cluster
  const int ncl = !cfgin && G->m / kThinDegree < G->n
                      ? cluster_ctas(ctx, (const void*)sssp_cluster_kernel, sizeof(SsspClShared))
                      : 0;
  a.staged = ncl > 0;
  gsrb::GridBarrier gb = make_barrier(ctx, c, 0, (uint32_t)grid, 0, 0);
  void* args[] = {&gb, &a};
  if (!ctx->events[62]) GSRB_CUDA(cudaEventCreate(&ctx->events[62]));
  if (!ctx->events[63]) GSRB_CUDA(cudaEventCreate(&ctx->events[63]));
  // refused before anything is enqueued that writes the caller's array
  gsrb_status_t st = require_coresident(ctx, fn, grid, c.threads, 0, c.cluster);
  if (st) return st;
  const size_t smem = with_stage<IdStage>(ctx, fn, grid, c, c.cluster);
  a.stage = smem != 0;
  GSRB_CUDA(cudaEventRecord(ctx->events[62], ctx->stream));
  if (!a.staged) {
    GSRB_CUDA(cudaMemsetAsync(G->flags, 0, 128, ctx->stream));
  } else {
    uint32_t* flags = G->flags;
    uint32_t prefetch = ((uint64_t)G->m * 2 + G->n) * 4 <= (uint64_t)ctx->l2_bytes / 4 * 3 ? 1u : 0u;
    void* iargs[] = {&a, &flags, &prefetch};
    st = launch_plain(ctx, (const void*)sssp_init_kernel, dim3(ctx->num_sms * 2), dim3(512), 0, iargs);
    if (st) return st;
    unsigned long long timeout_ns = gb.timeout_ns;
    void* cargs[] = {&a, &timeout_ns};
    st = launch_persistent(ctx, (const void*)sssp_cluster_kernel, ncl, kClThreads, sizeof(SsspClShared), ncl, 0, cargs);
  }
  if (!st) st = launch_persistent(ctx, fn, grid, c.threads, smem, c.cluster, coop_of(c), args);
  if (st) {
    cudaStreamSynchronize(ctx->stream);  // nothing writes the caller's array after the return
    return st;
  }
  GSRB_CUDA(cudaEventRecord(ctx->events[63], ctx->stream));
  st = finish_stats(ctx, G, stats);
  if (stats) stats->launch = launch;
  return st;
}

gsrb_status_t gsrb_pagerank(gsrb_ctx_t ctx, gsrb_graph_t G, float alpha, int32_t iters, float* d_rank,
                            const gsrb_cfg_t* cfgin, gsrb_traversal_stats_t* stats) {
  if (!ctx || !G || !d_rank || iters < 0 || !(alpha >= 0.f && alpha < 1.f)) return GSRB_ERR_ARG;
  if (!G->symmetric) return GSRB_ERR_UNSUPPORTED;  // a row is summed as the vertex's in-edges
  gsrb_cfg_t c = graph_cfg(ctx, cfgin);
  const void* fn = pr_fn(c.variant);
  if (!fn) return GSRB_ERR_UNSUPPORTED;
  const int grid = grid_of(ctx, c);
  if (grid % c.cluster || c.threads % 32 || grid > 148 * 32) return GSRB_ERR_ARG;
  PrArgs a;
  a.g = dev_csr(G);
  a.alpha = alpha;
  a.iters = iters;
  a.rank = d_rank;
  a.contrib[0] = G->contrib[0];
  a.contrib[1] = G->contrib[1];
  a.pull = pull_args(G, c);
  a.out = G->flags + 4;
  G->last_delta = 0;
  std::lock_guard<std::mutex> g(ctx->mu);
  GSRB_CUDA(cudaMemsetAsync(G->flags, 0, 128, ctx->stream));
  if (G->nhubs) GSRB_CUDA(cudaMemsetAsync(G->hub_done, 0, sizeof(uint32_t) * G->nhubs, ctx->stream));
  gsrb::GridBarrier gb = make_barrier(ctx, c, 0, (uint32_t)grid, 0, 0);
  void* args[] = {&gb, &a};
  if (!ctx->events[62]) GSRB_CUDA(cudaEventCreate(&ctx->events[62]));
  if (!ctx->events[63]) GSRB_CUDA(cudaEventCreate(&ctx->events[63]));
  GSRB_CUDA(cudaEventRecord(ctx->events[62], ctx->stream));
  gsrb_status_t st = launch_persistent(ctx, fn, grid, c.threads, 0, c.cluster, coop_of(c), args);
  if (st) return st;
  GSRB_CUDA(cudaEventRecord(ctx->events[63], ctx->stream));
  return finish_stats(ctx, G, stats);
}

gsrb_status_t gsrb_pagerank_residual(gsrb_ctx_t ctx, gsrb_graph_t G, float alpha, float epsilon, int32_t max_iters,
                                     float* d_rank, const gsrb_cfg_t* cfgin, gsrb_traversal_stats_t* stats) {
  if (!ctx || !G || !d_rank || max_iters < 0 || !(alpha >= 0.f && alpha < 1.f) || !(epsilon > 0.f))
    return GSRB_ERR_ARG;
  gsrb_cfg_t c = graph_cfg(ctx, cfgin);
  const void* fn = prr_fn(c.variant);
  if (!fn) return GSRB_ERR_UNSUPPORTED;
  const int grid = grid_of(ctx, c);
  if (grid % c.cluster || c.threads % 32) return GSRB_ERR_ARG;
  PrrArgs a;
  a.g = dev_csr(G);
  a.alpha = alpha;
  a.eps = epsilon;
  a.max_iters = max_iters;
  a.p = d_rank;
  a.pull = pull_args(G, c);
  a.symmetric = G->symmetric;
  const size_t smem = with_stage<IdStage>(ctx, fn, grid, c, c.cluster);
  a.stage = smem != 0;
  a.r = G->contrib[0];
  a.hub_upd = G->contrib[1];
  a.share[0] = G->contrib[1];
  a.share[1] = reinterpret_cast<float*>(G->far[0]);  // (SSSP's, free here)
  a.mark = G->mark;
  a.q[0] = G->q[0];
  a.q[1] = G->q[1];
  a.hq[0] = G->hq[0];
  a.hq[1] = G->hq[1];
  a.cnt = G->cnt;
  a.overflow = G->flags;
  a.out = G->flags + 4;
  a.out_edges = (unsigned long long*)((char*)G->flags + 64);
  G->last_delta = 0;
  std::lock_guard<std::mutex> g(ctx->mu);
  GSRB_CUDA(cudaMemsetAsync(G->flags, 0, 128, ctx->stream));
  if (G->nhubs) GSRB_CUDA(cudaMemsetAsync(G->hub_done, 0, sizeof(uint32_t) * G->nhubs, ctx->stream));
  gsrb::GridBarrier gb = make_barrier(ctx, c, 0, (uint32_t)grid, 0, 0);
  void* args[] = {&gb, &a};
  if (!ctx->events[62]) GSRB_CUDA(cudaEventCreate(&ctx->events[62]));
  if (!ctx->events[63]) GSRB_CUDA(cudaEventCreate(&ctx->events[63]));
  GSRB_CUDA(cudaEventRecord(ctx->events[62], ctx->stream));
  gsrb_status_t st = launch_persistent(ctx, fn, grid, c.threads, smem, c.cluster, coop_of(c), args);
  if (st) return st;
  GSRB_CUDA(cudaEventRecord(ctx->events[63], ctx->stream));
  return finish_stats(ctx, G, stats);
}

}  // extern "C"

// ---------------------------------------------------------------- batches ----
struct gsrb_batch {
  gsrb_ctx* ctx = nullptr;
  std::vector<gsrb_graph*> graphs;
  gsrb_cfg_t cfg;
  int grid = 0;
  std::vector<uint32_t> first, count;
  BatchDesc* h_desc = nullptr;  // pinned; read by the last live call's copy until `copied`
  cudaEvent_t copied = nullptr;
  // A captured call's copy reads its source at every replay, so each has a
  // pinned block of its own, kept until the batch is freed.
  std::vector<BatchDesc*> h_captured;
  BatchDesc* d_desc = nullptr;
  uint16_t* d_cta_inst = nullptr;
};

namespace {

BfsArgs bfs_args(gsrb_graph* G, uint32_t src, int32_t* level, int32_t mode, bool stage) {
  BfsArgs a;
  a.g = dev_csr(G);
  a.src = src;
  a.level = level;
  a.q[0] = G->q[0];
  a.q[1] = G->q[1];
  a.hq[0] = G->hq[0];
  a.hq[1] = G->hq[1];
  a.cnt = G->cnt;
  a.overflow = G->flags;
  a.trace = G->trace;
  a.trace_cap = G->trace_cap;
  a.mlp = G->mlp;
  a.mode = mode;
  a.alpha = 15.f;
  a.beta = 18.f;
  a.out = G->flags + 4;
  a.out_edges = (unsigned long long*)((char*)G->flags + 64);
  a.solo = G->flags + 8;
  a.symmetric = G->symmetric;
  a.lb = false;
  a.lb_pre = G->lb_pre;
  a.lb_own = G->lb_own;
  a.lb_part = G->lb_part;
  a.phase = G->flags + 20;
  a.staged = false;
  a.stage = stage;
  return a;
}

SsspArgs sssp_args(gsrb_graph* G, uint32_t src, int32_t* dist, int32_t delta, bool stage) {
  SsspArgs a;
  a.g = dev_csr(G);
  a.src = src;
  a.dist = dist;
  for (int k = 0; k < 2; ++k) {
    a.q[k] = G->q[k];
    a.hq[k] = G->hq[k];
    a.far[k] = G->far[k];
  }
  a.mark = G->mark;
  a.fmark = G->fmark;
  a.cnt = G->cnt;
  a.fcnt = G->fcnt;
  a.overflow = G->flags;
  a.trace = G->trace;
  a.trace_cap = G->trace_cap;
  a.delta = delta;
  a.out = G->flags + 4;
  a.out_edges = (unsigned long long*)((char*)G->flags + 64);
  a.phase = G->flags + 20;
  a.state = G->flags + 8;
  a.staged = false;
  a.stage = stage;
  return a;
}

gsrb_status_t batch_launch(gsrb_batch* B, const uint32_t* srcs, int32_t* const* outs, int kind, int32_t param) {
  if (!B || !srcs || !outs) return GSRB_ERR_ARG;
  const int k = (int)B->graphs.size();
  for (int i = 0; i < k; ++i)
    if (!outs[i] || srcs[i] >= B->graphs[i]->n) return GSRB_ERR_ARG;
  if (kind == 0 && param == GSRB_BFS_LEARNED)
    for (int i = 0; i < k; ++i)
      if (!B->graphs[i]->mlp_set) return GSRB_ERR_STATE;
  // SSSP with the learned bucket width: every instance its own (host-side
  // plan from the graph's statistics; nothing is read from the device)
  std::vector<int32_t> deltas((size_t)k, param);
  if (kind == 1 && param == GSRB_SSSP_DELTA_LEARNED)
    for (int i = 0; i < k; ++i) {
      gsrb_status_t st = gsrb_graph_sssp_plan(B->graphs[i], srcs[i], &deltas[i], nullptr, nullptr);
      if (st) return st;
    }
  gsrb_ctx* ctx = B->ctx;
  const void* fn = batch_fn(B->cfg.variant, kind);
  if (!fn) return GSRB_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> g(ctx->mu);
  const size_t smem = kind == 0 ? with_stage<BfsStage>(ctx, fn, B->grid, B->cfg, 1)
                                : with_stage<IdStage>(ctx, fn, B->grid, B->cfg, 1);
  std::vector<BatchDesc> desc((size_t)k);
  for (int i = 0; i < k; ++i) {
    BatchDesc& d = desc[i];
    memset(&d, 0, sizeof(d));
    // slot 1 + i and, for the group-counter variants, groups starting at the
    // instance's first CTA (an instance never has more groups than CTAs)
    d.gb = make_barrier(ctx, B->cfg, 1 + i, B->count[i], B->first[i], B->first[i]);
    d.first = B->first[i];
    d.count = B->count[i];
    d.kind = (uint32_t)kind;
    if (kind == 0) {
      d.bfs = bfs_args(B->graphs[i], srcs[i], outs[i], param, smem != 0);
      B->graphs[i]->last_delta = 0;
    }
    else {
      d.sssp = sssp_args(B->graphs[i], srcs[i], outs[i], deltas[i], smem != 0);
      B->graphs[i]->last_delta = deltas[i];
    }
  }
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  GSRB_CUDA(cudaStreamIsCapturing(ctx->stream, &capturing));
  const BatchDesc* src = B->h_desc;
  if (capturing != cudaStreamCaptureStatusNone) {
    BatchDesc* block = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // (an allocation is not part of what is recorded)
    GSRB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t e = cudaMallocHost(&block, sizeof(BatchDesc) * (size_t)k);
    GSRB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    GSRB_CUDA(e);
    B->h_captured.push_back(block);
    memcpy(block, desc.data(), sizeof(BatchDesc) * (size_t)k);
    src = block;
  } else if (memcmp(B->h_desc, desc.data(), sizeof(BatchDesc) * (size_t)k) != 0) {
    // The copy of an earlier call may not have run yet (calls are asynchronous):
    // its source is rewritten only when the descriptors differ, and after it.
    if (B->copied) GSRB_CUDA(cudaEventSynchronize(B->copied));
    memcpy(B->h_desc, desc.data(), sizeof(BatchDesc) * (size_t)k);
  }
  for (int i = 0; i < k; ++i) GSRB_CUDA(cudaMemsetAsync(B->graphs[i]->flags, 0, 128, ctx->stream));
  GSRB_CUDA(cudaMemcpyAsync(B->d_desc, src, sizeof(BatchDesc) * k, cudaMemcpyHostToDevice, ctx->stream));
  if (capturing == cudaStreamCaptureStatusNone) {
    if (!B->copied) GSRB_CUDA(cudaEventCreateWithFlags(&B->copied, cudaEventDisableTiming));
    GSRB_CUDA(cudaEventRecord(B->copied, ctx->stream));
  }
  const BatchDesc* dd = B->d_desc;
  const uint16_t* ci = B->d_cta_inst;
  void* args[] = {(void*)&dd, (void*)&ci};
  return launch_persistent(ctx, fn, B->grid, B->cfg.threads, smem, 1, coop_of(B->cfg), args);
}

}  // namespace

extern "C" {

gsrb_status_t gsrb_batch_create(gsrb_ctx_t ctx, const gsrb_graph_t* graphs, int32_t k, const gsrb_cfg_t* cfgin,
                                gsrb_batch_t* out) {
  if (!ctx || !graphs || !out || k <= 0 || k > kSlots - 1) return GSRB_ERR_ARG;
  gsrb_cfg_t c = resolve_cfg(ctx, cfgin);
  if (!cfgin) {
    c.variant = gsrb::V_FANOUT;
    c.ctas_per_sm = 2;
    c.threads = 512;
  }
  c.cluster = 1;
  if (!batch_fn(c.variant, 0)) return GSRB_ERR_UNSUPPORTED;
  if (c.threads % 32 || c.threads > kGraphMaxThreads) return GSRB_ERR_ARG;
  const int grid = grid_of(ctx, c);
  if (grid < k || grid > 65535) return GSRB_ERR_ARG;
  gsrb_batch* B = new gsrb_batch();
  B->ctx = ctx;
  B->cfg = c;
  B->grid = grid;
  for (int i = 0; i < k; ++i) {
    if (!graphs[i]) {
      delete B;
      return GSRB_ERR_ARG;
    }
    B->graphs.push_back(graphs[i]);
  }
  // CTAs in proportion to each instance's edges (+ vertices), at least one each
  std::vector<double> w(k);
  double W = 0;
  for (int i = 0; i < k; ++i) {
    w[i] = (double)graphs[i]->m + (double)graphs[i]->n;
    W += w[i];
  }
  std::vector<uint32_t> cnt(k, 1);
  int left = grid - k;
  std::vector<std::pair<double, int>> rem;
  for (int i = 0; i < k; ++i) {
    const double share = W > 0 ? left * w[i] / W : 0.0;
    const uint32_t extra = (uint32_t)share;
    cnt[i] += extra;
    rem.push_back({share - extra, i});
  }
  int used = 0;
  for (int i = 0; i < k; ++i) used += (int)cnt[i];
  std::sort(rem.begin(), rem.end(), [](const std::pair<double, int>& a, const std::pair<double, int>& b) {
    return a.first > b.first || (a.first == b.first && a.second < b.second);
  });
  for (size_t j = 0; used < grid && j < rem.size(); ++j, ++used) cnt[rem[j].second] += 1;
  std::vector<uint16_t> inst(grid);
  uint32_t f = 0;
  for (int i = 0; i < k; ++i) {
    B->first.push_back(f);
    B->count.push_back(cnt[i]);
    for (uint32_t j = 0; j < cnt[i]; ++j) inst[f + j] = (uint16_t)i;
    f += cnt[i];
  }
  cudaError_t e = cudaMallocHost(&B->h_desc, sizeof(BatchDesc) * k);
  if (!e) memset(B->h_desc, 0, sizeof(BatchDesc) * k);
  if (!e) e = cudaMalloc(&B->d_desc, sizeof(BatchDesc) * k);
  if (!e) e = cudaMalloc(&B->d_cta_inst, sizeof(uint16_t) * grid);
  if (!e) e = cudaMemcpy(B->d_cta_inst, inst.data(), sizeof(uint16_t) * grid, cudaMemcpyHostToDevice);
  if (e) {
    gsrb_batch_free(B);
    return cuda_err(e, "batch_create");
  }
  *out = B;
  return GSRB_OK;
}

gsrb_status_t gsrb_batch_free(gsrb_batch_t B) {
  if (!B) return GSRB_ERR_ARG;
  if (B->ctx) cudaStreamSynchronize(B->ctx->stream);
  if (B->copied) cudaEventDestroy(B->copied);
  if (B->h_desc) cudaFreeHost(B->h_desc);
  for (BatchDesc* d : B->h_captured) cudaFreeHost(d);
  if (B->d_desc) cudaFree(B->d_desc);
  if (B->d_cta_inst) cudaFree(B->d_cta_inst);
  delete B;
  return GSRB_OK;
}

gsrb_status_t gsrb_batch_layout(gsrb_batch_t B, uint32_t* first, uint32_t* count) {
  if (!B) return GSRB_ERR_ARG;
  for (size_t i = 0; i < B->graphs.size(); ++i) {
    if (first) first[i] = B->first[i];
    if (count) count[i] = B->count[i];
  }
  return GSRB_OK;
}

gsrb_status_t gsrb_batch_bfs(gsrb_batch_t B, const uint32_t* srcs, int32_t* const* d_levels, int32_t mode) {
  if (mode < 0 || mode > GSRB_BFS_TOPO) return GSRB_ERR_ARG;
  return batch_launch(B, srcs, d_levels, 0, mode);
}

gsrb_status_t gsrb_batch_sssp(gsrb_batch_t B, const uint32_t* srcs, int32_t* const* d_dists, int32_t delta) {
  if (delta < 0) return GSRB_ERR_ARG;
  return batch_launch(B, srcs, d_dists, 1, delta);
}

gsrb_status_t gsrb_batch_stats(gsrb_batch_t B, gsrb_traversal_stats_t* stats) {
  if (!B) return GSRB_ERR_ARG;
  std::lock_guard<std::mutex> g(B->ctx->mu);
  for (size_t i = 0; i < B->graphs.size(); ++i) GSRB_CUDA(copy_status(B->ctx, B->graphs[i], (int)i));
  GSRB_CUDA(cudaStreamSynchronize(B->ctx->stream));
  gsrb_status_t worst = GSRB_OK;
  for (size_t i = 0; i < B->graphs.size(); ++i) {
    gsrb_status_t st = stats_of(B->graphs[i], B->ctx->h_status + 32 * i, stats ? &stats[i] : nullptr, 0.f);
    if (st && !worst) worst = st;
  }
  return worst;
}

// ---- CUDA graphs: capture the context stream's work once, replay it ----------
gsrb_status_t gsrb_capture_begin(gsrb_ctx_t ctx) {
  if (!ctx) return GSRB_ERR_ARG;
  std::lock_guard<std::mutex> g(ctx->mu);
  GSRB_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
  ctx->writer_open = true;  // recorded and live calls do not follow one another
  return GSRB_OK;
}

gsrb_status_t gsrb_capture_end(gsrb_ctx_t ctx, gsrb_exec_t* out) {
  if (!ctx || !out) return GSRB_ERR_ARG;
  cudaGraph_t graph = nullptr;
  {
    std::lock_guard<std::mutex> g(ctx->mu);
    GSRB_CUDA(cudaStreamEndCapture(ctx->stream, &graph));
    ctx->writer_open = true;
  }
  cudaGraphExec_t exec = nullptr;
  cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e) return cuda_err(e, "cudaGraphInstantiate");
  *out = (gsrb_exec_t)exec;
  return GSRB_OK;
}

gsrb_status_t gsrb_exec_launch(gsrb_ctx_t ctx, gsrb_exec_t exec) {
  if (!ctx || !exec) return GSRB_ERR_ARG;
  std::lock_guard<std::mutex> g(ctx->mu);
  GSRB_CUDA(cudaGraphLaunch((cudaGraphExec_t)exec, ctx->stream));
  ctx->writer_open = true;  // (the replay may end in a kernel that lets the next one in)
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return GSRB_OK;
}

gsrb_status_t gsrb_exec_free(gsrb_exec_t exec) {
  if (exec) GSRB_CUDA(cudaGraphExecDestroy((cudaGraphExec_t)exec));
  return GSRB_OK;
}

}  // extern "C"
