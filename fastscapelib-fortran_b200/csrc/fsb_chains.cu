// Heavy-path chain schedule of the receiver forest and the single-flow tree
// sweeps that run on it (lake fill, drainage area, stream power law).
//
// The tree recurrences of the reference are sequential loops over the stack:
//   hwater fill           src/FlowRouting.f90:73-89  (root -> leaves)
//   drainage area         src/FlowRouting.f90:123-143 (leaves -> root)
//   implicit SPL, g == 0  src/StreamPowerLaw.f90:291-373 (root -> leaves)
// Each node only needs its receiver (top-down) or its donors (bottom-up), so
// any schedule that respects the tree gives the same per-node arithmetic.
//
// Schedule.  Every node's heavy child is its donor with the largest subtree
// (first in ascending node order on ties).  A heavy-first preorder lays every
// heavy path out contiguously; a "chain" is one heavy path, from its head (a
// root or a light child) to a leaf.  A chain depends only on its head's parent
// (top-down) or on the chains hanging off it (bottom-up); its "light depth" --
// the number of light edges above it, at most log2(nn) -- therefore orders the
// chains.  They are dealt out by light depth (increasing for top-down sweeps,
// decreasing for bottom-up), by three kinds of workers:
//   * chains of one node (two thirds of all) take no part in the waiting: a
//     kernel with a thread per node computes them after (top-down) or before
//     (bottom-up) the others;
//   * chains of kLong nodes or more get a warp each: 32 nodes' data arrive with
//     one load per lane while the recurrence runs through the previous 32 on
//     values shuffled from their lanes, so a node costs its arithmetic, not a
//     memory round trip;
//   * the others get a lane each; a lane that waits for its chain's parent does
//     not hold up its warp mates.
// Every wait targets a chain of another light depth that is earlier in both
// lists, so the sweeps cannot deadlock.  A published value says itself that
// it has arrived: the arrays start as all ones (a NaN no result has: see
// fsb::publishable), values are written and polled with relaxed accesses at
// GPU scope, and no flags or fences are needed.
//
// Measured (B200), per step: 1023x767 single flow on a cell size without a
// closed form for the area: area 2.29 -> 0.26 ms, stream power 1.70 -> 0.20,
// schedule and fill 0.65 -> 0.22; 513x511 with n = 1.37: stream power 1.94 -> 0.24;
// 2049^2 schedule and fill 2.37 -> 0.87.  Against 32 chains of any length per
// warp that waited together, flags behind a fence at GPU scope (770 cycles per
// 8 or 16 nodes), powers evaluated on the chain, radix-sorted tickets and three
// read-backs.  What bounds a sweep now is the recurrence along the longest
// root-to-leaf path (a quotient or Newton's iterations per node) and ten or so
// hand-offs between chains of about 1 us.
//
// Heavy-first positions come from path sums over the receiver forest (a scan
// over the DFS preorder): pos(k) = sum over the root->k path of each node's
// offset within its parent's subtree (1 + sizes of the siblings laid out
// before it).
#include <algorithm>
#include <climits>
#include <cmath>

#include "fsb_kernels.cuh"

namespace fsb {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kLong = kLongChain;  // nodes of a chain that gets a warp of its own
constexpr int kDepths = 32;        // light depths (at most log2(nn) <= 28)
constexpr int kClasses = 32;       // length classes (powers of two, longest first)
constexpr int kBuckets = kDepths * kClasses;
// ticket counts and cursors: kBuckets of the long chains, kDepths of the short ones
constexpr int kHist = kBuckets + kDepths;
static_assert(kHist == kChainHist, "the arena holds three of them");

// ---- schedule ---------------------------------------------------------------

// offset of k inside its parent's heavy-first layout and whether it heads a
// chain, as path-sum marks: node k's subtree is the interval [pos(k), pos(k) +
// size(k)) of the DFS preorder, so adding w(k) at pos(k) and subtracting it
// at pos(k) + size(k) makes the prefix sum at pos(k) the sum over k's
// ancestors and k.  w = (light flag << kOffBits) | offset: offsets sum to a
// heavy-first position and light flags to a light depth (< 32), so the two
// fields never carry into each other; the marks wrap and cancel exactly.
// 32-bit words hold grids below 2^27 nodes, 64-bit ones the others.
template <class U>
constexpr int kOffBits = sizeof(U) == 4 ? 27 : 32;

template <class U>
__global__ void k_path_marks(int nn, const int* __restrict__ rec, const int* __restrict__ ndon,
                             const int* __restrict__ don, const int* __restrict__ pos, const int* __restrict__ size,
                             U* __restrict__ marks, unsigned char* __restrict__ head, int* __restrict__ err) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const int r = rec[k], p = pos[k], e = p + size[k];
    U off = 1, light = 0;
    bool hd = true;
    if (r == k) {
      off = (U)p;  // roots ascending: the earlier roots' trees fill [0, pos)
    } else {
      const int nd = ndon[r];
      if (nd > 1) {
        const int4* row = reinterpret_cast<const int4*>(don + (size_t)r * 8);
        const int4 a = __ldg(row), b = __ldg(row + 1);
        const int d[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        int hv = -1, hs = -1, before = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i < nd) {
            const int s = __ldg(&size[d[i]]);
            if (s > hs) { hs = s; hv = d[i]; }
            if (d[i] < k) before += s;
          }
        hd = hv != k;
        if (hd) {
          light = 1;
          off = 1u + (U)before + (hv < k ? (U)0 : (U)hs);  // the heavy child comes first
        }
      } else {
        hd = false;  // the only donor
      }
    }
    head[k] = hd ? 1 : 0;
    if (p < 0 || e > nn || e <= p) {
      atomicExch(err, DEV_STACK_ERROR);
      continue;
    }
    const U w = (light << kOffBits<U>) | off;
    atomicAdd(&marks[p], w);
    atomicAdd(&marks[e], (U)0 - w);
  }
}

// after an exclusive scan of the marks: the heavy-first order, and by position
// the chain starts and light depths
template <class U>
__global__ void k_hf_order(int nn, const U* __restrict__ scan, const int* __restrict__ pos,
                           const unsigned char* __restrict__ head, int* __restrict__ ord, int* __restrict__ flag,
                           unsigned char* __restrict__ depth, int* __restrict__ err) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const U s = scan[pos[k] + 1];
    const U off = s & (((U)1 << kOffBits<U>) - 1);
    if (off >= (U)nn) { atomicExch(err, DEV_STACK_ERROR); continue; }
    ord[off] = k;
    flag[off] = head[k];
    depth[off] = (unsigned char)min((unsigned)(s >> kOffBits<U>), (unsigned)kDepths - 1u);
    if (k == 0) flag[nn] = 0;
  }
}

__global__ void k_chain_list(int nn, const int* __restrict__ flag, const int* __restrict__ scan,
                             int* __restrict__ cstart) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nn; p += gridDim.x * blockDim.x)
    if (flag[p]) cstart[scan[p]] = p;
}

// bucket of a chain of `len` >= 2 nodes: the long ones by depth, then longest first
__device__ __forceinline__ int chain_bucket(int len, int depth) {
  if (len < kLong) return kBuckets + depth;
  return depth * kClasses + __clz(len);
}
// the same with decreasing depth (bottom-up)
__device__ __forceinline__ int reversed(int b) {
  if (b >= kBuckets) return kBuckets + (kDepths - 1 - (b - kBuckets));
  return (kDepths - 1 - b / kClasses) * kClasses + b % kClasses;
}

// Chains per bucket.  Counted per block in shared memory: the buckets are
// few, and one global atomic per block and bucket replaces one per chain.
constexpr int kChainBlock = 256, kChainsPerBlock = 8 * kChainBlock;
__global__ void __launch_bounds__(kChainBlock) k_chain_hist(int nn, const int* __restrict__ nchains,
                                                            const int* __restrict__ cstart,
                                                            const unsigned char* __restrict__ depth,
                                                            int* __restrict__ hist) {
  __shared__ int sh[kHist];
  const int n = *nchains;
  for (int t = threadIdx.x; t < kHist; t += kChainBlock) sh[t] = 0;
  __syncthreads();
  for (int c = blockIdx.x * kChainsPerBlock + threadIdx.x, i = 0; i < 8 && c < n; ++i, c += kChainBlock) {
    const int s = cstart[c], e = c + 1 < n ? cstart[c + 1] : nn;
    if (e - s > 1) atomicAdd(&sh[chain_bucket(e - s, depth[s])], 1);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kHist; t += kChainBlock)
    if (sh[t]) atomicAdd(&hist[t], sh[t]);
}

// exclusive prefix of the bucket counts, top-down and bottom-up order, and the
// two lists' lengths (one block of kBuckets threads)
__global__ void __launch_bounds__(kBuckets) k_chain_offsets(const int* __restrict__ hist, int* __restrict__ cur_td,
                                                            int* __restrict__ cur_bu, int* __restrict__ totals) {
  __shared__ int warp_sum[2][32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (int dir = 0; dir < 2; ++dir) {
    int* cur = dir ? cur_bu : cur_td;
    const int v = hist[dir ? reversed(t) : t];
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[dir][w] = x;
    __syncthreads();
    if (w == 0) {
      int s = warp_sum[dir][lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, s, o);
        if (lane >= o) s += y;
      }
      warp_sum[dir][lane] = s;
    }
    __syncthreads();
    cur[t] = x - v + (w ? warp_sum[dir][w - 1] : 0);  // cursors are in this direction's order
    if (t == kBuckets - 1) totals[0] = warp_sum[dir][31];
    if (w == 0) {  // the short chains
      const int b = kBuckets + lane;
      const int sv = hist[dir ? reversed(b) : b];
      int sx = sv;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, sx, o);
        if (lane >= o) sx += y;
      }
      cur[b] = sx - sv;
      if (lane == 31) totals[1] = sx;
    }
  }
}

// tickets {first position, end, head, its receiver}, both directions; within a
// bucket in any order
__global__ void __launch_bounds__(kChainBlock) k_chain_tickets(int nn, const int* __restrict__ nchains,
                                                               const int* __restrict__ cstart,
                                                               const unsigned char* __restrict__ depth,
                                                               const int* __restrict__ ord, const int* __restrict__ rec,
                                                               int* cur_td, int* cur_bu, int4* __restrict__ td_long,
                                                               int4* __restrict__ td_short, int4* __restrict__ bu_long,
                                                               int4* __restrict__ bu_short) {
  __shared__ int cnt[kHist], base_td[kHist], base_bu[kHist];
  const int n = *nchains;
  if (blockIdx.x * kChainsPerBlock >= n) return;
  for (int t = threadIdx.x; t < kHist; t += kChainBlock) cnt[t] = 0;
  __syncthreads();
  int b[8], rank[8], st[8], en[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = blockIdx.x * kChainsPerBlock + i * kChainBlock + threadIdx.x;
    b[i] = -1;
    if (c < n) {
      st[i] = cstart[c];
      en[i] = c + 1 < n ? cstart[c + 1] : nn;
      if (en[i] - st[i] > 1) {
        b[i] = chain_bucket(en[i] - st[i], depth[st[i]]);
        rank[i] = atomicAdd(&cnt[b[i]], 1);
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kHist; t += kChainBlock)
    if (cnt[t]) {
      base_td[t] = atomicAdd(&cur_td[t], cnt[t]);
      base_bu[t] = atomicAdd(&cur_bu[reversed(t)], cnt[t]);
    }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (b[i] >= 0) {
      const int k0 = ord[st[i]];
      const int4 t = make_int4(st[i], en[i], k0, rec[k0]);
      (b[i] < kBuckets ? td_long : td_short)[base_td[b[i]] + rank[i]] = t;
      (b[i] < kBuckets ? bu_long : bu_short)[base_bu[b[i]] + rank[i]] = t;
    }
}

// ---- sweeps -------------------------------------------------------------------

struct ChainView {
  const int* ord;  // heavy-first order
  const int4 *tk_long, *tk_short;
  const int* totals;   // long, short chains
  unsigned* ticket;    // next long, next short chain
  int* err;
};

// Values travel between chains in arrays that start as all ones.
__device__ __forceinline__ bool arrived(double v) { return __double_as_longlong(v) != -1ll; }

// Bounded waiting: true when the caller must give up (a wait here or elsewhere failed).
struct Patience {
  int spins = 0, back = 32;
  __device__ bool over(int* err) {
    if (++spins > kSpinLimit) {
      atomicCAS(err, 0, DEV_SPIN_LIMIT);  // an earlier error is the cause
      return true;
    }
    return (spins & 63) == 0 && *(volatile int*)err != 0;
  }
  __device__ void rest() {
    __nanosleep(back);
    if (back < 256) back <<= 1;
  }
};

constexpr int kSweepThreads = 128, kSoloWarps = 2;  // per block: warps for long chains; the others' lanes take short ones

// Top-down sweep.  Op:
//   Node load(k)            what the recurrence needs of node k
//   Node shfl(node, lane)   that of another lane
//   bool poll(r, State&)    the state after receiver r; false if not there yet
//   State root()            the state before a root
//   void step(State&, node, k, first, store)
//                           node k's value; first: k is a root; store: write it out
template <class Op>
__global__ void __launch_bounds__(kSweepThreads) k_top_down(ChainView cv, Op op) {
  using Node = typename Op::Node;
  using State = typename Op::State;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < kSoloWarps) {
    const int total = cv.totals[0];
    for (;;) {
      unsigned t = 0;
      if (lane == 0) t = atomicAdd(&cv.ticket[0], 1u);
      t = __shfl_sync(FULL, t, 0);
      if ((int)t >= total) return;
      const int4 tk = cv.tk_long[t];
      const int s = tk.x, e = tk.y;
      const bool root = tk.z == tk.w;
      // nodes of this chunk, of the next one, and the indices of the one after
      int k = s + lane < e ? cv.ord[s + lane] : -1;
      int k2 = s + 32 + lane < e ? cv.ord[s + 32 + lane] : -1;
      Node nd{}, nd2{};
      if (k >= 0) nd = op.load(k);
      State st = op.root();
      if (!root) {
        Patience pat;
        while (!__all_sync(FULL, op.poll(tk.w, st))) {  // a value that has arrived is final: the lanes agree
          if (__any_sync(FULL, pat.over(cv.err))) return;
          pat.rest();
        }
      }
      for (int p = s; p < e; p += 32) {
        const int k3 = p + 64 + lane < e ? cv.ord[p + 64 + lane] : -1;
        if (k2 >= 0) nd2 = op.load(k2);
        const int n = min(32, e - p);
        for (int i = 0; i < n; ++i)
          op.step(st, op.shfl(nd, i), __shfl_sync(FULL, k, i), root && p == s && i == 0, lane == i);
        k = k2;
        nd = nd2;
        k2 = k3;
      }
    }
  }
  constexpr int kC = 4;
  const int total = cv.totals[1];
  int4 tk = make_int4(0, 0, 0, 0);
  int status = 0;  // 0 without a chain, 1 waiting, 2 walking, 3 no chain left
  State st = op.root();
  Patience pat;
  for (;;) {
    const unsigned idle = __ballot_sync(FULL, status == 0);
    if (idle) {
      unsigned t = 0;
      if (lane == 0) t = atomicAdd(&cv.ticket[1], (unsigned)__popc(idle));
      t = __shfl_sync(FULL, t, 0) + __popc(idle & ((1u << lane) - 1u));
      if (status == 0) {
        if ((int)t < total) {
          tk = cv.tk_short[t];
          status = tk.z == tk.w ? 2 : 1;
          st = op.root();
        } else {
          status = 3;
        }
      }
    }
    if (!__any_sync(FULL, status != 3)) return;
    if (status == 1 && op.poll(tk.w, st)) status = 2;
    if (status == 2) {
      int k[kC];
      Node nd[kC];
#pragma unroll
      for (int i = 0; i < kC; ++i) k[i] = tk.x + i < tk.y ? cv.ord[tk.x + i] : -1;
#pragma unroll
      for (int i = 0; i < kC; ++i)
        if (k[i] >= 0) nd[i] = op.load(k[i]);
#pragma unroll
      for (int i = 0; i < kC; ++i)
        if (k[i] >= 0) op.step(st, nd[i], k[i], k[i] == tk.w, true);
      tk.x += kC;
      if (tk.x >= tk.y) status = 0;
    }
    if (!__any_sync(FULL, status == 0 || status == 2)) {  // all of them wait
      if (__any_sync(FULL, pat.over(cv.err))) return;
      pat.rest();
    } else {
      pat = Patience{};
    }
  }
}

// chains of one node, after the others: everything they need is final
template <class Op>
__global__ void k_top_down_leaves(int nn, const int* __restrict__ rec, const int* __restrict__ ndon,
                                  const unsigned char* __restrict__ head, Op op, int* err) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    if (ndon[k] != 0 || !head[k]) continue;
    const int r = rec[k];
    typename Op::State st = op.root();
    if (r != k && !op.poll(r, st)) {
      atomicCAS(err, 0, DEV_SPIN_LIMIT);  // only after an error: the walkers have finished
      continue;
    }
    op.step(st, op.load(k), k, r == k, true);
  }
}

// hwater(k) = hwater(rec) > h(k) ? hwater(rec) + 1e-8 : h(k)
// (FlowRouting.f90:77-86); lake_depth = hwater - h.
struct FillOp {
  const double* __restrict__ h;
  double *hwater, *lake_depth;
  using Node = double;
  using State = double;
  __device__ Node load(int k) const { return __ldg(&h[k]); }
  __device__ Node shfl(Node n, int i) const { return __shfl_sync(FULL, n, i); }
  __device__ State root() const { return 0.0; }
  __device__ bool poll(int r, State& st) const {
    const double v = ld_relaxed_gpu(&hwater[r]);
    if (!arrived(v)) return false;
    st = v;
    return true;
  }
  __device__ void step(State& st, Node hk, int k, bool first, bool store) const {
    st = first ? hk : (st > hk ? st + 1.0e-8 : hk);
    if (store) {
      st_relaxed_gpu(&hwater[k], publishable(st));
      lake_depth[k] = st - hk;
    }
  }
};

// CopyChi (FastScape_ctx.f90:228-251) top down: chi(k) = chi(rec(k)) +
// (a0/a(k))^(m/n) * length(k) where a(k) > a0, else 0; a root starts from 0.
struct ChiOp {
  const double* __restrict__ a;
  const double* __restrict__ length;
  double a0, mn;
  double* chi;
  struct Node { double term, above; };
  using State = double;
  __device__ Node load(int k) const {
    const double ak = __ldg(&a[k]);
    return {pow(a0 / ak, mn) * __ldg(&length[k]), ak > a0 ? 1.0 : 0.0};
  }
  __device__ Node shfl(const Node& n, int i) const {
    return {__shfl_sync(FULL, n.term, i), __shfl_sync(FULL, n.above, i)};
  }
  __device__ State root() const { return 0.0; }
  __device__ bool poll(int r, State& st) const {
    const double v = ld_relaxed_gpu(&chi[r]);
    if (!arrived(v)) return false;
    st = v;
    return true;
  }
  __device__ void step(State& st, const Node& n, int k, bool, bool store) const {
    st = n.above != 0.0 ? st + n.term : 0.0;
    if (store) st_relaxed_gpu(&chi[k], publishable(st));
  }
};

// Single-flow erosion factor kf*dt*a^m/l^n of every node: the powers do not
// depend on the recurrence, so they stay off the chains.
__global__ void k_spl_factor(int nn, int n_is_one, const int* __restrict__ rec, const double* __restrict__ h,
                             const double* __restrict__ b, const double* __restrict__ kf,
                             const double* __restrict__ a, const double* __restrict__ length, double kfsed, double dt,
                             double m, double n, double* __restrict__ fact) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    double f = 0.0;
    if (rec[k] != k) {
      const double kfint = (kfsed > 0.0 && (h[k] - b[k]) > 1.0) ? kfsed : kf[k];
      const double l = length[k];
      f = n_is_one ? kfint * dt * pow(a[k], m) / l : kfint * dt * pow(a[k], m) / pow(l, n);
    }
    fact[k] = f;
  }
}

// Top-down single-flow stream power law (StreamPowerLaw.f90:291-373): writes
// hnew and water; h keeps ht.  MODE 0: n = 1; 1: n = 1.5 (x*sqrt(x) and
// sqrt(x)); 2: other n (one pow: x^n = x * x^(n-1)).  With GS (a Gauss-Seidel
// iteration of the g > 0 solve, :285-373) the deposition-corrected surface
// comes from `elev`, Newton starts from the current iterate `hstart`, and the
// lake bookkeeping is written: sill(k) = k for a node above its receiver's
// water, else sill(rec) with its volume contribution w_rcv - h(k) in
// contrib(k).  Without GS, elev = hstart = ht.
template <int MODE, bool GS>
struct SplOp {
  const double* __restrict__ h;
  const double* __restrict__ fact;
  double n, omega;
  double *hnew, *water;
  const double* __restrict__ elev;
  const double* __restrict__ hstart;
  int* sill;  // -1 until written
  double* contrib;
  int* err;
  struct Node { double ht, fact, elev, h0; };
  struct State {
    double h, w, ht;  // the receiver's new elevation, water and old elevation
    int sill;
  };
  __device__ Node load(int k) const {
    Node nd;
    nd.ht = __ldg(&h[k]);
    nd.fact = __ldg(&fact[k]);
    nd.elev = GS ? __ldg(&elev[k]) : nd.ht;
    nd.h0 = GS ? __ldg(&hstart[k]) : nd.ht;
    return nd;
  }
  __device__ Node shfl(const Node& nd, int i) const {
    Node o;
    o.ht = __shfl_sync(FULL, nd.ht, i);
    o.fact = __shfl_sync(FULL, nd.fact, i);
    o.elev = GS ? __shfl_sync(FULL, nd.elev, i) : o.ht;
    o.h0 = GS ? __shfl_sync(FULL, nd.h0, i) : o.ht;
    return o;
  }
  __device__ State root() const { return {0.0, 0.0, 0.0, 0}; }
  __device__ bool poll(int r, State& st) const {
    const double hv = ld_relaxed_gpu(&hnew[r]), wv = ld_relaxed_gpu(&water[r]);
    const int sv = GS ? ld_relaxed_gpu(&sill[r]) : 0;
    if (!arrived(hv) || !arrived(wv) || (GS && sv < 0)) return false;
    st.h = hv;
    st.w = wv;
    st.ht = __ldg(&h[r]);
    st.sill = sv;
    return true;
  }
  __device__ void step(State& st, const Node& nd, int k, bool first, bool store) const {
    const double ht = nd.ht, el = nd.elev;
    double hk = ht, wk = ht, ck = 0.0;
    int sk = k;
    if (!first) {
      hk = nd.h0;
      if (el > st.w) {
        if constexpr (MODE == 0) {
          double f = el, df = 1.0;
          f = f + nd.fact * st.h;
          df = df + nd.fact;
          hk = f / df;
        } else {
          const double tolp = 1.0e-3;
          double errp = 2.0 * tolp;
          int guard = 0;
          while (errp > tolp) {
            if (++guard > kNewtonLimit) {
              atomicExch(err, DEV_NEWTON_LIMIT);
              break;
            }
            double f = hk - el, df = 1.0;
            if (ht > st.ht) {
              const double x = fmax(0.0, hk - st.h);
              double pn, pn1;
              if constexpr (MODE == 1) {
                pn1 = sqrt(x);
                pn = x * pn1;
              } else if (x > 0.0) {
                pn1 = pow(x, n - 1.0);
                pn = x * pn1;
              } else {
                pn = pow(x, n);
                pn1 = pow(x, n - 1.0);
              }
              f = f + nd.fact * pn;
              df = df + nd.fact * n * pn1;
            }
            const double hn = hk - f / df;
            errp = fabs(hn - hk);
            hk = hk * (1.0 - omega) + hn * omega;
          }
        }
        if (hk < st.w) hk = st.w;
      } else {
        hk = el;
        sk = st.sill;
        ck = st.w - hk;
      }
      wk = fmax(st.w, hk);
    }
    if (store) {
      st_relaxed_gpu(&hnew[k], publishable(hk));
      st_relaxed_gpu(&water[k], publishable(wk));
      if (GS) {
        st_relaxed_gpu(&sill[k], sk);
        contrib[k] = ck;
      }
    }
    st.h = hk;
    st.w = wk;
    st.ht = ht;
    st.sill = sk;
  }
};

// ---- bottom-up --------------------------------------------------------------------
// v(k) = value(base(k) + v(d_m) + ... + v(d_1)), donors descending (the
// reverse-stack order of FlowRouting.f90:136-139).  Finishers:
//   AreaFin  drainage area; a root adds itself (FlowRouting.f90:136-139)
//   FluxFin  compute_fluxes' sediment flux: base erate, max(0, .) before the
//            value goes downstream, a root adds itself (FastScape_ctx.f90:864-869)
//   GsFin    the erosion sum of a Gauss-Seidel iteration with g > 0
//            (StreamPowerLaw.f90:262-280): base ht-hp; a lake sill's own
//            share is taken out and kept as lake_sediment
//   VolFin   lake water volume: a flooded node passes its contribution
//            (w_rcv - h) and its flooded donors' up to its receiver; every
//            node records what its donors pass as its volume (a sill's volume)
// aux(k): a further number of the node that value needs (kAux); flags bit 0: a
// root, bit 1: a property of the node.
struct AreaFin {
  const double* __restrict__ precip;
  double dxdy;
  static constexpr bool kAux = false;
  __device__ double base(int k) const { return dxdy * __ldg(&precip[k]); }
  __device__ double aux(int) const { return 0.0; }
  __device__ unsigned prop(int) const { return 0u; }
  __device__ double value(double acc, double, unsigned fl) const { return (fl & 1u) ? acc + acc : acc; }
  __device__ void side(int, double, double, unsigned) const {}
};
struct FluxFin {
  const double* __restrict__ erate;
  static constexpr bool kAux = false;
  __device__ double base(int k) const { return __ldg(&erate[k]); }
  __device__ double aux(int) const { return 0.0; }
  __device__ unsigned prop(int) const { return 0u; }
  __device__ double value(double acc, double, unsigned fl) const {
    acc = fmax(0.0, acc);
    return (fl & 1u) ? acc + acc : acc;
  }
  __device__ void side(int, double, double, unsigned) const {}
};
struct GsFin {
  const double* __restrict__ ht;
  const double* __restrict__ hp;
  const int* __restrict__ sill;
  double* lsed;
  static constexpr bool kAux = true;
  __device__ double base(int k) const { return __ldg(&ht[k]) - __ldg(&hp[k]); }
  __device__ double aux(int k) const { return base(k); }
  __device__ unsigned prop(int k) const { return __ldg(&sill[k]) == k ? 2u : 0u; }
  __device__ double value(double acc, double e, unsigned fl) const {
    if (fl & 1u) return acc;
    const double t = acc - e;
    return t + e;
  }
  __device__ void side(int k, double acc, double e, unsigned fl) const {
    if (fl & 1u) {
      lsed[k] = acc;
    } else if (fl & 2u) {
      const double t = acc - e;
      lsed[k] = t <= 0.0 ? 0.0 : t;
    }
  }
};
struct VolFin {
  const int* __restrict__ sill;
  const double* __restrict__ contrib;
  double* vol;
  static constexpr bool kAux = true;
  __device__ double base(int) const { return 0.0; }
  __device__ double aux(int k) const { return __ldg(&contrib[k]); }
  __device__ unsigned prop(int k) const { return __ldg(&sill[k]) != k ? 2u : 0u; }
  __device__ double value(double acc, double cb, unsigned fl) const { return fl == 2u ? cb + acc : 0.0; }
  __device__ void side(int k, double acc, double, unsigned) const { vol[k] = acc; }
};

// A node's donors: the sum down to the heavy one (descending) and the lighter
// values that follow it.
struct Gather {
  double first;    // base and the donors above the heavy child
  double rest[7];  // the donors below it, in order
  int nrest;
  // false while a value has not arrived
  __device__ __forceinline__ bool take(int k, int nd, int heavy, double base, const int* __restrict__ don,
                                       const double* a) {
    first = base;
    nrest = 0;
    if (nd < 2) return true;
    const int4* row = reinterpret_cast<const int4*>(don + (size_t)k * 8);
    const int4 x = __ldg(row), y = __ldg(row + 1);
    const int d[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < nd && d[i] != heavy) v[i] = ld_relaxed_gpu(&a[d[i]]);
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < nd && d[i] != heavy) ok &= arrived(v[i]);
    if (!ok) return false;
    bool below = false;
#pragma unroll
    for (int i = 7; i >= 0; --i)
      if (i < nd) {
        if (d[i] == heavy) {
          below = true;
        } else if (!below) {
          first = first + v[i];
        } else {
#pragma unroll
          for (int t = 0; t < 7; ++t)
            if (t == nrest) rest[t] = v[i];
          ++nrest;
        }
      }
    return true;
  }
};

template <class Fin>
__global__ void __launch_bounds__(kSweepThreads) k_bottom_up(ChainView cv, const int* __restrict__ rec,
                                                             const int* __restrict__ ndon,
                                                             const int* __restrict__ don, Fin fin, double* a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < kSoloWarps) {
    const int total = cv.totals[0];
    for (;;) {
      unsigned t = 0;
      if (lane == 0) t = atomicAdd(&cv.ticket[0], 1u);
      t = __shfl_sync(FULL, t, 0);
      if ((int)t >= total) return;
      const int4 tk = cv.tk_long[t];
      const int s = tk.x, e = tk.y;
      double ac = 0.0;
      // lane i of a chunk holds position hi - 1 - i; its heavy child is the position after
      int k = e - 1 - lane >= s ? cv.ord[e - 1 - lane] : -1;
      for (int hi = e; hi > s; hi -= 32) {
        const int n = min(32, hi - s);
        const int k2 = hi - 33 - lane >= s ? cv.ord[hi - 33 - lane] : -1;
        int heavy = __shfl_up_sync(FULL, k, 1);
        if (lane == 0) heavy = hi < e ? cv.ord[hi] : -1;
        double base = 0.0, aux = 0.0;
        int nd = 0;
        unsigned fl = 0;
        if (k >= 0) {
          nd = ndon[k];
          base = fin.base(k);
          if (Fin::kAux) aux = fin.aux(k);
          fl = (rec[k] == k ? 1u : 0u) | fin.prop(k);
        }
        Gather g;
        bool ready = k < 0 || g.take(k, nd, heavy, base, don, a);
        const bool inner = heavy >= 0;  // the chain's leaf has no child
        double acc_own = 0.0;
        int i = 0;
        Patience pat;
        while (i < n) {
          const unsigned rb = __ballot_sync(FULL, ready);
          const int upto = min(n, __ffs(~rb) ? __ffs(~rb) - 1 : 32);
          if (i >= upto) {  // the next node's donors are not all there
            if (__any_sync(FULL, pat.over(cv.err))) return;
            if (pat.spins > 4) pat.rest();
            if (!ready) ready = g.take(k, nd, heavy, base, don, a);
            continue;
          }
          for (; i < upto; ++i) {
            double acc = __shfl_sync(FULL, g.first, i);
            if (__shfl_sync(FULL, (int)inner, i)) acc = acc + ac;
            const int nr = __shfl_sync(FULL, g.nrest, i);
#pragma unroll
            for (int u = 0; u < 7; ++u) {
              if (u >= nr) break;
              acc = acc + __shfl_sync(FULL, g.rest[u], i);
            }
            const double ax = Fin::kAux ? __shfl_sync(FULL, aux, i) : 0.0;
            ac = fin.value(acc, ax, __shfl_sync(FULL, fl, i));
            if (lane == i) {
              acc_own = acc;
              st_relaxed_gpu(&a[k], publishable(ac));
            }
          }
        }
        if (k >= 0) fin.side(k, acc_own, aux, fl);
        k = k2;
      }
    }
  }
  const int total = cv.totals[1];
  int4 tk = make_int4(0, 0, 0, 0);
  int status = 0;  // 0 without a chain, 2 walking, 3 no chain left
  int child = -1;
  double ac = 0.0;
  Patience pat;
  for (;;) {
    const unsigned idle = __ballot_sync(FULL, status == 0);
    if (idle) {
      unsigned t = 0;
      if (lane == 0) t = atomicAdd(&cv.ticket[1], (unsigned)__popc(idle));
      t = __shfl_sync(FULL, t, 0) + __popc(idle & ((1u << lane) - 1u));
      if (status == 0) {
        if ((int)t < total) {
          tk = cv.tk_short[t];
          status = 2;
          child = -1;
        } else {
          status = 3;
        }
      }
    }
    if (!__any_sync(FULL, status != 3)) return;
    bool moved = false;
    if (status == 2) {
      const int k = cv.ord[tk.y - 1];
      const int nd = ndon[k];
      Gather g;
      if (g.take(k, nd, child, fin.base(k), don, a)) {
        double acc = g.first;
        if (child >= 0) acc = acc + ac;
#pragma unroll
        for (int u = 0; u < 7; ++u)
          if (u < g.nrest) acc = acc + g.rest[u];
        const double ax = Fin::kAux ? fin.aux(k) : 0.0;
        const unsigned fl = (rec[k] == k ? 1u : 0u) | fin.prop(k);
        ac = fin.value(acc, ax, fl);
        fin.side(k, acc, ax, fl);
        st_relaxed_gpu(&a[k], publishable(ac));
        child = k;
        moved = true;
        if (--tk.y <= tk.x) status = 0;
      }
    }
    if (!__any_sync(FULL, moved)) {
      if (__any_sync(FULL, pat.over(cv.err))) return;
      pat.rest();
    } else {
      pat = Patience{};
    }
  }
}

// chains of one node, before the others
template <class Fin>
__global__ void k_bottom_up_leaves(int nn, const int* __restrict__ rec, const int* __restrict__ ndon,
                                   const unsigned char* __restrict__ head, Fin fin, double* __restrict__ a) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    if (ndon[k] != 0 || !head[k]) continue;
    const double acc = fin.base(k), ax = Fin::kAux ? fin.aux(k) : 0.0;
    const unsigned fl = (rec[k] == k ? 1u : 0u) | fin.prop(k);
    fin.side(k, acc, ax, fl);
    a[k] = publishable(fin.value(acc, ax, fl));
  }
}

template <class U>
void path_sums(Ctx& c, U* marks, U* scan) {
  const int nn = c.nn;
  cudaStream_t st = c.stream;
  cudaMemsetAsync(marks, 0, sizeof(U) * ((size_t)nn + 1), st);
  k_path_marks<U><<<grid1d(nn), kBlock, 0, st>>>(nn, c.rec, c.ndon, c.don, c.pos, c.size, marks, c.ch_head, c.d_err);
  if constexpr (sizeof(U) == 4) exclusive_scan_u32(c, marks, scan, (size_t)nn + 1);
  else exclusive_scan_u64(c, marks, scan, (size_t)nn + 1);
  k_hf_order<U><<<grid1d(nn), kBlock, 0, st>>>(nn, scan, c.pos, c.ch_head, c.ch_ord, c.ch_flag, c.ch_depth, c.d_err);
  c.count_launch(2);
}

}  // namespace

// Builds the heavy-first order and both ticket lists for the current receiver
// forest (rec, ndon, don, stack positions and sizes must be current).
void build_chains(Ctx& c) {
  const int nn = c.nn;
  cudaStream_t st = c.stream;
  if (nn < 1 << 27) path_sums(c, reinterpret_cast<unsigned*>(c.ch_val), reinterpret_cast<unsigned*>(c.ch_val2));
  else path_sums(c, c.ch_val, c.ch_val2);
  int* scan = reinterpret_cast<int*>(c.ch_val);
  exclusive_scan_int(c, c.ch_flag, scan, (size_t)nn + 1);
  const int* nchains = scan + nn;
  k_chain_list<<<grid1d(nn), kBlock, 0, st>>>(nn, c.ch_flag, scan, c.ch_start);
  int *hist = c.ch_hist, *cur_td = hist + kHist, *cur_bu = cur_td + kHist;
  cudaMemsetAsync(hist, 0, sizeof(int) * kHist, st);
  const unsigned blocks = (unsigned)((nn + kChainsPerBlock - 1) / kChainsPerBlock);
  k_chain_hist<<<blocks, kChainBlock, 0, st>>>(nn, nchains, c.ch_start, c.ch_depth, hist);
  k_chain_offsets<<<1, kBuckets, 0, st>>>(hist, cur_td, cur_bu, c.ch_totals);
  k_chain_tickets<<<blocks, kChainBlock, 0, st>>>(nn, nchains, c.ch_start, c.ch_depth, c.ch_ord, c.rec, cur_td, cur_bu,
                                                  c.ch_tk[0], c.ch_tk[1], c.ch_tk[2], c.ch_tk[3]);
  c.count_launch(4);
}

void ensure_chains(Ctx& c) {
  if (!c.chains_valid) {
    build_chains(c);
    c.chains_valid = true;
  }
}

// Blocks of a chain sweep: one per 512 nodes up to 4 per SM; a quarter of that
// beside other instances (fsb_set_concurrency), whose kernels need the SMs that
// waiting blocks would hold.
static int sweep_blocks(const Ctx& c) {
  const int want = c.nn / (512 * c.launch_share) + 1;
  return std::min(want, 148 * 4);
}

static ChainView chain_view(Ctx& c, bool top_down) {
  cudaMemsetAsync(c.ticket, 0, 2 * sizeof(unsigned), c.stream);
  return ChainView{c.ch_ord, c.ch_tk[top_down ? 0 : 2], c.ch_tk[top_down ? 1 : 3], c.ch_totals, c.ticket, c.d_err};
}

template <class Op>
static void top_down(Ctx& c, const Op& op) {
  const ChainView cv = chain_view(c, true);
  k_top_down<Op><<<sweep_blocks(c), kSweepThreads, 0, c.stream>>>(cv, op);
  k_top_down_leaves<Op><<<grid1d(c.nn), kBlock, 0, c.stream>>>(c.nn, c.rec, c.ndon, c.ch_head, op, c.d_err);
  c.count_launch(2);
}

template <class Fin>
static void bottom_up(Ctx& c, const Fin& fin, double* a) {
  cudaMemsetAsync(a, 0xff, sizeof(double) * c.nn, c.stream);
  const ChainView cv = chain_view(c, false);
  k_bottom_up_leaves<Fin><<<grid1d(c.nn), kBlock, 0, c.stream>>>(c.nn, c.rec, c.ndon, c.ch_head, fin, a);
  k_bottom_up<Fin><<<sweep_blocks(c), kSweepThreads, 0, c.stream>>>(cv, c.rec, c.ndon, c.don, fin, a);
  c.count_launch(2);
}

void fill_chains(Ctx& c) {
  stage_begin(c, KT_FILL);
  cudaMemsetAsync(c.hwater, 0xff, sizeof(double) * c.nn, c.stream);
  top_down(c, FillOp{c.h, c.hwater, c.lake_depth});
  stage_end(c, KT_FILL);
}

void area_chains(Ctx& c) { bottom_up(c, AreaFin{c.precip, c.dx * c.dy}, c.a); }

void flux_chains(Ctx& c, double* flux) { bottom_up(c, FluxFin{c.erate}, flux); }

void chi_chains(Ctx& c, double a0, double mn, double* chi) {
  cudaMemsetAsync(chi, 0xff, sizeof(double) * c.nn, c.stream);
  top_down(c, ChiOp{c.a, c.length, a0, mn, chi});
}

template <int MODE, bool GS>
static void spl_mode(Ctx& c, const double* fact, double* hnew, const double* elev, const double* hstart, int* sill,
                     double* contrib) {
  top_down(c, SplOp<MODE, GS>{c.h, fact, c.n, 0.875 / c.n, hnew, c.water, elev, hstart, sill, contrib, c.d_err});
}

template <bool GS>
static void spl_sweep(Ctx& c, double* hnew, const double* elev, const double* hstart, int* sill, double* contrib) {
  const int n1 = fabs(c.n - 1.0) < 2.2250738585072014e-308;
  double* fact = reinterpret_cast<double*>(c.ch_val2);
  k_spl_factor<<<grid1d(c.nn), kBlock, 0, c.stream>>>(c.nn, n1, c.rec, c.h, c.b, c.kf, c.a, c.length, c.kfsed, c.dt,
                                                      c.m, c.n, fact);
  c.count_launch();
  cudaMemsetAsync(hnew, 0xff, sizeof(double) * c.nn, c.stream);
  cudaMemsetAsync(c.water, 0xff, sizeof(double) * c.nn, c.stream);
  if (GS) cudaMemsetAsync(sill, 0xff, sizeof(int) * c.nn, c.stream);
  if (n1) spl_mode<0, GS>(c, fact, hnew, elev, hstart, sill, contrib);
  else if (c.n == 1.5) spl_mode<1, GS>(c, fact, hnew, elev, hstart, sill, contrib);
  else spl_mode<2, GS>(c, fact, hnew, elev, hstart, sill, contrib);
}

void spl_chains(Ctx& c, double* hnew) { spl_sweep<false>(c, hnew, nullptr, nullptr, nullptr, nullptr); }

void spl_chains_gs(Ctx& c, const double* elev, const double* hstart, double* hnew, int* sill, double* contrib) {
  spl_sweep<true>(c, hnew, elev, hstart, sill, contrib);
}

void gs_erosion_chains(Ctx& c, const double* hp, const int* sill, double* lsed, double* dh) {
  bottom_up(c, GsFin{c.h, hp, sill, lsed}, dh);
}

void lake_volume_chains(Ctx& c, const int* sill, const double* contrib, double* vol, double* up) {
  bottom_up(c, VolFin{sill, contrib, vol}, up);
}

}  // namespace fsb
