// Flow routing kernels: uplift, steepest-descent receivers, donor lists and the
// depth-first stack (DFS preorder) of the receiver forest.
//
// Reference routines restated here (file:line in fastscapelib-fortran):
//   Uplift                 src/Uplift.f90:9-10
//   find_receiver          src/FlowRouting.f90:302-362
//   find_donor             src/FlowRouting.f90:366-389 (= loc_min_3_find_donors,
//                          src/LocalMinima.f90:881-900)
//   find_stack(+recursion) src/FlowRouting.f90:393-443 (= loc_min_3_find_stack,
//                          src/LocalMinima.f90:904-923,1050-1067)
//
// The stack is the DFS preorder of the receiver forest with roots in ascending
// node order and children (donors) in ascending node order.  Instead of the
// reference's recursion it is built from the Euler tour of the forest: every
// node k contributes an enter event E(k)=2k and an exit event X(k)=2k+1, the
// tour successor of each event is local information (first donor, next
// sibling, parent, next root), and list ranking (in tiles first) counts the
// enter events from each event to the end of the tour.  That count gives the
// preorder position and the subtree size of every node exactly.
#include "fsb_kernels.cuh"

namespace fsb {

// ---------------------------------------------------------------------------
// Uplift: h += u*dt ; b += u*dt   (no FMA: the library is built --fmad=false)
__global__ void k_uplift(int nn, double dt, const double* __restrict__ u, double* __restrict__ h,
                         double* __restrict__ b) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const double du = u[k] * dt;
    h[k] = h[k] + du;
    b[k] = b[k] + du;
  }
}

// find_receiver: one thread per node, 3x3 stencil, jj outer / ii inner, the
// first strictly steeper neighbour wins (smax starts at tiny(1d0)).  Lengths
// come from the 3x3 table `ltab` computed on the host exactly like the
// reference's sqrt((dx*ii)**2+(dy*jj)**2).
__global__ void k_find_receiver(Bounds bd, const double* __restrict__ h, const double* __restrict__ ltab,
                                int* __restrict__ rec, double* __restrict__ length) {
  const int nx = bd.nx, ny = bd.ny;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  const int ij = i + j * nx;
  int r = ij;
  double len = 0.0;
  if (i >= bd.i1 && i <= bd.i2 && j >= bd.j1 && j <= bd.j2) {
    const double hij = h[ij];
    double smax = 2.2250738585072014e-308;
#pragma unroll
    for (int jj = -1; jj <= 1; ++jj) {
      const int jjj = wrap_clamp(j + jj, ny, bd.ycyc);
#pragma unroll
      for (int ii = -1; ii <= 1; ++ii) {
        const int iii = wrap_clamp(i + ii, nx, bd.xcyc);
        const int ijk = iii + jjj * nx;
        if (ijk != ij) {
          const double l = ltab[(jj + 1) * 3 + (ii + 1)];
          const double slope = (hij - h[ijk]) / l;
          if (slope > smax) {
            smax = slope;
            r = ijk;
            len = l;
          }
        }
      }
    }
  }
  rec[ij] = r;
  length[ij] = len;
}

// Donor lists by gathering: the receiver of any node is one of its 3x3
// (wrapped) neighbours, so node k's donors are the neighbours d with
// rec[d]==k and d!=k.  They are emitted in ascending node order, which is the
// order of the reference's scatter loop over ij=1..nn.
__global__ void k_find_donors(Bounds bd, const int* __restrict__ rec, int* __restrict__ ndon,
                              int* __restrict__ don) {
  const int nx = bd.nx, ny = bd.ny;
  const int nn = nx * ny;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const int j = k / nx, i = k - j * nx;
    if (i > 0 && i < nx - 1 && j > 0 && j < ny - 1) {  // the neighbours in ascending order
      const int q[8] = {k - nx - 1, k - nx, k - nx + 1, k - 1, k + 1, k + nx - 1, k + nx, k + nx + 1};
      int r[8], d[8], n = 0;
#pragma unroll
      for (int t = 0; t < 8; ++t) r[t] = rec[q[t]];
#pragma unroll
      for (int t = 0; t < 8; ++t) d[t] = -1;
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (r[t] == k) {
#pragma unroll
          for (int u = 0; u <= t; ++u)
            if (u == n) d[u] = q[t];
          ++n;
        }
      ndon[k] = n;
      int4* row = reinterpret_cast<int4*>(don + (size_t)k * 8);
      row[0] = make_int4(d[0], d[1], d[2], d[3]);
      row[1] = make_int4(d[4], d[5], d[6], d[7]);
      continue;
    }
    int cand[8];
    int nc = 0;
    // Distinct neighbours in the wrapped 3x3 block (rows/columns that fall off
    // a non-cyclic edge do not exist).
    int rows[3], nr = 0, cols[3], ncl = 0;
    for (int d = -1; d <= 1; ++d) {
      int jj = j + d;
      if (jj < 0) { if (!bd.ycyc) continue; jj += ny; }
      if (jj >= ny) { if (!bd.ycyc) continue; jj -= ny; }
      bool dup = false;
      for (int t = 0; t < nr; ++t) dup |= rows[t] == jj;
      if (!dup) rows[nr++] = jj;
    }
    for (int d = -1; d <= 1; ++d) {
      int ii = i + d;
      if (ii < 0) { if (!bd.xcyc) continue; ii += nx; }
      if (ii >= nx) { if (!bd.xcyc) continue; ii -= nx; }
      bool dup = false;
      for (int t = 0; t < ncl; ++t) dup |= cols[t] == ii;
      if (!dup) cols[ncl++] = ii;
    }
    for (int a = 0; a < nr; ++a)
      for (int c = 0; c < ncl; ++c) {
        const int q = cols[c] + rows[a] * nx;
        if (q != k && rec[q] == k && nc < 8) cand[nc++] = q;
      }
    // insertion sort (<= 8 entries)
    for (int x = 1; x < nc; ++x) {
      const int v = cand[x];
      int y = x - 1;
      while (y >= 0 && cand[y] > v) { cand[y + 1] = cand[y]; --y; }
      cand[y + 1] = v;
    }
    ndon[k] = nc;
    for (int x = 0; x < 8; ++x) don[(size_t)k * 8 + x] = x < nc ? cand[x] : -1;
  }
}

// root flags (rec==self) for the compaction of the ascending root list
__global__ void k_root_flags(int nn, const int* __restrict__ rec, int* __restrict__ flag) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x)
    flag[k] = rec[k] == k ? 1 : 0;
}

// After an exclusive scan of the root flags: rank of each root and root list.
__global__ void k_root_list(int nn, const int* __restrict__ rec, const int* __restrict__ scan,
                            int* __restrict__ roots, int* __restrict__ root_rank) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x)
    if (rec[k] == k) {
      roots[scan[k]] = k;
      root_rank[k] = scan[k];
    }
}

// ---- list ranking by sublist walks (long lists) --------------------------------
// Entry e's result is the suffix sum of the weights from e to its list's end.
// Splitters: one of every STRIDE entries and every head (an entry that is no
// entry's successor).  In the basin tree's list it is drawn from the group's number:
// the way back along a chain of basins sorted by height visits odd entries only,
// and with every STRIDE-th entry met no splitter at all (B200, 3 x 60000 nodes: one
// walk of 18,000 steps, 2.7 ms of a LocalMinima of 3.6, now 0.95).  The elements of
// the Euler tour's paths come in the order of atomics; there the first of every
// group does, and drawing it costs the stack of 12 x 30000 nodes 10 %.  Each splitter walks its sublist up to the next
// splitter, writing for every entry (splitter id << 32 | prefix), the prefix
// being the weights before the entry within the sublist, and records
// (next splitter id << 32 | sublist total).  The splitters' list is ranked in
// the same way, down to a list that one block ranks in shared memory; entry
// e's result is its splitter's suffix sum minus its prefix.  O(n) work.
// Ranking by pointer jumping alone, or over the first splitters, took one
// launch per doubling: 42 launches and 133 us of 101^2's step, now 9 and 81,
// the basin tree's list among them.

// Head slots of a splitter list that no head took are inert: no list holds
// them, and in the next list they must not pass for heads themselves (counted
// as heads they fill that list's slots, one level after the other).
constexpr unsigned kInert = 0xfffffffeu;

// flags every entry that is some entry's successor, and the inert ones; the
// next list's head slots start inert
__global__ void k_rank_pred(size_t n, const unsigned long long* __restrict__ lst, unsigned char* __restrict__ pred,
                            unsigned long long* __restrict__ sub, unsigned long long* __restrict__ spl, size_t s0) {
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (size_t e = tid; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const unsigned nx = (unsigned)(lst[e] >> 32);
    if (nx < n) pred[nx] = 1;
    if (nx == kInert) {
      pred[e] = 1;
      sub[e] = 0;  // not walked unless a splitter; k_rank_final reads it
    }
  }
  if (tid < (size_t)kRankMaxHeads) spl[s0 + tid] = (unsigned long long)kInert << 32;
}

// splitter of group t of a list of n
template <int STRIDE, bool DRAWN>
__host__ __device__ inline size_t rank_splitter(unsigned t, size_t n) {
  if (!DRAWN) return (size_t)t * STRIDE;
  unsigned x = t * 0x9e3779b1u;
  x ^= x >> 15;
  x *= 0x85ebca77u;
  const size_t base = (size_t)t * STRIDE, e = base + (x >> (STRIDE == 16 ? 28 : 30));
  return e < n ? e : base;
}

// one sublist walk from splitter entry e with splitter id `id`; every step is
// one dependent load, and the walk ends within n steps
template <int STRIDE, bool DRAWN>
__device__ void rank_walk(size_t n, const unsigned long long* __restrict__ lst, unsigned long long* __restrict__ sub,
                          unsigned long long* __restrict__ spl, size_t e, unsigned id, int* err) {
  const unsigned END = 0xffffffffu;
  unsigned pre = 0, nid = END;
  size_t x = e;
  unsigned long long cur = lst[x];
  for (size_t steps = 0;; ++steps) {
    sub[x] = ((unsigned long long)id << 32) | pre;
    pre += (unsigned)cur;
    const unsigned nx = (unsigned)(cur >> 32);
    if (nx == END) break;
    if (nx == kInert) {
      nid = kInert;
      break;
    }
    if (nx >= n || steps >= n) {  // not a list
      atomicExch(err, DEV_STACK_ERROR);
      break;
    }
    cur = lst[nx];  // on its way while the splitter is told
    if (nx == rank_splitter<STRIDE, DRAWN>(nx / STRIDE, n)) {
      nid = nx / STRIDE;
      break;
    }
    x = nx;
  }
  spl[id] = ((unsigned long long)nid << 32) | pre;
}

// thread t: the splitter of group t, then any head among its other entries (one
// load of their flags)
template <int STRIDE, bool DRAWN>
__global__ void k_rank_walk(size_t n, size_t s0, const unsigned long long* __restrict__ lst,
                            const unsigned char* __restrict__ pred, unsigned long long* __restrict__ sub,
                            unsigned long long* __restrict__ spl, unsigned* nheads, int* err) {
  static_assert(STRIDE == 16 || STRIDE == 4, "one word of flags per splitter");
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < s0; t += (size_t)gridDim.x * blockDim.x) {
    const size_t base = t * STRIDE, own = rank_splitter<STRIDE, DRAWN>((unsigned)t, n);
    rank_walk<STRIDE, DRAWN>(n, lst, sub, spl, own, (unsigned)t, err);
    unsigned f[STRIDE / 4];
    if constexpr (STRIDE == 16) {
      const uint4 f4 = *reinterpret_cast<const uint4*>(pred + base);
      f[0] = f4.x; f[1] = f4.y; f[2] = f4.z; f[3] = f4.w;
    } else {
      f[0] = *reinterpret_cast<const unsigned*>(pred + base);
    }
#pragma unroll
    for (int j = 0; j < STRIDE; ++j) {
      const size_t e = base + j;
      if (e >= n || e == own || ((f[j >> 2] >> (8 * (j & 3))) & 0xffu) != 0u) continue;
      const unsigned h = atomicAdd(nheads, 1u);
      if (h >= (unsigned)kRankMaxHeads) {
        atomicExch(err, DEV_OVERFLOW);
        continue;
      }
      rank_walk<STRIDE, DRAWN>(n, lst, sub, spl, e, (unsigned)(s0 + h), err);
    }
  }
}

// Pointer jumping over a whole list in one block's shared memory.
constexpr int kRankThreads = 512, kRankEach = kRankBlock / kRankThreads;
__global__ void __launch_bounds__(kRankThreads, 2) k_rank_block(int n, unsigned long long* __restrict__ lst) {
  extern __shared__ unsigned long long rank_sh[];
  const unsigned END = 0xffffffffu;
  const int tid = threadIdx.x;
  for (int e = tid; e < n; e += kRankThreads) rank_sh[e] = lst[e];
  __syncthreads();
  for (int r = 1; r < 2 * n; r <<= 1) {  // after round i a value covers 2^i entries
    unsigned long long v[kRankEach];
    bool moved = false;
#pragma unroll
    for (int i = 0; i < kRankEach; ++i) {
      const int e = tid + i * kRankThreads;
      if (e >= n) break;
      v[i] = rank_sh[e];
      const unsigned nx = (unsigned)(v[i] >> 32);
      if (nx == END || nx >= (unsigned)n) continue;
      const unsigned long long nb = rank_sh[nx];
      v[i] = (nb & 0xffffffff00000000ull) | (unsigned)((unsigned)v[i] + (unsigned)nb);
      moved = true;
    }
    if (!__syncthreads_or(moved)) break;
#pragma unroll
    for (int i = 0; i < kRankEach; ++i) {
      const int e = tid + i * kRankThreads;
      if (e >= n) break;
      rank_sh[e] = v[i];
    }
    __syncthreads();
  }
  for (int e = tid; e < n; e += kRankThreads) lst[e] = rank_sh[e];
}

// a device that refuses the block's shared memory: the step reports it
__global__ void k_rank_refused(int* err) { *err = DEV_OVERFLOW; }

__global__ void k_rank_final(size_t n, const unsigned long long* __restrict__ sub,
                             const unsigned long long* __restrict__ vs, unsigned long long* __restrict__ out) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const unsigned long long s = sub[e];
    out[e] = (unsigned long long)((unsigned)vs[s >> 32] - (unsigned)s);
  }
}

// ---- Euler tour, ranked in tiles first -----------------------------------------
// The tour visits entry 2k when it enters node k (weight 1) and 2k+1 when it
// leaves (weight 0): 2k is followed by the first donor's entry or by 2k+1, 2k+1
// by the next donor of k's receiver, by the receiver's exit, or for a root by
// the next root.  Suffix sums of the weights give the stack's positions.
// Successors are nearly always neighbours, so a block takes a tile of 2048 nodes
// and jumps pointers in shared memory: every entry learns the last entry of its
// path inside the tile and the weight up to there.  Only the paths go to the list
// ranking, one element each.  A path can leave a tile from its two outermost rings
// of nodes (donors and receivers are one node away, siblings two) or from the last
// root of a row, hence TourTiles::slots.
//
// Measured (B200): walking all 2 nn entries in random order took 595 us twice
// per step of 2049^2, the tiles and their paths' ranking 190.  The stack of
// 1023x767 329 -> 151 us, of 101^2 68 -> 62; the stack after LocalMinima gains
// more, its walks being longer.  Strips' tiles follow their shorter side: tiles of
// 64 x 32 gave a strip under 12 nodes wide a longer list than the 2 nn entries (3 x
// 60000: stack 126 us with those, 165 so, 80 with tiles of 4 x 512).
constexpr int kTourThreads = 512;

__global__ void __launch_bounds__(kTourThreads) k_tour_tiles(int nx, int ny, TourTiles tt,
                                                             const int* __restrict__ rec,
                                                             const int* __restrict__ ndon,
                                                             const int* __restrict__ don,
                                                             const int* __restrict__ roots,
                                                             const int* __restrict__ root_rank,
                                                             const int* __restrict__ nroots,
                                                             unsigned* __restrict__ head_slot,
                                                             unsigned* __restrict__ info,
                                                             unsigned* __restrict__ list, int* __restrict__ err) {
  constexpr unsigned END = 0xffffffffu;
  constexpr int kEach = kTourNodes / kTourThreads;
  __shared__ unsigned path[2 * kTourNodes];  // furthest entry known << 16 | weight before it
  __shared__ unsigned short slot[2 * kTourNodes];
  __shared__ unsigned char inner[2 * kTourNodes];  // has a predecessor in the tile
  __shared__ int count;
  const int tid = threadIdx.x;
  const int tx = 1 << tt.lx, ty = 1 << tt.ly, x0 = blockIdx.x << tt.lx, y0 = blockIdx.y << tt.ly;
  const unsigned tile = blockIdx.y * gridDim.x + blockIdx.x, first = tile * tt.slots;
  const int R = *nroots;
  if (tid == 0) count = 0;
  for (int e = tid; e < 2 * kTourNodes / 4; e += kTourThreads) reinterpret_cast<unsigned*>(inner)[e] = 0u;
  unsigned next[2 * kEach];
  bool valid[kEach];
  int node[kEach];
#pragma unroll
  for (int n = 0; n < kEach; ++n) {
    const int ln = tid + n * kTourThreads, x = x0 + (ln & (tx - 1)), y = y0 + (ln >> tt.lx);
    valid[n] = x < nx && y < ny;
    const int k = x + y * nx;
    node[n] = k;
    if (!valid[n]) continue;
    next[2 * n] = ndon[k] > 0 ? 2u * (unsigned)don[(size_t)k * 8] : 2u * (unsigned)k + 1u;
    const int r = rec[k];
    if (r != k) {
      const int4* row = reinterpret_cast<const int4*>(don + (size_t)r * 8);
      const int4 a = row[0], b = row[1];
      const int d[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      const int nd = ndon[r];
      unsigned nxt = 2u * (unsigned)r + 1u;
#pragma unroll
      for (int i = 0; i < 7; ++i)
        if (d[i] == k && i + 1 < nd) nxt = 2u * (unsigned)d[i + 1];
      next[2 * n + 1] = nxt;
    } else {
      const int rr = root_rank[k];
      next[2 * n + 1] = rr + 1 < R ? 2u * (unsigned)roots[rr + 1] : END;
    }
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < kEach; ++n)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int e = 2 * (tid + n * kTourThreads) + b;
      unsigned to = (unsigned)e;  // the path's last entry points to itself
      if (valid[n] && next[2 * n + b] != END) {
        const int q = (int)(next[2 * n + b] >> 1), qy = q / nx, lx = q - qy * nx - x0, ly = qy - y0;
        if (lx >= 0 && lx < tx && ly >= 0 && ly < ty) {
          to = 2u * (unsigned)((ly << tt.lx) + lx) + (next[2 * n + b] & 1u);
          inner[to] = 1;
        }
      }
      path[e] = to << 16 | (to == (unsigned)e || b ? 0u : 1u);
      slot[e] = 0;
    }
  __syncthreads();
  // a word is read and written whole and is right before and after every jump,
  // so the jumps need no order; 2 * kTourNodes entries take 12 doublings
  for (int round = 0; round < 13; ++round) {
    bool moved = false;
#pragma unroll
    for (int n = 0; n < 2 * kEach; ++n) {
      const unsigned e = 2u * (tid + (n >> 1) * kTourThreads) + (n & 1);
      const unsigned u = *(volatile unsigned*)&path[e], v = *(volatile unsigned*)&path[u >> 16];
      if (v >> 16 != u >> 16) {
        *(volatile unsigned*)&path[e] = (v & 0xffff0000u) | ((u & 0xffffu) + (v & 0xffffu));
        moved = true;
      }
    }
    if (!__syncthreads_or(moved)) break;
  }
#pragma unroll
  for (int n = 0; n < kEach; ++n)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const unsigned e = 2u * (tid + n * kTourThreads) + b;
      if (valid[n] && path[e] >> 16 == e) {
        const int s = atomicAdd(&count, 1);
        if (s < tt.slots) {
          slot[e] = (unsigned short)s;
          list[2 * (size_t)(first + s) + 1] = next[2 * n + b];
        } else {
          atomicExch(err, DEV_OVERFLOW);
        }
      }
    }
  __syncthreads();
  for (int s = count + tid; s < tt.slots; s += kTourThreads) {
    list[2 * (size_t)(first + s)] = 0u;
    list[2 * (size_t)(first + s) + 1] = kInert;
  }
#pragma unroll
  for (int n = 0; n < kEach; ++n) {
    if (!valid[n]) continue;
    unsigned word[2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const unsigned e = 2u * (tid + n * kTourThreads) + b, u = path[e], t = u >> 16;
      const unsigned s = slot[t], w = (u & 0xffffu) + (t & 1u ? 0u : 1u);
      word[b] = s << 16 | w;
      if (!inner[e]) {  // the path's first entry
        head_slot[2 * (size_t)node[n] + b] = first + s;
        list[2 * (size_t)(first + s)] = w;
      }
    }
    reinterpret_cast<uint2*>(info)[node[n]] = make_uint2(word[0], word[1]);
  }
}

// the paths' successors become list elements; keeps the paths' weights
__global__ void k_tour_link(int nn, size_t n, const unsigned* __restrict__ head_slot,
                            unsigned long long* __restrict__ list, unsigned* __restrict__ weight) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const unsigned long long v = list[i];
    const unsigned s = (unsigned)(v >> 32);
    weight[i] = (unsigned)v;
    if (s < 2u * (unsigned)nn) list[i] = (unsigned long long)head_slot[s] << 32 | (unsigned)v;
  }
}

// preorder position and subtree size from the ranks of the enter/exit entries
__global__ void k_stack_from_tiles(int nx, int ny, TourTiles tt, const unsigned* __restrict__ info,
                                   const unsigned long long* __restrict__ ranks, const unsigned* __restrict__ weight,
                                   int* __restrict__ pos, int* __restrict__ size, int* __restrict__ stack,
                                   int* __restrict__ err) {
  const int nn = nx * ny;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const int y = k / nx, x = k - y * nx;
    const size_t first = (size_t)((y >> tt.ly) * tt.tiles_x + (x >> tt.lx)) * tt.slots;
    const uint2 w = reinterpret_cast<const uint2*>(info)[k];
    const size_t se = first + (w.x >> 16), sx = first + (w.y >> 16);
    // from the path's first entry, less what lies before this one
    const unsigned re = (unsigned)ranks[se] - weight[se] + (w.x & 0xffffu);
    const unsigned rx = (unsigned)ranks[sx] - weight[sx] + (w.y & 0xffffu);
    const int p = nn - (int)re;
    if (p < 0 || p >= nn) { atomicExch(err, DEV_STACK_ERROR); continue; }
    pos[k] = p;
    size[k] = (int)(re - rx);
    stack[p] = k;
  }
}

// ---------------------------------------------------------------------------
// host launchers

void launch_uplift(Ctx& c) {
  k_uplift<<<grid1d(c.nn), kBlock, 0, c.stream>>>(c.nn, c.dt, c.u, c.h, c.b);
  c.count_launch();
}

void launch_find_receiver(Ctx& c, const double* h, int* rec, double* length) {
  dim3 blk(32, 8);
  dim3 grd((c.nx + 31) / 32, (c.ny + 7) / 8);
  k_find_receiver<<<grd, blk, 0, c.stream>>>(c.bd, h, c.ltab, rec, length);
  c.count_launch();
}

void launch_find_donors(Ctx& c, const int* rec, int* ndon, int* don) {
  k_find_donors<<<grid1d(c.nn), kBlock, 0, c.stream>>>(c.bd, rec, ndon, don);
  c.count_launch();
}

// Ranks list a (n packed entries) in place; sub holds n entries, ws the scratch
// of the shorter lists.  DRAWN: the splitters of every level are.
template <bool DRAWN>
static void rank_list(Ctx& c, size_t n, unsigned long long* a, unsigned long long* sub, unsigned long long* ws) {
  if (n <= (size_t)kRankBlock) {
    int len = (int)n;
    void* args[] = {&len, &a};
    if (!BigSmem<k_rank_block>::launch(1, kRankThreads, sizeof(unsigned long long) * n,
                                       (int)sizeof(unsigned long long) * kRankBlock, c.stream, args))
      k_rank_refused<<<1, 1, 0, c.stream>>>(c.d_err);
    c.count_launch();
    return;
  }
  // a splitter every 16 entries, or every 4 where that is enough: the longest
  // sublist, about stride * ln(splitters) entries, is the walk's time
  const bool coarse = n > 4 * ((size_t)kRankBlock - kRankMaxHeads);
  const size_t stride = coarse ? 16 : 4, s0 = (n + stride - 1) / stride, n1 = s0 + kRankMaxHeads;
  unsigned long long* spl = ws;
  cudaMemsetAsync(c.s_rank_pred, 0, s0 * stride, c.stream);  // whole flag words past n too
  cudaMemsetAsync(c.s_rank_nheads, 0, sizeof(unsigned), c.stream);
  k_rank_pred<<<grid1d(n), kBlock, 0, c.stream>>>(n, a, c.s_rank_pred, sub, spl, s0);
  const unsigned blocks = (unsigned)((s0 + 127) / 128);
  const auto walk = coarse ? k_rank_walk<16, DRAWN> : k_rank_walk<4, DRAWN>;
  walk<<<blocks, 128, 0, c.stream>>>(n, s0, a, c.s_rank_pred, sub, spl, c.s_rank_nheads, c.d_err);
  rank_list<DRAWN>(c, n1, spl, ws + n1, ws + 2 * n1);
  k_rank_final<<<grid1d(n), kBlock, 0, c.stream>>>(n, sub, spl, a);
  c.count_launch(3);
}

// Suffix sums of `n` <= 2*nn packed entries (succ << 32 | weight) in the low
// words of the returned buffer, a; b holds as many entries of scratch.
unsigned long long* list_rank(Ctx& c, size_t n, unsigned long long* a, unsigned long long* b) {
  rank_list<true>(c, n, a, b, c.s_rank_ws);
  return a;
}

// Builds ndon/don/stack(+pos,size) for the receiver array `rec`.
void build_stack(Ctx& c, const int* rec, int* ndon, int* don, int* stack, int* pos, int* size) {
  const int nn = c.nn;
  launch_find_donors(c, rec, ndon, don);
  k_root_flags<<<grid1d(nn), kBlock, 0, c.stream>>>(nn, rec, c.s_flag);
  c.count_launch();
  exclusive_scan_int(c, c.s_flag, c.s_scan, nn + 1);  // s_scan[nn] = number of roots
  k_root_list<<<grid1d(nn), kBlock, 0, c.stream>>>(nn, rec, c.s_scan, c.s_roots, c.s_root_rank);
  c.count_launch();
  const TourTiles tt(c.nx, c.ny);
  const dim3 tiles(tt.tiles_x, tt.tiles_y);
  const size_t n = tt.elements();
  unsigned* head_slot = reinterpret_cast<unsigned*>(c.s_list_a);
  unsigned* info = head_slot + 2 * (size_t)nn;
  k_tour_tiles<<<tiles, kTourThreads, 0, c.stream>>>(c.nx, c.ny, tt, rec, ndon, don, c.s_roots, c.s_root_rank, c.s_scan + nn,
                                                     head_slot, info, reinterpret_cast<unsigned*>(c.s_tour), c.d_err);
  k_tour_link<<<grid1d(n), kBlock, 0, c.stream>>>(nn, n, head_slot, c.s_tour, c.s_tour_weight);
  rank_list<false>(c, n, c.s_tour, c.s_tour_sub, c.s_rank_ws);
  k_stack_from_tiles<<<grid1d(nn), kBlock, 0, c.stream>>>(c.nx, c.ny, tt, info, c.s_tour, c.s_tour_weight, pos, size, stack,
                                                          c.d_err);
  c.count_launch(3);
}

}  // namespace fsb
