// Region-owned sweeps of the multiple-flow receiver DAG: drainage area and
// the implicit stream power law with g == 0.
//
// Reference loops restated (fastscapelib-fortran file:line):
//   FlowAccumulation (MFD)   src/FlowRouting.f90:97-119
//   StreamPowerLaw (MFD)     src/StreamPowerLaw.f90:89-177 (g == 0: one
//                            Gauss-Seidel pass, elev = ht)
//
// Both sweeps are recurrences along the receiver DAG whose critical path is
// about three grid sides long, so their time is the number of hops on that
// path times the latency of one hop, plus what the nodes of the wave front
// cost the SMs that own them.  The grid is cut into square tiles dealt out
// over one CTA per SM (cooperative launch, all co-resident), so that the
// front, wherever it runs, is spread over all SMs.  A CTA keeps its nodes'
// dependency counters in shared memory and hands ready nodes to its warps
// through a queue that its L1 serves; eight lanes compute one node.  What a
// node needs beyond its inputs' values is one 96-byte record, built in
// parallel before the sweep and brought into L1 by the nodes it waits for.
// A value that crosses a tile edge is written into a mailbox cell of the
// neighbouring tile, whose CTA polls a flag bit per cell: the value itself
// says whether it has arrived, so no fence beyond CTA scope runs during a
// sweep (a fence at GPU scope would empty the SM's L1).  The arithmetic of a
// node, including the order of its sums, is that of the queue engine in
// fsb_flow.cu, so both engines give bit-identical results in FP64 (the mixed form's
// FP32 sweeps are this engine's alone).
//
// What bounds them (2049^2, B200, a trace of every node's start and end
// followed back from the last one): the path is about 6,000 hops, 90 % of
// them continuations inside one warp.  A stream-power hop is about 750 cycles
// for each Newton iteration (a root, two exchanges, sixteen additions in
// order, a quotient) and about 800 between the value and the next node's
// start; an area hop about 950 (records come from DRAM there) and 500.  150
// hops cross a tile, at 4,000 to 6,000 cycles each.  DRAM is idle.  Against the form
// with one tile per CTA, a warp per node and inboxes behind GPU-scope fences:
// area 6.9 -> 5.8 ms, stream power 12.0 -> 6.9 ms; 4097^2 (which took the
// queue engine) 36.1 -> 17.1 and 54.9 -> 20.6 ms with their records; 2049x1537
// closed basins, n = 1: 7.6 -> 6.1 and 24.0 -> 7.3 ms.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <type_traits>

#include "fsb_kernels.cuh"

namespace fsb {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr unsigned long long kRegionTimeLimitNs = 4000000000ull;  // a sweep giving up: 4 s

// Threads of a sweep CTA (warp 0 polls the flag words, the others compute
// nodes).  2049^2, B200: 384 threads 5.9 + 7.9 ms (area + stream power), 512
// threads 5.8 + 7.3, 768 threads 5.8 + 7.5.
constexpr int kThreads = 512;
// Grids whose records (96 bytes a node) L2 does not keep: the area sweep then brings
// the records two hops on into L2.  With / without that code, random surfaces:
// 1025^2 2.91 / 2.81 ms, 2049^2 5.46 / 5.84, 4097^2 30.2 / 32.9; reliefs 2.50 / 2.36,
// 5.29 / 5.23, 14.0 / 14.2.
constexpr int kL2Records = 1 << 20;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Loads under a predicate, without a branch (0 where it is off); the SM's L1
// may serve them (values written by this CTA)
__device__ __forceinline__ double ld_l1_if(const double* p, bool on) {
  double v;
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n mov.f64 %0, 0d0000000000000000;\n @q ld.global.f64 %0, [%1];\n}"
      : "=d"(v)
      : "l"(p), "r"((unsigned)on)
      : "memory");
  return v;
}
__device__ __forceinline__ float ld_l1_if(const float* p, bool on) {
  float v;
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n mov.f32 %0, 0f00000000;\n @q ld.global.f32 %0, [%1];\n}"
               : "=f"(v)
               : "l"(p), "r"((unsigned)on)
               : "memory");
  return v;
}
// the same for data written before the kernel; v keeps its value where the
// predicate is off
__device__ __forceinline__ void ldg_if(int4& v, const int4* p, bool on) {
  asm("{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n @q ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];\n}"
      : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
      : "l"(p), "r"((unsigned)on));
}
__device__ __forceinline__ void ldg_if(double& v, const double* p, bool on) {
  asm("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q ld.global.nc.f64 %0, [%1];\n}" : "+d"(v) : "l"(p), "r"((unsigned)on));
}
__device__ __forceinline__ void ldg_if(float& v, const float* p, bool on) {
  asm("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q ld.global.nc.f32 %0, [%1];\n}" : "+f"(v) : "l"(p), "r"((unsigned)on));
}
__device__ __forceinline__ void st_value(double* p, double v) {
  asm volatile("st.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_value(float* p, float v) {
  asm volatile("st.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_value(double2* p, double2 v) {
  asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
// queue entries: written and polled by one CTA, so L1 may hold them
__device__ __forceinline__ long long ld_queue(const long long* p) {
  long long v;
  asm volatile("ld.relaxed.cta.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_queue(long long* p, long long v) {
  asm volatile("st.relaxed.cta.global.s64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Brings the 32-byte sector at p into L1: a 16-byte copy whose destination
// nobody reads (prefetch.global.L1 left the sector in L2 only: the consumer's
// load still took an L2 round trip)
__device__ __forceinline__ void touch_l1_if(unsigned scratch, const void* p, bool on) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q cp.async.ca.shared.global [%0], [%1], 16;\n}" ::"r"(scratch),
      "l"(p), "r"((unsigned)on)
      : "memory");
}

// brings a record into L2
__device__ __forceinline__ void prefetch_l2_if(const void* p, bool on) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %1, 0;\n @q cp.async.bulk.prefetch.L2.global [%0], 64;\n}" ::"l"(p),
               "r"((unsigned)on)
               : "memory");
}

// four flag words
__device__ __forceinline__ void ld_flags(const unsigned* p, unsigned (&v)[4]) {
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "l"(p)
               : "memory");
}

// mailbox cells: every word is all ones until its value has arrived
__device__ __forceinline__ bool mail_read(const double* p, double& v) {
  v = ld_relaxed_gpu(p);
  return __double_as_longlong(v) != -1ll;
}
__device__ __forceinline__ bool mail_read(const float* p, float& v) {
  v = __int_as_float(ld_relaxed_gpu(reinterpret_cast<const int*>(p)));
  return __float_as_int(v) != -1;
}
__device__ __forceinline__ bool mail_read(const double2* p, double2& v) {
  const double* d = reinterpret_cast<const double*>(p);
  v.x = ld_relaxed_gpu(d);
  v.y = ld_relaxed_gpu(d + 1);
  return __double_as_longlong(v.x) != -1ll && __double_as_longlong(v.y) != -1ll;
}
__device__ __forceinline__ void mail_write(double* p, double v) { st_relaxed_gpu(p, publishable(v)); }
__device__ __forceinline__ void mail_write(float* p, float v) {
  const int b = __float_as_int(v);
  st_relaxed_gpu(reinterpret_cast<int*>(p), b == -1 ? 0x7fc00000 : b);
}
__device__ __forceinline__ void mail_write(double2* p, double2 v) {
  double* d = reinterpret_cast<double*>(p);
  st_relaxed_gpu(d, publishable(v.x));
  st_relaxed_gpu(d + 1, publishable(v.y));
}

// The eight neighbours in the order of the reference's loops (jj outer, ii
// inner, FlowRouting.f90:200-236): direction t, and 7 - t is its opposite.
// dir_code packs the offset as (dj + 1) << 2 | (di + 1).
__host__ __device__ constexpr int dir_di(int t) { return (t + (t >> 2)) % 3 - 1; }
__host__ __device__ constexpr int dir_dj(int t) { return (t + (t >> 2)) / 3 - 1; }
__host__ __device__ constexpr unsigned dir_code(int t) { return (unsigned)((dir_dj(t) + 1) << 2 | (dir_di(t) + 1)); }
// direction of offset (di, dj), not (0, 0)
__device__ __forceinline__ int dir_of(int di, int dj) {
  const int c = 3 * (dj + 1) + di + 1;
  return c - (c > 4 ? 1 : 0);
}

// One record per node: a 16-byte header, then the coefficients of its present
// inputs (at most 8, in input order).
//   codes  offset of input s (dir_code) in bits 4s..4s+3
//   meta   bits 0-3 number of inputs (stream power: kNoRec a root, kNoMrec no
//          receivers); 4-7 tile edges the node lies on (kWest ...); 8-15
//          directions of the dependents; 16-19 stream power: offset of rec(k)
//          and 20 whether it lies in another tile; 21-23 the dependent to
//          continue with; 24-31 inputs that lie in another tile
//   base   area: dx*dy*precip(k); stream power: ht(k)
//   c      area: summed weight of the donor's slots targeting k
//          stream power: kf*dt*(a*w)^m/l^n of the gated receiver slot
constexpr unsigned kNoMrec = 14, kNoRec = 15;
constexpr unsigned kWest = 1, kEast = 2, kSouth = 4, kNorth = 8;
// the edges beyond which the neighbour in direction (di, dj) lies in another tile
__device__ __forceinline__ unsigned edges_of(int di, int dj) {
  return (di < 0 ? kWest : di > 0 ? kEast : 0u) | (dj < 0 ? kSouth : dj > 0 ? kNorth : 0u);
}
template <class T>
struct RecordFields {
  unsigned codes, meta;
  double base;
  T c[8];
};
template <class T>
struct __align__(32) RecordT : RecordFields<T> {};
static_assert(sizeof(RecordT<double>) == 96 && sizeof(RecordT<float>) == 64, "whole 32-byte sectors");

// ---- record builders --------------------------------------------------------

// neighbour of (i, j) in direction t; false when it lies beyond a non-cyclic edge
__device__ __forceinline__ bool nbr_at(const Bounds& bd, int i, int j, int t, int& q) {
  int x = i + dir_di(t), y = j + dir_dj(t);
  if (x < 0) { if (!bd.xcyc) return false; x += bd.nx; }
  if (x >= bd.nx) { if (!bd.xcyc) return false; x -= bd.nx; }
  if (y < 0) { if (!bd.ycyc) return false; y += bd.ny; }
  if (y >= bd.ny) { if (!bd.ycyc) return false; y -= bd.ny; }
  q = x + y * bd.nx;
  return true;
}

// direction of q from k = (i, j), reporting a node that is no neighbour (-1)
__device__ inline int dir_to(const Bounds& bd, int i, int j, int q, int* err) {
  const int qj = q / bd.nx, qi = q - qj * bd.nx;
  int di = qi - i, dj = qj - j;
  if (di > 1) di -= bd.nx; else if (di < -1) di += bd.nx;
  if (dj > 1) dj -= bd.ny; else if (dj < -1) dj += bd.ny;
  if (di < -1 || di > 1 || dj < -1 || dj > 1 || (di == 0 && dj == 0)) {
    atomicExch(err, DEV_NOT_ADJACENT);
    return -1;
  }
  return dir_of(di, dj);
}

// the edges of its tile (or of the grid) that (i, j) lies on
__device__ __forceinline__ unsigned tile_edges(const Bounds& bd, int ts, int i, int j) {
  const int x = i & (ts - 1), y = j & (ts - 1);
  return (x == 0 ? kWest : 0u) | (x == ts - 1 || i == bd.nx - 1 ? kEast : 0u) | (y == 0 ? kSouth : 0u) |
         (y == ts - 1 || j == bd.ny - 1 ? kNorth : 0u);
}

// mmask[k] (k_mfd_receivers): bits 0-7 the loop directions that hold a
// receiver slot, in slot order; bits 8-15 the directions of the distinct
// receivers.  The two differ only beside a free, non-cyclic edge, where the
// reference lists a clamped neighbour again.

// A block builds the records of 32 x 8 nodes in shared memory and stores them as
// whole lines; built in place, word by word, k_acc_records took 328 us and
// k_spl_records 580 of 2049^2, now 236 and 462.
constexpr int kRecPitch = 104;  // bytes per record there: an odd number of double words
// node: its place among the block's 256.  The staged form carries the fields'
// own alignment only: at this pitch the compiler must not take the 16-byte
// header for one store.
template <class T>
__device__ __forceinline__ RecordFields<T>* staged_record(unsigned char* sm, int node) {
  using Staged = RecordFields<T>;
  static_assert(kRecPitch % alignof(Staged) == 0 && sizeof(RecordT<T>) <= kRecPitch, "every staged record is aligned");
  return reinterpret_cast<Staged*>(sm + node * kRecPitch);
}
template <class T>
__device__ __forceinline__ void store_records(const Bounds& bd, const unsigned char* sm, RecordT<T>* __restrict__ rec) {
  constexpr int kWords = sizeof(RecordT<T>) / 8;
  const int x0 = blockIdx.x * 32, row = blockIdx.y * 8 + threadIdx.y;  // a row of records per warp
  if (row >= bd.ny) return;
  const int words = min(32, bd.nx - x0) * kWords;
  double* out = reinterpret_cast<double*>(rec + (size_t)row * bd.nx + x0);
  for (int e = threadIdx.x; e < words; e += 32)
    out[e] = *reinterpret_cast<const double*>(sm + (threadIdx.y * 32 + e / kWords) * kRecPitch + e % kWords * 8);
}

// Area: inputs are k's distinct donors in direction order with the summed
// weight of their slots targeting k; dependents are k's distinct receivers.
template <class T>
__global__ void __launch_bounds__(256) k_acc_records(Bounds bd, int ts, double dxdy, const int* __restrict__ mmask,
                                                     const int* __restrict__ mrec, const double* __restrict__ mwrec,
                                                     const double* __restrict__ precip, RecordT<T>* __restrict__ rec,
                                                     unsigned short* __restrict__ wmeta) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
  __shared__ __align__(16) unsigned char sm[256 * kRecPitch];
  if (i < bd.nx && j < bd.ny) {
    const int k = i + j * bd.nx;
    const unsigned edges = tile_edges(bd, ts, i, j);
    unsigned codes = 0, far = 0;
    int n = 0;
    RecordFields<T>* r = staged_record<T>(sm, threadIdx.y * 32 + threadIdx.x);
  #pragma unroll
    for (int t = 0; t < 8; ++t) {
      int d;
      if (!nbr_at(bd, i, j, t, d)) continue;
      const int m = __ldg(&mmask[d]);
      const int ot = 7 - t;
      if (!((m >> (8 + ot)) & 1)) continue;
      const size_t o = (size_t)d * 8;
      double w;
      if ((m & 255) == (m >> 8)) {
        w = __ldg(&mwrec[o + __popc(m & ((1 << ot) - 1))]);
      } else {  // beside a free edge: d may list k twice
        const int nr = __popc(m & 255);
        int hits = 0;
        w = 0.0;
        for (int s = 0; s < nr; ++s)
          if (mrec[o + s] == k) {
            const double ws = mwrec[o + s];
            w = hits ? w + ws : ws;
            ++hits;
          }
      }
      codes |= dir_code(t) << (4 * n);
      far |= ((edges & edges_of(dir_di(t), dir_dj(t))) ? 1u : 0u) << n;
      r->c[n++] = (T)w;
    }
    const unsigned deps = (unsigned)(mmask[k] >> 8) & 255u;
    r->codes = codes;
    r->meta = (unsigned)n | (edges << 4) | (deps << 8) | (far << 24);
    r->base = dxdy * precip[k];
    wmeta[k] = (unsigned short)((unsigned)n | (deps << 8));
  }
  __syncwarp();
  store_records(bd, sm, rec);
}

// Stream power: inputs are k's gated receiver slots (ht(k) >= ht(q) for n = 1,
// > otherwise: the terms StreamPowerLaw.f90:108-114 / 152-158 include), in
// mrec slot order, duplicates kept; the counter also waits for rec(k), whose
// water the node compares against.  Dependents are the donors that read
// k's new elevation (gated) or its water (rec == k).
template <class T>
__global__ void __launch_bounds__(256) k_spl_records(
    Bounds bd, int ts, int n_is_one, double kfsed, double dt, double m, const int* __restrict__ recv,
    const int* __restrict__ mmask, const int* __restrict__ mrec, const double* __restrict__ mwrec,
    const double* __restrict__ mlrec, const double* __restrict__ h, const double* __restrict__ b,
    const double* __restrict__ kf, const double* __restrict__ a, const double* __restrict__ ltab,
    const T* __restrict__ lpow, RecordT<T>* __restrict__ rec, unsigned short* __restrict__ wmeta, int* err) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
  __shared__ __align__(16) unsigned char sm[256 * kRecPitch];
  __shared__ double factor[256];  // kf*dt
  __shared__ unsigned char slots[8][256];  // a row's slots whose powers are wanted: node << 3 | slot
  __shared__ unsigned short lens[256];  // two bits per slot
  const int me = threadIdx.y * 32 + threadIdx.x;
  int n = 0;
  if (i < bd.nx && j < bd.ny) {
    const int k = i + j * bd.nx;
    const double htk = h[k];
    const int mk = mmask[k];
    const int r = recv[k];
    const unsigned edges = tile_edges(bd, ts, i, j);
    unsigned codes = 0, waits = 0, far = 0, rcode = 0, lengths = 0;
    RecordFields<T>* out = staged_record<T>(sm, me);
    if (r != k) {
      factor[me] = ((kfsed > 0.0 && (htk - b[k]) > 1.0) ? kfsed : kf[k]) * dt;
      const double ak = a[k];
      const int nr = __popc(mk & 255);
      const size_t o = (size_t)k * 8;
      const bool plain = (mk & 255) == (mk >> 8);
      int dirs = mk & 255;
      for (int s = 0; s < nr; ++s) {
        int t = __ffs(dirs) - 1;  // the loop direction of slot s
        dirs &= dirs - 1;
        int q;
        double l;
        if (plain) {
          nbr_at(bd, i, j, t, q);
          l = __ldg(&ltab[t + (t >> 2)]);
        } else {  // a clamped neighbour keeps the length of its loop direction
          q = mrec[o + s];
          l = mlrec[o + s];
          t = dir_to(bd, i, j, q, err);
          if (t < 0) continue;
        }
        if (!(n_is_one ? (htk >= h[q]) : (htk > h[q]))) continue;
        const double w = mwrec[o + s];
        // the length is one of three values (diagonal at 0, dy at 1, dx at 3; equal
        // values have equal powers)
        const unsigned len = l == __ldg(&ltab[0]) ? 0u : l == __ldg(&ltab[1]) ? 1u : 3u;
        lengths |= len << (2 * n);
        codes |= dir_code(t) << (4 * n);
        far |= ((edges & edges_of((t + (t >> 2)) % 3 - 1, (t + (t >> 2)) / 3 - 1)) ? 1u : 0u) << n;
        waits |= 1u << t;
        out->c[n++] = (T)(ak * w);
      }
      const int rd = dir_to(bd, i, j, r, err);
      if (rd >= 0) {
        rcode = dir_code(rd) | ((edges & edges_of((rd + (rd >> 2)) % 3 - 1, (rd + (rd >> 2)) / 3 - 1)) ? 16u : 0u);
        waits |= 1u << rd;
      }
    }
    unsigned deps = 0, prefer = 0;
    double amax = -1.0;  // the dependent with the largest area has the longest way up behind it
  #pragma unroll
    for (int t = 0; t < 8; ++t) {
      int d;
      if (!nbr_at(bd, i, j, t, d)) continue;
      const int rd = __ldg(&recv[d]);
      if (rd == d) continue;
      const bool hits = (__ldg(&mmask[d]) >> (15 - t)) & 1;
      const bool gated = hits && (n_is_one ? (h[d] >= htk) : (h[d] > htk));
      if (gated || rd == k) {
        deps |= 1u << t;
        const double ad = __ldg(&a[d]);
        if (ad > amax) {
          amax = ad;
          prefer = (unsigned)t;
        }
      }
    }
    out->codes = codes;
    const unsigned ni = r == k ? kNoRec : (mk & 255) ? (unsigned)n : kNoMrec;
    out->meta = ni | (edges << 4) | (deps << 8) | (rcode << 16) | (prefer << 21) | (far << 24);
    out->base = htk;
    lens[me] = (unsigned short)lengths;
    wmeta[k] = (unsigned short)((unsigned)__popc(waits) | (deps << 8));
  }
  // the erosion factors: one power each, dealt over the lanes whatever the nodes
  // of the row they belong to
  int before = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, before, o);
    if ((int)threadIdx.x >= o) before += v;
  }
  const int total = __shfl_sync(0xffffffffu, before, 31);
  before -= n;
  for (int t = 0; t < n; ++t) slots[threadIdx.y][before + t] = (unsigned char)(threadIdx.x << 3 | t);
  __syncwarp();
  for (int e = threadIdx.x; e < total; e += 32) {
    const int slot = slots[threadIdx.y][e] & 7, node = threadIdx.y * 32 + (slots[threadIdx.y][e] >> 3);
    T* const c = &staged_record<T>(sm, node)->c[slot];
    const int len = (lens[node] >> (2 * slot)) & 3;
    const double kk = factor[node], l = __ldg(&ltab[len]);
    const T ln = __ldg(&lpow[len]), aw = *c;
    if constexpr (sizeof(T) == sizeof(double)) {
      *c = n_is_one ? kk * pow(aw, m) / l : kk * pow(aw, m) / ln;
    } else {  // mixed precision: the erosion factor in FP32
      const float kf32 = (float)kk, l32 = (float)l;
      *c = n_is_one ? kf32 * powf(aw, (float)m) / l32 : kf32 * powf(aw, (float)m) / ln;
    }
  }
  __syncwarp();
  store_records(bd, sm, rec);
}

// l^n for the nine neighbour lengths of find_receiver / find_mult_rec, with
// the same pow the per-node expression used (so the factors are unchanged)
__global__ void k_length_pow(const double* __restrict__ ltab, double n, double* __restrict__ lpow,
                             float* __restrict__ lpowf) {
  const int e = threadIdx.x;
  if (e < 9) {
    lpow[e] = pow(ltab[e], n);
    lpowf[e] = powf((float)ltab[e], (float)n);
  }
}

// ---- node operations: eight lanes per node -------------------------------------
// A node is computed by a segment of eight lanes of a warp: lane t holds input
// t of the node's record, loads its value and forms term t; the terms then
// meet in the warp's row of shared memory (two 16-byte accesses per term
// instead of shuffling the halves of two doubles) and every lane adds them up
// in input order -- the order of the queue engine in fsb_flow.cu -- so all
// eight do the same scalar arithmetic.  All segments of a warp execute the
// same instruction stream: a segment without a node, or whose node needs
// fewer Newton iterations, runs along without effect.
//
// Inputs of this tile are read through L1 (a store updates the line, which
// the node's inputs bring in before it is computed), those of other tiles
// from this tile's mailbox.
constexpr int kSegLanes = 8, kSegs = 32 / kSegLanes;
constexpr int kRowStride = 8 * 16 + 16;  // bytes of a segment's terms, padded against bank conflicts

// a tile of this CTA: its first node, its size
struct TileInfo {
  int x0, y0, w, h;
};

// Cells of the rim around a w x h tile of side 2^LT: the row above, the row
// below, then the left and the right column.
template <int LT>
struct Rim {
  static constexpr int kTS = 1 << LT;
  static constexpr int kCells = rim_cells(LT), kWords = rim_words(LT);
  __device__ static __forceinline__ int index(int x, int y, int w, int h) {
    if (y < 0) return x + 1;
    if (y >= h) return kTS + 3 + x;
    return 2 * (kTS + 2) + (x < 0 ? y : kTS + y);
  }
  // false for a cell that a w x h tile does not have
  __device__ static __forceinline__ bool coords(int c, int w, int h, int& x, int& y) {
    if (c < kTS + 2) { x = c - 1; y = -1; return x <= w; }
    if (c < 2 * (kTS + 2)) { x = c - (kTS + 3); y = h; return x <= w; }
    if (c < 2 * (kTS + 2) + kTS) { x = -1; y = c - 2 * (kTS + 2); return y < h; }
    x = w; y = c - 2 * (kTS + 2) - kTS;
    return c < 4 * kTS + 4 && y < h;
  }
};

// What a lane knows about its segment's node: natural index k, local index id
// (tile of this CTA << 2*LT | y << LT | x), and where cross-tile inputs lie.
template <class V, int LT>
struct NodeCtx {
  int k, id, nx;
  int sl;                // lane within the segment
  unsigned char* row;    // the segment's terms in shared memory
  const TileInfo* tab;   // shared memory
  const V* mbox;         // all tiles' cells
  int tile0, tile_step;
  __device__ __forceinline__ int near(unsigned code) const {
    return k + ((int)(code >> 2) - 1) * nx + (int)(code & 3u) - 1;
  }
  __device__ __forceinline__ const V* far(unsigned code) const {
    const int slot = id >> (2 * LT);
    const int lx = id & ((1 << LT) - 1), ly = (id >> LT) & ((1 << LT) - 1);
    const TileInfo ti = tab[slot];
    return mbox + (size_t)(tile0 + slot * tile_step) * Rim<LT>::kCells +
           Rim<LT>::index(lx + (int)(code & 3u) - 1, ly + (int)(code >> 2) - 1, ti.w, ti.h);
  }
  // every lane's term(s), in input order
  template <class T, class F>
  __device__ __forceinline__ void exchange(T a, F add) const {
    T* r = reinterpret_cast<T*>(row);
    __syncwarp();
    r[sl] = a;
    __syncwarp();
    struct __align__(16) Quad { T v[16 / sizeof(T)]; } v[8 * sizeof(T) / 16];
#pragma unroll
    for (int i = 0; i < (int)(8 * sizeof(T) / 16); ++i) v[i] = reinterpret_cast<const Quad*>(row)[i];
#pragma unroll
    for (int s = 0; s < 8; ++s) add(v[s / (16 / sizeof(T))].v[s % (16 / sizeof(T))]);
  }
  template <class T, class F>
  __device__ __forceinline__ void exchange(T a, T b, F add) const {
    struct __align__(2 * sizeof(T)) Pair { T a, b; };
    Pair* r = reinterpret_cast<Pair*>(row);
    __syncwarp();
    r[sl] = Pair{a, b};
    __syncwarp();
    Pair v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = r[s];
#pragma unroll
    for (int s = 0; s < 8; ++s) add(v[s].a, v[s].b);
  }
};

// The record of this lane's node (without inputs and dependents for an idle
// segment).  It is loaded as soon as the node is known, before the previous
// node's bookkeeping is finished.
template <class T>
struct Slot {
  int4 hd = {0, 0, 0, 0};
  T c = 0;
  unsigned codes, meta;
  double base;
  __device__ __forceinline__ void load(const RecordT<T>* r, bool on, int sl) {
    ldg_if(hd, reinterpret_cast<const int4*>(r), on);
    ldg_if(c, &r->c[sl], on);
  }
  __device__ __forceinline__ void open(bool on) {
    codes = (unsigned)hd.x;
    meta = on ? (unsigned)hd.y : kNoRec;
    base = __hiloint2double(hd.w, hd.z);
  }
  // inputs of the node; whether this lane has one, its offset, whether it lies in another tile
  __device__ __forceinline__ unsigned n() const { return meta & 15u; }
  __device__ __forceinline__ bool mine(int sl) const { return (unsigned)sl < n() && n() < kNoMrec; }
  __device__ __forceinline__ unsigned code(int sl) const { return (codes >> (4 * sl)) & 15u; }
  __device__ __forceinline__ bool far(int sl) const { return (meta >> (24 + sl)) & 1u; }
};

// a(k) = dx*dy*precip(k) + sum over donors of a(d)*w(d->k) (FlowRouting.f90:109-115)
template <class T_>
struct AccOp {
  using T = T_;
  using Value = T_;
  static constexpr int kId = sizeof(T_) == sizeof(double) ? 0 : 1;
  static constexpr bool kPrefer = false;  // records name a dependent to continue with
  const RecordT<T>* rec;
  T* val;
  template <int LT, class Touch>
  __device__ __forceinline__ unsigned run(const NodeCtx<T, LT>& nc, const Slot<T>& sl, bool on, T& out, Touch touch) const {
    const unsigned code = sl.code(nc.sl);
    const bool mine = sl.mine(nc.sl), far = mine && sl.far(nc.sl);
    T x = ld_l1_if(val + nc.near(code), mine && !far);
    if (far) mail_read(nc.far(code), x);
    touch(sl.meta);
    T acc = (T)sl.base;
    nc.exchange(mine ? x * sl.c : T(0), [&](T a) { acc = acc + a; });
    if (on && nc.sl == 0) st_value(val + nc.k, acc);
    out = acc;
    return sl.meta;
  }
};

// implicit stream power law over the multiple receivers with g == 0
// (StreamPowerLaw.f90:92-177): hw[k] = (new h, water).  MODE 0: n = 1, closed
// form; 1: n = 1.5, whose powers are x*sqrt(x) and sqrt(x) (sqrt is correctly
// rounded); 2: other n, x*x^(n-1) with one pow for x > 0.
//
// T = double: the reference's arithmetic.  T = float (mixed precision): the
// solve for the increment d = h - ht in FP32.  Elevations, water levels and
// the h update stay FP64; the distances to the receivers' new elevations,
// ht(k) - h(q), are taken in FP64 and rounded once.  n = 1: d =
// -sum f*(ht - hq) / (1 + sum f), the closed form of StreamPowerLaw.f90:108-118
// rewritten for the increment; otherwise Newton on d (x = max(0, ht - hq + d),
// :146-162) with the reference's tolerance and relaxation.
// x^n and x^(n-1) for x >= 0
template <int MODE>
__device__ __forceinline__ void newton_pow(double x, double n, double& pn, double& pn1) {
  pn1 = MODE == 1 ? sqrt(x) : pow(x, n - 1.0);
  pn = MODE == 1 || x > 0.0 ? x * pn1 : pow(x, n);
}
template <int MODE>
__device__ __forceinline__ void newton_pow(float x, float n, float& pn, float& pn1) {
  pn1 = MODE == 1 ? sqrtf(x) : powf(x, n - 1.0f);
  pn = MODE == 1 || x > 0.0f ? x * pn1 : powf(x, n);
}

template <class T_, int MODE>
struct SplOp {
  using T = T_;
  using Value = double2;
  static constexpr bool kPrefer = true;
  static constexpr int kId = 2 + MODE + (sizeof(T_) == sizeof(double) ? 0 : 3);
  const RecordT<T>* rec;
  double2* val;
  T n, omega;
  int* err;
  template <int LT, class Touch>
  __device__ __forceinline__ unsigned run(const NodeCtx<double2, LT>& nc, const Slot<T>& sl, bool on, double2& out,
                                             Touch touch) const {
    constexpr bool kInc = sizeof(T) == sizeof(float);  // solve for the increment
    const unsigned ni = sl.n(), code = sl.code(nc.sl), rc = (sl.meta >> 16) & 15u;
    const bool has_rec = ni != kNoRec, mine = sl.mine(nc.sl);
    const bool far = mine && sl.far(nc.sl), rfar = (sl.meta >> 20) & 1u;
    const double ht = sl.base;
    double hq = ld_l1_if(&val[nc.near(code)].x, mine && !far);
    double wr = ld_l1_if(&val[nc.near(rc)].y, has_rec && !rfar);
    if (far || (has_rec && rfar)) {
      if (far) hq = ld_relaxed_gpu(&nc.far(code)->x);
      if (has_rec && rfar) wr = ld_relaxed_gpu(&nc.far(rc)->y);
    }
    touch(sl.meta);
    const bool above = has_rec && ht > wr;
    const bool solve = above && ni != kNoMrec;
    // the unknown: h itself, or its increment over ht; q: h or ht - h of the receiver
    T u = kInc ? T(0) : (T)ht;
    const T q = kInc ? (T)(ht - hq) : (T)hq;
    if constexpr (MODE == 0) {
      T f = kInc ? T(0) : (T)ht, df = 1;
      nc.exchange(mine ? sl.c * q : T(0), mine ? sl.c : T(0), [&](T a, T b) {
        f = f + a;
        df = df + b;
      });
      if (solve) u = kInc ? -f / df : f / df;
    } else {
      const T tolp = (T)1.0e-3;
      bool go = solve;
      int guard = 0;
      while (__any_sync(FULL, go)) {
        if (go && ++guard > kNewtonLimit) {
          if (nc.sl == 0) atomicExch(err, DEV_NEWTON_LIMIT);
          go = false;
        }
        T x = 1, pn, pn1;  // lanes without an input run on 1: a root of 0 takes a slow path
        if (mine) {
          if constexpr (kInc) x = fmaxf(0.0f, q + u);
          else x = fmax(0.0, u - q);
        }
        newton_pow<MODE>(x, n, pn, pn1);
        T f = kInc ? u : u - (T)ht, df = 1;
        const T tf = mine ? sl.c * pn : T(0), tdf = mine ? sl.c * n * pn1 : T(0);
        nc.exchange(tf, tdf, [&](T a, T b) {
          f = f + a;
          df = df + b;
        });
        if (go) {
          const T un = u - f / df;
          const T errp = kInc ? (T)fabsf((float)(un - u)) : (T)fabs((double)(un - u));
          u = u * (T(1) - omega) + un * omega;
          go = errp > tolp;
        }
      }
    }
    double hk = ht, wk = ht;
    if (has_rec) {
      if (above) {
        if (solve) hk = kInc ? ht + (double)u : (double)u;
        if (hk < wr) hk = wr;
      }
      wk = fmax(wr, hk);
    }
    out = make_double2(hk, wk);
    if (on && nc.sl == 0) st_value(val + nc.k, out);
    return sl.meta;
  }
};

// ---- the sweep kernel ------------------------------------------------------------
// One CTA per SM; CTA c owns tiles c, c + C, c + 2C, ...  Shared memory: a
// counter byte per node, the directions in which each rim cell's node has
// dependents in the tile, the flag words already seen.  Warp 0 polls the flag
// words of the CTA's tiles; every segment of the other warps computes one node
// at a time: its lanes release the node's dependents (lane t the one in
// direction t), it continues with the first one made ready and queues the
// others.  A warp without work claims one queue
// entry ahead and waits for it, so that a new entry wakes an idle warp at
// once; entries beyond those that idle warps wait for are taken by whichever
// warp comes round next, up to four at a time.  A CTA ends when all its
// nodes are done; every wait is bounded by a 4 s limit, after which the sweep
// reports DEV_SPIN_LIMIT.
template <class Op, int LT>
__global__ void __launch_bounds__(kThreads, 1)
    k_region_sweep(Op op, TileMap tm, const unsigned short* __restrict__ wmeta, long long* queue,
                   typename Op::Value* mbox, unsigned* flags, int* err) {
  using V = typename Op::Value;
  using R = Rim<LT>;
  constexpr int kTS = 1 << LT, kNodes = kTS * kTS;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int qhead, qtail, ndone, stop, count_sh;
  __shared__ __align__(16) int4 scratch;
  __shared__ __align__(16) unsigned char terms[kThreads / 32][kSegs * kRowStride];
  const int nC = gridDim.x;
  const int tiles = tm.tiles();
  const int ns = (tiles - (int)blockIdx.x + nC - 1) / nC;  // tiles of this CTA
  unsigned* cnt = reinterpret_cast<unsigned*>(smem);
  unsigned char* rim = smem + tm.ns * kNodes;                                        // tm.ns * R::kCells
  unsigned* seen = reinterpret_cast<unsigned*>(rim + tm.ns * R::kCells);            // tm.ns * R::kWords
  TileInfo* tab = reinterpret_cast<TileInfo*>(seen + tm.ns * R::kWords);  // tm.ns
  long long* q = queue + (size_t)blockIdx.x * tm.cta_nodes;
  asm volatile("" : "+l"(q));  // kept, not worked out anew for every look (1 to 2 % of a sweep)
  const unsigned long long t0 = global_ns();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kWarps = kThreads / 32;

  if (threadIdx.x == 0) {
    qhead = 0;
    qtail = 0;
    ndone = 0;
    stop = 0;
    count_sh = 0;
  }
  __syncthreads();
  for (int s = threadIdx.x; s < ns; s += kThreads) {
    const int t = (int)blockIdx.x + s * nC;
    TileInfo ti;
    ti.x0 = (t % tm.ntx) * kTS;
    ti.y0 = (t / tm.ntx) * kTS;
    ti.w = min(kTS, tm.nx - ti.x0);
    ti.h = min(kTS, tm.ny - ti.y0);
    tab[s] = ti;
    atomicAdd(&count_sh, ti.w * ti.h);
  }
  __syncthreads();
  const int count = count_sh;
  for (int row = warp; row < ns * kTS; row += kWarps) {
    const int s = row >> LT, y = row & (kTS - 1);
    const TileInfo ti = tab[s];
    if (y >= ti.h) continue;
    for (int xb = 0; xb < ti.w; xb += 32) {
      const int x = xb + lane;
      const int k = ti.x0 + x + (ti.y0 + y) * tm.nx;
      int c = 255;
      if (x < ti.w) {
        c = wmeta[k] & 255;
        smem[(row << LT) + x] = (unsigned char)c;
      }
      const unsigned m = __ballot_sync(FULL, c == 0);
      if (m) {
        int p = 0;
        if (lane == 0) p = atomicAdd(&qtail, __popc(m));
        p = __shfl_sync(FULL, p, 0) + __popc(m & ((1u << lane) - 1u));
        if (c == 0) st_queue(q + p, (long long)k << 32 | ((row << LT) + x));
      }
    }
  }
  for (int e = threadIdx.x; e < ns * R::kCells; e += kThreads) {
    const int s = e / R::kCells, c = e - s * R::kCells;
    const TileInfo ti = tab[s];
    int x, y;
    unsigned m = 0;
    if (R::coords(c, ti.w, ti.h, x, y)) {
      // a cell beyond a non-cyclic edge names a node on the other side, which
      // has no dependents in the directions that lead here
      int X = ti.x0 + x, Y = ti.y0 + y;
      X += X < 0 ? tm.nx : (X >= tm.nx ? -tm.nx : 0);
      Y += Y < 0 ? tm.ny : (Y >= tm.ny ? -tm.ny : 0);
      const unsigned deps = wmeta[X + Y * tm.nx] >> 8;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int ax = x + dir_di(t), ay = y + dir_dj(t);
        if (((deps >> t) & 1u) && ax >= 0 && ax < ti.w && ay >= 0 && ay < ti.h) m |= 1u << t;
      }
    }
    rim[e] = (unsigned char)m;
  }
  for (int e = threadIdx.x; e < ns * R::kWords; e += kThreads) seen[e] = 0u;
  __syncthreads();

  auto push = [&](int p, int k, int id) {
    if (p < count) st_queue(q + p, (long long)k << 32 | id);
    else atomicExch(err, DEV_OVERFLOW);
  };
  // decrements the counter of local node l; true when the node became ready
  auto release = [&](int l) {
    const unsigned sh = 8u * (unsigned)(l & 3);
    const unsigned old = atomicSub(&cnt[l >> 2], 1u << sh);
    return ((old >> sh) & 0xffu) == 1u;
  };
  // periodic checks of the time limit and of failures elsewhere (one lane)
  auto should_stop = [&](int& ticks) {
    if (*(volatile int*)&stop) return true;
    if (++ticks < 256) return false;
    ticks = 0;
    if (*(volatile int*)err != 0) {
      *(volatile int*)&stop = 1;
      return true;
    }
    if (global_ns() - t0 > kRegionTimeLimitNs) {
      atomicExch(err, DEV_SPIN_LIMIT);
      *(volatile int*)&stop = 1;
      return true;
    }
    return false;
  };

  if (warp == 0) {
    int ticks = 0;
    for (;;) {
      bool any = false;
      for (int e0 = 0; e0 < ns * (R::kWords / 4); e0 += 32) {
        const int e = e0 + lane;
        unsigned nw[4] = {0u, 0u, 0u, 0u};
        if (e < ns * (R::kWords / 4)) {
          const int s = e / (R::kWords / 4), w4 = e - s * (R::kWords / 4);
          ld_flags(flags + ((size_t)blockIdx.x + (size_t)s * nC) * R::kWords + 4 * w4, nw);
#pragma unroll
          for (int i = 0; i < 4; ++i) nw[i] &= ~seen[4 * e + i];
        }
        // the warp takes the words with news one after the other, a cell per lane
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          unsigned lanes = __ballot_sync(FULL, nw[i] != 0u);
          while (lanes) {
            const int src = __ffs(lanes) - 1;
            lanes &= lanes - 1u;
            const unsigned bits = __shfl_sync(FULL, nw[i], src);
            const int word = 4 * (e0 + src) + i;
            bool got = false;
            if ((bits >> lane) & 1u) {
              const int s = word / R::kWords, c = 32 * (word - s * R::kWords) + lane;
              V v;
              got = mail_read(mbox + ((size_t)blockIdx.x + (size_t)s * nC) * R::kCells + c, v);  // or the flag overtook it
              if (got) {
                const TileInfo ti = tab[s];
                int x, y;
                R::coords(c, ti.w, ti.h, x, y);
                unsigned m = rim[s * R::kCells + c];
                __threadfence_block();
                while (m) {
                  const int t = __ffs(m) - 1;
                  m &= m - 1u;
                  const int c3 = t + (t >> 2);
                  const int lx = x + c3 % 3 - 1, ly = y + c3 / 3 - 1;
                  const int id = (s << (2 * LT)) | (ly << LT) | lx;
                  if (release(id)) {
                    __threadfence_block();
                    push(atomicAdd(&qtail, 1), ti.x0 + lx + (ti.y0 + ly) * tm.nx, id);
                  }
                }
              }
            }
            const unsigned in = __ballot_sync(FULL, got);
            if (lane == 0) seen[word] |= in;
            any |= in != 0u;
          }
        }
        __syncwarp();
      }
      if (!any) {
        int quit = 0;
        if (lane == 0) quit = *(volatile int*)&ndone >= count || should_stop(ticks);
        if (__shfl_sync(FULL, quit, 0)) return;
        __nanosleep(20);
      }
    }
  }

  const unsigned scr = (unsigned)__cvta_generic_to_shared(&scratch);
  const int sl = lane & (kSegLanes - 1), base = lane - sl;
  const int di = (sl + (sl >> 2)) % 3 - 1, dj = (sl + (sl >> 2)) / 3 - 1;  // this lane's direction
  const int kstep = dj * tm.nx + di, lstep = dj * kTS + di;
  const unsigned my_edges = edges_of(di, dj);
  const int nn = tm.nx * tm.ny;
  const bool far_ahead = nn > kL2Records;
  int k = 0, id = -1, slot = -1, ticks = 0;  // the same in all lanes of a segment
  int backlog = 0;  // entries queued beyond the claims, as last seen (the same in all lanes)
  int hops = 0;
  int done = 0;     // nodes computed by this segment and not yet counted (its first lane)
  Slot<typename Op::T> rec;
  for (;;) {
    // a warp without work claims one entry ahead; segments of a working warp
    // take entries that are queued beyond the waiting warps' claims
    const unsigned busy = __ballot_sync(FULL, id >= 0 || slot >= 0);
    if (busy == 0u || (backlog > 0 && busy != FULL)) {
      const unsigned open = ~busy & 0x01010101u;  // one bit per open segment
      const int want = backlog > 0 ? min(__popc(open), max(1, backlog >> 4)) : 1;
      int b0 = 0;
      if (lane == 0) b0 = atomicAdd(&qhead, want);
      b0 = __shfl_sync(FULL, b0, 0);
      const int rank = __popc(open & ((1u << base) - 1u));
      if (((open >> base) & 1u) && rank < want) slot = b0 + rank;
    }
    const bool poll = sl == 0 && slot >= 0 && slot < count;  // a segment's first lane looks
    long long v = -1;
    if (poll) v = ld_queue(q + slot);
    if (!__any_sync(FULL, id >= 0)) {  // nothing to do until an entry comes
      if (done) {
        atomicAdd(&ndone, done);
        done = 0;
      }
      const int mine = __reduce_max_sync(FULL, slot);
      int tries = 0;
      while (!__any_sync(FULL, v >= 0)) {
        // the next pushes fill the entries right after the tail: warps that
        // wait further ahead look less often
        const int ahead = mine - *(volatile int*)&qtail;
        if (ahead > 2) __nanosleep(ahead > 6 ? 200 : 40);
        if ((++tries & 7) == 0) {
          int quit = 0;
          if (lane == 0) quit = *(volatile int*)&ndone >= count || should_stop(ticks);
          if (__shfl_sync(FULL, quit, 0)) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            return;
          }
        }
        if (poll) v = ld_queue(q + slot);
      }
    }
    v = __shfl_sync(FULL, v, base);
    if (v >= 0) {
      k = (int)(v >> 32);
      id = (int)v;
      slot = -1;
      rec.load(op.rec + k, true, sl);
    }
    const bool waiting = __any_sync(FULL, slot >= 0);
    bool go;
    do {  // chains of nodes, while nothing waits for this warp's idle segments
      __threadfence_block();  // acquire: the producers' values
      const bool on = id >= 0;
      V out;
      rec.open(on);
      const NodeCtx<V, LT> nc{k, id, tm.nx, sl, &terms[warp][(lane >> 3) * kRowStride], tab, mbox, (int)blockIdx.x, nC};
      const unsigned meta = op.run(nc, rec, on, out, [&](unsigned m) {
        // bring what the dependents will read into L1
        const bool t = ((m >> (8 + sl)) & 1u) && !((m >> 4) & my_edges);
        const char* p = reinterpret_cast<const char*>(op.rec + (k + kstep));
        touch_l1_if(scr, p, t);
        touch_l1_if(scr, p + 32, t);
        if (sizeof(typename Op::T) == 8) touch_l1_if(scr, p + 64, t);
        if (!Op::kPrefer && far_ahead) {  // the area's nodes wait long for their last input: L2 may have lost what comes after
          const char* p2 = reinterpret_cast<const char*>(op.rec + (k + 2 * kstep));
          prefetch_l2_if(p2, t && (unsigned)(k + 2 * kstep) < (unsigned)nn);
        }
        touch_l1_if(scr, reinterpret_cast<const void*>(reinterpret_cast<size_t>(op.val + (k + kstep)) & ~(size_t)15), t);
      });
      __syncwarp();
      __threadfence_block();  // release: the node's value before its dependents' counters
      const bool dep = on && ((meta >> (8 + sl)) & 1u), cross = (meta >> 4) & my_edges;
      const unsigned prefer = (meta >> 21) & 7u;
      bool ready = false;
      if (dep && !cross) ready = release(id + lstep);
      const unsigned all = __ballot_sync(FULL, ready);
      unsigned rm = (all >> base) & 0xffu;
      if (Op::kPrefer && ((rm >> prefer) & 1u)) rm = 1u << prefer;
      const int first = (base + __ffs(rm) - 1) & 31;  // any lane where none is ready
      const bool queued = ready && lane != first;
      int qp = 0;
      if (queued) {
        __threadfence_block();  // the other producers' values too
        qp = atomicAdd(&qtail, 1);
      }
      const int nk = __shfl_sync(FULL, k + kstep, first), nid = __shfl_sync(FULL, id + lstep, first);
      rec.load(op.rec + nk, rm != 0u, sl);
      if (queued) push(qp, k + kstep, id + lstep);
      if (dep && cross) {  // the value into the neighbouring tile's cell, then its flag
        const TileInfo ti = tab[id >> (2 * LT)];
        int X = ti.x0 + (id & (kTS - 1)) + di, Y = ti.y0 + ((id >> LT) & (kTS - 1)) + dj;
        X += X < 0 ? tm.nx : (X >= tm.nx ? -tm.nx : 0);
        Y += Y < 0 ? tm.ny : (Y >= tm.ny ? -tm.ny : 0);
        const int ox = X >> LT, oy = Y >> LT;
        const int ow = min(kTS, tm.nx - ox * kTS), oh = min(kTS, tm.ny - oy * kTS);
        const int c = R::index((X & (kTS - 1)) - di, (Y & (kTS - 1)) - dj, ow, oh);
        const size_t tile = (size_t)oy * tm.ntx + ox;
        mail_write(mbox + tile * R::kCells + c, out);
        // Around a cyclic side that one tile spans the node is this CTA's own: its
        // counter is at hand, and warp 0 need not hear of it (area of 3 x 3736 nodes,
        // flow along it: 6.4 -> 4.1 ms, of 60000 x 20 264 -> 165)
        if (ox == ti.x0 >> LT && oy == ti.y0 >> LT) {
          const int l = (id >> (2 * LT) << (2 * LT)) | ((Y & (kTS - 1)) << LT) | (X & (kTS - 1));
          __threadfence_block();  // the cell before the counter
          if (release(l)) {
            __threadfence_block();
            push(atomicAdd(&qtail, 1), X + Y * tm.nx, l);
          }
        } else {
          atomicOr(&flags[tile * R::kWords + (c >> 5)], 1u << (c & 31));
        }
      }
      done += on && sl == 0;
      k = nk;
      id = rm ? nid : -1;
      // on with the chains while every segment has a node, or none of the idle
      // ones has anything to do (looked up every fourth node)
      const bool full = (all & 0xffu) && (all & 0xff00u) && (all & 0xff0000u) && (all & 0xff000000u);
      go = full || (all && !waiting && ((++hops & 3) || !__any_sync(FULL, *(volatile int*)&qtail > *(volatile int*)&qhead)));
    } while (go);
    backlog = __shfl_sync(FULL, *(volatile int*)&qtail - *(volatile int*)&qhead, 0);
  }
}

// natural-order FP64 area from the mixed form's FP32 values
__global__ void k_widen(int nn, const float* __restrict__ v, double* __restrict__ a) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) a[k] = (double)v[k];
}

// StreamPowerLaw.f90:380-393 with g == 0: b=min(h,b), etot=etot+ht-h,
// erate=(ht-h)/dt, Sedflux=ht-h, from the (h, water) pairs
__global__ void k_spl_finish_hw(int nn, double dt, const double2* __restrict__ hw, double* __restrict__ h,
                                double* __restrict__ b, double* __restrict__ etot, double* __restrict__ erate,
                                double* __restrict__ sedflux) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const double ht = h[k], hn = hw[k].x;
    b[k] = fmin(hn, b[k]);
    etot[k] = etot[k] + ht - hn;
    erate[k] = (ht - hn) / dt;
    sedflux[k] = ht - hn;
    h[k] = hn;
  }
}

constexpr int kMaxSmem = 212 * 1024;  // dynamic shared memory of a sweep CTA at most

int region_smem(const TileMap& tm) {
  return tm.ns * ((1 << 2 * tm.lt) + rim_cells(tm.lt) + 4 * rim_words(tm.lt) + (int)sizeof(TileInfo));
}

// whether every CTA of this sweep kernel can be co-resident
template <class Op, int LT>
bool region_fits(const TileMap& tm) {
  const int smem = region_smem(tm);
  if (smem > kMaxSmem) return false;
  // the permitted maximum covers every plan, so instances with different
  // plans never undo each other's setting
  using Big = BigSmem<k_region_sweep<Op, LT>>;
  int dev = 0, sms = 0, per_sm = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) {
    cudaGetLastError();
    return false;
  }
  for (int t = 0; t < 2 && per_sm == 0; ++t)
    if (!Big::allow(kMaxSmem, t == 1) ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_region_sweep<Op, LT>, kThreads, (size_t)smem) !=
            cudaSuccess) {
      cudaGetLastError();
      per_sm = 0;
    }
  return per_sm * sms >= tm.nctas;
}

// whether the sweep of Op can run on the plan (checked once per instance)
template <class Op, int LT>
bool region_usable(Ctx& c, const TileMap& tm) {
  if (tm.ntx == 0) return false;
  signed char& st = c.region_ok[Op::kId];
  if (st == 0) st = region_fits<Op, LT>(tm) ? 1 : -1;
  return st > 0;
}

// Launches the sweep of op; false when the launch is refused (the queue engine
// of fsb_flow.cu then runs).
template <int LT, class Op>
bool launch_region(Ctx& c, const TileMap& plan, Op op) {
  using V = typename Op::Value;
  TileMap tm = plan;
  const size_t tiles = (size_t)tm.tiles();
  cudaMemsetAsync(c.rl_queue, 0xff, sizeof(long long) * tm.queue_entries(), c.stream);
  cudaMemsetAsync(c.rl_flags, 0, sizeof(unsigned) * tiles * rim_words(LT), c.stream);
  cudaMemsetAsync(c.rl_mbox, 0xff, sizeof(V) * tiles * rim_cells(LT), c.stream);
  const unsigned short* wmeta = c.rl_wmeta;
  long long* queue = c.rl_queue;
  V* mbox = reinterpret_cast<V*>(c.rl_mbox);
  unsigned* flags = c.rl_flags;
  int* err = c.d_err;
  void* args[] = {&op, &tm, &wmeta, &queue, &mbox, &flags, &err};
  const int timer = Op::kPrefer ? KT_SPL_SWEEP : KT_AREA_SWEEP;
  stage_begin(c, timer);
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_region_sweep<Op, LT>, dim3(tm.nctas), dim3(kThreads),
                                                    args, (size_t)region_smem(tm), c.stream);
  if (e != cudaSuccess) {  // e.g. the GPU is shared and the CTAs no longer fit
    cudaGetLastError();
    c.region_ok[Op::kId] = -1;
    return false;
  }
  stage_end(c, timer);  // the timers count sweeps that ran here
  c.count_launch();
  return true;
}

dim3 grid2d(const Ctx& c) { return dim3((c.nx + 31) / 32, (c.ny + 7) / 8); }

template <class T, int LT>
bool accumulate_t(Ctx& c) {
  using Op = AccOp<T>;
  const TileMap& tm = c.tplan[LT - kLogTileMin];
  if (!region_usable<Op, LT>(c, tm)) return false;
  RecordT<T>* rec = static_cast<RecordT<T>*>(c.mfd_line);
  T* val = sizeof(T) == sizeof(double) ? reinterpret_cast<T*>(c.a) : reinterpret_cast<T*>(c.hw);
  k_acc_records<T><<<grid2d(c), dim3(32, 8), 0, c.stream>>>(c.bd, 1 << LT, c.dx * c.dy, c.mdmask, c.mrec, c.mwrec,
                                                            c.precip, rec, c.rl_wmeta);
  c.count_launch();
  if (!launch_region<LT>(c, tm, Op{rec, val})) return false;
  if (sizeof(T) == sizeof(float)) {
    k_widen<<<grid1d(c.nn), kBlock, 0, c.stream>>>(c.nn, reinterpret_cast<float*>(c.hw), c.a);
    c.count_launch();
  }
  return true;
}

template <class T, int MODE, int LT>
bool stream_power_t(Ctx& c) {
  using Op = SplOp<T, MODE>;
  const TileMap& tm = c.tplan[LT - kLogTileMin];
  if (!region_usable<Op, LT>(c, tm)) return false;
  RecordT<T>* rec = static_cast<RecordT<T>*>(c.mfd_line);
  double2* hw = reinterpret_cast<double2*>(c.hw);
  double* lpow = c.ltab + 16;
  float* lpowf = reinterpret_cast<float*>(c.ltab + 32);
  const T* lp;
  if constexpr (sizeof(T) == sizeof(double)) lp = lpow; else lp = lpowf;
  k_length_pow<<<1, 32, 0, c.stream>>>(c.ltab, c.n, lpow, lpowf);
  k_spl_records<T><<<grid2d(c), dim3(32, 8), 0, c.stream>>>(c.bd, 1 << LT, MODE == 0, c.kfsed, c.dt, c.m, c.rec,
                                                            c.mdmask, c.mrec, c.mwrec, c.mlrec, c.h, c.b, c.kf, c.a,
                                                            c.ltab, lp, rec, c.rl_wmeta, c.d_err);
  c.count_launch(2);
  if (!launch_region<LT>(c, tm, Op{rec, hw, (T)c.n, (T)(0.875 / c.n), c.d_err})) return false;
  k_spl_finish_hw<<<grid1d(c.nn), kBlock, 0, c.stream>>>(c.nn, c.dt, hw, c.h, c.b, c.etot, c.erate, c.sedflux);
  c.count_launch();
  return true;
}

template <class T, int LT>
bool stream_power_n(Ctx& c) {
  if (fabs(c.n - 1.0) < DBL_MIN) return stream_power_t<T, 0, LT>(c);
  return c.n == 1.5 ? stream_power_t<T, 1, LT>(c) : stream_power_t<T, 2, LT>(c);
}

}  // namespace

// Tile plan: the grid's tiles of side 2^lt over at most one CTA per SM.  Tiles
// so many that a CTA's counters exceed its shared memory leave ntx at 0: the
// queue engine runs.
TileMap plan_tiles(int nx, int ny, int lt, int sms) {
  TileMap tm;
  tm.nx = nx;
  tm.ny = ny;
  tm.lt = lt;
  tm.ntx = (nx + (1 << lt) - 1) >> lt;
  tm.nty = (ny + (1 << lt) - 1) >> lt;
  tm.nctas = std::min(std::max(1, sms), tm.tiles());
  tm.ns = (tm.tiles() + tm.nctas - 1) / tm.nctas;
  if (region_smem(tm) > kMaxSmem) tm.ntx = 0;
  else tm.cta_nodes = tm.ns * std::min(1 << lt, nx) * std::min(1 << lt, ny);
  return tm;
}

// Tile sides.  Smaller tiles spread the front over more SMs and halve the
// nodes that share an SM; larger ones have fewer crossings, and the area's
// nodes, all sources at once, are spread anyway.  B200, side 32 / 64: area
// 257^2 0.48 / 0.53 ms, 1025x769 3.05 / 2.88, 2049^2 6.4 / 5.8, and around the
// border (random surfaces) 385^2 0.81 / 0.83, 513^2 0.83 / 0.83, 577^2 1.46 / 1.42,
// 641^2 1.34 / 1.26; stream power (n = 1.5) 0.69 / 0.84, 3.98 / 4.27, 6.9 / 7.3,
// 4097^2 18.0 / 18.0.
// A strip that one larger tile spans and a smaller one does not takes the larger:
// its flow runs along it, and every row of nodes would wait for a crossing
// (4000x33, a cone: area 11.3 / 5.5 ms, stream power 15.7 / 10.8; 256x50, a ramp:
// 1.07 / 0.68 and 1.32 / 1.01).  Short ones have more to lose without a slope
// (128x64, a relief: 0.18 / 0.24 and 0.31 / 0.50).
static bool larger_tiles(const Ctx& c, bool area) {
  constexpr int kSmall = 1 << kLogTileMin;
  const int across = std::min(c.nx, c.ny), along = std::max(c.nx, c.ny);
  if (across > kSmall && across <= 2 * kSmall && along >= 8 * kSmall) return true;
  return area && c.nn > 1 << 18;
}

// The mixed form's sweeps run in FP32 on up to 296 blocks of 256 x 128 nodes (9.7e6)
// and in FP64 beyond: the rounding of the areas grows with the number of nodes
// that drain through one, and elevations with them (relative error of h after a
// step of 3001^2: 4.5e-7; of 4097^2 2.3e-5 with FP32 sweeps, 2.3e-7 without).
static bool fp32_sweeps(const Ctx& c) { return c.mixed && ((c.nx + 255) / 256) * ((c.ny + 127) / 128) <= 296; }

bool region_accumulate(Ctx& c) {
  const bool f32 = fp32_sweeps(c);
  if (!larger_tiles(c, true)) return f32 ? accumulate_t<float, 5>(c) : accumulate_t<double, 5>(c);
  return f32 ? accumulate_t<float, 6>(c) : accumulate_t<double, 6>(c);
}

bool region_stream_power(Ctx& c) {
  const bool f32 = fp32_sweeps(c);
  if (!larger_tiles(c, false)) return f32 ? stream_power_n<float, 5>(c) : stream_power_n<double, 5>(c);
  return f32 ? stream_power_n<float, 6>(c) : stream_power_n<double, 6>(c);
}

}  // namespace fsb
