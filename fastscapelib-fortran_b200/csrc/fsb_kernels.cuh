// Device-resident state of one continental-step instance and the launchers
// that operate on it.  One Ctx mirrors the reference's FastScapeContext module
// (src/FastScape_ctx.f90:9-36) for the arrays the continental step touches.
#pragma once

#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <cstddef>
#include <string>
#include <utility>

#include "fsb_common.cuh"

namespace fsb {

constexpr int kBlock = 256;
constexpr int kSlotStride = 16;  // doubles per node in Ctx::slots

inline unsigned grid1d(size_t n, int block = kBlock) {
  size_t g = (n + block - 1) / block;
  if (g > 148u * 64u) g = 148u * 64u;  // grid-stride loops beyond 64 blocks per SM
  if (g == 0) g = 1;
  return (unsigned)g;
}

// Tiles of the region-owned sweeps (fsb_region.cu): squares of 2^lt nodes a
// side, tile ty*ntx + tx, dealt out over nctas CTAs (tile t to CTA t % nctas).
constexpr int kLogTileMin = 5, kTilePlans = 2;  // sides 32 and 64
// per tile: mailbox cells, one for each node around it, and flag words, one bit per cell
__host__ __device__ constexpr int rim_cells(int lt) { return ((4 << lt) + 4 + 15) & ~15; }
__host__ __device__ constexpr int rim_words(int lt) { return (rim_cells(lt) + 127) / 128 * 4; }
struct TileMap {
  int nx = 0, ny = 0, lt = 0;
  int ntx = 0, nty = 0;  // ntx == 0: no plan
  int nctas = 0, ns = 0;  // CTAs, tiles per CTA at most
  int cta_nodes = 0;      // nodes of a CTA's tiles at most (a strip does not fill them)
  __host__ __device__ int tiles() const { return ntx * nty; }
  size_t queue_entries() const { return (size_t)nctas * cta_nodes; }
};

// heavy-path chains (fsb_chains.cu): nodes of a long one; ticket buckets (32
// light depths x 32 length classes of the long chains, 32 depths of the others)
constexpr int kLongChain = 16, kChainHist = 32 * 32 + 32;

struct Ctx {
  // ---- configuration (setters of FastScape_ctx.f90) ----
  int nx = 0, ny = 0, nn = 0;
  int ibc = 1111;
  Bounds bd{};
  double xl = 0, yl = 0, dt = 0, kfsed = -1, m = 0, n = 1, kdsed = -1, g1 = 0, g2 = 0, p = 0;
  double dx = 0, dy = 0;
  bool sfd = false, runSPL = false, runDiffusion = false, runUplift = false;
  bool setup_done = false;
  // mixed precision (fsb_set_precision): FP32 weights, area, Newton iterations
  // and tridiagonal solves; FP64 state, h update and residuals
  bool mixed = false;
  int launch_share = 1;  // 1: alone on the device; 4: beside other instances (persistent sweeps take 1/4 the blocks)
  bool capture = false;  // keep LocalMinima intermediates of the last step
  bool routed = false;   // a step has built receivers, stack, chains and area
  bool precip_uniform = true;  // every node has precipitation precip_value (SetUp: 1)
  double precip_value = 1.0;
  int step = 0;
  cudaStream_t stream = 0;
  long long launches = 0;  // kernels launched by this instance
  void count_launch(long long k = 1) { launches += k; }

  // ---- device arena ----
  char* arena = nullptr;
  size_t arena_bytes = 0;
  bool owns_arena = false;

  // ---- persistent fields (nn each unless noted) ----
  double *h = nullptr, *b = nullptr, *u = nullptr, *kf = nullptr, *kd = nullptr, *precip = nullptr;
  double *etot = nullptr, *erate = nullptr, *a = nullptr, *length = nullptr, *lake_depth = nullptr;
  double *hwater = nullptr, *sedflux = nullptr;
  double *catch0 = nullptr, *catchv = nullptr;  // catchment seeds (SetUp) and labels (ctx:17,94)
  double* red = nullptr;                         // 3*512 partial sums + 3 results (reductions)
  double* g = nullptr;                           // sediment parameter per node (ctx:17), kept across steps
  double *vx = nullptr, *vy = nullptr;           // advection velocities (ctx:17, SetV)
  bool runAdvect = false;
  bool g_positive = false;                       // max(g) > 0 at the last stream-power call
  int ngs = 0;                                   // Gauss-Seidel iterations of the last call
  int *rec = nullptr, *ndon = nullptr, *don = nullptr /*8*nn*/, *stack = nullptr;
  int *pos = nullptr, *size = nullptr;
  int *mrec = nullptr /*8*nn*/, *mnrec = nullptr, *mstack = nullptr, *mdmask = nullptr;
  double *mwrec = nullptr /*8*nn*/, *mlrec = nullptr /*8*nn*/;
  double* ltab = nullptr;  // 9 neighbour lengths of find_receiver / find_mult_rec

  // ---- captured intermediates (debug / parity) ----
  int *rec_pre = nullptr, *stack_pre = nullptr, *basins = nullptr, *outlets = nullptr;
  double* length_pre = nullptr;

  // ---- scratch ----
  int *s_flag = nullptr, *s_scan = nullptr, *s_roots = nullptr, *s_root_rank = nullptr;
  unsigned long long *s_list_a = nullptr, *s_list_b = nullptr;  // 2*nn each
  // the Euler tour's paths through the tiles (TourTiles::elements of them): list, walks, weights
  unsigned long long *s_tour = nullptr, *s_tour_sub = nullptr;
  unsigned* s_tour_weight = nullptr;
  // list ranking by sublist walks: predecessor flags, the shorter lists and the count of list heads
  unsigned char* s_rank_pred = nullptr;
  unsigned long long* s_rank_ws = nullptr;
  unsigned* s_rank_nheads = nullptr;
  // LocalMinima
  size_t conn_cap = 0;       // capacity of edge arrays
  size_t hash_cap = 0;       // capacity (power of two) of the basin-pair hash
  unsigned long long *ht_key = nullptr, *ht_wmin = nullptr;
  unsigned *ht_first = nullptr, *ht_best = nullptr;
  int *e_b1 = nullptr, *e_b2 = nullptr, *e_n1 = nullptr, *e_n2 = nullptr;
  double* e_w = nullptr;
  unsigned *e_key = nullptr, *e_key2 = nullptr;
  int *e_idx = nullptr, *e_idx2 = nullptr;
  int *o_b1 = nullptr, *o_b2 = nullptr, *o_n1 = nullptr, *o_n2 = nullptr;  // oriented copies
  int *r_b1 = nullptr, *r_b2 = nullptr, *r_n1 = nullptr, *r_n2 = nullptr;  // unsorted edges
  double* r_w = nullptr;
  int* nr_bsum = nullptr;  // per-block stopper totals of the cooperative NR sort
  int nr_bsum_cap = 0;
  int *nr_idx = nullptr, *nr_idx2 = nullptr, *nr_lf = nullptr, *nr_rf = nullptr, *nr_ls = nullptr,
      *nr_rs = nullptr, *nr_lpos = nullptr, *nr_rpos = nullptr, *nr_segof = nullptr;
  int *nr_seg = nullptr, *nr_seg2 = nullptr;  // segments: pairs (l, ir), 1-based
  int *nr_small = nullptr;                    // small segments (l, ir)
  int *nr_med = nullptr;                      // queue of the segments (l, ir) that blocks take
  double* nr_piv = nullptr;
  int* nr_segmeta = nullptr;  // per segment: pv, i, j, T
  int* nr_child = nullptr;    // per level segment: i, left id, right id, j (cooperative levels)
  int *e_rank = nullptr, *e_inmst = nullptr, *tree = nullptr;
  int *mst_comp = nullptr, *mst_min = nullptr, *mst_next = nullptr;
  int *arc_deg = nullptr, *arc_start = nullptr, *arc_slot = nullptr, *arc_adj = nullptr;
  // MFD order
  unsigned long long *o_keys = nullptr, *o_keys2 = nullptr;
  int *o_vals = nullptr, *o_vals2 = nullptr, *o_pos = nullptr;
  // heavy-path chain schedule (fsb_chains.cu)
  unsigned long long *ch_val = nullptr, *ch_val2 = nullptr;  // nn+1 each; scratch between the schedule's steps
  int *ch_ord = nullptr, *ch_flag = nullptr, *ch_start = nullptr, *ch_hist = nullptr, *ch_totals = nullptr;
  unsigned char *ch_head = nullptr, *ch_depth = nullptr;
  int4* ch_tk[4] = {};  // tickets: top-down long, short; bottom-up long, short chains
  bool chains_valid = false;  // the chain schedule matches the current forest
  // last-arriver sweeps (multiple flow)
  int *la_queue = nullptr, *la_cnt = nullptr, *cnt_acc = nullptr, *cnt_spl = nullptr;
  // one record per node (area, then stream power): 128 bytes of the queue engine, 96 or
  // 64 of the region sweeps
  void* mfd_line = nullptr;
  double* hw = nullptr;      // (elevation, water surface) pairs of the stream-power sweep
  double* slots = nullptr;   // kSlotStride input slots per node of the multiple-flow sweeps
  // region-owned sweeps (fsb_region.cu)
  TileMap tplan[kTilePlans];  // per tile side
  signed char region_ok[8] = {};  // per sweep op: 0 unchecked, 1 usable, -1 not
  unsigned short* rl_wmeta = nullptr;  // per node: inputs to wait for | dependents' directions << 8
  unsigned* rl_flags = nullptr;        // rim_words per tile
  double* rl_mbox = nullptr;           // rim_cells mailbox cells of up to 16 bytes per tile
  long long* rl_queue = nullptr;       // ready nodes: natural index << 32 | index within the CTA
  unsigned* la_ctl = nullptr;  // head, tail, done count
  int* s_scan2 = nullptr;
  // sweeps
  unsigned* ticket = nullptr;
  double* water = nullptr;
  double* hnew = nullptr;  // elevation written by the stream-power sweep
  // diffusion scratch: kdint, tridiagonal coefficients, forward factors, x-pass result
  double *dK = nullptr, *dA = nullptr, *dB = nullptr, *dC = nullptr, *dF = nullptr, *dG = nullptr, *dZ = nullptr;
  // counters on device and their pinned host mirror
  int* d_err = nullptr;   // device error word
  int* d_cnt = nullptr;   // small device counters
  int* h_cnt = nullptr;   // pinned host mirror of d_cnt
  void* cub_tmp = nullptr;
  size_t cub_tmp_bytes = 0;

  // last LocalMinima counts (host)
  int nbasins = 0, basin0 = 0, nconn = 0, tree_size = 0, nlocmin_before = 0, nlocmin_after = 0;

  // per-stage device timing (CUDA events on the instance's stream)
  // stages: uplift receivers stack locmin fill mfd accum spl diffusion advection;
  // then single kernels inside them: the area sweep, the stream-power sweep,
  // the row and the column tridiagonal solves of the diffusion, the lake fill
  // sweep
  static constexpr int kStages = 15;
  bool profile = false;
  cudaEvent_t ev_begin[kStages] = {}, ev_end[kStages] = {};
  bool ev_pending[kStages] = {};
  double stage_ms[kStages] = {};
  long long stage_calls[kStages] = {};

  std::string err;
};

// Dynamic shared memory beyond 48 KB.  cudaFuncSetAttribute holds up the other
// threads' launches (24 grids on 16 streams: 120 ms with three calls per
// instance, 92 without), so each kernel asks once per device; a
// refused launch asks again (the device's context may have been made anew).
template <auto Kernel>
struct BigSmem {
  static inline std::atomic<unsigned long long> devices{0};
  static bool allow(int bytes, bool again = false) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!again && (devices.load(std::memory_order_relaxed) & bit)) return true;
    if (cudaFuncSetAttribute((const void*)Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    devices.fetch_or(bit);
    return true;
  }
  // launches Kernel with up to `most` bytes; false when the device refuses it
  static bool launch(unsigned blocks, unsigned threads, size_t bytes, int most, cudaStream_t st, void** args) {
    for (int t = 0; t < 2; ++t) {
      if (!allow(most, t == 1)) return false;
      if (cudaLaunchKernel((const void*)Kernel, dim3(blocks), dim3(threads), args, bytes, st) == cudaSuccess) return true;
      cudaGetLastError();
    }
    return false;
  }
};

// per-stage / per-kernel CUDA events while profiling is on (fsb_api.cu)
enum { KT_AREA_SWEEP = 10, KT_SPL_SWEEP = 11, KT_THOMAS_ROWS = 12, KT_THOMAS_COLS = 13, KT_FILL = 14 };
void stage_begin(Ctx& c, int s);
void stage_end(Ctx& c, int s);

// sets the message fsb_last_error() returns; returns 1 (fsb_api.cu)
int report_error(const std::string& msg);

// routing (fsb_routing.cu)
void launch_uplift(Ctx& c);
void launch_find_receiver(Ctx& c, const double* h, int* rec, double* length);
void launch_find_donors(Ctx& c, const int* rec, int* ndon, int* don);
void build_stack(Ctx& c, const int* rec, int* ndon, int* don, int* stack, int* pos, int* size);
unsigned long long* list_rank(Ctx& c, size_t n, unsigned long long* a, unsigned long long* b);
// list ranking by sublist walks: a splitter every 16 or 4 entries plus each
// list head (at most kRankMaxHeads heads); a block ranks up to kRankBlock entries
constexpr int kRankMaxHeads = 4, kRankBlock = 8192;
// Tiles of the Euler tour (fsb_routing.cu): 2048 nodes, 64 x 32, or as wide (high)
// as a narrower grid's power of two and so much higher (wider), and list elements
// per tile: paths leave a tile from the two outermost rows and columns beyond
// which the grid goes on, or from the last root of a row.
constexpr int kTourNodes = 2048;
struct TourTiles {
  int lx = 6, ly = 5;  // log2 of the sides
  int tiles_x, tiles_y, slots;
  TourTiles(int nx, int ny) {
    while (lx > 2 && nx <= 1 << (lx - 1)) --lx, ++ly;
    if (lx == 6)
      while (ly > 2 && ny <= 1 << (ly - 1)) --ly, ++lx;
    tiles_x = ((nx - 1) >> lx) + 1;
    tiles_y = ((ny - 1) >> ly) + 1;
    const int inner = ((1 << lx) - (tiles_x > 1 ? 4 : 0)) * ((1 << ly) - (tiles_y > 1 ? 4 : 0));
    slots = 2 * (kTourNodes - inner) + (1 << ly);
  }
  size_t elements() const { return (size_t)tiles_x * tiles_y * slots; }
};
// scratch entries below a list of n: per level its splitters and their walk's results
inline size_t rank_scratch(size_t n) {
  size_t total = 0;
  while (n > (size_t)kRankBlock) {
    const size_t stride = n > 4 * ((size_t)kRankBlock - kRankMaxHeads) ? 16 : 4;
    n = (n + stride - 1) / stride + kRankMaxHeads;
    total += 2 * n;
  }
  return total + 2 * kRankBlock;  // a shorter list may take the finer stride and one level more
}

// primitives (fsb_prims.cu)
void exclusive_scan_int(Ctx& c, const int* in, int* out, size_t n);
void exclusive_scan_u32(Ctx& c, const unsigned* in, unsigned* out, size_t n);
void exclusive_scan_u64(Ctx& c, const unsigned long long* in, unsigned long long* out, size_t n);
void inclusive_scan_int(Ctx& c, const int* in, int* out, size_t n);
void sort_pairs_u32(Ctx& c, const unsigned* kin, unsigned* kout, const int* vin, int* vout, size_t n, int end_bit);
void sort_pairs_u64(Ctx& c, const unsigned long long* kin, unsigned long long* kout, const int* vin,
                    int* vout, size_t n);
size_t cub_temp_bytes_needed(size_t nn, size_t nconn);
void fetch_counters(Ctx& c, int n);  // d_cnt[0..n) -> h_cnt (synchronises the stream)

// LocalMinima (fsb_locmin.cu); returns false and sets c.err on failure
bool local_minima(Ctx& c);

// chains (fsb_chains.cu)
void build_chains(Ctx& c);          // heavy-first order + ticket lists of the current forest
void ensure_chains(Ctx& c);         // build_chains unless the schedule is current
void fill_chains(Ctx& c);
void area_chains(Ctx& c);
void spl_chains(Ctx& c, double* hnew);
void flux_chains(Ctx& c, double* flux);               // compute_fluxes' flux, single flow
void chi_chains(Ctx& c, double a0, double mn, double* chi);
void flux_mfd(Ctx& c, double* flux);                  // compute_fluxes' flux, multiple flow
// tridiagonal systems s0..s1-1, element t of system s at [t*L + s], F solved in place
// region-owned multiple-flow sweeps (fsb_region.cu); false: not usable, the
// queue engine of fsb_flow.cu runs instead
TileMap plan_tiles(int nx, int ny, int lt, int sms);
bool region_accumulate(Ctx& c);
bool region_stream_power(Ctx& c);
void thomas_lines(Ctx& c, int N, int L, int s0, int s1, const double* A, const double* B, const double* C,
                  double* const* F, double* G);
void advect(Ctx& c);  // fsb_advect.cu
int write_vtk(Ctx& c, const double* f_dev, double vex, const char* dir);  // fsb_vtk.cu
// the stream power law with the sediment term g > 0 (fsb_sediment.cu)
bool gs_active(const Ctx& c);
int stream_power_gs(Ctx& c);
void spl_chains_gs(Ctx& c, const double* elev, const double* hstart, double* hnew, int* sill, double* contrib);
void gs_erosion_chains(Ctx& c, const double* hp, const int* sill, double* lsed, double* dh);
void lake_volume_chains(Ctx& c, const int* sill, const double* contrib, double* vol, double* up);
void gs_erosion_mfd(Ctx& c, const double* e, const int* sill, double* lsed, double* dh);
void spl_mfd_gs(Ctx& c, const double* elev, const double* hstart, int* sill, double* contrib);
// derived fields (fsb_derived.cu)
void catchment(Ctx& c);                               // catch = catch0 of the root, before LocalMinima
void slope_field(Ctx& c, double* out);
void curvature_field(Ctx& c, double* out);
void add_layers(Ctx& c, const double* dh);
void flux_sums(Ctx& c, const double* flux, double* part, double* out3);

// flow (fsb_flow.cu)
void fill_sweep(Ctx& c);            // hwater along the stack (SFD lake fill / MFD h0)
void mfd_receivers(Ctx& c);         // find_mult_rec: mrec, mnrec, mlrec, mwrec, order
void accumulate(Ctx& c);            // drainage area
void stream_power(Ctx& c);          // implicit stream power law (g == 0)
void diffusion(Ctx& c);             // ADI hillslope diffusion
void diffusion_raw(const Bounds& bd, double dx, double dy, double dt, double kdsed, const double* kd, double* h,
                   double* b, double* etot, double* erate, double* scratch, int* err, cudaStream_t st);

}  // namespace fsb
