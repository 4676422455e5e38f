// Drift and cell binning, the counting sort by cell, and the packed FP32
// copies that the pair passes read. Replaces the FDPS tree build and the j
// gather of TreeForForceShort::Gather (src/main.cpp:124-132, 173-174) and
// performs drift_and_predict (driftkick.hpp:6-27) in the same pass.
#include <algorithm>

#include "row_ops.cuh"

namespace idpd {

// Whether the centre-of-mass drift removal is due for some replica, into the condition of
// its IF node; the whole block takes part.
__device__ __forceinline__ void set_cm_cond(const StepConds& c, const uint32_t* rep_time, int R) {
  int any = 0;
  for (int r = threadIdx.x; r < R; r += blockDim.x) any |= (rep_time[r] % kCmCorr) == 0u;
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) cudaGraphSetConditional(c.cm, any ? 1u : 0u);
}

// One thread per storage row: optional drift, then cell index and arrival slot.
__global__ void __launch_bounds__(kRowBlock) k_drift_bin(DevState d, int do_drift, int nrep,
                                                         StepConds conds) {
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int i = d.blk_row[blockIdx.x] + threadIdx.x, end = R->row_off + R->n;
  chain_wait();
  if (conds.cm_on && blockIdx.x == 0) set_cm_cond(conds, d.rep_time, nrep);
  if (i >= end) return;
  double p[3] = {d.px[i], d.py[i], d.pz[i]}, ds[3];
  if (do_drift) drift_row(d, R, i, p, ds);
  bin_row(d, R, i, p);
}

// Steps that keep the neighbour lists: drift, and the largest squared
// displacement since the last rebuild into the rebuild record.
//
// What bounds the elementwise kernels (this one, the pack, the kick): at 10^6 particles
// the FP64 unit (74 - 80 % busy, DRAM 11 - 19 %), so their products, conversions and
// comparisons, and six of the drift's nine sums, run in integer instructions
// (fp64_int.cuh); the sums left to the unit run beside them (all nine on it 59 us, six
// 52, none 56). 998k particles, us in a launch list: drift 75 -> 52, pack 61 -> 27, kick
// 31 -> 21; with the bonded forces of 984k beads 73 -> 52, 60 -> 34, 45 -> 41.
__global__ void __launch_bounds__(kRowBlock, 8) k_drift_disp(DevState d) {
  __shared__ float wmax[kRowBlock / 32];
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int i = d.blk_row[blockIdx.x] + threadIdx.x, end = R->row_off + R->n;
  chain_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) d.overflow[1] = 0;
  float m = 0.0f;
  if (i < end) {
    const uint32_t s = d.rank[i];
    const double r0[3] = {d.drx[s], d.dry[s], d.drz[s]};
    double p[3] = {d.px[i], d.py[i], d.pz[i]}, ds[3];
    drift_row(d, R, i, p, ds);
    m = displacement2(d, ds, r0);
  }
  note_displacement(d, m, wmax);
}

// (Taken by the drift's last block instead, behind a counter, it was no faster below 400k
// rows, and at 1M the drift grew by 5 us.)
__global__ void __launch_bounds__(256) k_vl_decide(VerletDev* v, const uint32_t* rep_time,
                                                   int nrep, StepConds conds) {
  chain_begin();
  if (threadIdx.x == 0) {
    const int rb = v->force || __uint_as_float(v->maxd2) > v->thr2;
    v->rebuild = rb;
    v->force = 0;
    v->maxd2 = 0u;
    v->rebuilds += (unsigned)rb;
    if (conds.on) cudaGraphSetConditional(conds.rebuild, rb ? 1u : 0u);
  }
  if (conds.cm_on) set_cm_cond(conds, rep_time, nrep);
}

// The binning of k_drift_bin on a rebuild step (positions already drifted).
__global__ void __launch_bounds__(kRowBlock) k_bin_gated(DevState d) {
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int i = d.blk_row[blockIdx.x] + threadIdx.x, end = R->row_off + R->n;
  chain_wait();
  if (!d.vdev->rebuild || i >= end) return;
  const double p[3] = {d.px[i], d.py[i], d.pz[i]};
  bin_row(d, R, i, p);
}

void launch_drift_disp(const DevState& d, int nblk, const Chain& st) {
  if (nblk > 0) launch(st, k_drift_disp, nblk, kRowBlock, 0, d);
}

void launch_vl_decide(const DevState& d, int R, const StepConds& c, const Chain& st) {
  launch(st, k_vl_decide, 1, 256, 0, d.vdev, d.rep_time, R, c);
}

void launch_bin_gated(const DevState& d, int nblk, const Chain& st) {
  if (nblk > 0) launch(st, k_bin_gated, nblk, kRowBlock, 0, d);
}

// ---------------------------------------------------------------- scan
constexpr int kScanThreads = 1024;
constexpr int kScanPerThread = 4;
constexpr int kScanTile = kScanThreads * kScanPerThread;

__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[w] = incl;
  __syncthreads();
  if (w == 0) {
    int s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
    int si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, si, o);
      if (lane >= o) si += t;
    }
    warp_sums[lane] = si - s;
    if (lane == 31) warp_sums[32] = si;
  }
  __syncthreads();
  total = warp_sums[32];
  const int res = incl - v + warp_sums[w];
  __syncthreads();
  return res;
}

// One tile's exclusive scan into start; returns its total.
__device__ __forceinline__ int scan_tile(const int* cnt, int* start, int base, int ncell, int* ws) {
  int c[kScanPerThread];
  int sum = 0;
#pragma unroll
  for (int k = 0; k < kScanPerThread; k++) {
    c[k] = (base + k < ncell) ? cnt[base + k] : 0;
    sum += c[k];
  }
  int total;
  int run = block_exclusive_scan(sum, ws, total);
#pragma unroll
  for (int k = 0; k < kScanPerThread; k++) {
    if (base + k < ncell) start[base + k] = run;
    run += c[k];
  }
  return total;
}

// Exclusive scan of the cell counts. A block per tile of 4,096 cells writes its tile's scan
// and total (k_scan_tiles); then each block adds the totals before its tile
// (k_scan_finish). Up to kScanOneBlock cells (T = 1 or 4 tiles) one block does it all, its
// tiles side by side between the same two barriers: one launch instead of two (13k cells,
// us: the tiles one after the other 6.9, 16 consecutive cells per thread 9.9, this 4.8; a step
// of 50k particles 73.3 -> 69.8, of 62k beads 139 -> 137). cnt and start are 16-byte aligned.
constexpr int kScanOneBlock = 4 * kScanTile;

template <int T>
__global__ void __launch_bounds__(kScanThreads) k_scan_small(int* cnt, int* start, int ncell,
                                                             int n_tot, const RepDev* last,
                                                             const int* gate, int* overflow) {
  __shared__ int ws[T][32], totals[T];
  chain_begin();
  if (gate && !*gate) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int c[T][kScanPerThread], sum[T], incl[T];
#pragma unroll
  for (int t = 0; t < T; t++) {
    const int base = t * kScanTile + (int)threadIdx.x * kScanPerThread;
    if (base + kScanPerThread <= ncell) {
      const int4 v = *reinterpret_cast<const int4*>(cnt + base);
      c[t][0] = v.x; c[t][1] = v.y; c[t][2] = v.z; c[t][3] = v.w;
    } else {
#pragma unroll
      for (int k = 0; k < kScanPerThread; k++) c[t][k] = base + k < ncell ? cnt[base + k] : 0;
    }
  }
#pragma unroll
  for (int t = 0; t < T; t++) {
    sum[t] = c[t][0] + c[t][1] + c[t][2] + c[t][3];
    incl[t] = sum[t];
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (int t = 0; t < T; t++) {
      const int v = __shfl_up_sync(0xffffffffu, incl[t], o);
      if (lane >= o) incl[t] += v;
    }
  }
  if (lane == 31) {
#pragma unroll
    for (int t = 0; t < T; t++) ws[t][w] = incl[t];
  }
  __syncthreads();
  if (w < T) {  // warp t scans tile t's warps
    const int s = ws[w][lane];
    int si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, si, o);
      if (lane >= o) si += v;
    }
    ws[w][lane] = si - s;
    if (lane == 31) totals[w] = si;
  }
  __syncthreads();
  int before = 0;
#pragma unroll
  for (int t = 0; t < T; t++) {
    const int base = t * kScanTile + (int)threadIdx.x * kScanPerThread;
    int4 v;
    v.x = before + ws[t][w] + incl[t] - sum[t];
    v.y = v.x + c[t][0];
    v.z = v.y + c[t][1];
    v.w = v.z + c[t][2];
    before += totals[t];
    if (base + kScanPerThread <= ncell) {
      *reinterpret_cast<int4*>(start + base) = v;
      *reinterpret_cast<int4*>(cnt + base) = make_int4(0, 0, 0, 0);  // ready for the next binning
    } else {
      const int x[kScanPerThread] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < kScanPerThread; k++) {
        if (base + k < ncell) {
          start[base + k] = x[k];
          cnt[base + k] = 0;
        }
      }
    }
  }
  if (threadIdx.x == 0) {
    start[ncell] = last ? last->row_off + last->n : n_tot;
    if (overflow) *overflow = 0;  // of the lists built next
  }
}
static_assert(kScanPerThread == 4 && kScanThreads == 1024, "a tile's scan");

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const int* cnt, int* start, int* part,
                                                             int ncell, const int* gate) {
  __shared__ int ws[33];
  chain_begin();
  if (gate && !*gate) return;
  const int total = scan_tile(cnt, start, blockIdx.x * kScanTile + threadIdx.x * kScanPerThread,
                              ncell, ws);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_finish(int* cnt, int* start, const int* part,
                                                              int ncell, int n_tot,
                                                              const RepDev* last,
                                                              const int* gate, int* overflow) {
  __shared__ int ws[33];
  chain_begin();
  if (gate && !*gate) return;
  int before = 0;
  for (int p = threadIdx.x; p < blockIdx.x; p += kScanThreads) before += part[p];
  int off;
  block_exclusive_scan(before, ws, off);
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanPerThread;
#pragma unroll
  for (int k = 0; k < kScanPerThread; k++) {
    if (base + k < ncell) {
      start[base + k] += off;
      cnt[base + k] = 0;  // ready for the next binning
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    start[ncell] = last ? last->row_off + last->n : n_tot;
    if (overflow) *overflow = 0;  // of the lists built next
  }
}

static void launch_scan_of(int* cnt, int* start, int* part, int ncell, int n_tot,
                           const RepDev* last, const int* gate, int* overflow, const Chain& st) {
  if (ncell <= kScanOneBlock) {
    launch(st, ncell <= kScanTile ? k_scan_small<1> : k_scan_small<4>, 1, kScanThreads, 0, cnt,
           start, ncell, n_tot, last, gate, overflow);
    return;
  }
  const int nb = (ncell + kScanTile - 1) / kScanTile;
  launch(st, k_scan_tiles, nb, kScanThreads, 0, cnt, start, part, ncell, gate);
  launch(Chain(st.st, true), k_scan_finish, nb, kScanThreads, 0, cnt, start, part, ncell, n_tot,
         last, gate, overflow);
}

void launch_scan(const DevState& d, int ncell_tot, int last_rep, const Chain& st,
                 const int* gate) {
  launch_scan_of(d.cell_cnt, d.cell_start, d.scan_part, ncell_tot, 0, d.reps + last_rep, gate,
                 d.overflow, st);
}

// ------------------------------------------------- scatter / sort / pack
__global__ void __launch_bounds__(kRowBlock) k_scatter(DevState d, const int* gate) {
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int i = d.blk_row[blockIdx.x] + threadIdx.x, end = R->row_off + R->n;
  chain_wait();
  if ((gate && !*gate) || i >= end) return;
  const uint32_t s = (uint32_t)d.cell_start[d.key[i]] + d.slot[i];
  d.arrival[s] = (uint32_t)i;
}

// Rows of one cell in ascending storage row: the order a stable counting
// sort gives, independent of the arrival order of the atomics (rows given as x y z
// triples; the step's rows are placed by k_sort_pack). A warp per
// cell: each of up to 128 rows finds its place by counting the smaller rows
// (rows are distinct); a larger cell is sorted by one lane in place.
__device__ __forceinline__ void sort_cell(uint32_t* perm, int b, int e, int lane) {
  const int n = e - b;
  if (n <= 1) return;
  if (n <= 128) {
    uint32_t v[4];
    int rank[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      v[q] = 32 * q + lane < n ? perm[b + 32 * q + lane] : 0xFFFFFFFFu;
      rank[q] = 0;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (32 * q >= n) break;  // warp-uniform
      for (int j = 0; j < 32; j++) {
        const uint32_t x = __shfl_sync(0xffffffffu, v[q], j);
#pragma unroll
        for (int m = 0; m < 4; m++) rank[m] += x < v[m];
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (32 * q + lane < n) perm[b + rank[q]] = v[q];
    __syncwarp();
    return;
  }
  if (lane == 0) {
    for (int k = b + 1; k < e; k++) {
      const uint32_t v = perm[k];
      int m = k - 1;
      while (m >= b && perm[m] > v) {
        perm[m + 1] = perm[m];
        m--;
      }
      perm[m + 1] = v;
    }
  }
  __syncwarp();
}

constexpr int kSortWarps = 8;
constexpr int kSortBlocks = 1216;  // 8 per SM of a GB300; the cells are strided over them

__global__ void __launch_bounds__(32 * kSortWarps) k_cell_sort(uint32_t* perm, const int* start,
                                                               int ncell) {
  const int lane = threadIdx.x & 31;
  for (int c = blockIdx.x * kSortWarps + (threadIdx.x >> 5); c < ncell; c += gridDim.x * kSortWarps)
    sort_cell(perm, start[c], start[c + 1], lane);
}

// Offset of x from its frame cell's origin o, at the periodic image nearest
// to the cell (a particle that crossed the box edge since the cells were
// built keeps its old cell). For a particle inside its cell, x - o is exact
// in FP64 (Sterbenz: x lies in [o, 2o] or o = 0).
__device__ __forceinline__ double cell_offset(double x, double o, double L, double half) {
  double v = __dsub_rn(x, o);
  if (abs_above(v, half)) v = plain_add(v, f64_bits(v) >> 63 ? L : -L);
  return v;
}

// The FP32 copies of storage row i at sorted slot s, in cell key: cell-local position,
// velocity and ids; zero: kZero* bits of what the passes after it add to.
__device__ __forceinline__ void pack_row(const DevState& d, const RepDev* R, uint32_t i, int s,
                                         uint32_t key, int zero) {
  int cx, cy, cz;
  cell_xyz((int)key - R->cell_off, R->nc, cx, cy, cz);
  cx >>= R->rshift;  // frame cell
  cy >>= R->rshift;
  cz >>= R->rshift;
  // the float split keeps 48 bits for the near-cutoff pair terms
  float lx, ly, lz, ex, ey, ez;
  split_double(cell_offset(d.px[i], mul_int_f64(cx, R->cs[0]), R->box[0], R->half_box[0]), lx, ex);
  split_double(cell_offset(d.py[i], mul_int_f64(cy, R->cs[1]), R->box[1], R->half_box[1]), ly, ey);
  split_double(cell_offset(d.pz[i], mul_int_f64(cz, R->cs[2]), R->box[2], R->half_box[2]), lz, ez);
  d.posf[s] = make_float4(lx, ly, lz, __uint_as_float(d.prop[i]));
  d.poslo[s] = make_float4(ex, ey, ez, 0.0f);
  d.velf[s] = make_float4(to_f32(d.vx[i]), to_f32(d.vy[i]), to_f32(d.vz[i]),
                          __uint_as_float(d.id[i]));
  if (d.svel) {  // FP64 engine-algorithm arm
    double* v = d.svel + 4 * (size_t)s;
    v[0] = d.vx[i];
    v[1] = d.vy[i];
    v[2] = d.vz[i];
  }
  const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (zero & kZeroForce) {
    float4* f = reinterpret_cast<float4*>(d.fq + 4 * (size_t)s);
    f[0] = z;
    f[1] = z;
  }
  if (zero & kZeroVirial) {
    float4* f = reinterpret_cast<float4*>(d.pq + 4 * (size_t)s);
    f[0] = z;
    f[1] = z;
  }
  if (zero & kZeroMarks) d.phit[s] = 0;
}

// One thread per arrival slot: the row's place in its cell, the order of ascending storage
// rows that a stable counting sort gives, is the number of smaller rows in the cell (the
// cell's rows are the neighbouring threads', so the reads are broadcasts), and its FP32
// copies are written there. One kernel instead of a sort by cell (a warp each) and a
// pass over the sorted rows. gate (may be null): device flag; when 0 the slots keep the
// rows and cells of the last rebuild, and only the copies are written.
__global__ void __launch_bounds__(kRowBlock) k_sort_pack(DevState d, int zero, const int* gate) {
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int k = d.blk_row[blockIdx.x] + threadIdx.x, end = R->row_off + R->n;
  chain_wait();
  const bool sort = !gate || *gate;
  if (k >= end) return;
  if (!sort) {
    pack_row(d, R, d.perm[k], k, d.scell[k], zero);
    return;
  }
  const uint32_t i = d.arrival[k], key = d.key[i];
  const int b = d.cell_start[key], e = d.cell_start[key + 1];
  int s = b;
  for (int q = b; q < e; q++) s += d.arrival[q] < i;
  d.perm[s] = i;
  d.rank[i] = (uint32_t)s;
  d.scell[s] = key;
  pack_row(d, R, i, s, key, zero);
}

// The copies alone, in a step whose rebuild is in an IF node (packed: device flag; when set
// k_sort_pack wrote them there).
__global__ void __launch_bounds__(kRowBlock) k_pack(DevState d, int zero, const int* packed) {
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int s = d.blk_row[blockIdx.x] + threadIdx.x, end = R->row_off + R->n;
  chain_wait();
  if (*packed || s >= end) return;
  pack_row(d, R, d.perm[s], s, d.scell[s], zero);
}

void launch_scan_raw(int* cnt, int* start, int* part, int ncell, int n_tot, cudaStream_t st) {
  launch_scan_of(cnt, start, part, ncell, n_tot, nullptr, nullptr, nullptr, st);
}

void launch_cell_sort_raw(uint32_t* perm, const int* start, int ncell, cudaStream_t st) {
  if (ncell > 0)
    k_cell_sort<<<std::min((ncell + kSortWarps - 1) / kSortWarps, kSortBlocks), 32 * kSortWarps,
                  0, st>>>(perm, start, ncell);
}

// Cell index and arrival slot of rows given as x y z triples (one grid, no
// replicas): the binning of k_drift_bin without the drift.
__global__ void __launch_bounds__(256) k_bin_rows(const double* pos, int n, double ix, double iy,
                                                  double iz, int nx, int ny, int nz,
                                                  uint32_t* cell, uint32_t* slot, int* cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* p = pos + 3 * (size_t)i;
  const int cx = cell_index(p[0], ix, nx);
  const int cy = cell_index(p[1], iy, ny);
  const int cz = cell_index(p[2], iz, nz);
  const uint32_t c = (uint32_t)((cz * ny + cy) * nx + cx);
  cell[i] = c;
  slot[i] = (uint32_t)atomicAdd(&cnt[c], 1);
}

__global__ void __launch_bounds__(256) k_scatter_rows(const uint32_t* cell, const uint32_t* slot,
                                                      const int* start, int n, uint32_t* perm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  perm[(uint32_t)start[cell[i]] + slot[i]] = (uint32_t)i;
}

void launch_bin_rows(const double* pos, int n, const double inv_cs[3], const int nc[3],
                     uint32_t* cell, uint32_t* slot, int* cnt, cudaStream_t st) {
  if (n > 0)
    k_bin_rows<<<(n + 255) / 256, 256, 0, st>>>(pos, n, inv_cs[0], inv_cs[1], inv_cs[2], nc[0],
                                                nc[1], nc[2], cell, slot, cnt);
}

void launch_scatter_rows(const uint32_t* cell, const uint32_t* slot, const int* start, int n,
                         uint32_t* perm, cudaStream_t st) {
  if (n > 0) k_scatter_rows<<<(n + 255) / 256, 256, 0, st>>>(cell, slot, start, n, perm);
}

void launch_drift_bin(const DevState& d, int nblk, bool do_drift, int R, const StepConds& c,
                      const Chain& st) {
  if (nblk > 0) launch(st, k_drift_bin, nblk, kRowBlock, 0, d, do_drift ? 1 : 0, R, c);
}

void launch_scatter_sort_pack(const DevState& d, int nblk, int zero, const Chain& st,
                              const int* gate) {
  if (nblk == 0) return;
  launch(st, k_scatter, nblk, kRowBlock, 0, d, gate);
  launch(Chain(st.st, true), k_sort_pack, nblk, kRowBlock, 0, d, zero, gate);
}

void launch_pack(const DevState& d, int nblk, int zero, const Chain& st, const int* packed) {
  if (nblk > 0) launch(st, k_pack, nblk, kRowBlock, 0, d, zero, packed);
}

// ------------------------------------------------------------- reorder
// Moves every storage-order field into sorted order: gathered into o's buffers of the same
// shape, the topology rewritten to the new rows, and copied back (captured steps hold d's
// pointers) together with the maps between storage, sorted and upload rows. The copy
// back was 18 copies and two more launches, 80 us more every 100 steps of a small system.
__global__ void __launch_bounds__(kRowBlock) k_reorder_gather(DevState d, DevState o) {
  const int r = d.blk_rep[blockIdx.x];
  const int s = d.blk_row[blockIdx.x] + threadIdx.x;
  const RepDev* R = d.reps + r;
  if (s >= R->row_off + R->n) return;
  const uint32_t i = d.perm[s];
  o.px[s] = d.px[i]; o.py[s] = d.py[i]; o.pz[s] = d.pz[i];
  o.vx[s] = d.vx[i]; o.vy[s] = d.vy[i]; o.vz[s] = d.vz[i];
  o.ax[s] = d.ax[i]; o.ay[s] = d.ay[i]; o.az[s] = d.az[i];
  o.dsx[s] = d.dsx[i]; o.dsy[s] = d.dsy[i]; o.dsz[s] = d.dsz[i];
  o.id[s] = d.id[i]; o.prop[s] = d.prop[i]; o.amp_id[s] = d.amp_id[i]; o.unit[s] = d.unit[i];
  o.orig[s] = d.orig[i];
  o.key[s] = d.key[i];
}

__global__ void k_reorder_topol(uint32_t* topol, const uint32_t* rank, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) topol[k] = rank[topol[k]];
}

__global__ void __launch_bounds__(kRowBlock) k_reorder_back(DevState d, DevState o) {
  const int r = d.blk_rep[blockIdx.x];
  const int s = d.blk_row[blockIdx.x] + threadIdx.x;
  const RepDev* R = d.reps + r;
  if (s >= R->row_off + R->n) return;
  d.px[s] = o.px[s]; d.py[s] = o.py[s]; d.pz[s] = o.pz[s];
  d.vx[s] = o.vx[s]; d.vy[s] = o.vy[s]; d.vz[s] = o.vz[s];
  d.ax[s] = o.ax[s]; d.ay[s] = o.ay[s]; d.az[s] = o.az[s];
  d.dsx[s] = o.dsx[s]; d.dsy[s] = o.dsy[s]; d.dsz[s] = o.dsz[s];
  d.id[s] = o.id[s]; d.prop[s] = o.prop[s]; d.amp_id[s] = o.amp_id[s]; d.unit[s] = o.unit[s];
  const uint32_t up = o.orig[s];
  d.orig[s] = up;
  d.key[s] = o.key[s];
  d.loc[up] = (uint32_t)s;
  d.perm[s] = (uint32_t)s;
  d.rank[s] = (uint32_t)s;
}

void launch_reorder(const DevState& d, const DevState& o, int nblk, int n_topol, cudaStream_t st) {
  if (nblk == 0) return;
  k_reorder_gather<<<nblk, kRowBlock, 0, st>>>(d, o);
  if (n_topol > 0) k_reorder_topol<<<(n_topol + 255) / 256, 256, 0, st>>>(d.topol, d.rank, n_topol);
  k_reorder_back<<<nblk, kRowBlock, 0, st>>>(d, o);
}

}  // namespace idpd
