// The two MDPD passes over the cell list:
//   pass 1, CalcDensity::operator() (nbdf_calculator.hpp:11-60);
//   pass 2, CalcForceEpEpDPD::operator() (nbdf_calculator.hpp:63-145).
//
// FP32 passes (the engine): each pair is taken once, by the particle that
// owns it (owns()), and its term goes to both particles. Pair vectors come
// from cell-local FP32 coordinates; cutoff decisions within kGuard of the
// cutoff are re-taken in FP64 from the FP64 positions as the reference takes
// them; pairs within 0.01 of the cutoff take 1 - r from the compensated
// (hi + lo) coordinates; every pair term is summed as a 64-bit fixed-point
// integer, so the result is independent of the visiting order, of the cell
// size and of the launch shape.
//
// FP64 passes (the plain single-system baseline): one thread per particle,
// FP64 throughout, FP64 sums in cell order.
#include <algorithm>

#include "cell_reach.hpp"
#include "pair_lists.cuh"

namespace idpd {

// ------------------------------------------------------------- pass 1
// Two kernels. k_pair_build finds each particle's owned candidates (owns()) from the
// cells: the kept lists on rebuild steps, or, without kept lists, on every step the
// owned pairs within the cutoff themselves, straight into the lists of pass 2.
// k_density_list goes over those lists: it takes each pair's density weight to both
// particles and, over kept lists, tests each candidate and writes the pairs within the
// cutoff as the list of pass 2. k_dens_finalize turns the fixed-point sums into the
// FP32 densities. The rows whose list overflowed are swept by k_density_over.

// The lists' densities, LP lanes per particle (LP 4, 8, 16 or 32). The warp sorts the
// rows of its chunk by list length and takes them 32 / LP at a time, so that short
// lists (a liquid at density 6 keeps ~20 owned candidates per particle) do not leave
// lanes idle and neighbours in that order run about as long; every LP gives the same
// densities and pass-2 lists bit for bit. KNOWN: the lists hold the pairs within the
// cutoff 1 already (pass 2's own, no kept lists). MARKS: the precursor conversion's
// marks (phit): a pair of prop_from and prop_near within the cutoff marks the
// prop_from particle. Rows whose list overflowed are left to k_density_over; a replica
// of another form (WARREN or not) to the other launch.
//
// What bounds it: instruction issue and the latency of the candidates' rows. The sums
// lie per property, so that the weights a group's lanes send to neighbouring rows share
// 32-byte sectors (one sector of four sums per row before, the SM's request port 50 %
// busy); frame offsets come from a table, the form is a template argument and a lane
// without a candidate needs no test of its own. 984k-bead membrane (8 lanes) 510 -> 407
// us, 998k-particle liquid (4 lanes) 197 -> 173 us.
template <bool MARKS, bool WARREN, bool KNOWN, int LP>
__global__ void __launch_bounds__(kRowBlock, 10) k_density_list(DevState d, int rows) {
  constexpr int G = 32 / LP;  // particles per warp at a time
  __shared__ OffTable OT;
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  if (threadIdx.x < 64) fill_off_table(OT, *R, threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int h = lane / LP, sl = lane % LP;
  const int s0 = d.blk_row[blockIdx.x] + 32 * wid + rows * blockIdx.y;
  const int nrow = min(rows, R->row_off + R->n - s0);
  const float cutd2 = WARREN ? R->wrd * R->wrd : 1.0f;  // density cutoff^2
  const float inv_rd = R->winv_rd, wnorm = R->wnorm, pre = R->dens_prescale;
  const bool prec = MARKS && R->prec_on;
  const bool other_form = (R->form == IDPD_FORM_WARREN_K) != WARREN;
  chain_wait();
  if (other_form || nrow <= 0) return;
  const uint32_t gmask = (LP == 32 ? 0xffffffffu : ((1u << LP) - 1u)) << (LP * h);
  const uint32_t group_lt = ((1u << lane) - 1u) & gmask;
  const uint16_t* len = KNOWN ? d.nbn : d.vn;
  // the chunk's rows sorted by list length, those without one (overflowed, or past the
  // end) last: key = length << 5 | row - s0
  uint32_t key = 0xffffffffu;
  if (lane < nrow) {
    const uint32_t n = (uint32_t)len[s0 + lane];
    if (n != kNbrFallback) key = (n << 5) | (uint32_t)lane;
  }
  const int nact = __popc(__ballot_sync(0xffffffffu, key != 0xffffffffu));
  key = warp_sort_asc(key, lane);
  for (int i2 = 0; i2 < nact; i2 += G) {
    const uint32_t ki = __shfl_sync(0xffffffffu, key, i2 + h);
    const bool act = i2 + h < nact;
    const int s = act ? s0 + (int)(ki & 31u) : s0;
    const int nv = act ? (int)(ki >> 5) : 0;
    const int nmax = (int)(__shfl_sync(0xffffffffu, key, min(i2 + G, nact) - 1) >> 5);
    const float4 pi = d.posf[s];
    const uint32_t pri = fbits(pi.w);
    const uint32_t none = (uint32_t)s | (kOffNone << kRowBits);
    unsigned long long* other = d.dsum + (pri & 3u) * d.dstride;
    int nl = 0;  // owned pairs within the cutoff
    bool hit = false;
    uint32_t q0 = 0, q1 = 0, q2 = 0;
    const uint32_t* list = KNOWN ? d.nbl + (size_t)s * kNbrCap : d.vl + (size_t)s * kVerletCap;
    uint32_t* out = d.nbl + (size_t)s * kNbrCap;
    uint32_t e_next = sl < nv ? list[sl] : none;  // one round ahead
    for (int k0 = 0; k0 < nmax; k0 += LP) {
      const uint32_t e = e_next;
      e_next = k0 + LP + sl < nv ? list[k0 + LP + sl] : none;
      const int t = (int)(e & kRowMask);
      const float4 pj = __ldg(d.posf + t);
      const auto o = OT.at(e >> kRowBits);  // far away on a lane without a candidate
      const float dr2 = dist2((pi.x - o.x) - pj.x, (pi.y - o.y) - pj.y, (pi.z - o.z) - pj.z);
      bool in1 = dr2 < (KNOWN ? 4.0f : 1.0f);
      bool ind = in1 && dr2 < cutd2 && dr2 >= 1.0e-10f;
      const bool near1 = !KNOWN && fabsf(dr2 - 1.0f) <= kGuard;
      const bool near2 = dr2 < 1.0e-10f || (WARREN && fabsf(dr2 - cutd2) <= kGuard);
      // rare: the FP64 decisions of the reference near the cutoffs and at
      // coincident positions
      if (__any_sync(0xffffffffu, near1 || near2)) {
        if (near1 || near2) {
          const double e2 = exact_dr2(d, R, d.perm[s], d.perm[t]);
          const double cutd2d = WARREN ? (double)R->wrd * (double)R->wrd : 1.0;
          if (near1) in1 = e2 < 1.0;
          ind = in1 && (near2 ? (e2 < cutd2d && e2 != 0.0) : (dr2 < cutd2 && dr2 >= 1.0e-10f));
        }
      }
      const uint32_t prj = fbits(pj.w);
      const uint32_t w = ind ? dens_weight(dr2, WARREN, inv_rd, wnorm, pre) : 0u;
      add_weight(q0, q1, q2, prj, w);
      red_add_if(ind, reinterpret_cast<long long*>(other + t), (long long)w);
      if (MARKS && prec && in1) {
        hit |= pri == R->prec_from && prj == R->prec_near;
        if (prj == R->prec_from && pri == R->prec_near) d.phit[t] = 1;
      }
      if (!KNOWN) {
        const uint32_t mask = __ballot_sync(0xffffffffu, in1);
        const int pos = nl + __popc(mask & group_lt);
        if (in1 && pos < kNbrCap) out[pos] = e;
        nl += __popc(mask & gmask);
      }
    }
    if (KNOWN) nl = nv;
    // the totals of each group's lanes: a list holds at most 512 entries and each weight is
    // below 2^23 (2^23 within 3e-8 of the particle, not for 512 partners), so a total fits 32 bits
#pragma unroll
    for (int o = 1; o < LP; o <<= 1) {
      q0 += __shfl_xor_sync(0xffffffffu, q0, o);
      q1 += __shfl_xor_sync(0xffffffffu, q1, o);
      q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    }
    const uint32_t q = sl == 0 ? q0 : (sl == 1 ? q1 : q2);
    red_add_if(act && sl < 3 && q != 0u,
               reinterpret_cast<long long*>(d.dsum + (sl < 3 ? sl : 0) * d.dstride + s), (long long)q);
    if (MARKS) hit = (__ballot_sync(0xffffffffu, hit) & gmask) != 0u;
    if (sl == 0 && act) {
      if (!KNOWN) {
        d.nbn[s] = nl <= kNbrCap ? (uint16_t)nl : (uint16_t)kNbrFallback;
        if (nl > kNbrCap) d.overflow[1] = 1;
      }
      d.npair[s] = 2u * (uint32_t)nl;  // ordered pairs: each owned pair counts twice
      if (MARKS && hit) d.phit[s] = 1;
    }
  }
}
static_assert((long long)kVerletCap * (1ll << 23) <= (1ll << 32) &&
              (long long)kNbrCap * (1ll << 23) <= (1ll << 32), "32-bit totals of pass 1");

// Pass 1 of the rows whose list overflowed (VERLET: the kept list, with the ownership
// of its build; else the pass-2 list), one warp per 32-row chunk, a row at a time:
// phase A sweeps the neighbour segments 32 candidates at a time and appends the owned
// pairs within the cutoff 1 to a list in shared memory; phase B takes the density
// weights from that list with every lane busy and copies the list out for pass 2 (a
// particle whose list overflows takes its weights during a second sweep). Shared
// memory: per warp the neighbour segments and the list (dens_sweep_smem_bytes). A few
// CTAs per SM stride over the row blocks and leave at once when the build had no such
// list: with a CTA per row block, reading the list lengths, the empty pass took 12 us
// at 10^6 particles (and pass 2's walk of its overflowed lists 16).
constexpr size_t dens_sweep_smem_bytes() {
  return kWarps * (sizeof(SegTable) + kNbrCap * sizeof(uint32_t));
}

template <int REACH, bool VERLET, bool MARKS>
__global__ void __launch_bounds__(kRowBlock) k_density_over(DevState d, int nblk) {
  extern __shared__ __align__(16) unsigned char dens_smem[];
  chain_begin();
  if (!d.overflow[0]) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  SegTable& S = reinterpret_cast<SegTable*>(dens_smem)[wid];
  uint32_t* L = reinterpret_cast<uint32_t*>(dens_smem + kWarps * sizeof(SegTable)) + wid * kNbrCap;
  for (int rb = blockIdx.x; rb < nblk; rb += gridDim.x) {
    const int r = d.blk_rep[rb];
    const RepDev* R = d.reps + r;
    const int s0 = d.blk_row[rb] + 32 * wid;
    const int s_end = min(s0 + 32, R->row_off + R->n);
    const uint16_t* len = VERLET ? d.vn : d.nbn;
    uint32_t todo = __ballot_sync(0xffffffffu, s0 + lane < s_end && len[s0 + lane] == kNbrFallback);
    const bool warren = R->form == IDPD_FORM_WARREN_K;
    const float cutd2 = R->wrd * R->wrd;  // density cutoff^2 (1 unless Warren)
    const double cutd2d = (double)R->wrd * (double)R->wrd;
    const float inv_rd = R->winv_rd, wnorm = R->wnorm, pre = R->dens_prescale;
    const float csx = R->cs_f[0], csy = R->cs_f[1], csz = R->cs_f[2];
    const bool prec = MARKS && R->prec_on;
    constexpr int nseg = 2 * (2 * REACH + 1) * (2 * REACH + 1);
    const uint32_t lt_mask = (1u << lane) - 1u;
    int cached = -1;
    for (; todo; todo &= todo - 1) {
      const int s = s0 + __ffs(todo) - 1;
      const float4 pi = d.posf[s];
      const uint32_t si = d.perm[s], pri = fbits(pi.w);
      const float ki = VERLET ? d.okey[s] : pi.x;  // the ownership key of the step
      int nl = 0;  // owned pairs within the cutoff
      bool hit = false;
      // 64-bit sums: one lane can take every pair of a long second sweep
      unsigned long long q0 = 0, q1 = 0, q2 = 0;
      // weight of one owned candidate, to both particles; called by every lane
      // together (valid = false for lanes without one) so that the rare FP64
      // recheck is warp-uniform
      auto test = [&](bool valid, int t, int dx, int dy, int dz, float4 pj, bool list_known) {
        const float ex = (pi.x - (float)dx * csx) - pj.x;
        const float ey = (pi.y - (float)dy * csy) - pj.y;
        const float ez = (pi.z - (float)dz * csz) - pj.z;
        const float dr2 = dist2(ex, ey, ez);
        bool in1 = valid && (list_known || dr2 < 1.0f);
        bool ind = in1 && dr2 < cutd2 && dr2 >= 1.0e-10f;
        const bool near1 = valid && !list_known && fabsf(dr2 - 1.0f) <= kGuard;
        const bool near2 = valid && ((warren && fabsf(dr2 - cutd2) <= kGuard) || dr2 < 1.0e-10f);
        if (__any_sync(0xffffffffu, near1 || near2)) {
          if (near1 || near2) {
            const double e2 = exact_dr2(d, R, si, d.perm[t]);
            if (near1) in1 = e2 < 1.0;
            ind = in1 && (near2 ? (e2 < cutd2d && e2 != 0.0) : (dr2 < cutd2 && dr2 >= 1.0e-10f));
          }
        }
        const uint32_t prj = fbits(pj.w);
        if (ind) {
          const uint32_t w = dens_weight(dr2, warren, inv_rd, wnorm, pre);
          add_weight(q0, q1, q2, prj, w);
          atomicAdd(d.dsum + (pri & 3u) * d.dstride + t, (unsigned long long)w);
        }
        if (MARKS && prec && in1) {
          hit |= pri == R->prec_from && prj == R->prec_near;
          if (prj == R->prec_from && pri == R->prec_near) d.phit[t] = 1;
        }
      };
      const int cell = (int)d.scell[s];
      if (cell != cached) {
        int cx, cy, cz;
        cell_xyz(cell - R->cell_off, R->nc, cx, cy, cz);
        __syncwarp();
        build_segments(S, d, R, cx, cy, cz, lane);
        __syncwarp();
        cached = cell;
      }
      // ---- phase A: the owned pairs within the cutoff 1
#pragma unroll 1
      for (int g = 0; g < nseg; g++) {
        const int tb = S.tb[g], te = S.te[g];
        if (tb >= te) continue;
        const int code = S.code[g];
        int b[2 * REACH];
#pragma unroll
        for (int q = 0; q < 2 * REACH; q++) b[q] = S.bnd[g][q];
        const int fx0 = (code & 7) - 4, dy = ((code >> 3) & 7) - 4, dz = ((code >> 6) & 7) - 4;
        const float by = pi.y - (float)dy * csy, bz = pi.z - (float)dz * csz;
        for (int t0 = tb; t0 < te; t0 += 32) {
          const int t = t0 + lane;
          bool in1 = false, near = false;
          int ddx = 0;
          if (t < te && t != s) {
            const float4 pj = __ldg(d.posf + t);
            ddx = frame_step<REACH>(t, b);
            if (owns(fx0 + ddx, VERLET ? d.okey[t] : pj.x, ki, t, s)) {
              const float dr2 =
                  dist2((pi.x - (float)(fx0 + ddx) * csx) - pj.x, by - pj.y, bz - pj.z);
              in1 = dr2 < 1.0f;
              near = fabsf(dr2 - 1.0f) <= kGuard;
            }
          }
          if (__any_sync(0xffffffffu, near)) {
            if (near) in1 = exact_dr2(d, R, si, d.perm[t]) < 1.0;
          }
          const uint32_t mask = __ballot_sync(0xffffffffu, in1);
          if (in1) {
            const int pos = nl + __popc(mask & lt_mask);
            if (pos < kNbrCap) L[pos] = make_entry(t, fx0 + ddx, dy, dz);
          }
          nl += __popc(mask);
        }
      }
      __syncwarp();
      const bool fits = nl <= kNbrCap;
      // ---- phase B: density weights
      if (fits) {
        for (int k0 = 0; k0 < nl; k0 += 32) {
          const int k = k0 + lane;
          const bool valid = k < nl;
          int t = s, dx = 0, dy = 0, dz = 0;
          if (valid) read_entry(L[k], t, dx, dy, dz);
          test(valid, t, dx, dy, dz, valid ? __ldg(d.posf + t) : pi, true);
        }
      } else {
        if (nl > kDensPairsMax && lane == 0) atomicCAS(d.err, 0, kErrDensPairs);
#pragma unroll 1
        for (int g = 0; g < nseg; g++) {
          const int tb = S.tb[g], te = S.te[g];
          if (tb >= te) continue;
          const int code = S.code[g];
          int b[2 * REACH];
#pragma unroll
          for (int q = 0; q < 2 * REACH; q++) b[q] = S.bnd[g][q];
          const int fx0 = (code & 7) - 4, dy = ((code >> 3) & 7) - 4, dz = ((code >> 6) & 7) - 4;
          for (int t0 = tb; t0 < te; t0 += 32) {
            const int t = t0 + lane;
            const int dx = fx0 + frame_step<REACH>(t, b);
            const float4 pj = t < te ? __ldg(d.posf + t) : pi;
            const bool valid = t < te && t != s && owns(dx, VERLET ? d.okey[t] : pj.x, ki, t, s);
            test(valid, valid ? t : s, dx, dy, dz, pj, false);
          }
        }
      }
      __syncwarp();
      if (fits) {  // list out for pass 2, coalesced
        uint32_t* out = d.nbl + (size_t)s * kNbrCap;
        for (int k = lane; k < nl; k += 32) out[k] = L[k];
      }
      unsigned long long a0 = q0, a1 = q1, a2 = q2;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
      }
      if (MARKS) hit = __any_sync(0xffffffffu, hit);
      if (lane == 0) {
        if (a0) atomicAdd(d.dsum + s, a0);
        if (a1) atomicAdd(d.dsum + d.dstride + s, a1);
        if (a2) atomicAdd(d.dsum + 2 * d.dstride + s, a2);
        d.nbn[s] = fits ? (uint16_t)nl : (uint16_t)kNbrFallback;
        if (!fits) d.overflow[1] = 1;
        d.npair[s] = 2u * (uint32_t)nl;  // ordered pairs: each owned pair counts twice
        if (MARKS && hit) d.phit[s] = 1;
      }
      __syncwarp();
    }
  }
}

// The FP32 densities of pass 1 from its fixed-point sums (and the fixed-point
// densities of the fine-grained API); the sums are zeroed for the next pass.
__global__ void __launch_bounds__(kRowBlock) k_dens_finalize(DevState d) {
  chain_launch();
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int s = d.blk_row[blockIdx.x] + threadIdx.x, end = R->row_off + R->n;
  const float u = R->dens_unscale_f;
  chain_wait();
  if (s >= end) return;
  unsigned long long *q0 = d.dsum + s, *q1 = q0 + d.dstride, *q2 = q1 + d.dstride;
  const long long a0 = (long long)*q0, a1 = (long long)*q1, a2 = (long long)*q2;
  d.densf[s] = make_float4(fix_to_float(a0, u), fix_to_float(a1, u), fix_to_float(a2, u), 0.0f);
  if (d.dqx) {
    d.dqx[s] = a0;
    d.dqy[s] = a1;
    d.dqz[s] = a2;
  }
  *q0 = *q1 = *q2 = 0ull;
}

// The forward half of a cell's stencil as one range of candidates: per (dy, dz) row of
// search cells the run from the particle's own frame cell column to the stencil's +x
// end (the -x frame column is never owned), its part beyond the box edge apart. A
// candidate's frame offset in x is 0 or 1.
struct HalfStencil {
  struct alignas(16) Part {
    int shift;      // row - candidate number
    int end;        // candidates up to and including this part
    int fwd;        // first row whose x offset is 1
    uint32_t code;  // the frame offsets y and z of a list entry
    float oy, oz;   // the same in length
  } part[kMaxSeg];
};

// Lane k < (2m+1)^2 sets up row k (two parts); returns the number of candidates.
__device__ __forceinline__ int half_stencil(HalfStencil& S, const DevState& d, const RepDev* R,
                                            int cx, int cy, int cz, int lane) {
  const int m = R->reach, w = 2 * m + 1, rs = R->rshift;
  const int nx = R->nc[0], ny = R->nc[1], nz = R->nc[2];
  int n0 = 0, n1 = 0, b0 = 0, b1 = 0, f0 = 0x7fffffff, fy = 0, fz = 0;
  if (lane < w * w) {
    const int dz = lane / w - m, dy = lane % w - m;
    const int qz = cz + dz, wz = qz < 0 ? qz + nz : (qz >= nz ? qz - nz : qz);
    const int qy = cy + dy, wy = qy < 0 ? qy + ny : (qy >= ny ? qy - ny : qy);
    const int* start = d.cell_start + R->cell_off + (wz * ny + wy) * nx;
    const int lo = cx & ~(m - 1), hi = cx + m;  // lo: first search cell of the frame cell
    b0 = start[lo];
    n0 = start[min(hi, nx - 1) + 1] - b0;
    if (lo + m < nx) f0 = start[lo + m];
    if (hi >= nx) {  // beyond the edge: the next frame cell
      b1 = start[0];
      n1 = start[hi - nx + 1] - b1;
    }
    fy = (qy >> rs) - (cy >> rs);
    fz = (qz >> rs) - (cz >> rs);
  }
  int end = n0 + n1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += v;
  }
  if (lane < w * w) {
    const uint32_t code = make_entry(0, -1, fy, fz);
    const float oy = (float)fy * R->cs_f[1], oz = (float)fz * R->cs_f[2];
    S.part[2 * lane] = {b0 - (end - n1 - n0), end - n1, f0, code, oy, oz};
    S.part[2 * lane + 1] = {b1 - (end - n1), end, b1, code, oy, oz};
  }
  return __shfl_sync(0xffffffffu, end, 31);
}

// Two particles of a batch, as the packed FP32 instructions take them, and the lengths of
// their lists so far: xy = (x, x', y, y'), zn = (z, z', length, length').
struct BatchPair {
  float4 xy, zn;
  __device__ __forceinline__ void set(int which, float x, float y, float z) {
    (&xy.x)[which] = x;
    (&xy.z)[which] = y;
    (&zn.x)[which] = z;
    (&zn.z)[which] = __int_as_float(0);
  }
  __device__ __forceinline__ int length(int which) const { return __float_as_int((&zn.z)[which]); }
};

// The lists from the cells. KEPT: the kept lists (rebuild steps only), every owned
// candidate closer than 1 + skin in FP32 (with a margin: the list only has to hold
// every pair that can come within the cutoff before the next rebuild); it also keeps
// the cell-local x of the build (okey) and each row's delta_sumr for the displacement
// test. Else (no kept lists, every step): the owned pairs within the cutoff, decisions
// near it re-taken in FP64, straight into the lists of pass 2.
//
// The particles of one cell share its candidates and, per candidate, the frame
// offset, so a warp takes one cell at a time and up to 32 of its particles at once:
// each lane holds one candidate, every particle of the batch is tested against the 32
// (one ballot per particle), and the lanes whose candidate is in range append it to
// that particle's list in one coalesced store. The candidates of all the stencil's rows
// are numbered through, so that each load round has 32 of them (by segment, a round
// held a liquid's 26 to 40 in one or two loads); those farther than 1 + skin from the
// batch's bounding box (about a quarter) are dropped and the others queued into full
// rounds. Each warp builds the lists of its own chunk of `rows` rows, one cell's share of
// it at a time (a cell split between chunks is set up by each).
//
// What bounds it: instruction issue of the tests, about 25 instructions per particle and 32
// candidates. Two particles are tested together, so that the distances take the packed
// FP32 instructions, each rounded as the scalar one (984k-bead membrane 620 -> 531 us per
// rebuild, 998k-particle liquid 329 -> 298, 131k beads without kept lists 163 -> 152 us of
// pass 1). Fewer registers (a cap for 10 or 12 CTAs per SM) cost 6 and 12 %, loads of the
// next candidates one round ahead 5 %, a cell's candidates shared by the CTA's warps 3 to
// 20 % below 100k rows. Kept lists, per rebuild, against a sweep of each particle's cells:
// 984k beads 742 us, the liquid 441, 8k beads 105 (now 27).
// Without kept lists it replaces a sweep of each particle's own 27 cells by one warp
// (pass 1 in all: 400k-particle liquid 766 -> 173 us, 131k-bead membrane 543 -> 152 us, 31k
// beads with solvent 397 -> 55 us, 3k particles 206 -> 20 us).
template <bool KEPT>
__global__ void __launch_bounds__(kRowBlock) k_pair_build(DevState d, int rows) {
  __shared__ HalfStencil seg[kWarps];
  __shared__ BatchPair batch[kWarps][16];
  __shared__ float4 qpos[kWarps][64];
  __shared__ uint32_t qent[kWarps][64];
  chain_launch();
  if (KEPT) {  // (the constants' loads held over the wait cost rebuilds 2 %)
    chain_wait();
    if (!d.vdev->rebuild) return;
  }
  const RepDev* R = d.reps + d.blk_rep[blockIdx.x];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  HalfStencil& S = seg[wid];
  BatchPair* P = batch[wid];
  float4* QX = qpos[wid];
  uint32_t* QE = qent[wid];
  uint32_t* lists = KEPT ? d.vl : d.nbl;
  constexpr int cap = KEPT ? kVerletCap : kNbrCap;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const int s0 = d.blk_row[blockIdx.x] + 32 * wid + rows * blockIdx.y;
  const int s_end = min(s0 + rows, R->row_off + R->n);
  const float csx = R->cs_f[0];
  if (!KEPT) {
    chain_wait();
    if (blockIdx.x + blockIdx.y == 0 && threadIdx.x == 0) d.overflow[1] = 0;
  }
  const float prune2 = KEPT ? d.vdev->rv2 : 1.0f + 1.0e-4f;
  const float rv2 = KEPT ? prune2 : 1.0f;
  // the chunk's rows cell by cell: [cs, ce) are the chunk's rows of one cell
  for (int cs = s0; cs < s_end;) {
    const int cell = (int)d.scell[cs];
    const int ce = min(d.cell_start[cell + 1], s_end);
    int cx, cy, cz;
    cell_xyz(cell - R->cell_off, R->nc, cx, cy, cz);
    __syncwarp();
    const int total = half_stencil(S, d, R, cx, cy, cz, lane);
    for (int b0 = cs; b0 < ce; b0 += 32) {
      const int nb = min(32, ce - b0);
      const int me = b0 + lane;  // the lane's particle (lane < nb)
      __syncwarp();
      const float4 pm = lane < nb ? d.posf[me] : d.posf[b0];
      P[lane >> 1].set(lane & 1, lane < nb ? pm.x : 1.0e18f, pm.y, pm.z);
      float lox = pm.x, hix = pm.x, loy = pm.y, hiy = pm.y, loz = pm.z, hiz = pm.z;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lox = fminf(lox, __shfl_xor_sync(0xffffffffu, lox, o));
        hix = fmaxf(hix, __shfl_xor_sync(0xffffffffu, hix, o));
        loy = fminf(loy, __shfl_xor_sync(0xffffffffu, loy, o));
        hiy = fmaxf(hiy, __shfl_xor_sync(0xffffffffu, hiy, o));
        loz = fminf(loz, __shfl_xor_sync(0xffffffffu, loz, o));
        hiz = fmaxf(hiz, __shfl_xor_sync(0xffffffffu, hiz, o));
      }
      __syncwarp();
      int qn = 0;  // candidates queued for the next full round
      // tests the 32 queued candidates against every particle of the batch, two at a
      // time: the lanes whose candidate is in range of a particle write it to its
      // list, consecutive lanes to consecutive slots
      auto round = [&](float qx, float qy, float qz, uint32_t e, int t) {
        // owns(): a candidate of the next frame column is owned by all, else qx is its
        // cell-local x (a particle never owns itself)
        const float qk = ((e >> kRowBits) & 3u) == 2u ? 3.0e38f : qx;
        const f32x2 nx = pack2(-qx, -qx), ny = pack2(-qy, -qy), nz = pack2(-qz, -qz);
#pragma unroll 1
        for (int k = 0; k < nb; k += 2) {
          const float4 xy = P[k >> 1].xy, zn = P[k >> 1].zn;
          const f32x2 ex = add2(pack2(xy.x, xy.y), nx), ey = add2(pack2(xy.z, xy.w), ny),
                      ez = add2(pack2(zn.x, zn.y), nz);
          float d0, d1;  // dist2() of both
          unpack2(fma2(ez, ez, fma2(ex, ex, mul2(ey, ey))), d0, d1);
          const bool own0 = (qk > xy.x) | ((qk == xy.x) & (t > b0 + k));
          const bool own1 = (qk > xy.y) | ((qk == xy.y) & (t > b0 + k + 1));
          bool in0 = (d0 < rv2) & own0, in1 = (d1 < rv2) & own1;
          if (!KEPT) {
            const bool near0 = (fabsf(d0 - 1.0f) <= kGuard) & own0;
            const bool near1 = (fabsf(d1 - 1.0f) <= kGuard) & own1;
            if (__any_sync(0xffffffffu, near0 | near1)) {
              if (near0) in0 = exact_dr2(d, R, d.perm[b0 + k], d.perm[t]) < 1.0;
              if (near1) in1 = exact_dr2(d, R, d.perm[b0 + k + 1], d.perm[t]) < 1.0;
            }
          }
          const uint32_t m0 = __ballot_sync(0xffffffffu, in0);
          const uint32_t m1 = __ballot_sync(0xffffffffu, in1);
          const int n0 = __float_as_int(zn.z), n1 = __float_as_int(zn.w);
          const int at0 = n0 + __popc(m0 & lt_mask), at1 = n1 + __popc(m1 & lt_mask);
          uint32_t* list = lists + (size_t)(b0 + k) * cap;
          if (in0 && at0 < cap) list[at0] = e;
          if (in1 && at1 < cap) list[cap + at1] = e;
          if (lane == 0)
            *reinterpret_cast<float2*>(&P[k >> 1].zn.z) =
                make_float2(__int_as_float(n0 + __popc(m0)), __int_as_float(n1 + __popc(m1)));
        }
        __syncwarp();
      };
      int g = 0;  // the lane's part of the stencil
      HalfStencil::Part part = S.part[0];
      for (int k0 = 0; k0 < total; k0 += 32) {
        const int c = k0 + lane;
        bool keep = false;
        float qx = 0.0f, qy = 0.0f, qz = 0.0f;
        uint32_t e = 0;
        int t = 0;
        if (c < total) {
          while (c >= part.end) part = S.part[++g];
          t = c + part.shift;
          // the candidate in the frame of the cell's particles
          const float4 pj = __ldg(d.posf + t);
          const bool fx = t >= part.fwd;
          qx = fx ? csx + pj.x : pj.x;
          qy = part.oy + pj.y;
          qz = part.oz + pj.z;
          e = (uint32_t)t | part.code | (fx ? 2u : 1u) << kRowBits;
          const float ox = fmaxf(fmaxf(lox - qx, qx - hix), 0.0f);
          const float oy = fmaxf(fmaxf(loy - qy, qy - hiy), 0.0f);
          const float oz = fmaxf(fmaxf(loz - qz, qz - hiz), 0.0f);
          keep = ox * ox + oy * oy + oz * oz < prune2;
        }
        const uint32_t mask = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int at = qn + __popc(mask & lt_mask);
          QX[at] = make_float4(qx, qy, qz, __int_as_float(t));
          QE[at] = e;
        }
        qn += __popc(mask);
        if (qn >= 32) {
          __syncwarp();
          const float4 q = QX[lane];
          const uint32_t qe = QE[lane];
          __syncwarp();
          if (lane < qn - 32) {
            QX[lane] = QX[32 + lane];
            QE[lane] = QE[32 + lane];
          }
          __syncwarp();
          qn -= 32;
          round(q.x, q.y, q.z, qe, __float_as_int(q.w));
        }
      }
      __syncwarp();
      if (qn > 0) {  // the last, partial round (absent lanes far away)
        float4 q = make_float4(1.0e18f, 0.0f, 0.0f, __int_as_float(-1));
        uint32_t qe = 0;
        if (lane < qn) {
          q = QX[lane];
          qe = QE[lane];
        }
        round(q.x, q.y, q.z, qe, __float_as_int(q.w));
      }
      __syncwarp();
      if (lane < nb) {
        const int cnt = P[lane >> 1].length(lane & 1);
        (KEPT ? d.vn : d.nbn)[me] = cnt <= cap ? (uint16_t)cnt : (uint16_t)kNbrFallback;
        if (cnt > cap) d.overflow[0] = 1;
        if (KEPT) {
          d.okey[me] = pm.x;
          const uint32_t i = d.perm[me];
          d.drx[me] = d.dsx[i];
          d.dry[me] = d.dsy[i];
          d.drz[me] = d.dsz[i];
        }
      }
    }
    cs = ce;
  }
}

void launch_verlet_build(const DevState& d, int nblk, const Chain& st) {
  const int rows = build_rows(nblk);
  if (nblk > 0) launch(st, k_pair_build<true>, dim3(nblk, 32 / rows), kRowBlock, 0, d, rows);
}

// Plain FP64 pass 1 of one sorted row: FP64 positions of the storage rows,
// FP64 sums. Returns the row's ordered pairs within the cutoff 1.
__device__ __forceinline__ unsigned int density_f64_row(const DevState& d, int r, int s,
                                                        const RepDev* R) {
  const RepTab64* T = d.tab64 + r;
  const uint32_t i = d.perm[s];
  const double xi = d.px[i], yi = d.py[i], zi = d.pz[i];
  int cx, cy, cz;
  cell_xyz((int)d.scell[s] - R->cell_off, R->nc, cx, cy, cz);
  const bool warren = R->form == IDPD_FORM_WARREN_K;
  const double rd = T->wrd;
  const double cut2 = warren ? rd * rd : 1.0;
  const double wn = 15.0 / (2.0 * 3.14159265358979323846 * rd * rd * rd);
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  unsigned int np = 0;  // ordered pairs within the cutoff 1
  for_each_cell(R, R->reach, cx, cy, cz, [&](int cn, int, int, int, int sx, int sy, int sz) {
    const double shx = (double)sx * R->box[0], shy = (double)sy * R->box[1],
                 shz = (double)sz * R->box[2];
    for (int t = d.cell_start[cn]; t < d.cell_start[cn + 1]; t++) {
      const uint32_t j = d.perm[t];
      const double ex = xi - (d.px[j] + shx), ey = yi - (d.py[j] + shy), ez = zi - (d.pz[j] + shz);
      const double dr2 = ex * ex + ey * ey + ez * ez;
      np += (dr2 < 1.0 && t != s) ? 1u : 0u;
      if (dr2 < cut2 && dr2 != 0.0) {
        const double dr = sqrt(dr2);
        double w;
        if (warren) {
          const double u = 1.0 - dr / rd;
          w = wn * (u * u);
        } else {
          w = (1.0 - dr) * (1.0 - dr);
        }
        const uint32_t pr = d.prop[j];
        if (pr == 0) a0 += w;
        else if (pr == 1) a1 += w;
        else a2 += w;
      }
    }
  });
  d.dens64[3 * s] = a0;
  d.dens64[3 * s + 1] = a1;
  d.dens64[3 * s + 2] = a2;
  d.densf[s] = make_float4((float)a0, (float)a1, (float)a2, 0.0f);
  if (d.dqx) {
    d.dqx[s] = __double2ll_rn(a0 / R->dens_unscale);
    d.dqy[s] = __double2ll_rn(a1 / R->dens_unscale);
    d.dqz[s] = __double2ll_rn(a2 / R->dens_unscale);
  }
  return np;
}

__global__ void __launch_bounds__(kRowBlock) k_density_f64(DevState d) {
  chain_begin();
  const int r = d.blk_rep[blockIdx.x];
  const int s = d.blk_row[blockIdx.x] + threadIdx.x;
  const RepDev* R = d.reps + r;
  if (s < R->row_off + R->n) d.npair[s] = density_f64_row(d, r, s, R);
}

template <bool MARKS, bool WARREN, bool KNOWN>
void launch_density_lists(const DevState& d, int nblk, int lanes, const Chain& st) {
  const int rows = chunk_rows(nblk, lanes);
  void (*k)(DevState, int) = lanes == 4    ? k_density_list<MARKS, WARREN, KNOWN, 4>
                             : lanes == 8  ? k_density_list<MARKS, WARREN, KNOWN, 8>
                             : lanes == 16 ? k_density_list<MARKS, WARREN, KNOWN, 16>
                                           : k_density_list<MARKS, WARREN, KNOWN, 32>;
  launch(st, k, dim3(nblk, 32 / rows), kRowBlock, 0, d, rows);
}

template <int REACH, bool VERLET, bool MARKS>
void launch_density_f32(const DevState& d, int nblk, int lanes, int form_mask, Chain st) {
  if (!VERLET) {
    const int rows = build_rows(nblk);
    launch(st, k_pair_build<false>, dim3(nblk, 32 / rows), kRowBlock, 0, d, rows);
    st.chained = true;
    // whatever the tuning's lanes for kept lists. Us per step at 16 / 8 / 4 lanes: liquids, 3k
    // 32.9 / 33.5 / 34.4, 6k 36.5 / 37.2 / 37.2, 50k 74.9 / 73.3 / 72.9, 400k 324 / 311 / 304; 31k
    // mixed 100.0 / 99.3 / 104.4, 131k membrane 279 / 277 / 281
    lanes = nblk * kRowBlock < 16384 ? 16 : 8;
  }
  if (form_mask & (1 << IDPD_FORM_WARREN_K)) {
    launch_density_lists<MARKS, true, !VERLET>(d, nblk, lanes, st);
    st.chained = true;
  }
  if (form_mask & ~(1 << IDPD_FORM_WARREN_K)) {
    launch_density_lists<MARKS, false, !VERLET>(d, nblk, lanes, st);
    st.chained = true;
  }
  launch(st, k_density_over<REACH, VERLET, MARKS>, std::min(nblk, kRareBlocks), kRowBlock,
         dens_sweep_smem_bytes(), d, nblk);
}

template <bool MARKS>
void launch_density_f32(const DevState& d, int nblk, int reach, bool verlet, int lanes,
                        int form_mask, const Chain& st) {
  if (reach == 2 && verlet)
    launch_density_f32<2, true, MARKS>(d, nblk, lanes, form_mask, st);
  else if (reach == 2)
    launch_density_f32<2, false, MARKS>(d, nblk, lanes, form_mask, st);
  else if (verlet)
    launch_density_f32<1, true, MARKS>(d, nblk, lanes, form_mask, st);
  else
    launch_density_f32<1, false, MARKS>(d, nblk, lanes, form_mask, st);
}

// The reference's pair expression in FP64 (nbdf_calculator.hpp:84-132): the
// pair force over dr, for one pair within the cutoff, with the FP64 tables
// and the reference's FP64 Box-Muller.
__device__ __forceinline__ double pair_cf64(const RepTab64* T, int form, uint32_t pri,
                                            uint32_t prj, double dr2, double ex, double ey,
                                            double ez, double dvx, double dvy, double dvz,
                                            double di0, double di1, double di2, double dj0,
                                            double dj1, double dj2, uint32_t idi, uint32_t idj,
                                            uint32_t seed) {
  Saru sr(idi < idj ? idi : idj, idi < idj ? idj : idi, seed);
  const double rnd = saru_nrml_f64(sr);
  const double dr = sqrt(dr2);
  const double inv_dr = 1.0 / dr;
  const double w = 1.0 - dr;
  const int k = pri * 3 + prj;
  double cons;
  if (form == IDPD_FORM_PAIRWISE_K) {
    cons = 25.0 * w;
  } else if (form == IDPD_FORM_WARREN_K) {
    const double rho = (di0 + dj0) + (di1 + dj1) + (di2 + dj2);
    const double wb = dr < T->wrd ? 1.0 - dr / T->wrd : 0.0;
    cons = T->wa * w + T->wb * rho * wb;
  } else {
    const double cf_pair = T->cf_c[k] * (dr - kArcD) * (double)(dr >= kArcD);
    double cf_mbd = 0.0;
    cf_mbd += T->cf_m[3 * k] * (di0 + dj0);
    cf_mbd += T->cf_m[3 * k + 1] * (di1 + dj1);
    cf_mbd += T->cf_m[3 * k + 2] * (di2 + dj2);
    cons = (cf_pair + cf_mbd) * w;
  }
  return (cons + T->cf_r[k] * sqrt(w) * rnd -
          T->cf_g[k] * w * (ex * dvx + ey * dvy + ez * dvz) * inv_dr) *
         inv_dr;
}

// Plain FP64 pass 2 (the FP64 baseline): the reference's arithmetic on the
// FP64 rows with the FP64 coefficient tables, FP64 sums in cell order,
// stored in the engine's fixed point.
template <bool PRESS>
__global__ void __launch_bounds__(kRowBlock) k_force_f64(DevState d) {
  chain_begin();
  const int r = d.blk_rep[blockIdx.x];
  const int s = d.blk_row[blockIdx.x] + threadIdx.x;
  const RepDev* R = d.reps + r;
  if (s >= R->row_off + R->n) return;
  const RepTab64* T = d.tab64 + r;
  const uint32_t i = d.perm[s];
  const double xi = d.px[i], yi = d.py[i], zi = d.pz[i];
  const double vxi = d.vx[i], vyi = d.vy[i], vzi = d.vz[i];
  const uint32_t idi = d.id[i], pri = d.prop[i];
  const double di0 = d.dens64[3 * s], di1 = d.dens64[3 * s + 1], di2 = d.dens64[3 * s + 2];
  const uint32_t seed = R->seed + d.rep_time[r];
  const int form = R->form;
  int cx, cy, cz;
  cell_xyz((int)d.scell[s] - R->cell_off, R->nc, cx, cy, cz);
  double f0 = 0.0, f1 = 0.0, f2 = 0.0, p0 = 0.0, p1 = 0.0, p2 = 0.0;
  for_each_cell(R, R->reach, cx, cy, cz, [&](int cn, int, int, int, int sx, int sy, int sz) {
    const double shx = (double)sx * R->box[0], shy = (double)sy * R->box[1],
                 shz = (double)sz * R->box[2];
    for (int t = d.cell_start[cn]; t < d.cell_start[cn + 1]; t++) {
      const uint32_t j = d.perm[t];
      if (d.id[j] == idi) continue;
      const double ex = xi - (d.px[j] + shx), ey = yi - (d.py[j] + shy), ez = zi - (d.pz[j] + shz);
      const double dr2 = ex * ex + ey * ey + ez * ez;
      if (dr2 < 1.0) {
        const double all = pair_cf64(T, form, pri, d.prop[j], dr2, ex, ey, ez, vxi - d.vx[j],
                                     vyi - d.vy[j], vzi - d.vz[j], di0, di1, di2,
                                     d.dens64[3 * t], d.dens64[3 * t + 1], d.dens64[3 * t + 2],
                                     idi, d.id[j], seed);
        f0 += all * ex;
        f1 += all * ey;
        f2 += all * ez;
        if (PRESS) {
          p0 += all * ex * ex;
          p1 += all * ey * ey;
          p2 += all * ez * ez;
        }
      }
    }
  });
  long long* q = d.fq + 4 * (size_t)s;
  q[0] = __double2ll_rn(f0 * kForceScale);
  q[1] = __double2ll_rn(f1 * kForceScale);
  q[2] = __double2ll_rn(f2 * kForceScale);
  if (PRESS) {
    long long* pq = d.pq + 4 * (size_t)s;
    pq[0] = __double2ll_rn(p0 * kForceScale);
    pq[1] = __double2ll_rn(p1 * kForceScale);
    pq[2] = __double2ll_rn(p2 * kForceScale);
  }
}

// ================================================ FP64 engine algorithm
// The engine's algorithm with every pair term in FP64 (IDPD_CFG_FP64_KEPT):
// the same kept lists and rebuild schedule, the same ownership rule (each
// pair once, its term to both particles) and 64-bit fixed-point sums
// (densities in 2^-40, forces in 2^-26), with FP64 pair vectors from the
// cell-local coordinates (hi + lo of the packed split, exact to 2^-47
// relative), FP64 velocities and densities, the FP64 tables and the
// reference's FP64 Box-Muller. Pair-set decisions within 1e-10 of a cutoff
// take the reference's own FP64 distance. One warp per particle, cell reach 1.

__device__ __forceinline__ void pos64(const DevState& d, int s, double& x, double& y, double& z) {
  const float4 h = __ldg(d.posf + s), l = __ldg(d.poslo + s);
  x = (double)h.x + (double)l.x;
  y = (double)h.y + (double)l.y;
  z = (double)h.z + (double)l.z;
}

constexpr double kBand64 = 1.0e-10;

// Pass 1: over the kept list (VERLET) or the 27 cells, the owned candidates;
// each pair's weight goes to both particles, the pairs within the cutoff to
// the list of pass 2.
template <bool VERLET>
__global__ void __launch_bounds__(kRowBlock) k_density_kept64(DevState d) {
  chain_begin();
  const int r = d.blk_rep[blockIdx.x];
  const RepDev* R = d.reps + r;
  const RepTab64* T = d.tab64 + r;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int s0 = d.blk_row[blockIdx.x] + 32 * wid;
  const int s_end = min(s0 + 32, R->row_off + R->n);
  const bool warren = R->form == IDPD_FORM_WARREN_K;
  const double rd = T->wrd, cut2 = warren ? rd * rd : 1.0;
  const double wn = 15.0 / (2.0 * 3.14159265358979323846 * rd * rd * rd);
  const double csx = R->cs[0], csy = R->cs[1], csz = R->cs[2];
  const uint32_t lt_mask = (1u << lane) - 1u;
  for (int s = s0; s < s_end; s++) {
    double xi, yi, zi;
    pos64(d, s, xi, yi, zi);
    const uint32_t si = d.perm[s], pri = fbits(d.posf[s].w);
    const float ki = VERLET ? d.okey[s] : d.posf[s].x;
    long long q0 = 0, q1 = 0, q2 = 0;
    int nl = 0;
    uint32_t* out = d.nbl + (size_t)s * kNbrCap;
    // one owned candidate per lane, every lane together
    auto take = [&](bool valid, int t, int dx, int dy, int dz) {
      double dr2 = 4.0;
      uint32_t prj = 0;
      if (valid) {
        double xj, yj, zj;
        pos64(d, t, xj, yj, zj);
        prj = fbits(__ldg(d.posf + t).w);
        const double ex = (xi - (double)dx * csx) - xj, ey = (yi - (double)dy * csy) - yj,
                     ez = (zi - (double)dz * csz) - zj;
        dr2 = ex * ex + ey * ey + ez * ez;
      }
      bool in1 = valid && dr2 < 1.0;
      bool ind = valid && dr2 < cut2 && dr2 != 0.0;
      const bool near = valid && (fabs(dr2 - 1.0) < kBand64 || fabs(dr2 - cut2) < kBand64 ||
                                  dr2 < kBand64);
      if (__any_sync(0xffffffffu, near)) {
        if (near) {
          const double e2 = exact_dr2(d, R, si, d.perm[t]);
          in1 = e2 < 1.0;
          ind = e2 < cut2 && e2 != 0.0;
        }
      }
      if (ind) {
        const double dr = sqrt(dr2);
        double w;
        if (warren) {
          const double u = 1.0 - dr / rd;
          w = wn * (u * u);
        } else {
          w = (1.0 - dr) * (1.0 - dr);
        }
        const long long qw = __double2ll_rn(w * kDensScale);
        q0 += prj == 0 ? qw : 0ll;
        q1 += prj == 1 ? qw : 0ll;
        q2 += prj == 2 ? qw : 0ll;
        atomicAdd(d.dsum + (pri & 3u) * d.dstride + t, (unsigned long long)qw);
      }
      const uint32_t m = __ballot_sync(0xffffffffu, in1);
      if (in1) {
        const int pos = nl + __popc(m & lt_mask);
        if (pos < kNbrCap) out[pos] = make_entry(t, dx, dy, dz);
      }
      nl += __popc(m);
    };
    const uint32_t nv = VERLET ? (uint32_t)d.vn[s] : kNbrFallback;
    if (VERLET && nv != kNbrFallback) {
      const uint32_t* vl = d.vl + (size_t)s * kVerletCap;
      for (int k0 = 0; k0 < (int)nv; k0 += 32) {
        const int k = k0 + lane;
        const bool valid = k < (int)nv;
        int t = s, dx = 0, dy = 0, dz = 0;
        if (valid) read_entry(vl[k], t, dx, dy, dz);
        take(valid, t, dx, dy, dz);
      }
    } else {  // the 27 cells of the particle's cell (the build's cells with kept lists)
      int cx, cy, cz;
      cell_xyz((int)d.scell[s] - R->cell_off, R->nc, cx, cy, cz);
      for_each_cell(R, 1, cx, cy, cz, [&](int cn, int dx, int dy, int dz, int, int, int) {
        const int tb = d.cell_start[cn], te = d.cell_start[cn + 1];
        for (int t0 = tb; t0 < te; t0 += 32) {
          const int t = t0 + lane;
          const bool valid =
              t < te && t != s && owns(dx, VERLET ? d.okey[t] : __ldg(d.posf + t).x, ki, t, s);
          take(valid, valid ? t : s, dx, dy, dz);
        }
      });
    }
    q0 = warp_sum_ll(q0);
    q1 = warp_sum_ll(q1);
    q2 = warp_sum_ll(q2);
    if (lane == 0) {
      if (q0) atomicAdd(d.dsum + s, (unsigned long long)q0);
      if (q1) atomicAdd(d.dsum + d.dstride + s, (unsigned long long)q1);
      if (q2) atomicAdd(d.dsum + 2 * d.dstride + s, (unsigned long long)q2);
      d.nbn[s] = nl <= kNbrCap ? (uint16_t)nl : (uint16_t)kNbrFallback;
      d.npair[s] = 2u * (uint32_t)nl;
    }
    __syncwarp();
  }
}

// The FP64 densities of k_density_kept64 from its 2^-40 fixed-point sums
// (zeroed for the next pass).
__global__ void __launch_bounds__(kRowBlock) k_dens_finalize64(DevState d) {
  chain_begin();
  const int r = d.blk_rep[blockIdx.x];
  const int s = d.blk_row[blockIdx.x] + threadIdx.x;
  const RepDev* R = d.reps + r;
  if (s >= R->row_off + R->n) return;
  unsigned long long *q0 = d.dsum + s, *q1 = q0 + d.dstride, *q2 = q1 + d.dstride;
  const double a0 = (double)(long long)*q0 * kDensUnscale,
               a1 = (double)(long long)*q1 * kDensUnscale,
               a2 = (double)(long long)*q2 * kDensUnscale;
  d.dens64[3 * s] = a0;
  d.dens64[3 * s + 1] = a1;
  d.dens64[3 * s + 2] = a2;
  d.densf[s] = make_float4((float)a0, (float)a1, (float)a2, 0.0f);
  if (d.dqx) {
    d.dqx[s] = __double2ll_rn(a0 / R->dens_unscale);
    d.dqy[s] = __double2ll_rn(a1 / R->dens_unscale);
    d.dqz[s] = __double2ll_rn(a2 / R->dens_unscale);
  }
  *q0 = *q1 = *q2 = 0ull;
}

// Pass 2: over the pass-1 list (or, when it overflowed, the owned pairs
// within the cutoff of the 27 cells), each pair's FP64 term rounded once to
// the 2^-26 fixed point: +q to the owner, -q to the other particle (the
// virial a e e to both). The sums start at zero (launch_force).
template <bool PRESS, bool VERLET>
__global__ void __launch_bounds__(kRowBlock) k_force_kept64(DevState d) {
  chain_begin();
  const int r = d.blk_rep[blockIdx.x];
  const RepDev* R = d.reps + r;
  const RepTab64* T = d.tab64 + r;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int s0 = d.blk_row[blockIdx.x] + 32 * wid;
  const int s_end = min(s0 + 32, R->row_off + R->n);
  const uint32_t seed = R->seed + d.rep_time[r];
  const int form = R->form;
  const double csx = R->cs[0], csy = R->cs[1], csz = R->cs[2];
  for (int s = s0; s < s_end; s++) {
    double xi, yi, zi;
    pos64(d, s, xi, yi, zi);
    const double* vi = d.svel + 4 * (size_t)s;
    const double vxi = vi[0], vyi = vi[1], vzi = vi[2];
    const double di0 = d.dens64[3 * s], di1 = d.dens64[3 * s + 1], di2 = d.dens64[3 * s + 2];
    const uint32_t idi = fbits(d.velf[s].w), pri = fbits(d.posf[s].w), si = d.perm[s];
    long long f[6] = {0, 0, 0, 0, 0, 0};
    auto eval = [&](int t, int dx, int dy, int dz) {
      const uint32_t idj = fbits(__ldg(d.velf + t).w);
      if (idj == idi) return;
      double xj, yj, zj;
      pos64(d, t, xj, yj, zj);
      const double ex = (xi - (double)dx * csx) - xj, ey = (yi - (double)dy * csy) - yj,
                   ez = (zi - (double)dz * csz) - zj;
      const double* vj = d.svel + 4 * (size_t)t;
      const double all = pair_cf64(T, form, pri, fbits(__ldg(d.posf + t).w),
                                   ex * ex + ey * ey + ez * ez, ex, ey, ez, vxi - vj[0],
                                   vyi - vj[1], vzi - vj[2], di0, di1, di2, d.dens64[3 * t],
                                   d.dens64[3 * t + 1], d.dens64[3 * t + 2], idi, idj, seed);
      const double g[3] = {all * ex, all * ey, all * ez};
      const double e[3] = {ex, ey, ez};
      long long* q = d.fq + 4 * (size_t)t;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const long long x = __double2ll_rn(g[c] * kForceScale);
        f[c] += x;
        red_add(q + c, -x);
      }
      if (PRESS) {
        long long* pq = d.pq + 4 * (size_t)t;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const long long x = __double2ll_rn(g[c] * e[c] * kForceScale);
          f[3 + c] += x;
          red_add(pq + c, x);
        }
      }
    };
    const uint32_t nu = d.nbn[s];
    if (nu != kNbrFallback) {
      const uint32_t* list = d.nbl + (size_t)s * kNbrCap;
      for (int k = lane; k < (int)nu; k += 32) {
        int t, dx, dy, dz;
        read_entry(list[k], t, dx, dy, dz);
        eval(t, dx, dy, dz);
      }
    } else {  // the list did not fit: the owned pairs within the cutoff of the 27 cells
      const float ki = VERLET ? d.okey[s] : d.posf[s].x;
      int cx, cy, cz;
      cell_xyz((int)d.scell[s] - R->cell_off, R->nc, cx, cy, cz);
      for_each_cell(R, 1, cx, cy, cz, [&](int cn, int dx, int dy, int dz, int, int, int) {
        const int tb = d.cell_start[cn], te = d.cell_start[cn + 1];
        for (int t0 = tb; t0 < te; t0 += 32) {
          const int t = t0 + lane;
          bool in = false, near = false;
          if (t < te && t != s &&
              owns(dx, VERLET ? d.okey[t] : __ldg(d.posf + t).x, ki, t, s)) {
            double xj, yj, zj;
            pos64(d, t, xj, yj, zj);
            const double ex = (xi - (double)dx * csx) - xj, ey = (yi - (double)dy * csy) - yj,
                         ez = (zi - (double)dz * csz) - zj;
            const double dr2 = ex * ex + ey * ey + ez * ez;
            in = dr2 < 1.0;
            near = fabs(dr2 - 1.0) < kBand64;
          }
          if (__any_sync(0xffffffffu, near)) {
            if (near) in = exact_dr2(d, R, si, d.perm[t]) < 1.0;
          }
          if (in) eval(t, dx, dy, dz);
        }
      });
    }
#pragma unroll
    for (int c = 0; c < (PRESS ? 6 : 3); c++) f[c] = warp_sum_ll(f[c]);
    if (lane == 0) {
      long long* q = d.fq + 4 * (size_t)s;
      red_add(q, f[0]);
      red_add(q + 1, f[1]);
      red_add(q + 2, f[2]);
      if (PRESS) {
        long long* pq = d.pq + 4 * (size_t)s;
        red_add(pq, f[3]);
        red_add(pq + 1, f[4]);
        red_add(pq + 2, f[5]);
      }
    }
    __syncwarp();
  }
}


// Sum of the per-row pair counts of rows [row0, row0 + n) (idpd_pair_count).
__global__ void __launch_bounds__(256) k_sum_pairs(const uint32_t* npair, int row0, int n,
                                                   unsigned long long* out) {
  unsigned long long v = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    v += npair[row0 + i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

void launch_sum_pairs(const uint32_t* npair, int row0, int n, unsigned long long* out,
                      cudaStream_t st) {
  cudaMemsetAsync(out, 0, sizeof(unsigned long long), st);
  if (n > 0) k_sum_pairs<<<std::min((n + 255) / 256, 1024), 256, 0, st>>>(npair, row0, n, out);
}

void launch_force_fp64(const DevState& d, int nblk, int mode, bool with_press, bool kept,
                       const Chain& st) {
  void (*k)(DevState);
  if (mode == kPairsF64Kept)
    k = with_press ? (kept ? k_force_kept64<true, true> : k_force_kept64<true, false>)
                   : (kept ? k_force_kept64<false, true> : k_force_kept64<false, false>);
  else
    k = with_press ? k_force_f64<true> : k_force_f64<false>;
  launch(st, k, nblk, kRowBlock, 0, d);
}

void launch_density(const DevState& d, int nblk, int mode, int reach, bool verlet, bool marks,
                    size_t rows, int form_mask, const Chain& st, int lanes, bool zeroed) {
  if (nblk == 0) return;
  if (mode == kPairsF64) {
    launch(st, k_density_f64, nblk, kRowBlock, 0, d);
    return;
  }
  if (mode == kPairsF64Kept) {
    launch(st, verlet ? k_density_kept64<true> : k_density_kept64<false>, nblk, kRowBlock, 0, d);
    launch(Chain(st.st, true), k_dens_finalize64, nblk, kRowBlock, 0, d);
    return;
  }
  if (marks) {
    if (!zeroed) cudaMemsetAsync(d.phit, 0, rows, st.st);
    launch_density_f32<true>(d, nblk, reach, verlet, lanes, form_mask,
                             zeroed ? st : Chain(st.st));
  } else {
    launch_density_f32<false>(d, nblk, reach, verlet, lanes, form_mask, st);
  }
  launch(Chain(st.st, true), k_dens_finalize, nblk, kRowBlock, 0, d);
}

// ------------------------------------------- precursor conversion
// idpd_precursor: one warp per 32-row chunk, a particle at a time. A
// particle of prop_from looks for a particle of prop_near within the cutoff:
// the mark pass 1 left when it took such a pair (phit), or (FP64 arm) a sweep
// of the cells around it with the reference's FP64 distance. The draw is Saru(id, time, seed).u32() (saruprng.hpp:239-255,
// 322-333); properties change in the FP64 rows, so the pair passes see them
// from the next step's packing on.
__global__ void __launch_bounds__(kRowBlock) k_precursor(DevState d, int marks) {
  chain_begin();
  const int r = d.blk_rep[blockIdx.x];
  const RepDev* R = d.reps + r;
  if (!R->prec_on) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int s0 = d.blk_row[blockIdx.x] + 32 * wid;
  const int s_end = min(s0 + 32, R->row_off + R->n);
  const uint32_t from = R->prec_from, near_prop = R->prec_near;
  for (int s = s0; s < s_end; s++) {
    if (fbits(d.posf[s].w) != from) continue;
    bool near = false;
    if (marks) {
      near = d.phit[s] != 0;
    } else {
      const uint32_t i = d.perm[s];
      int cx, cy, cz;
      cell_xyz((int)d.scell[s] - R->cell_off, R->nc, cx, cy, cz);
      for_each_cell(R, R->reach, cx, cy, cz, [&](int c, int, int, int, int, int, int) {
        for (int t = d.cell_start[c] + lane; t < d.cell_start[c + 1]; t += 32)
          if (t != s && fbits(d.posf[t].w) == near_prop && exact_dr2(d, R, i, d.perm[t]) < 1.0)
            near = true;
      });
    }
    if (__any_sync(0xffffffffu, near) && lane == 0) {
      Saru g(fbits(d.velf[s].w), d.rep_time[r], R->prec_seed);
      if (g.next() < R->prec_thr) {
        d.prop[d.perm[s]] = R->prec_to;
        atomicAdd(d.prec_count + r, 1ull);
      }
    }
  }
}

void launch_precursor(const DevState& d, int nblk, bool marks, const Chain& st) {
  if (nblk > 0) launch(st, k_precursor, nblk, kRowBlock, 0, d, marks ? 1 : 0);
}

// -------------------------------------------- neighbour centre of mass
// The hydrophilic / hydrophobic neighbour sums of pass 1
// (nbdf_calculator.hpp:23-51) and FPDPD::copyFromForce (ptcl_class.hpp:53-57),
// for the fine-grained API and the chemistry: reach one more than the pair
// stencil (radius rn_c = 1.2), positions summed relative to the row's cell
// origin in 2^-40 fixed point, written per storage row.
//
// A warp per particle. Its lanes set up the (dy, dz) rows of cells, whose runs of
// x-consecutive cells are contiguous (two parts at the box edge), without those farther
// than rn_c from the particle; the candidates of all parts are numbered through and
// taken 32 at a time, one ahead. Bound by instruction issue (25 rounds and ~300
// instructions of sums a particle): 21k beads with solvent 88 us, the whole density call
// 384 -> 163 us against one thread per particle over 125 cells one by one. rows: rows
// per warp.
constexpr int kMaxComPart = 2 * (2 * (kMaxReach + 1) + 1) * (2 * (kMaxReach + 1) + 1);  // 98
struct ComParts {
  int tb[kMaxComPart];   // first row
  int end[kMaxComPart];  // candidates up to and including this part
  int x0[kMaxComPart];   // the part's cells' x, unwrapped, less their index
  int off[kMaxComPart];  // frame offsets fy + 8 | (fz + 8) << 8
};

__global__ void __launch_bounds__(kRowBlock) k_com(DevState d, double* cm, uint32_t* cnt_out,
                                                   int rows) {
  __shared__ ComParts parts[kWarps];
  const int r = d.blk_rep[blockIdx.x];
  const RepDev* R = d.reps + r;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  ComParts& S = parts[wid];
  const int m = R->reach + 1, w = 2 * m + 1;
  if (R->nc[0] < w || R->nc[1] < w || R->nc[2] < w) {
    if (threadIdx.x == 0) atomicCAS(d.err, 0, kErrComBox);
    return;
  }
  const int s0 = d.blk_row[blockIdx.x] + 32 * wid + rows * blockIdx.y;
  const int s_end = min(s0 + rows, R->row_off + R->n);
  const float rn2 = 1.44f;
  const double rn2d = 1.2 * 1.2;
  const int rs = R->rshift;
  const int nx = R->nc[0], ny = R->nc[1], nz = R->nc[2];
  const float csx = R->cs_f[0], csy = R->cs_f[1], csz = R->cs_f[2];
  const float sub = rs ? 0.5f : 1.0f;  // sides of a search cell per frame cell
  const float inv_side = 1.0f / (csx * sub);
  for (int s = s0; s < s_end; s++) {
    const float4 pi = d.posf[s];
    const uint32_t i = d.perm[s];
    int cx, cy, cz;
    cell_xyz((int)d.scell[s] - R->cell_off, R->nc, cx, cy, cz);
    __syncwarp();
    int total = 0;
    for (int k0 = 0; k0 < w * w; k0 += 32) {
      const int k = k0 + lane;
      int n0 = 0, n1 = 0, b0 = 0, b1 = 0, x0 = 0, off = 0, s1 = 0;
      if (k < w * w) {
        const int qy = cy + k % w - m, qz = cz + k / w - m;
        // the row's slab in the coordinates of the particle's frame cell, and its gap to
        // the particle, less a margin for the rounding
        const float y0 = (float)(qy - ((cy >> rs) << rs)) * (csy * sub);
        const float z0 = (float)(qz - ((cz >> rs) << rs)) * (csz * sub);
        const float gy = fmaxf(fmaxf(y0 - pi.y, pi.y - (y0 + csy * sub)), 0.0f);
        const float gz = fmaxf(fmaxf(z0 - pi.z, pi.z - (z0 + csz * sub)), 0.0f);
        const float rem2 = rn2 + 1.0e-3f - (gy * gy + gz * gz);
        if (rem2 >= 0.0f) {
          // the cells of the row that come within rn_c, from cx - ml to cx + mr
          const float rem = sqrtf(rem2);
          const int c0 = cx - ((cx >> rs) << rs);
          const int ml = cells_left(pi.x, rem, inv_side, c0, m);
          const int mr = cells_right(pi.x, rem, inv_side, c0, m);
          const int wy = qy < 0 ? qy + ny : (qy >= ny ? qy - ny : qy);
          const int wz = qz < 0 ? qz + nz : (qz >= nz ? qz - nz : qz);
          const int c00 = R->cell_off + (wz * ny + wy) * nx;
          const int* start = d.cell_start + c00;
          x0 = -c00;
          const int lo = max(cx - ml, 0), hi = min(cx + mr, nx - 1);
          b0 = start[lo];
          n0 = start[hi + 1] - b0;
          if (cx - ml < 0) {  // the part beyond the left edge, or the right one
            b1 = start[cx - ml + nx];
            n1 = start[nx] - b1;
            s1 = -1;
          } else if (cx + mr >= nx) {
            b1 = start[0];
            n1 = start[cx + mr - nx + 1] - b1;
            s1 = 1;
          }
          off = ((qy >> rs) - (cy >> rs) + 8) | ((qz >> rs) - (cz >> rs) + 8) << 8;
        }
      }
      int end = n0 + n1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
      }
      end += total;
      if (k < w * w) {
        S.tb[2 * k] = b0;
        S.end[2 * k] = end - n1;
        S.x0[2 * k] = x0;
        S.off[2 * k] = off;
        S.tb[2 * k + 1] = b1;
        S.end[2 * k + 1] = end;
        S.x0[2 * k + 1] = x0 + s1 * nx;
        S.off[2 * k + 1] = off;
      }
      total = __shfl_sync(0xffffffffu, end, 31);
    }
    __syncwarp();
    long long hl[3] = {0, 0, 0}, hb[3] = {0, 0, 0};
    uint32_t cl = 0, cb = 0;
    int g = 0, gb = 0;
    // one candidate ahead: row, part's offsets, position, cell
    int t_next = s, off_next = 0, x_next = 0;
    float4 p_next = pi;
    auto load = [&](int c) {
      if (c >= total) return;
      while (c >= S.end[g]) gb = S.end[g++];
      t_next = S.tb[g] + (c - gb);
      off_next = S.off[g];
      p_next = d.posf[t_next];
      x_next = (int)d.scell[t_next] + S.x0[g];
    };
    load(lane);
    for (int c = lane; c < total; c += 32) {
      const int t = t_next, off = off_next;
      const float4 pj = p_next;
      const int tx = x_next;
      load(c + 32);
      if (t == s) continue;
      const int fx = (tx >> rs) - (cx >> rs), fy = (off & 255) - 8, fz = (off >> 8 & 255) - 8;
      const float jx = pj.x + (float)fx * csx, jy = pj.y + (float)fy * csy,
                  jz = pj.z + (float)fz * csz;
      const float dr2 = dist2(pi.x - jx, pi.y - jy, pi.z - jz);
      if (dr2 >= rn2 + kGuard) continue;
      bool in_b = dr2 < rn2, in_l = dr2 < 1.0f;
      if (fabsf(dr2 - rn2) <= kGuard || fabsf(dr2 - 1.0f) <= kGuard || dr2 < 1.0e-10f) {
        const double e2 = exact_dr2(d, R, i, d.perm[t]);
        in_b = e2 < rn2d && e2 != 0.0;
        in_l = in_b && e2 < 1.0;
      }
      const uint32_t pr = fbits(pj.w);
      const bool is_b = in_b && pr == 1, is_l = in_l && pr == 0;
      if (is_b || is_l) {
        const long long q[3] = {fix_pos(jx), fix_pos(jy), fix_pos(jz)};
#pragma unroll
        for (int k = 0; k < 3; k++) {
          hb[k] += is_b ? q[k] : 0ll;
          hl[k] += is_b ? 0ll : q[k];
        }
        cb += is_b;
        cl += !is_b;
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 3; k++) {
      hl[k] = warp_sum_ll(hl[k]);
      hb[k] = warp_sum_ll(hb[k]);
    }
    cl = __reduce_add_sync(0xffffffffu, cl) + 1u;
    cb = __reduce_add_sync(0xffffffffu, cb);
    if (lane < 3) {
      // the hydrophilic sum starts at the row itself with count 1 (nbdf_calculator.hpp:23-24)
      const float own = lane == 0 ? pi.x : (lane == 1 ? pi.y : pi.z);
      const long long sl = (lane == 0 ? hl[0] : (lane == 1 ? hl[1] : hl[2])) +
                           fix_pos(own);
      const long long sb = lane == 0 ? hb[0] : (lane == 1 ? hb[1] : hb[2]);
      const int c = lane == 0 ? cx : (lane == 1 ? cy : cz);
      const double org = (double)(c >> rs) * R->cs[lane];
      cm[6 * (size_t)i + lane] = org + ((double)sl / kPosScale) / (double)cl;
      cm[6 * (size_t)i + 3 + lane] = org + ((double)sb / kPosScale) / (double)cb;
      if (lane < 2) cnt_out[2 * (size_t)i + lane] = lane ? cb : cl;
    }
  }
}

void launch_com(const DevState& d, int nblk, double* cm_out, uint32_t* cnt_out, cudaStream_t st) {
  if (nblk == 0) return;
  int rows = 32;  // four waves of warps, one row each when there are fewer
  while (rows > 1 && (long long)nblk * kRowBlock < 4ll * rows * kWaveWarps) rows >>= 1;
  k_com<<<dim3(nblk, 32 / rows), kRowBlock, 0, st>>>(d, cm_out, cnt_out, rows);
}

}  // namespace idpd
