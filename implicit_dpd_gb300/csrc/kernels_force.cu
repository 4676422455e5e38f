// Pass 2 of the FP32 engine, CalcForceEpEpDPD::operator()
// (nbdf_calculator.hpp:63-145) with each pair taken once, by the particle
// that owns it, over the pass-1 lists; and the dispatch of every pass-2 arm.
#include <algorithm>

#include "pair_lists.cuh"

namespace idpd {

// ------------------------------------------------------------- pass 2

// 1 - dr for a pair close to the cutoff, from the double-float cell-local
// coordinates (hi + lo) and the double-float cell side: every step below is
// an error-free transform or acts on terms below 1e-7, so 1 - dr^2 carries
// an absolute error near 1e-13 instead of the 1e-7 of the FP32 pair vector.
// The random term's sqrt(1 - r) amplifies the latter when r is near 1.
__device__ __forceinline__ float near_cut_w(float4 pi, float4 li, float4 pj, float4 lj, int dx,
                                            int dy, int dz, const RepDev* R, float dr) {
  const float hi_i[3] = {pi.x, pi.y, pi.z}, lo_i[3] = {li.x, li.y, li.z};
  const float hi_j[3] = {pj.x, pj.y, pj.z}, lo_j[3] = {lj.x, lj.y, lj.z};
  const int dk[3] = {dx, dy, dz};
  float p[3], err = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float e1, e2, pe;
    const float s = two_sum(hi_i[k], -hi_j[k], e1);
    const float t = two_sum(s, -(float)dk[k] * R->cs_f[k], e2);
    const float lo = e1 + e2 + (lo_i[k] - lo_j[k]) - (float)dk[k] * R->cs_lo[k];
    p[k] = two_prod(t, t, pe);
    err += pe + 2.0f * t * lo;
  }
  float ea, eb;
  const float s1 = two_sum(p[0], p[1], ea);
  const float s2 = two_sum(s1, p[2], eb);
  const float w2 = (1.0f - s2) - (err + ea + eb);  // 1 - s2 is exact for s2 in [0.5, 2]
  return w2 / (1.0f + dr);
}

// The pair vector of a close pair from the double-float cell-local
// coordinates: the FP32 difference of the hi parts carries an absolute error
// near 1e-7, which is a large part of a vector a few hundredths long.
__device__ __forceinline__ void close_pair_vector(float4 pi, float4 li, float4 pj, float4 lj, int dx,
                                                  int dy, int dz, const RepDev* R, float& ex,
                                                  float& ey, float& ez) {
  const float hi_i[3] = {pi.x, pi.y, pi.z}, lo_i[3] = {li.x, li.y, li.z};
  const float hi_j[3] = {pj.x, pj.y, pj.z}, lo_j[3] = {lj.x, lj.y, lj.z};
  const int dk[3] = {dx, dy, dz};
  float e[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float e1, e2;
    const float s = two_sum(hi_i[k], -hi_j[k], e1);
    const float t = two_sum(s, -(float)dk[k] * R->cs_f[k], e2);
    e[k] = t + (e1 + e2 + (lo_i[k] - lo_j[k]) - (float)dk[k] * R->cs_lo[k]);
  }
  ex = e[0];
  ey = e[1];
  ez = e[2];
}

// Pairs closer than 0.1 take their pair vector from close_pair_vector.
constexpr float kCloseCut2 = 0.01f;

// The particle of one (half) warp in pass 2 and its fixed-point sums.
struct PairI {
  float4 pi, vi, di;
  uint32_t idi, pri, seed;
  int row;  // the particle's row (its low position parts are read near the cutoff)
  long long fx, fy, fz, px, py, pz;
};

__device__ __forceinline__ void load_row(PairI& I, const DevState& d, int s) {
  I.pi = d.posf[s];
  I.vi = d.velf[s];
  I.di = d.densf[s];
  I.row = s;
  I.idi = fbits(I.vi.w);
  I.pri = fbits(I.pi.w);
}

// The terms of the four pairs of a quad of lanes (4 q .. 4 q + 3, one particle's)
// turned from one pair per lane to one component per lane: on return w[j] of
// lane 4 q + c is component c (x, y, z; nothing for c = 3) of lane 4 q + j's pair.
// Two butterfly exchanges; every lane of the warp takes part.
__device__ __forceinline__ void quad_components(float x, float y, float z, int c, float w[4]) {
  const bool odd = c & 1, up = c & 2;
  float r = __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
  const float a0 = odd ? r : x, a1 = odd ? y : r;   // component c & 1 of the even, odd lane's pair
  const float a3 = __shfl_xor_sync(0xffffffffu, z, 1);  // even lanes: z of the odd lane's pair
  r = __shfl_xor_sync(0xffffffffu, up ? a0 : z, 2);
  w[0] = up ? r : a0;
  w[2] = up ? z : r;
  r = __shfl_xor_sync(0xffffffffu, up ? a1 : a3, 2);
  w[1] = up ? r : a1;
  w[3] = up ? a3 : r;
}

// Component c of the terms of a quad's four pairs, converted to fixed point
// once for both particles: the owner's 64-bit sum S takes -x (the virial, the
// same for both, +x) and the sum of the other particle of pair j, row t[j], x by
// atomic add. The three lanes of a quad that hold x, y and z address one row at a
// time, so a row's three adds leave the SM as one access of its 32-byte sector.
// The terms are below 65536. lim: pairs of the quad that exist (0 on the lane without a
// component); sums points at component c of row 0.
template <bool VIRIAL>
__device__ __forceinline__ void quad_both(const float w[4], const int t[4], int lim,
                                          long long* sums, long long& S) {
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const long long x = fix_force_small(w[j]);
    S = VIRIAL ? S + x : S - x;
    red_add_if(j < lim, sums + 4 * (size_t)t[j], x);
  }
}

// A term too large for the fast conversion (or none at all: NaN), one lane on its own:
// v goes to the other particle's sum, -v (VIRIAL: v) to the owner's.
template <bool VIRIAL>
__device__ __forceinline__ void big_both(float v, long long* owner, long long* other) {
  const long long x = fix_force(v);
  red_add(other, x);
  red_add(owner, VIRIAL ? x : -x);
}

// One owned pair of a pass-1 list (fast path of pass 2), given the other
// particle's three rows (posf, velf, densf): the force on the other particle
// over the pair vector, and the pair vector. The pair arithmetic runs in FP32
// (the compensated forms near the cutoff and for close pairs). A pair of equal
// ids contributes nothing (nbdf_calculator.hpp:84), nor does a lane without a pair.
template <bool PRESS, int FORM>
__device__ __forceinline__ float owned_pair(const DevState& d, const RepDev* R, const PairTables& T,
                                            const OffTable& OT, const PairI& I, uint32_t e,
                                            bool valid, float4 pj, float4 vj, float4 dj, float& ex,
                                            float& ey, float& ez) {
  const int t = (int)(e & kRowMask);
  const auto o = OT.at(e >> kRowBits);
  ex = (I.pi.x - o.x) - pj.x;
  ey = (I.pi.y - o.y) - pj.y;
  ez = (I.pi.z - o.z) - pj.z;
  float dr2 = dist2(ex, ey, ez);
  float inv_dr, dr, w;
  if (valid && (dr2 < kCloseCut2 || dr2 > kNearCut2)) {  // rare: the compensated forms
    int tt, dx, dy, dz;
    read_entry(e, tt, dx, dy, dz);
    const float4 li = __ldg(d.poslo + I.row), lj = __ldg(d.poslo + t);
    if (dr2 < kCloseCut2) {
      close_pair_vector(I.pi, li, pj, lj, dx, dy, dz, R, ex, ey, ez);
      dr2 = ex * ex + ey * ey + ez * ez;
    }
    inv_dr = rsqrt_approx(dr2);
    dr = dr2 * inv_dr;
    w = 1.0f - dr;
    if (dr2 > kNearCut2)  // admitted pairs have 1 - r >= 0 up to ~1e-13
      w = fmaxf(near_cut_w(I.pi, li, pj, lj, dx, dy, dz, R, dr), 0.0f);
  } else {
    inv_dr = rsqrt_approx(dr2);
    dr = dr2 * inv_dr;
    w = 1.0f - dr;
  }
  const uint32_t idj = fbits(vj.w);
  const float a = pair_cf<FORM, PRESS>(T, R, I.pri, fbits(pj.w), dr, inv_dr, w, ex, ey, ez, I.vi, vj,
                                I.di, dj, I.idi, idj, I.seed);
  return valid && idj != I.idi ? -a : 0.0f;  // the other particle's force is -a e
}

// The force and virial terms of one pair (the pair arithmetic of pass 2),
// from the side of the particle that owns the pair (a pair of equal ids is
// skipped, nbdf_calculator.hpp:84); 64-bit path.
template <bool PRESS, int FORM>
__device__ __forceinline__ bool pair_terms(const DevState& d, const RepDev* R, const PairTables& T,
                                           const PairI& I, int t, int dx, int dy, int dz,
                                           float g[6]) {
  const float4 vj = __ldg(d.velf + t);
  const float4 pj = __ldg(d.posf + t);
  const float4 dj = __ldg(d.densf + t);
  const uint32_t idj = fbits(vj.w);
  if (idj == I.idi) return false;
  float ex = (I.pi.x - (float)dx * R->cs_f[0]) - pj.x;
  float ey = (I.pi.y - (float)dy * R->cs_f[1]) - pj.y;
  float ez = (I.pi.z - (float)dz * R->cs_f[2]) - pj.z;
  float dr2 = dist2(ex, ey, ez);
  if (dr2 < kCloseCut2) {
    close_pair_vector(I.pi, __ldg(d.poslo + I.row), pj, __ldg(d.poslo + t), dx, dy, dz, R, ex, ey,
                      ez);
    dr2 = dist2(ex, ey, ez);
  }
  const float inv_dr = rsqrt_approx(dr2);
  const float dr = dr2 * inv_dr;
  float w = 1.0f - dr;
  if (dr2 > kNearCut2)  // admitted pairs have 1 - r >= 0 up to ~1e-13
    w = fmaxf(near_cut_w(I.pi, __ldg(d.poslo + I.row), pj, __ldg(d.poslo + t), dx, dy, dz, R, dr),
              0.0f);
  const float a = pair_cf<FORM, false>(T, R, I.pri, fbits(pj.w), dr, inv_dr, w, ex, ey, ez, I.vi, vj,
                                I.di, dj, I.idi, idj, I.seed);
  if (!isfinite(a)) atomicCAS(d.err, 0, kErrNonFinite);
  g[0] = a * ex;
  g[1] = a * ey;
  g[2] = a * ez;
  if (PRESS) {
    g[3] = g[0] * ex;
    g[4] = g[1] * ey;
    g[5] = g[2] * ez;
  }
  return true;
}

// The other particle's share of one pair term: the force -g (the exact
// negation of the owner's fixed-point term) and the virial +g e.
template <bool PRESS>
__device__ __forceinline__ void add_to_other(const DevState& d, int t, const float g[6]) {
  long long* q = d.fq + 4 * (size_t)t;
  red_add(q, -fix_force(g[0]));
  red_add(q + 1, -fix_force(g[1]));
  red_add(q + 2, -fix_force(g[2]));
  if (PRESS) {
    long long* pq = d.pq + 4 * (size_t)t;
    red_add(pq, fix_force(g[3]));
    red_add(pq + 1, fix_force(g[4]));
    red_add(pq + 2, fix_force(g[5]));
  }
}

// One owned pair added to the owner's 64-bit sums (the lane's share) and to
// the other particle's sums in memory.
template <bool PRESS, int FORM>
__device__ __forceinline__ void eval_pair(const DevState& d, const RepDev* R, const PairTables& T,
                                          PairI& I, int t, int dx, int dy, int dz) {
  float g[6];
  if (!pair_terms<PRESS, FORM>(d, R, T, I, t, dx, dy, dz, g)) return;
  I.fx += fix_force(g[0]);
  I.fy += fix_force(g[1]);
  I.fz += fix_force(g[2]);
  if (PRESS) {
    I.px += fix_force(g[3]);
    I.py += fix_force(g[4]);
    I.pz += fix_force(g[5]);
  }
  add_to_other<PRESS>(d, t, g);
}

// A component's total over the lanes of its group that hold it (every fourth
// lane of the LP).
template <int LP>
__device__ __forceinline__ long long group_total(long long v) {
#pragma unroll
  for (int o = 4; o < LP; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Shared memory of pass 2 (dynamic, sized by the launch): per 128-row block
// its replica's tables, per warp the segments and the queue of the
// cell-walk path.
struct ForceBlockSmem {
  PairTables T;
  OffTable OT;
};
struct ForceWarpSmem {
  SegTable seg;
  uint32_t qt[64], qc[64];
};

size_t force_smem_bytes(int fb) { return (size_t)fb * sizeof(ForceBlockSmem); }

// Each pair is evaluated once, by the particle that owns it (owns()), and
// its term goes to both particles (Newton's third law in exact fixed point: the
// sums equal those of the reference's two evaluations up to the FP32
// rounding of one of them). A warp takes the particles of its chunk 32 / LP
// at a time, LP lanes each, over their pass-1 lists (owned pairs only),
// grouped by list length (the chunk sorted by length, neighbours in that
// order share a warp) so that the groups run about as long; each lane reads
// its next list entry one round ahead. The sums start at zero (launch_force)
// and every term arrives by atomic add. A particle whose list overflowed is
// left to k_force_walk, so that this pass keeps no walk state, and only the
// replica tables in shared memory, which leaves the SM's L1 the room to cache
// the other particles' rows (with the walk's 7.6 KB of shared memory per CTA in
// the same kernel the pass took 1.15 ms instead of 1.08 on membrane_1m).
// One launch per pair form present: a warp whose replica has another form
// returns at once.
//
// What bounds it: instruction issue (70 % of the slots, ~340 instructions per 32
// pairs) with the other particles' row loads behind it. The three adds to the other
// particle bound it before: a lane that adds x, y and z of its own pair sends three
// instructions of 32 scattered sectors each, which kept the L2's atomic unit 50 % and
// L1 76 % busy. With the terms turned inside each quad of lanes (quad_components), one
// instruction adds x, y and z of eight rows in eight sectors: a third of the sectors,
// atomic unit 16 %, long-scoreboard stalls 4.3 -> 2.4 per issue, L1 hit rate 22 -> 39 %;
// 984k-bead membrane 976 -> 836 us, 998k-particle liquid 248 -> 207 us (786 and 174 with
// the cheaper conversion and with large terms taken out of the common path). A register cap
// of 72 or 92 instead of 64 (7 or 5 CTAs per SM) gave 852 and 935 us on that membrane.
//
// Pass 2 over the rows s0 .. s0 + rows - 1 of replica r (one warp's chunk, rows
// <= 32), the particles whose pass-1 list fit: G particles at a time, LP lanes each.
template <bool PRESS, int FORM, int LP>
__device__ __forceinline__ void force_rows(const DevState& d, int s0, int rows, int r,
                                           const RepDev* R, const PairTables& T,
                                           const OffTable& OT, int lane) {
  constexpr int G = 32 / LP;  // particles per warp at a time
  const int h = lane / LP, sl = lane % LP, c = lane & 3;
  const int nrow = min(rows, R->row_off + R->n - s0);
  if (nrow <= 0) return;
  PairI I;
  I.seed = R->seed + d.rep_time[r];
  // the chunk's rows sorted by the length of their lists (overflowed lists
  // count 0, lanes without a row come last): key = length << 5 | row - s0
  uint32_t key = 0xffffffffu;
  if (lane < nrow) {
    const uint32_t n = (uint32_t)d.nbn[s0 + lane];
    key = ((n != kNbrFallback ? n : 0u) << 5) | (uint32_t)lane;
  }
  key = warp_sort_asc(key, lane);
  for (int i2 = 0; i2 < nrow; i2 += G) {
    // ---- G particles, LP lanes each: the owned pairs of the lists
    const uint32_t ki = __shfl_sync(0xffffffffu, key, i2 + h);
    const bool act = i2 + h < nrow;
    const int s = act ? s0 + (int)(ki & 31u) : s0;
    const int nu = act ? (int)(ki >> 5) : 0;
    const int nmax = (int)(__shfl_sync(0xffffffffu, key, min(i2 + G, nrow) - 1) >> 5);
    load_row(I, d, s);
    const uint32_t* list = d.nbl + (size_t)s * kNbrCap;
    long long F = 0, V = 0;
    uint32_t e_next = sl < nu ? __ldg(list + sl) : make_entry(s, 0, 0, 0);  // one round ahead
    for (int k0 = 0; k0 < nmax; k0 += LP) {
      const int k = k0 + sl;
      const bool valid = k < nu;
      const uint32_t e = valid ? e_next : make_entry(s, 0, 0, 0);
      if (k + LP < nu) e_next = __ldg(list + k + LP);
      const int t = (int)(e & kRowMask);
      float ex, ey, ez;
      float an = owned_pair<PRESS, FORM>(d, R, T, OT, I, e, valid, __ldg(d.posf + t),
                                        __ldg(d.velf + t), __ldg(d.densf + t), ex, ey, ez);
      // |e| <= 1 up to rounding: below this no component reaches 65536
      const bool big = !(fabsf(an) < 60000.0f);
      if (__any_sync(0xffffffffu, big)) {
        if (big) {
          if (!isfinite(an)) atomicCAS(d.err, 0, kErrNonFinite);
          const float g[3] = {an * ex, an * ey, an * ez}, x[3] = {ex, ey, ez};
#pragma unroll
          for (int q = 0; q < 3; q++) {
            big_both<false>(g[q], d.fq + 4 * (size_t)s + q, d.fq + 4 * (size_t)t + q);
            if (PRESS)
              big_both<true>(-g[q] * x[q], d.pq + 4 * (size_t)s + q, d.pq + 4 * (size_t)t + q);
          }
          an = 0.0f;
        }
      }
      const float gx = an * ex, gy = an * ey, gz = an * ez;
      int tq[4];
#pragma unroll
      for (int j = 0; j < 4; j++) tq[j] = __shfl_sync(0xffffffffu, t, j, 4);
      const int lim = c < 3 ? nu - (k - c) : 0;
      float w[4];
      quad_components(gx, gy, gz, c, w);
      quad_both<false>(w, tq, lim, d.fq + c, F);
      if (PRESS) {  // the virial a e e, the same for both particles
        quad_components(-gx * ex, -gy * ey, -gz * ez, c, w);
        quad_both<true>(w, tq, lim, d.pq + c, V);
      }
    }
    F = group_total<LP>(F);
    if (PRESS) V = group_total<LP>(V);
    red_add_if(sl < 3 && nu > 0, d.fq + 4 * (size_t)s + c, F);
    if (PRESS) red_add_if(sl < 3 && nu > 0, d.pq + 4 * (size_t)s + c, V);
  }
}

// Pass 2 for the particles of the chunk s0 .. s0 + 31 whose pass-1 list did
// not fit (more than kNbrCap owned pairs, only at extreme densities): one at
// a time, the whole warp walks the particle's cells again and queues its
// owned in-range pairs in shared memory; each term goes to both particles.
template <int REACH, bool PRESS, int FORM>
__device__ __forceinline__ void force_walk_rows(const DevState& d, int kept, int s0, int r,
                                                const RepDev* R, const PairTables& T,
                                                ForceWarpSmem& W, int lane) {
  const int s_end = min(s0 + 32, R->row_off + R->n);
  if (s0 >= s_end) return;
  SegTable& S = W.seg;
  uint32_t* QT = W.qt;
  uint32_t* QC = W.qc;
  PairI I;
  I.seed = R->seed + d.rep_time[r];
  constexpr int nseg = 2 * (2 * REACH + 1) * (2 * REACH + 1);
  const uint32_t lt_mask = (1u << lane) - 1u;
  int cached = -1;
  uint32_t slow = __ballot_sync(0xffffffffu, s0 + lane < s_end && d.nbn[s0 + lane] == kNbrFallback);
  while (slow) {
    const int ss = s0 + __ffs(slow) - 1;
    slow &= slow - 1;
    load_row(I, d, ss);
    I.fx = I.fy = I.fz = I.px = I.py = I.pz = 0;
    const int cell = (int)d.scell[ss];
    if (cell != cached) {  // the segments of the particle's cell (only this path walks cells)
      int cx, cy, cz;
      cell_xyz(cell - R->cell_off, R->nc, cx, cy, cz);
      __syncwarp();
      build_segments(S, d, R, cx, cy, cz, lane);
      __syncwarp();
      cached = cell;
    }
    int qn = 0;
#pragma unroll 1
    for (int g = 0; g < nseg; g++) {
      const int tb = S.tb[g], te = S.te[g];
      if (tb >= te) continue;
      const int code = S.code[g];
      int b[2 * REACH];
#pragma unroll
      for (int q = 0; q < 2 * REACH; q++) b[q] = S.bnd[g][q];
      const int fx0 = (code & 7) - 4, dy = ((code >> 3) & 7) - 4, dz = ((code >> 6) & 7) - 4;
      const float by = I.pi.y - (float)dy * R->cs_f[1], bz = I.pi.z - (float)dz * R->cs_f[2];
      for (int t0 = tb; t0 < te; t0 += 32) {
        const int t = t0 + lane;
        bool in = false, own = false;
        int dx = 0;
        bool near = false;
        if (t < te && t != ss) {
          const float4 pj = __ldg(d.posf + t);
          dx = fx0 + frame_step<REACH>(t, b);
          const float ex = (I.pi.x - (float)dx * R->cs_f[0]) - pj.x, ey = by - pj.y,
                      ez = bz - pj.z;
          const float dr2 = ex * ex + ey * ey + ez * ez;
          in = dr2 < 1.0f;
          near = fabsf(dr2 - 1.0f) <= kGuard;
          own = owns(dx, kept ? d.okey[t] : pj.x, kept ? d.okey[ss] : I.pi.x, t, ss);
        }
        if (__any_sync(0xffffffffu, near) && near) {
          in = exact_dr2(d, R, d.perm[ss], d.perm[t]) < 1.0;
        }
        in = in && own;  // the pairs this particle owns
        const uint32_t mask = __ballot_sync(0xffffffffu, in);
        if (in) {
          const int pos = qn + __popc(mask & lt_mask);
          QT[pos] = (uint32_t)t;
          QC[pos] = pack_code(dx, code);
        }
        qn += __popc(mask);
        if (qn >= 32) {
          __syncwarp();
          const PairCode pc = unpack_code(QC[lane]);
          eval_pair<PRESS, FORM>(d, R, T, I, (int)QT[lane], pc.dx, pc.dy, pc.dz);
          __syncwarp();
          if (lane < qn - 32) {
            QT[lane] = QT[32 + lane];
            QC[lane] = QC[32 + lane];
          }
          __syncwarp();
          qn -= 32;
        }
      }
    }
    __syncwarp();
    if (lane < qn) {
      const PairCode pc = unpack_code(QC[lane]);
      eval_pair<PRESS, FORM>(d, R, T, I, (int)QT[lane], pc.dx, pc.dy, pc.dz);
    }
    __syncwarp();
    const long long fx = warp_sum_ll(I.fx), fy = warp_sum_ll(I.fy), fz = warp_sum_ll(I.fz);
    long long px = 0, py = 0, pz = 0;
    if (PRESS) {
      px = warp_sum_ll(I.px);
      py = warp_sum_ll(I.py);
      pz = warp_sum_ll(I.pz);
    }
    if (lane == 0) {
      long long* q = d.fq + 4 * (size_t)ss;
      red_add(q, fx);
      red_add(q + 1, fy);
      red_add(q + 2, fz);
      if (PRESS) {
        long long* pq = d.pq + 4 * (size_t)ss;
        red_add(pq, px);
        red_add(pq + 1, py);
        red_add(pq + 2, pz);
      }
    }
  }
}

// Pass 2, grid order: CTA b takes row blocks b fb .. b fb + fb - 1, one warp
// per 32-row chunk. Its shared memory is the replica tables only (1.2 KB per
// row block), which leaves most of the SM's 256 KB of L1 and shared memory
// to the L1 that caches the other particles' rows.
template <bool PRESS, int FORM, int LP>
__global__ void __launch_bounds__(1024, 1) k_force_f32(DevState d, int nblk, int rows) {
  extern __shared__ __align__(16) unsigned char force_smem[];
  chain_launch();
  ForceBlockSmem* BS = reinterpret_cast<ForceBlockSmem*>(force_smem);
  const int fb = blockDim.x >> 7;  // 128-row blocks of this CTA
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int rbl = wid / kWarps;              // the warp's row block within the CTA
  const int rb = blockIdx.x * fb + rbl;      // in the row-block map
  const int r = rb < nblk ? d.blk_rep[rb] : 0;
  const RepDev* R = d.reps + r;
  if (rb < nblk) {
    const int tb = threadIdx.x & (kRowBlock - 1);
    if (tb < 9) fill_pair_table(BS[rbl].T, *R, tb);
    if (tb < 64) fill_off_table(BS[rbl].OT, *R, tb);
  }
  __syncthreads();
  const bool mine = rb < nblk && R->form == FORM;
  const int row0 = mine ? d.blk_row[rb] : 0;
  chain_wait();
  if (!mine) return;
  force_rows<PRESS, FORM, LP>(d, row0 + 32 * (wid % kWarps) + rows * blockIdx.y,
                                     rows, r, R, BS[rbl].T, BS[rbl].OT, lane);
}

// Pass 2 of the particles whose list overflowed (force_walk_rows), one warp
// per 32-row chunk; a few CTAs per SM stride over the row blocks and leave at once
// when no list did.
template <int REACH, bool PRESS, int FORM>
__global__ void __launch_bounds__(kRowBlock) k_force_walk(DevState d, int kept, int nblk) {
  __shared__ ForceBlockSmem B;
  __shared__ ForceWarpSmem W[kWarps];
  chain_begin();
  if (!d.overflow[1]) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int rb = blockIdx.x; rb < nblk; rb += gridDim.x) {
    const int r = d.blk_rep[rb];
    const RepDev* R = d.reps + r;
    __syncthreads();
    if (threadIdx.x < 9) fill_pair_table(B.T, *R, threadIdx.x);
    __syncthreads();
    if (R->form == FORM)
      force_walk_rows<REACH, PRESS, FORM>(d, kept, d.blk_row[rb] + 32 * wid, r, R, B.T, W[wid],
                                          lane);
  }
}

// Pass 2 of one pair form: the shape of the tuning (lanes per particle,
// row blocks per CTA); the observation steps (PRESS) run 16 lanes, one row
// block per CTA.
template <int REACH, int FORM, bool PRESS, int LP>
void launch_force_kernel(const DevState& d, int nblk, int kept, int fb, const Chain& st) {
  const int rows = chunk_rows(nblk, LP);
  launch(st, k_force_f32<PRESS, FORM, LP>, dim3((nblk + fb - 1) / fb, 32 / rows), kRowBlock * fb,
         force_smem_bytes(fb), d, nblk, rows);
  launch(Chain(st.st, true), k_force_walk<REACH, PRESS, FORM>, std::min(nblk, kRareBlocks),
         kRowBlock, 0, d, kept, nblk);
}

template <int FORM, bool PRESS, int LP>
void launch_force_shape(const DevState& d, int nblk, int reach, int kept, int fb,
                        const Chain& st) {
  if (reach == 2)
    launch_force_kernel<2, FORM, PRESS, LP>(d, nblk, kept, fb, st);
  else
    launch_force_kernel<1, FORM, PRESS, LP>(d, nblk, kept, fb, st);
}

template <int FORM>
void launch_force_form(const DevState& d, int nblk, bool with_press, const PairTuning& tu,
                       int kept, Chain& st) {
  const int fb = tu.fblk == 2 || tu.fblk == 4 ? tu.fblk : 1;
  if (with_press)
    launch_force_shape<FORM, true, 16>(d, nblk, tu.reach, kept, 1, st);
  else if (tu.lanes == 4)
    launch_force_shape<FORM, false, 4>(d, nblk, tu.reach, kept, fb, st);
  else if (tu.lanes == 8)
    launch_force_shape<FORM, false, 8>(d, nblk, tu.reach, kept, fb, st);
  else if (tu.lanes == 32)
    launch_force_shape<FORM, false, 32>(d, nblk, tu.reach, kept, fb, st);
  else
    launch_force_shape<FORM, false, 16>(d, nblk, tu.reach, kept, fb, st);
  st.chained = true;
}

void launch_force(const DevState& d, int nblk, int mode, bool with_press, bool kept,
                  const PairTuning& tu, int form_mask, size_t rows, const Chain& st, bool zeroed) {
  if (nblk == 0) return;
  Chain c = st;
  if (mode != kPairsF64 && !zeroed) {
    cudaMemsetAsync(d.fq, 0, 4 * rows * sizeof(long long), st.st);
    if (with_press) cudaMemsetAsync(d.pq, 0, 4 * rows * sizeof(long long), st.st);
    c.chained = false;
  }
  if (mode != kPairsF32) {
    launch_force_fp64(d, nblk, mode, with_press, kept, c);
    return;
  }
  if (form_mask & (1 << IDPD_FORM_MDPD_K))
    launch_force_form<IDPD_FORM_MDPD_K>(d, nblk, with_press, tu, kept ? 1 : 0, c);
  if (form_mask & (1 << IDPD_FORM_PAIRWISE_K))
    launch_force_form<IDPD_FORM_PAIRWISE_K>(d, nblk, with_press, tu, kept ? 1 : 0, c);
  if (form_mask & (1 << IDPD_FORM_WARREN_K))
    launch_force_form<IDPD_FORM_WARREN_K>(d, nblk, with_press, tu, kept ? 1 : 0, c);
}

}  // namespace idpd
