// The drift of one storage row and what follows it in the same kernel: the displacement
// since the last list rebuild, or the binning.
#pragma once

#include "state.cuh"

namespace idpd {

// Periodic wrap of driftkick.hpp:19-21, t - floor(t / L) L with the
// reference's rounding. Rows that stay inside [0, hi) keep t unchanged
// without touching the FP64 pipe (the sign bit and the bit pattern order of
// non-negative doubles decide it); all others take the reference expression.
__device__ __forceinline__ double wrap_pbc(double t, double L, double iL, long long hi_bits) {
  const long long b = __double_as_longlong(t);
  if (b >= 0 && b < hi_bits) return t;
  const double f = floor(plain_mul(t, iL));
  return plain_add(t, -plain_mul(f, L));
}

// drift_and_predict of one storage row (driftkick.hpp:6-27), from its velocity v and
// kv = a dt/2; p holds the row's position on entry and the new one on return, ds its new
// delta_sumr.
__device__ __forceinline__ void drift_row(const DevState& d, const RepDev* R, int i, double v[3],
                                          const double kv[3], double p[3], double ds[3]) {
  const double dt = R->dt;
  ds[0] = d.dsx[i];
  ds[1] = d.dsy[i];
  ds[2] = d.dsz[i];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    v[k] = add_f64(v[k], kv[k]);
    const double dr = mul_f64(v[k], dt);
    const double t = __dadd_rn(p[k], dr);
    ds[k] = add_f64(ds[k], dr);
    // hi = L (1 - 2^-50): below it t / L rounds below 1 and floor() is 0.
    const double L = R->box[k];
    const long long hi = __double_as_longlong(L) - 4;
    p[k] = wrap_pbc(t, L, R->ibox[k], hi);
  }
  d.vx[i] = v[0]; d.vy[i] = v[1]; d.vz[i] = v[2];
  d.dsx[i] = ds[0]; d.dsy[i] = ds[1]; d.dsz[i] = ds[2];
  d.px[i] = p[0]; d.py[i] = p[1]; d.pz[i] = p[2];
}

// The same from the row's stored velocity and acceleration.
__device__ __forceinline__ void drift_row(const DevState& d, const RepDev* R, int i, double p[3],
                                          double ds[3]) {
  const double h = R->half_dt;
  double v[3] = {d.vx[i], d.vy[i], d.vz[i]};
  const double a[3] = {d.ax[i], d.ay[i], d.az[i]};
  const double kv[3] = {mul_f64(a[0], h), mul_f64(a[1], h), mul_f64(a[2], h)};
  drift_row(d, R, i, v, kv, p, ds);
}

// a - b as a float, to about 2^-32 (far beyond any skin where that cannot be told).
__device__ __forceinline__ float diff_f32(double a, double b) {
  const long long q = to_fix(a) - to_fix(b);
  const bool ok = in_fix(a) && in_fix(b) && q == (long long)(int)q;
  return ok ? __int2float_rn((int)q) * 2.3283064365386963e-10f : 1.0e3f;
}

// The squared displacement of row i since the last rebuild (delta_sumr ds against that of
// the rebuild, r0, accumulates every drift, unwrapped). It only has to fall on the right
// side of the threshold: taken in FP32, and again in FP64 close to it.
__device__ __forceinline__ float displacement2(const DevState& d, const double ds[3],
                                               const double r0[3]) {
  const float fx = diff_f32(ds[0], r0[0]), fy = diff_f32(ds[1], r0[1]), fz = diff_f32(ds[2], r0[2]);
  float m = fx * fx + fy * fy + fz * fz;
  const float thr2 = d.vdev->thr2;
  if (fabsf(m - thr2) < 1.0e-3f * thr2) {
    const double ex = plain_add(ds[0], -r0[0]), ey = plain_add(ds[1], -r0[1]),
                 ez = plain_add(ds[2], -r0[2]);
    m = plain_f32(ex * ex + ey * ey + ez * ez);
  }
  return m;
}

// The largest of a block's displacements m into the rebuild record; every thread takes part.
__device__ __forceinline__ void note_displacement(const DevState& d, float m, float* wmax) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float b = 0.0f;
    for (int w = 0; w < kRowBlock / 32; w++) b = fmaxf(b, wmax[w]);
    // non-negative floats order like their bit patterns; the running maximum
    // is read first, so only blocks that raise it take the (single-address) atomic
    const unsigned int bb = __float_as_uint(b);
    if (b > 0.0f && bb > *(volatile unsigned int*)&d.vdev->maxd2) atomicMax(&d.vdev->maxd2, bb);
  }
}

// Cell index and arrival slot of row i at position p.
__device__ __forceinline__ void bin_row(const DevState& d, const RepDev* R, int i,
                                        const double p[3]) {
  const int cx = cell_index(p[0], R->inv_cs[0], R->nc[0]);
  const int cy = cell_index(p[1], R->inv_cs[1], R->nc[1]);
  const int cz = cell_index(p[2], R->inv_cs[2], R->nc[2]);
  const uint32_t key = (uint32_t)(R->cell_off + (cz * R->nc[1] + cy) * R->nc[0] + cx);
  d.key[i] = key;
  d.slot[i] = (uint32_t)atomicAdd(&d.cell_cnt[key], 1);
}

}  // namespace idpd
