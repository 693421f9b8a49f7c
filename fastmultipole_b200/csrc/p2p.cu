// p2p.cu -- near-field (P2P) kernels over the target-sorted direct list.
//
// Kernels of the reference's point systems:
//   Laplace point source  (test/gravitational.jl:80-104): phi += q/(4 pi r),
//     grad += q dx/(4 pi r^3), pairs with r^2 = 0 skipped, no hessian;
//   vortex particle       (test/vortex.jl:83-128): u = (dx x Gamma)/(4 pi r^3)
//     and the 9-term velocity gradient.
// k_p2p (direct list): one CTA per target leaf, source bodies gathered into
// warp-private shared-memory batches, lanes split between targets and sources
// by the leaf's size (details at the kernel).  k_direct (all pairs): one CTA
// per block of targets and share of the sources, staged through shared memory.  FP64 is the
// drop-in arithmetic; the MIXED variant moves every body relative to a nearby
// centre in FP64, then evaluates the kernel in FP32 (rsqrt on the SFU),
// summing blocks of sources in FP32 and the block partials in FP64.
#include <climits>
#include <algorithm>
#include <type_traits>

#include "context.cuh"

namespace fmmb {

namespace {

constexpr int kP2PThreads = 128;
// targets per thread held in registers: 4 for point sources (4 accumulators),
// 2 for vortex particles (up to 12 accumulators)
template <int KIND>
__host__ __device__ constexpr int tpt() { return KIND == FMM_POINT_SOURCE ? 4 : 2; }

__device__ __forceinline__ double rsq(double x) { return rsqrt(x); }

// ---------------------------------------------------------------------------
// Direct-list P2P.  One CTA of kWarps warps owns one direct-list row (a target leaf), or an
// item: a tile of its targets and a share of its source leaves.  Each warp takes its part of
// the source leaves and gathers up to batch_bodies() bodies of consecutive leaves of its share (many
// small leaves, or a piece of a large one) into its own shared-memory batch,
// converted once per body (to FP32 relative to the target leaf centre on the
// mixed path).  Targets sit in registers, kTPT per lane.  A target tile holds
// up to 32 * kTPT targets; the lanes split into TS lanes along the tile times
// 32 / TS slices along the batch, TS the smallest power of two that covers the
// tile, so a leaf of 5 bodies keeps every lane busy as a leaf of 64 does.
// Slices are summed by shuffles, warps through shared memory.  The mixed path
// sums each batch in FP32 and the batches in FP64.  On the packed FP32 path, rows
// of small target leaves (at most 8 bodies on average) take one warp each instead of
// a CTA, so that the per-row setup and the cross-warp sum do not dominate their work.
constexpr int kWarps = 4;
// Launches of up to kItemRowsPerSM rows per SM whose rows are long are cut into items of about equal
// work, some kItemWaves for every CTA that the SMs hold at a time: one tile of a row's targets x a share
// of the row's source leaves (at least kItemSources bodies), whose sums are added in order by k_p2p_sum.
// With a CTA of 4 or 16 warps per row the few rows of large leaves (up to three tiles) and the long
// rows of probe leaves were still running when the others had finished.  10,000 bodies FP64: near
// field 273 -> 113 us and 50 us to cut and to add; 300k vortex ring FP64: 28.2 -> 25.5 ms (whole
// solves).  More rows than that fill the GPU by themselves (1e6 bodies: 62.0 ms either way).
constexpr int kItemRowsPerSM = 64, kItemWaves = 4, kItemSources = 256;
// Body pairs per row (on average) from which rows are cut; to cut and to add takes some 40 us.  Near field
// whole / cut: 4,096 rows of 3,000 pairs FP64 0.07 / 0.13 ms; 64 rows of 15,600 0.036 / 0.055; 407 uneven rows
// of 20,000 (up to 210,000) 0.129 / 0.082; 512 even rows of 27,000 0.070 / 0.091, mixed 0.100 / 0.095; 64 rows of
// 62,000, vortex particles, 0.10 / 0.07; 574 rows of 80,000 0.24 / 0.16; one row of 1.6e6 1.28 / 0.09.
constexpr double kItemRowPairs = 1.6e4;
// A body's gathering into a batch, in target slots of its pairs.  Without it the second tile of a row of 68
// targets got a sixteenth of the shares of the first and took the longest: 4,333 probes and 189,460 vortex
// particles, gradients on, mixed: near field 2.25 ms, 1.42 with it (1.41 and 1.45 with two and four times as
// many slots); gradients off 1.13 and 0.78
constexpr int kGatherSlotsF32 = 16, kGatherSlotsF64 = 4;
constexpr int kTPT = 2;
constexpr unsigned kAll = 0xffffffffu;

template <int KIND>
struct Batch {
  static constexpr int n = KIND == FMM_POINT_SOURCE ? 256 : 128;  // bodies per warp batch
  static constexpr int nv = KIND == FMM_POINT_SOURCE ? 4 : 6;     // values per body: x y z + strengths
};

// FP32 point sources evaluate two targets per lane with packed f32x2 arithmetic;
// their batch holds per body {-x, -x, -y, -y}, {-z, -z, q, q} (ready-made pairs)
template <class R, int KIND>
__host__ __device__ constexpr bool packed() { return sizeof(R) == 4 && KIND == FMM_POINT_SOURCE; }
// FP32 vortex particles: two targets per lane as well; batch per body {-x, -x, -y, -y},
// {-z, -z, G0, G0}, {G1, G1, G2, G2}
template <class R, int KIND>
__host__ __device__ constexpr bool packed_vortex() { return sizeof(R) == 4 && KIND == FMM_POINT_VORTEX; }
template <class R, int KIND>
__host__ __device__ constexpr int slots_per_body() {
  return packed<R, KIND>() ? 8 : packed_vortex<R, KIND>() ? 12 : Batch<KIND>::nv;
}
// bodies per warp batch: the packed batch is halved to keep the same shared memory per CTA
template <class R, int KIND>
__host__ __device__ constexpr int batch_bodies() { return packed<R, KIND>() ? 128 : Batch<KIND>::n; }

// 1/sqrt(x) on the SFU, denormal inputs flushed (rsqrt.approx.ftz.f32)
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// accumulated channels: Laplace phi, grad (3); vortex u (3) if GS, grad u (9) if HS
template <int KIND, bool GS, bool HS>
__host__ __device__ constexpr int n_chan() {
  return KIND == FMM_POINT_SOURCE ? 4 : (GS ? 3 : 0) + (HS ? 9 : 0);
}
// acc13 row of channel a
template <int KIND, bool GS>
__device__ __forceinline__ int chan_row(int a) {
  return KIND == FMM_POINT_SOURCE ? a : (GS ? a + 1 : a + 4);
}

// r^-3 of an FP64 pair without a call, a branch or a special case.  y, about r^-1, is the SFU's
// approximation (rsqrt.approx.ftz.f64) with its low word cleared, so that u = y^2 is exact; with
// e = 1 - r^2 u (|e| below 2^-18) the binomial series of (1 - e)^(-3/2) and (1 - e)^-1
//   r^-3 = y^3 (1 + 3/2 e + 15/8 e^2 + 35/16 e^3 ...),  r^-2 = u (1 + e + e^2 + e^3 ...)
// are cut after e^2, below the rounding of a double.  r^2 = 0 gives y = 0 and all products
// zero, which skips the pair as the reference does.  Outside the range where y^3 and the
// products are normal numbers the sums come out non-finite or the caller must not get here
// (kFarHi, tiny_strength): such batches take the general arithmetic (self_batch_f64_*).
struct InvR {
  double u, e, r3;  // y^2, 1 - r^2 y^2, q r^-3 (q the factor given)
};
__device__ __forceinline__ InvR inv_r3(double r2, double q) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
  const int nz = __double2hiint(r2) | __double2loint(r2);
  y = __hiloint2double(nz ? __double2hiint(y) : 0, 0);
  InvR v;
  v.u = y * y;
  v.e = fma(-r2, v.u, 1.0);
  const double h = v.e * fma(v.e, 1.875, 1.5);
  const double w = (q * y) * v.u;
  v.r3 = fma(w, h, w);
  return v;
}

// bodies with a coordinate of at least 2^160 (high word of the double) take the general
// arithmetic: r^-5 and the products with it stay normal numbers below
constexpr int kFarHi = (1023 + 160) << 20;
__device__ __forceinline__ int hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }
// so do, where the potential is asked for, strengths below 2^-536 (not zero): the potential is
// (q r^-3) r^2, r below 2^162, and q r^-3 would be subnormal where q / r is not
constexpr int kTinyHi = (1023 - 536) << 20;
__device__ __forceinline__ bool tiny_strength(double q) {
  const int h = hi_abs(q);
  return h < kTinyHi && (h | __double2loint(q)) != 0;
}

// one source body on one target, Laplace, 17 FP64 operations: phi = (q / r^3) r^2
template <bool PS>
__device__ __forceinline__ void source_pair_f64(double tx, double ty, double tz, double sx, double sy, double sz,
                                                double q, double (&a)[4]) {
  const double dx = tx - sx, dy = ty - sy, dz = tz - sz;
  const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
  const double q3 = inv_r3(r2, q).r3;
  if (PS) a[0] = fma(q3, r2, a[0]);
  a[1] = fma(dx, q3, a[1]);
  a[2] = fma(dy, q3, a[2]);
  a[3] = fma(dz, q3, a[3]);
}

// How a packed batch treats pairs without r^2 > 0.  kUnguarded: they make the sums non-finite.
// kCoincident: 1 / r = 0, so that coincident bodies add nothing.  kSkip: they are left out whatever
// their offsets and strengths (NaN coordinates, infinite strengths) are.
enum : int { kUnguarded = 0, kCoincident, kSkip };
__device__ __forceinline__ float2 keep(float2 r2, float2 v) {
  return make_float2(r2.x > 0.f ? v.x : 0.f, r2.y > 0.f ? v.y : 0.f);
}

// One lane's slice of a packed batch on its two targets.
template <int GUARD, bool PS>
__device__ __forceinline__ void packed_batch(const float4* __restrict__ B4, int j0, int nb, int SS, float2 tx2,
                                             float2 ty2, float2 tz2, float2& ph, float2& gx, float2& gy, float2& gz) {
#pragma unroll 4
  for (int j = j0; j < nb; j += SS) {
    const float4 u = B4[2 * j], v = B4[2 * j + 1];
    float2 dx = __fadd2_rn(tx2, make_float2(u.x, u.y));
    float2 dy = __fadd2_rn(ty2, make_float2(u.z, u.w));
    float2 dz = __fadd2_rn(tz2, make_float2(v.x, v.y));
    float2 q = make_float2(v.z, v.w);
    float2 r2 = __fmul2_rn(dx, dx);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    if (GUARD == kSkip) dx = keep(r2, dx), dy = keep(r2, dy), dz = keep(r2, dz), q = keep(r2, q);
    float2 ri;
    if (GUARD) {
      ri.x = r2.x > 0.f ? rsqrt_ftz(r2.x) : 0.f;
      ri.y = r2.y > 0.f ? rsqrt_ftz(r2.y) : 0.f;
    } else {
      ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    }
    // q / r and q / r^3 = (q / r) (1 / r^2): the two products after the rsqrt are independent
    const float2 qr = __fmul2_rn(q, ri);
    const float2 ri2 = __fmul2_rn(ri, ri);
    if (PS) ph = __fadd2_rn(ph, qr);
    const float2 q3 = __fmul2_rn(qr, ri2);
    gx = __ffma2_rn(dx, q3, gx);
    gy = __ffma2_rn(dy, q3, gy);
    gz = __ffma2_rn(dz, q3, gz);
  }
}

// one source body on one target, vortex particles with the velocity gradient (FP64 path):
// velocity into u[0..2] (GS); the gradient as Q_ij += d_i (G x d)_j / r^5 and E_k += G_k / r^3,
// which the caller combines to -3 Q_ij + eps_jki E_k (r^2 / r^5 = 1 / r^3)
template <class R, bool GS>
__device__ __forceinline__ void vortex_pair_qe(R tx, R ty, R tz, R sx, R sy, R sz, R s0, R s1, R s2, R* u,
                                               R (&Q)[9], R (&E)[3]) {
  const R dx = tx - sx, dy = ty - sy, dz = tz - sz;
  const R r2 = dx * dx + dy * dy + dz * dz;
  if (r2 > R(0)) {
    const R rinv = rsq(r2);
    const R rinv2 = rinv * rinv;
    const R den = rinv * rinv2;
    const R cx = s1 * dz - s2 * dy, cy = s2 * dx - s0 * dz, cz = s0 * dy - s1 * dx;
    if (GS) {
      u[0] += cx * den;
      u[1] += cy * den;
      u[2] += cz * den;
    }
    const R d5 = den * rinv2;
    const R px = dx * d5, py = dy * d5, pz = dz * d5;
    Q[0] += px * cx;
    Q[1] += px * cy;
    Q[2] += px * cz;
    Q[3] += py * cx;
    Q[4] += py * cy;
    Q[5] += py * cz;
    Q[6] += pz * cx;
    Q[7] += pz * cy;
    Q[8] += pz * cz;
    E[0] += s0 * den;
    E[1] += s1 * den;
    E[2] += s2 * den;
  }
}

// the gradient channels g[0..8] (column-major d u_j / d x_i at 3 i + j) from Q and E
template <class R>
__device__ __forceinline__ void vortex_grad_from_qe(const R (&Q)[9], const R (&E)[3], R* g) {
  g[0] = R(-3) * Q[0];
  g[1] = R(-3) * Q[1] + E[2];
  g[2] = R(-3) * Q[2] - E[1];
  g[3] = R(-3) * Q[3] - E[2];
  g[4] = R(-3) * Q[4];
  g[5] = R(-3) * Q[5] + E[0];
  g[6] = R(-3) * Q[6] + E[1];
  g[7] = R(-3) * Q[7] - E[0];
  g[8] = R(-3) * Q[8];
}

// the same sums without the special cases (inv_r3), 38 FP64 operations with both outputs: the
// gradient is trace-free (d . (G x d) = 0 for every pair), so Q_zz is formed at the end as
// -(Q_xx + Q_yy)
template <bool GS, bool HS>
__device__ __forceinline__ void vortex_pair_f64(double tx, double ty, double tz, double sx, double sy, double sz,
                                                double s0, double s1, double s2, double (&u)[3], double (&Q)[9],
                                                double (&E)[3]) {
  const double dx = tx - sx, dy = ty - sy, dz = tz - sz;
  const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
  const InvR v = inv_r3(r2, 1.0);
  const double cx = fma(s1, dz, -(s2 * dy)), cy = fma(s2, dx, -(s0 * dz)), cz = fma(s0, dy, -(s1 * dx));
  if (GS) {
    u[0] = fma(cx, v.r3, u[0]);
    u[1] = fma(cy, v.r3, u[1]);
    u[2] = fma(cz, v.r3, u[2]);
  }
  if (HS) {
    const double d5 = v.r3 * fma(v.u, fma(v.e, v.e, v.e), v.u);
    const double px = dx * d5, py = dy * d5, pz = dz * d5;
    Q[0] = fma(px, cx, Q[0]);
    Q[1] = fma(px, cy, Q[1]);
    Q[2] = fma(px, cz, Q[2]);
    Q[3] = fma(py, cx, Q[3]);
    Q[4] = fma(py, cy, Q[4]);
    Q[5] = fma(py, cz, Q[5]);
    Q[6] = fma(pz, cx, Q[6]);
    Q[7] = fma(pz, cy, Q[7]);
    E[0] = fma(s0, v.r3, E[0]);
    E[1] = fma(s1, v.r3, E[1]);
    E[2] = fma(s2, v.r3, E[2]);
  }
}

// f32x2 with both halves negated
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// One lane's slice of a packed vortex batch on its two targets: velocity
// u = (G x d) / r^3 (GS) and its gradient (HS, the SMatrix column-major order of
// test/vortex.jl:83-128).  acc[a] receives channel a of the two targets.  The gradient
// du_j/dx_i = eps_jki G_k / r^3 - 3 d_i (G x d)_j / r^5 is summed as two parts, Q_ij =
// sum d_i (G x d)_j / r^5 and E_k = sum G_k / r^3, combined once per batch (r^2 / r^5 =
// 1 / r^3, so the six eps terms need three sums; the trace of Q vanishes, so Q_zz is not
// summed).
template <int GUARD, bool GS, bool HS, int NA>
__device__ __forceinline__ void packed_vortex_batch(const float4* __restrict__ B4, int j0, int nb, int SS,
                                                    float2 tx2, float2 ty2, float2 tz2, float2 (&acc)[NA]) {
  constexpr int h = GS ? 3 : 0;
  float2 u[3], Q[9], E[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) u[a] = E[a] = make_float2(0.f, 0.f);
#pragma unroll
  for (int a = 0; a < 9; ++a) Q[a] = make_float2(0.f, 0.f);
#pragma unroll 2
  for (int j = j0; j < nb; j += SS) {
    const float4 p = B4[3 * j], v = B4[3 * j + 1], w = B4[3 * j + 2];
    float2 dx = __fadd2_rn(tx2, make_float2(p.x, p.y));
    float2 dy = __fadd2_rn(ty2, make_float2(p.z, p.w));
    float2 dz = __fadd2_rn(tz2, make_float2(v.x, v.y));
    float2 g0 = make_float2(v.z, v.w), g1 = make_float2(w.x, w.y), g2 = make_float2(w.z, w.w);
    float2 r2 = __fmul2_rn(dx, dx);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    if (GUARD == kSkip) {
      dx = keep(r2, dx), dy = keep(r2, dy), dz = keep(r2, dz);
      g0 = keep(r2, g0), g1 = keep(r2, g1), g2 = keep(r2, g2);
    }
    float2 ri;
    if (GUARD) {
      ri.x = r2.x > 0.f ? rsqrt_ftz(r2.x) : 0.f;
      ri.y = r2.y > 0.f ? rsqrt_ftz(r2.y) : 0.f;
    } else {
      ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    }
    const float2 ri2 = __fmul2_rn(ri, ri);
    const float2 den = __fmul2_rn(ri, ri2);
    // c = G x d
    const float2 cx = __ffma2_rn(g1, dz, neg2(__fmul2_rn(g2, dy)));
    const float2 cy = __ffma2_rn(g2, dx, neg2(__fmul2_rn(g0, dz)));
    const float2 cz = __ffma2_rn(g0, dy, neg2(__fmul2_rn(g1, dx)));
    if (GS) {
      u[0] = __ffma2_rn(cx, den, u[0]);
      u[1] = __ffma2_rn(cy, den, u[1]);
      u[2] = __ffma2_rn(cz, den, u[2]);
    }
    if (HS) {
      const float2 d5 = __fmul2_rn(den, ri2);
      const float2 px = __fmul2_rn(dx, d5), py = __fmul2_rn(dy, d5), pz = __fmul2_rn(dz, d5);
      Q[0] = __ffma2_rn(px, cx, Q[0]);
      Q[1] = __ffma2_rn(px, cy, Q[1]);
      Q[2] = __ffma2_rn(px, cz, Q[2]);
      Q[3] = __ffma2_rn(py, cx, Q[3]);
      Q[4] = __ffma2_rn(py, cy, Q[4]);
      Q[5] = __ffma2_rn(py, cz, Q[5]);
      Q[6] = __ffma2_rn(pz, cx, Q[6]);
      Q[7] = __ffma2_rn(pz, cy, Q[7]);
      E[0] = __ffma2_rn(g0, den, E[0]);
      E[1] = __ffma2_rn(g1, den, E[1]);
      E[2] = __ffma2_rn(g2, den, E[2]);
    }
  }
  if (GS) {
    acc[0] = u[0];
    acc[1 % NA] = u[1];
    acc[2 % NA] = u[2];
  }
  if (HS) {
    // the gradient is trace-free: d . (G x d) = 0 for every pair, so Q_zz = -(Q_xx + Q_yy)
    Q[8] = neg2(__fadd2_rn(Q[0], Q[4]));
    const float2 m3 = make_float2(-3.f, -3.f);
    acc[(h + 0) % NA] = __fmul2_rn(m3, Q[0]);
    acc[(h + 1) % NA] = __ffma2_rn(m3, Q[1], E[2]);
    acc[(h + 2) % NA] = __ffma2_rn(m3, Q[2], neg2(E[1]));
    acc[(h + 3) % NA] = __ffma2_rn(m3, Q[3], neg2(E[2]));
    acc[(h + 4) % NA] = __fmul2_rn(m3, Q[4]);
    acc[(h + 5) % NA] = __ffma2_rn(m3, Q[5], E[0]);
    acc[(h + 6) % NA] = __ffma2_rn(m3, Q[6], E[1]);
    acc[(h + 7) % NA] = __ffma2_rn(m3, Q[7], neg2(E[0]));
    acc[(h + 8) % NA] = __fmul2_rn(m3, Q[8]);
  }
}

// The batch holding the target's own leaf on the mixed path runs in FP64: its closest
// pairs are the ones whose FP32 coordinates relative to the leaf centre (absolute error
// about 2^-24 of the leaf size) would give large relative errors, and a few such pairs
// dominate the error of the whole field.  The batch holds per body (x, y, z, q) (point
// sources) or (x, y, z, G0, G1, G2) (vortex particles) relative to the target leaf
// centre, in FP64 (the size of the packed FP32 record); the lane's targets are read again
// in FP64.
// the lane's two targets relative to the leaf centre in FP64
__device__ __forceinline__ void self_targets_f64(const double4* __restrict__ tpos, int first, int nt, int ti, int TS,
                                                 double ox, double oy, double oz, double (&tx)[2], double (&ty)[2],
                                                 double (&tz)[2]) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    tx[k] = ty[k] = tz[k] = 0.0;
    const int i = ti + k * TS;
    if (i < nt) {
      const double4 p = tpos[first + i];
      tx[k] = p.x - ox;
      ty[k] = p.y - oy;
      tz[k] = p.z - oz;
    }
  }
}

template <bool PS, int NA>
__device__ __noinline__ void self_batch_f64_source(const double4* __restrict__ Bd, int j0, int nb, int SS,
                                                      const double (&tx)[2], const double (&ty)[2],
                                                      const double (&tz)[2], double (&tot)[2][NA]) {
  for (int j = j0; j < nb; j += SS) {
    const double4 sp = Bd[j];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double dx = tx[k] - sp.x, dy = ty[k] - sp.y, dz = tz[k] - sp.z;
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 > 0.0) {
        const double ri = rsqrt(r2);
        const double qr = sp.w * ri;
        if (PS) tot[k][0] += qr;
        const double q3 = qr * ri * ri;
        tot[k][1 % NA] += dx * q3;
        tot[k][2 % NA] += dy * q3;
        tot[k][3 % NA] += dz * q3;
      }
    }
  }
}

template <bool GS, bool HS, int NA>
__device__ __noinline__ void self_batch_f64_vortex(const double2* __restrict__ Bd, int j0, int nb, int SS,
                                                      const double (&tx)[2], const double (&ty)[2],
                                                      const double (&tz)[2], double (&tot)[2][NA]) {
  constexpr int h = GS ? 3 : 0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    double u[3] = {0.0, 0.0, 0.0}, Q[9], E[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < 9; ++a) Q[a] = 0.0;
    for (int j = j0; j < nb; j += SS) {
      const double2 a = Bd[3 * j], b = Bd[3 * j + 1], c = Bd[3 * j + 2];
      vortex_pair_qe<double, GS>(tx[k], ty[k], tz[k], a.x, a.y, b.x, b.y, c.x, c.y, u, Q, E);
    }
    if (GS)
#pragma unroll
      for (int c = 0; c < 3; ++c) tot[k][c % NA] += u[c];
    if (HS) {
      double gr[9];
      vortex_grad_from_qe<double>(Q, E, gr);
#pragma unroll
      for (int a = 0; a < 9; ++a) tot[k][(h + a) % NA] += gr[a];
    }
  }
}

// Targets of the next tile of a row with rem targets left.  SUB (two targets per lane, expensive
// pairs): a remainder that would leave a quarter or more of its slots empty gives a full power of two
// first.  The sources are gathered once more for the rest, which the vortex kernels' 32 or more
// operations per pair outweigh.
template <bool SUB>
__host__ __device__ __forceinline__ int next_tile(int rem) {
  constexpr int most = 32 * kTPT;
  if (rem >= most) return most;
  if (SUB) {
    if (rem > most / 2 && rem <= most * 3 / 4) return most / 2;
    if (rem > most / 4 && rem <= most * 3 / 8) return most / 4;
  }
  return rem;
}
// (300k ring FP64 25.1 -> 23.8 ms, 2e6 ring mixed 210.4 -> 205.8 ms, 1e6 clustered bodies mixed 34.7 -> 34.5 ms.
// Not in mixed items, whose pairs cost less than gathering far-off sources twice: gradient of 2e5 sources
// 2.99 -> 3.22 ms; 1e4 probes around 2e5 vortex particles, near field 2.97 -> 4.03 ms)
template <class R, int KIND, bool ITEMS>
__host__ __device__ constexpr bool sub_tiles() {
  return sizeof(R) == 4 ? !ITEMS : KIND == FMM_POINT_VORTEX;
}

// Targets per lane of a tile of nt targets on the FP64 path: three where 3 x a power of two lanes
// leave fewer slots empty than 2 x (nt in (2^k, 3/2 2^k]).  Leaves are split by eight, so their sizes
// spread over a factor of eight and the slots matter: slots per pair 1.24 -> 1.11 (1e6 clustered
// bodies), 1.36 -> 1.15 (1e4 uniform).
__host__ __device__ __forceinline__ int targets_per_lane(int nt) {
  int n2 = 1, n3 = 1;
  while (n2 * 2 < nt) n2 <<= 1;
  while (n3 * 3 < nt) n3 <<= 1;
  return n3 * 3 < n2 * 2 ? 3 : 2;
}
template <class R, int KIND, bool HS>
__host__ __device__ constexpr int max_targets_per_lane() {
  return sizeof(R) == 4 || (KIND == FMM_POINT_VORTEX && HS) ? kTPT : 3;
}
template <int N>
__device__ __forceinline__ double pick(const double (&v)[N], int q) {
  return q == 0 ? v[0] : q == 1 ? v[1] : v[N - 1];
}
template <int N>
__device__ __forceinline__ double pick(const float (&v)[N], int) { return v[0]; }

// RW: one warp per row (rows of small leaves, kWarps rows per CTA), the warp adding its
// sums to the targets itself; otherwise one CTA per row or item, the warps splitting its sources.
// resident CTAs of the mixed instances: the registers the packed loop needs (the FP64
// branch of the batch holding the target's own leaf is a call, and must not raise them);
// the FP64 vortex CTA path takes 168 registers (3 CTAs per SM; 300k ring, order 12, whole solve:
// 28.6 ms, 28.8 with 2 CTAs, and 49.3 with 4, whose 128 registers spill inside the loop)
template <class R, int KIND, bool HS, bool RW>
__host__ __device__ constexpr int p2p_min_blocks() {
  static_assert(!RW || packed<R, KIND>(), "a warp per row: packed point sources only");
  if (sizeof(R) != 4) return (KIND == FMM_POINT_VORTEX && HS) ? 3 : 4;
  constexpr int regs = (KIND == FMM_POINT_VORTEX && HS) ? 128 : (RW ? 72 : 64);
  return 65536 / (regs * kWarps * 32);
}

template <class R, int KIND, bool PS, bool GS, bool HS, bool RW, bool ITEMS>
__global__ void __launch_bounds__(kWarps * 32, p2p_min_blocks<R, KIND, HS, RW>())
    k_p2p(const int* __restrict__ tgt_list, const int* __restrict__ off, int n_rows, const int* __restrict__ src_of,
          const int* __restrict__ t_start, const int* __restrict__ t_count, const double* __restrict__ t_center,
          const int* __restrict__ s_start, const int* __restrict__ s_count, const double4* __restrict__ tpos,
          const double4* __restrict__ spos, const double4* __restrict__ sstr, double* __restrict__ acc13,
          const int4* __restrict__ items, const int* __restrict__ n_items, double* __restrict__ item_sums,
          int exact_self) {
  // items (ITEMS, CTA path only), two int4 each: row, first target of the tile, source leaves [z, w); and the place of
  // the item's sums (unscaled) in item_sums, or -1 to add them to the targets
  constexpr int W = kWarps;
  static_assert(!(RW && ITEMS), "a warp per row takes whole rows");
  constexpr int NB = batch_bodies<R, KIND>(), NA = n_chan<KIND, GS, HS>();
  constexpr int NS = slots_per_body<R, KIND>();
  constexpr bool MIXED = sizeof(R) == 4;
  constexpr int KT = max_targets_per_lane<R, KIND, HS>();
  constexpr bool PACK = packed<R, KIND>();
  constexpr bool PACKV = packed_vortex<R, KIND>();
  // vortex particles with the gradient on the FP64 path sum it as two parts per target
  constexpr bool QE = !MIXED && KIND == FMM_POINT_VORTEX && HS;
  static_assert((!PACK && !PACKV) || kTPT == 2, "packed paths pair two targets per lane");
  extern __shared__ __align__(16) unsigned char p2p_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  R* B = reinterpret_cast<R*>(p2p_smem) + w * NS * NB;  // this warp's batch, NS values per body
  double* red = reinterpret_cast<double*>(p2p_smem + W * NS * NB * sizeof(R));  // [W][32 kTPT][NA]
  if (ITEMS && (int)blockIdx.x >= *n_items) return;
  const int4 it = ITEMS ? items[2 * blockIdx.x] : make_int4(0, 0, 0, 0);
  const int row = RW ? blockIdx.x * W + w : (ITEMS ? it.x : (int)blockIdx.x);
  if (RW && row >= n_rows) return;  // whole warps: no block barrier on the RW path
  const int t = tgt_list[row];
  const int l0 = ITEMS ? it.z : off[row], l1 = ITEMS ? it.w : off[row + 1];
  const int ts = t_start[t], tc = t_count[t];
  // this warp's share of the leaves.  CTA path: an equal contiguous range of the source bodies
  // (leaves in row order, split inside a leaf where a range ends), so the warps reach the
  // block's reduction together whatever the leaf sizes; point sources every W-th leaf (an even
  // split measured no faster there, and its registers spill at the packed loop's 64), except FP64
  // items, whose few leaves do not divide evenly.  One warp per row takes them all.
  constexpr bool BAL = !RW && (KIND == FMM_POINT_VORTEX || (!MIXED && ITEMS));
  constexpr int LS = (RW || BAL) ? 1 : W;  // stride of this warp's source leaves along the row
  int lb0 = l0 + ((RW || BAL) ? 0 : w), poff0 = 0, rem0 = INT_MAX;
  if (BAL) {
    long long total = 0;
    for (int i = l0 + lane; i < l1; i += 32) total += s_count[src_of[i]];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(kAll, total, o);
    const int b_lo = (int)(total * w / W), b_hi = (int)(total * (w + 1) / W);
    rem0 = b_hi - b_lo;
    int before = 0;  // bodies of the leaves ahead of the current 32
    for (int i0 = l0; i0 < l1 && rem0 > 0; i0 += 32) {
      const int i = i0 + lane;
      const int c = i < l1 ? s_count[src_of[i]] : 0;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += v;
      }
      const unsigned past = __ballot_sync(kAll, i < l1 && before + incl > b_lo);
      if (past) {  // the range starts inside leaf i0 + f
        const int f = __ffs(past) - 1;
        const int ex = __shfl_sync(kAll, incl - c, f);
        lb0 = i0 + f;
        poff0 = b_lo - before - ex;
        break;
      }
      before += __shfl_sync(kAll, incl, 31);
    }
  }
  const double ox = MIXED ? t_center[3 * t] : 0.0;
  const double oy = MIXED ? t_center[3 * t + 1] : 0.0;
  const double oz = MIXED ? t_center[3 * t + 2] : 0.0;
  constexpr bool SUB = sub_tiles<R, KIND, ITEMS || RW>() && KT == kTPT;
  for (int tile = ITEMS ? it.y : 0, nt; tile < tc; tile += nt) {
    nt = next_tile<SUB>(tc - tile);
    const int tpt = KT == 3 ? targets_per_lane(nt) : kTPT;
    int TS = 1;
    while (TS * tpt < nt) TS <<= 1;
    const int ti = lane & (TS - 1), slice = lane / TS, SS = 32 / TS;
    R tx[KT], ty[KT], tz[KT];
    int tfar = 0;  // FP64: largest high word of the lane's target coordinates
#pragma unroll
    for (int k = 0; k < KT; ++k) {
      tx[k] = ty[k] = tz[k] = R(0);
      int i = ti + k * TS;
      if (i < nt) {
        double4 p = tpos[ts + tile + i];
        tfar = max(tfar, max(hi_abs(p.x), max(hi_abs(p.y), hi_abs(p.z))));
        tx[k] = (R)(p.x - ox);
        ty[k] = (R)(p.y - oy);
        tz[k] = (R)(p.z - oz);
      }
    }
    R part[KT][NA];
    double tot[KT][NA];
    R us[KT][3], Qs[KT][9], Es[KT][3];  // FP64 vortex particles: velocity, gradient as two sums
    // FP64: a second pass in the general arithmetic when the first meets a pair out of its range
    for (bool general = false;; general = true) {
#pragma unroll
      for (int k = 0; k < KT; ++k) {
#pragma unroll
        for (int a = 0; a < NA; ++a) part[k][a] = R(0), tot[k][a] = 0.0;
#pragma unroll
        for (int a = 0; a < 9; ++a) Qs[k][a] = R(0);
#pragma unroll
        for (int a = 0; a < 3; ++a) us[k][a] = Es[k][a] = R(0);
      }
      // next source leaf of this warp, bodies of it already taken, bodies of the range still to take
      int lb = lb0, poff = poff0, rem = rem0;
      while (lb < l1 && rem > 0) {
        // candidate leaves lb + LS * lane; take the longest prefix that fits the batch and the range
        const int l = lb + LS * lane;
        int cnt = 0, sb = 0, sl = -1;
        if (l < l1) {
          sl = src_of[l];
          sb = s_start[sl];
          cnt = s_count[sl];
        }
        if (lane == 0) {
          sb += poff;
          cnt -= poff;
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          int v = __shfl_up_sync(kAll, incl, o);
          if (lane >= o) incl += v;
        }
        const int excl = incl - cnt;
        const int lim = min(NB, rem);
        int nl = __popc(__ballot_sync(kAll, l < l1 && incl <= lim));
        int nb;
        if (nl == 0) {  // the first leaf alone overflows the batch or ends the range: lim bodies of it
          nl = 1;
          nb = lim;
          poff += lim;
        } else {
          nb = __shfl_sync(kAll, incl, nl - 1);
          lb += LS * nl;
          poff = 0;
        }
        rem -= nb;
        // the batch holds the target branch's own bodies (coincident pairs certain)
        const bool self_batch = __any_sync(kAll, lane < nl && sl == t);
        // mixed path: that batch in FP64 (the solve's own near field; the influence estimate, which
        // only needs the magnitude of the field, keeps it in FP32 with the r^2 > 0 guard)
        // (vortex ring 2e6, p = 12: velocity error 8e-8 against 9e-7 with that batch in FP32, at the
        // same speed)
        const bool self_f64 = self_batch && exact_self != 0;
        int far = 0;  // FP64: largest high word of the coordinates
        // gather: body idx of the batch lies in candidate leaf k (largest k < nl with excl_k <= idx)
        for (int i0 = 0; i0 < nb; i0 += 32) {
          const int idx = i0 + lane;
          int k = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1) {
            int c = k + step;
            int e = __shfl_sync(kAll, excl, c & 31);
            if (c < nl && e <= idx) k = c;
          }
          const int ek = __shfl_sync(kAll, excl, k);
          const int sk = __shfl_sync(kAll, sb, k);
          if ((PACK || PACKV) && self_f64 && idx < nb) {
            // FP64 (x, y, z, q) / (x, y, z, G0), (G1, G2, -, -) relative to the target leaf centre
            const int body = sk + idx - ek;
            const double4 p = spos[body];
            const double4 g = sstr[body];
            if (PACK) {
              reinterpret_cast<double4*>(B)[idx] = make_double4(p.x - ox, p.y - oy, p.z - oz, g.x);
            } else {  // 48 bytes per body, the size of the packed FP32 record
              double2* Bd = reinterpret_cast<double2*>(B) + 3 * idx;
              Bd[0] = make_double2(p.x - ox, p.y - oy);
              Bd[1] = make_double2(p.z - oz, g.x);
              Bd[2] = make_double2(g.y, g.z);
            }
          } else if (PACK && idx < nb) {
            const int body = sk + idx - ek;
            const double4 p = spos[body];
            const float x = -(float)(p.x - ox), y = -(float)(p.y - oy), z = -(float)(p.z - oz), q = (float)sstr[body].x;
            float4* B4 = reinterpret_cast<float4*>(B);
            B4[2 * idx] = make_float4(x, x, y, y);
            B4[2 * idx + 1] = make_float4(z, z, q, q);
          } else if (PACKV && idx < nb) {
            const int body = sk + idx - ek;
            const double4 p = spos[body];
            const double4 g = sstr[body];
            const float x = -(float)(p.x - ox), y = -(float)(p.y - oy), z = -(float)(p.z - oz);
            const float g0 = (float)g.x, g1 = (float)g.y, g2 = (float)g.z;
            float4* B4 = reinterpret_cast<float4*>(B);
            B4[3 * idx] = make_float4(x, x, y, y);
            B4[3 * idx + 1] = make_float4(z, z, g0, g0);
            B4[3 * idx + 2] = make_float4(g1, g1, g2, g2);
          } else if (idx < nb) {
            const int body = sk + idx - ek;
            const double4 p = spos[body];
            const double4 q = sstr[body];
            far = max(far, max(hi_abs(p.x), max(hi_abs(p.y), hi_abs(p.z))));
            if constexpr (KIND == FMM_POINT_SOURCE) {
              if (PS && tiny_strength(q.x)) far = kFarHi;
              reinterpret_cast<double4*>(B)[idx] = make_double4(p.x, p.y, p.z, q.x);
            } else {
              double2* Bd = reinterpret_cast<double2*>(B) + 3 * idx;
              Bd[0] = make_double2(p.x, p.y);
              Bd[1] = make_double2(p.z, q.x);
              Bd[2] = make_double2(q.y, q.z);
            }
          }
        }
        __syncwarp();
        if constexpr (PACK) {
          // targets 0 and 1 of the lane in the two halves of every f32x2 operation
          const float4* B4 = reinterpret_cast<const float4*>(B);
          const float2 tx2 = make_float2((float)tx[0], (float)tx[1]);
          const float2 ty2 = make_float2((float)ty[0], (float)ty[1]);
          const float2 tz2 = make_float2((float)tz[0], (float)tz[1]);
          float2 ph = make_float2(0.f, 0.f), gx = ph, gy = ph, gz = ph;
          // the batch holding the target's own leaf runs in FP64 and skips coincident bodies;
          // the others run unguarded and, in the rare case that their sums come out non-finite
          // (bodies that coincide in FP32), repeat the batch with the r^2 > 0 guard
          if (self_f64) {
            double txd[2], tyd[2], tzd[2];
            self_targets_f64(tpos, ts + tile, nt, ti, TS, ox, oy, oz, txd, tyd, tzd);
            self_batch_f64_source<PS, NA>(reinterpret_cast<const double4*>(B), slice, nb, SS, txd, tyd, tzd, tot);
          } else if (self_batch) {
            packed_batch<kCoincident, PS>(B4, slice, nb, SS, tx2, ty2, tz2, ph, gx, gy, gz);
          } else {
            packed_batch<kUnguarded, PS>(B4, slice, nb, SS, tx2, ty2, tz2, ph, gx, gy, gz);
            if (!isfinite(ph.x + ph.y + gx.x + gx.y + gy.x + gy.y + gz.x + gz.y)) {
              ph = gx = gy = gz = make_float2(0.f, 0.f);
              packed_batch<kCoincident, PS>(B4, slice, nb, SS, tx2, ty2, tz2, ph, gx, gy, gz);
            }
          }
          part[0][0] += (R)ph.x;
          part[1][0] += (R)ph.y;
          part[0][1 % NA] += (R)gx.x;
          part[1][1 % NA] += (R)gx.y;
          part[0][2 % NA] += (R)gy.x;
          part[1][2 % NA] += (R)gy.y;
          part[0][3 % NA] += (R)gz.x;
          part[1][3 % NA] += (R)gz.y;
        } else if constexpr (PACKV) {
          const float2 tx2 = make_float2((float)tx[0], (float)tx[1]);
          const float2 ty2 = make_float2((float)ty[0], (float)ty[1]);
          const float2 tz2 = make_float2((float)tz[0], (float)tz[1]);
          const float4* B4 = reinterpret_cast<const float4*>(B);
          float2 acc[NA];
          // as on the point-source path: the batch holding the target's own leaf runs in FP64
          if (self_f64) {
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[a] = make_float2(0.f, 0.f);
            double txd[2], tyd[2], tzd[2];
            self_targets_f64(tpos, ts + tile, nt, ti, TS, ox, oy, oz, txd, tyd, tzd);
            self_batch_f64_vortex<GS, HS, NA>(reinterpret_cast<const double2*>(B), slice, nb, SS, txd, tyd, tzd, tot);
          } else if (self_batch) {
            packed_vortex_batch<kCoincident, GS, HS, NA>(B4, slice, nb, SS, tx2, ty2, tz2, acc);
          } else {
            packed_vortex_batch<kUnguarded, GS, HS, NA>(B4, slice, nb, SS, tx2, ty2, tz2, acc);
            float sum = 0.f;
#pragma unroll
            for (int a = 0; a < NA; ++a) sum += acc[a].x + acc[a].y;
            if (!isfinite(sum)) packed_vortex_batch<kCoincident, GS, HS, NA>(B4, slice, nb, SS, tx2, ty2, tz2, acc);
          }
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            part[0][a] += (R)acc[a].x;
            part[1][a] += (R)acc[a].y;
          }
        } else if constexpr (KIND == FMM_POINT_SOURCE) {
          const double4* Bd = reinterpret_cast<const double4*>(B);
          if (general || __any_sync(kAll, max(far, tfar) >= kFarHi)) {
            // two targets of the lane at a time (the third twice, counted once)
#pragma unroll 1
            for (int q = 0; q < tpt; q += 2) {
              const int q1 = min(q + 1, tpt - 1);
              const double gx[2] = {pick(tx, q), pick(tx, q1)}, gy[2] = {pick(ty, q), pick(ty, q1)};
              const double gz[2] = {pick(tz, q), pick(tz, q1)};
              double g2[2][NA];
#pragma unroll
              for (int a = 0; a < NA; ++a) g2[0][a] = g2[1][a] = 0.0;
              self_batch_f64_source<PS, NA>(Bd, slice, nb, SS, gx, gy, gz, g2);
#pragma unroll
              for (int k = 0; k < KT; ++k)
                if (k == q || (k == q + 1 && q1 == q + 1))
#pragma unroll
                  for (int a = 0; a < NA; ++a) tot[k][a] += g2[k == q ? 0 : 1][a];
            }
          } else {
            auto pairs = [&](auto n) {
#pragma unroll 2
              for (int j = slice; j < nb; j += SS) {
                const double4 b = Bd[j];
#pragma unroll
                for (int k = 0; k < n.value; ++k) source_pair_f64<PS>(tx[k], ty[k], tz[k], b.x, b.y, b.z, b.w, part[k]);
              }
            };
            if (tpt == 3)
              pairs(std::integral_constant<int, KT>());
            else
              pairs(std::integral_constant<int, 2>());
          }
        } else {
          const double2* Bd = reinterpret_cast<const double2*>(B);
          if (general || __any_sync(kAll, max(far, tfar) >= kFarHi)) {
            if constexpr (KT == 2) {
              const double gx[2] = {tx[0], tx[1]}, gy[2] = {ty[0], ty[1]}, gz[2] = {tz[0], tz[1]};
              self_batch_f64_vortex<GS, HS, NA>(Bd, slice, nb, SS, gx, gy, gz, tot);
            } else {
              // two targets of the lane at a time (the third twice, counted once)
#pragma unroll 1
              for (int q = 0; q < tpt; q += 2) {
                const int q1 = min(q + 1, tpt - 1);
                const double gx[2] = {pick(tx, q), pick(tx, q1)}, gy[2] = {pick(ty, q), pick(ty, q1)};
                const double gz[2] = {pick(tz, q), pick(tz, q1)};
                double g2[2][NA];
#pragma unroll
                for (int a = 0; a < NA; ++a) g2[0][a] = g2[1][a] = 0.0;
                self_batch_f64_vortex<GS, HS, NA>(Bd, slice, nb, SS, gx, gy, gz, g2);
#pragma unroll
                for (int k = 0; k < KT; ++k)
                  if (k == q || (k == q + 1 && q1 == q + 1))
#pragma unroll
                    for (int a = 0; a < NA; ++a) tot[k][a] += g2[k == q ? 0 : 1][a];
              }
            }
          } else {
            // (two targets: a third costs the gradient's kernel its registers, 25.5 -> 29.4 ms on the 300k ring)
            for (int j = slice; j < nb; j += SS) {
              const double2 a = Bd[3 * j], b = Bd[3 * j + 1], c = Bd[3 * j + 2];
#pragma unroll
              for (int k = 0; k < KT; ++k)
                if (KT == 2 || k < tpt)
                  vortex_pair_f64<GS, HS>(tx[k], ty[k], tz[k], a.x, a.y, b.x, b.y, c.x, c.y, us[k], Qs[k], Es[k]);
            }
          }
        }
        __syncwarp();
        if (MIXED) {
#pragma unroll
          for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int a = 0; a < NA; ++a) tot[k][a] += (double)part[k][a], part[k][a] = R(0);
        }
      }
      if constexpr (MIXED) {
        break;
      } else {
        bool finite = true;
#pragma unroll
        for (int k = 0; k < KT; ++k) {
          if constexpr (KIND == FMM_POINT_VORTEX && GS) {
#pragma unroll
            for (int a = 0; a < 3; ++a) part[k][a % NA] = us[k][a];
          }
          if constexpr (QE) {
            Qs[k][8] = -(Qs[k][0] + Qs[k][4]);
            vortex_grad_from_qe<double>(Qs[k], Es[k], &part[k][(GS ? 3 : 0) % NA]);
          }
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            tot[k][a] += part[k][a];
            finite = finite && isfinite(tot[k][a]);
          }
        }
        if (general || !__any_sync(kAll, !finite)) break;
      }
    }
    // slices -> lanes ti (< TS), then warps -> shared memory
    for (int o = TS; o < 32; o <<= 1)
#pragma unroll
      for (int k = 0; k < KT; ++k)
#pragma unroll
        for (int a = 0; a < NA; ++a) tot[k][a] += __shfl_xor_sync(kAll, tot[k][a], o);
    if constexpr (RW) {
      // one warp owns the row: its sums go to the targets directly
      if (slice == 0) {
#pragma unroll
        for (int k = 0; k < KT; ++k) {
          const int i = ti + k * TS;
          if (i < nt)
#pragma unroll
            for (int a = 0; a < NA; ++a) {
              if (KIND == FMM_POINT_SOURCE && a == 0 && !PS) continue;
              atomicAdd(acc13 + 13 * (int64_t)(ts + tile + i) + chan_row<KIND, GS>(a), tot[k][a] * kOneOver4Pi);
            }
        }
      }
      continue;
    }
    if (slice == 0) {
#pragma unroll
      for (int k = 0; k < KT; ++k) {
        int i = ti + k * TS;
        if (i < nt)
#pragma unroll
          for (int a = 0; a < NA; ++a) red[(w * 32 * kTPT + i) * NA + a] = tot[k][a];
      }
    }
    __syncthreads();
    const int out = ITEMS ? items[2 * blockIdx.x + 1].x : -1;
    for (int e = threadIdx.x; e < nt * NA; e += W * 32) {
      const int i = e / NA, a = e - i * NA;
      double v = 0;
#pragma unroll
      for (int q = 0; q < W; ++q) v += red[(q * 32 * kTPT + i) * NA + a];
      if (ITEMS && out >= 0) {
        item_sums[out + e] = v;
        continue;
      }
      if (KIND == FMM_POINT_SOURCE && a == 0 && !PS) continue;
      // atomic: under SelfTuning a non-leaf target branch and its own leaves can both own direct-list rows
      atomicAdd(acc13 + 13 * (int64_t)(ts + tile + i) + chan_row<KIND, GS>(a), v * kOneOver4Pi);
    }
    if (ITEMS) break;
    __syncthreads();
  }
}

template <class R, int KIND, bool GS, bool HS>
constexpr size_t p2p_smem_bytes() {
  constexpr int W = kWarps;
  return (size_t)W * slots_per_body<R, KIND>() * batch_bodies<R, KIND>() * sizeof(R) +
         (size_t)W * 32 * kTPT * n_chan<KIND, GS, HS>() * sizeof(double);
}

// All pairs.  A CTA owns kP2PThreads * tpt() consecutive targets, tpt() per thread, and the source
// chunks [y, y + 1) * per_split of kP2PThreads bodies, staged through shared memory.  With `part`
// the sources are split over gridDim.y CTAs, whose sums go to part[split][target][channel] and are
// added in split order by k_direct_sum: the targets of a subsample fill a fraction of the SMs
// (20,000 targets are 40 CTAs), the splits fill them.  Arithmetic of the near field: FP64 through
// the 17 / 38-operation pair (a CTA that meets a pair outside its range repeats its share in the
// general arithmetic), mixed through the packed pair relative to the CTA's first target, a chunk in
// FP32 and the chunks in FP64.  Bound by the FP64 / FP32 pipe (no traffic to speak of): 20,000 targets x
// 200,003 point sources in FP64 82.3 -> 4.74 ms (8.4e11 pairs/s, 0.77 of the FP64 pipe at 17 operations).
template <class R, int KIND, bool PS, bool GS, bool HS>
__global__ void __launch_bounds__(kP2PThreads) k_direct(const double4* __restrict__ tpos, int64_t nt_total,
                                                        const double4* __restrict__ spos,
                                                        const double4* __restrict__ sstr, int64_t ns, int per_split,
                                                        double* __restrict__ acc13, double* __restrict__ part) {
  constexpr int TPT = tpt<KIND>(), NA = n_chan<KIND, GS, HS>();
  constexpr bool MIXED = sizeof(R) == 4;
  constexpr bool SOURCE = KIND == FMM_POINT_SOURCE;
  // a body: FP64 (x, y, z, q) / (x, y, z, G); mixed the packed record of the same size
  __shared__ __align__(16) unsigned char sh[kP2PThreads * (SOURCE ? 32 : 48)];
  const int64_t base = (int64_t)blockIdx.x * kP2PThreads * TPT;
  double ox = 0, oy = 0, oz = 0;
  if (MIXED) {
    const double4 p = tpos[base];
    ox = p.x;
    oy = p.y;
    oz = p.z;
  }
  R tx[TPT], ty[TPT], tz[TPT];
  int far = 0;
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int64_t i = base + threadIdx.x + k * kP2PThreads;
    tx[k] = ty[k] = tz[k] = R(0);
    if (i < nt_total) {
      const double4 p = tpos[i];
      far = max(far, max(hi_abs(p.x), max(hi_abs(p.y), hi_abs(p.z))));
      tx[k] = (R)(p.x - ox);
      ty[k] = (R)(p.y - oy);
      tz[k] = (R)(p.z - oz);
    }
  }
  double tot[TPT][NA];
  const int64_t c_lo = (int64_t)blockIdx.y * per_split * kP2PThreads;
  const int64_t c_hi = min(ns, c_lo + (int64_t)per_split * kP2PThreads);
  for (bool general = false;; general = true) {  // FP64: a second pass in the general arithmetic
    double part64[TPT][4], us[TPT][3], Qs[TPT][9], Es[TPT][3];
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
#pragma unroll
      for (int a = 0; a < NA; ++a) tot[k][a] = 0.0;
#pragma unroll
      for (int a = 0; a < 4; ++a) part64[k][a] = 0.0;
#pragma unroll
      for (int a = 0; a < 9; ++a) Qs[k][a] = 0.0;
#pragma unroll
      for (int a = 0; a < 3; ++a) us[k][a] = Es[k][a] = 0.0;
    }
    for (int64_t c = c_lo; c < c_hi; c += kP2PThreads) {
      const int64_t j = c + threadIdx.x;
      if (j < c_hi) {
        const double4 p = spos[j];
        const double4 q = sstr[j];
        far = max(far, max(hi_abs(p.x), max(hi_abs(p.y), hi_abs(p.z))));
        if (SOURCE && PS && tiny_strength(q.x)) far = kFarHi;
        float4* F = reinterpret_cast<float4*>(sh) + (SOURCE ? 2 : 3) * threadIdx.x;
        double2* D = reinterpret_cast<double2*>(F);
        if (MIXED) {
          const float x = -(float)(p.x - ox), y = -(float)(p.y - oy), z = -(float)(p.z - oz), s = (float)q.x;
          F[0] = make_float4(x, x, y, y);
          F[1] = make_float4(z, z, s, s);
          if (!SOURCE) F[2] = make_float4((float)q.y, (float)q.y, (float)q.z, (float)q.z);
        } else {
          D[0] = make_double2(p.x, p.y);
          D[1] = make_double2(p.z, q.x);
          if (!SOURCE) D[2] = make_double2(q.y, q.z);
        }
      }
      __syncthreads();
      const int m = (int)min((int64_t)kP2PThreads, c_hi - c);
      if constexpr (MIXED) {
        const float4* B4 = reinterpret_cast<const float4*>(sh);
#pragma unroll
        for (int h = 0; h < TPT / 2; ++h) {
          const float2 tx2 = make_float2(tx[2 * h], tx[2 * h + 1]), ty2 = make_float2(ty[2 * h], ty[2 * h + 1]);
          const float2 tz2 = make_float2(tz[2 * h], tz[2 * h + 1]);
          float2 a[NA];
          // unguarded; a chunk whose sums are not finite again without the pairs that lack r^2 > 0
#pragma unroll 1
          for (int guard = 0; guard < 2; ++guard) {
#pragma unroll
            for (int q = 0; q < NA; ++q) a[q] = make_float2(0.f, 0.f);
            if constexpr (SOURCE) {
              if (guard)
                packed_batch<kSkip, PS>(B4, 0, m, 1, tx2, ty2, tz2, a[0], a[1 % NA], a[2 % NA], a[3 % NA]);
              else
                packed_batch<kUnguarded, PS>(B4, 0, m, 1, tx2, ty2, tz2, a[0], a[1 % NA], a[2 % NA], a[3 % NA]);
            } else {
              if (guard)
                packed_vortex_batch<kSkip, GS, HS, NA>(B4, 0, m, 1, tx2, ty2, tz2, a);
              else
                packed_vortex_batch<kUnguarded, GS, HS, NA>(B4, 0, m, 1, tx2, ty2, tz2, a);
            }
            float sum = 0.f;
#pragma unroll
            for (int q = 0; q < NA; ++q) sum += a[q].x + a[q].y;
            if (isfinite(sum)) break;
          }
#pragma unroll
          for (int q = 0; q < NA; ++q) {
            tot[2 * h][q] += (double)a[q].x;
            tot[2 * h + 1][q] += (double)a[q].y;
          }
        }
      } else if (general) {
#pragma unroll
        for (int h = 0; h < TPT / 2; ++h) {
          const double gx[2] = {tx[2 * h], tx[2 * h + 1]}, gy[2] = {ty[2 * h], ty[2 * h + 1]};
          const double gz[2] = {tz[2 * h], tz[2 * h + 1]};
          double t2[2][NA];
#pragma unroll
          for (int a = 0; a < NA; ++a) t2[0][a] = t2[1][a] = 0.0;
          if constexpr (SOURCE)
            self_batch_f64_source<PS, NA>(reinterpret_cast<const double4*>(sh), 0, m, 1, gx, gy, gz, t2);
          else
            self_batch_f64_vortex<GS, HS, NA>(reinterpret_cast<const double2*>(sh), 0, m, 1, gx, gy, gz, t2);
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            tot[2 * h][a] += t2[0][a];
            tot[2 * h + 1][a] += t2[1][a];
          }
        }
      } else if constexpr (SOURCE) {
        const double4* B = reinterpret_cast<const double4*>(sh);
#pragma unroll 1
        for (int jj = 0; jj < m; ++jj) {
          const double4 b = B[jj];
#pragma unroll
          for (int k = 0; k < TPT; ++k) source_pair_f64<PS>(tx[k], ty[k], tz[k], b.x, b.y, b.z, b.w, part64[k]);
        }
      } else {
        const double2* B = reinterpret_cast<const double2*>(sh);
#pragma unroll 1
        for (int jj = 0; jj < m; ++jj) {
          const double2 a = B[3 * jj], b = B[3 * jj + 1], d = B[3 * jj + 2];
#pragma unroll
          for (int k = 0; k < TPT; ++k)
            vortex_pair_f64<GS, HS>(tx[k], ty[k], tz[k], a.x, a.y, b.x, b.y, d.x, d.y, us[k], Qs[k], Es[k]);
        }
      }
      __syncthreads();
    }
    if (MIXED || general) break;
    bool bad = far >= kFarHi;
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
      if constexpr (SOURCE) {
#pragma unroll
        for (int a = 0; a < 4; ++a) tot[k][a % NA] = part64[k][a];
      } else {
        if constexpr (GS) {
#pragma unroll
          for (int a = 0; a < 3; ++a) tot[k][a % NA] = us[k][a];
        }
        if constexpr (HS) {
          Qs[k][8] = -(Qs[k][0] + Qs[k][4]);
          vortex_grad_from_qe<double>(Qs[k], Es[k], &tot[k][(GS ? 3 : 0) % NA]);
        }
      }
#pragma unroll
      for (int a = 0; a < NA; ++a) bad = bad || !isfinite(tot[k][a]);
    }
    if (!__syncthreads_or(bad)) break;
  }
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int64_t i = base + threadIdx.x + k * kP2PThreads;
    if (i >= nt_total) continue;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      if (part)
        part[((int64_t)blockIdx.y * nt_total + i) * NA + a] = tot[k][a];
      else if (!(SOURCE && a == 0 && !PS))
        acc13[13 * i + chan_row<KIND, GS>(a)] += tot[k][a] * kOneOver4Pi;
    }
  }
}

// sums of the source splits in split order
template <int KIND, bool PS, bool GS, int NA>
__global__ void k_direct_sum(const double* __restrict__ part, int n_split, int64_t nt, double* __restrict__ acc13) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nt * NA; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / NA;
    const int a = (int)(e - i * NA);
    if (KIND == FMM_POINT_SOURCE && a == 0 && !PS) continue;
    double v = 0.0;
    for (int s = 0; s < n_split; ++s) v += part[(int64_t)s * nt * NA + e];
    acc13[13 * i + chan_row<KIND, GS>(a)] += v * kOneOver4Pi;
  }
}

// source bodies of every row, one block each, eight loads of a thread in flight (a warp per row and a
// thread per sum in k_p2p_sum: 300 targets x 1e6 sources, 32,000 leaves a row, mixed, near field 1.03 ms;
// 0.57 now)
__global__ void k_p2p_row_sources(const int* __restrict__ off, const int* __restrict__ src_of,
                                  const int* __restrict__ s_count, int* __restrict__ n_src) {
  __shared__ int sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  int v = 0;
  const int e = off[blockIdx.x + 1];
#pragma unroll 8
  for (int i = off[blockIdx.x] + threadIdx.x; i < e; i += blockDim.x) v += s_count[src_of[i]];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&sum, v);
  __syncthreads();
  if (threadIdx.x == 0) n_src[blockIdx.x] = sum;
}

// what a source body costs a tile of nt targets, in target slots: those that the tile occupies (three: the
// FP64 kernels' choice of targets per lane) and its gathering (gather)
__device__ __forceinline__ int tile_cost(int nt, bool three, int gather) {
  const int tpt = three ? targets_per_lane(nt) : kTPT;
  int ts = 1;
  while (ts * tpt < nt) ts <<= 1;
  return ts * tpt + gather;
}

// The items of a launch, one block: every tile of a row is cut into shares of about the launch's
// work / goal slot pairs.  Items and their sums' places come from scans over the rows, so that the
// cut, and with it the order of every sum, depends on the tree and the lists alone.
constexpr int kPlanThreads = 1024;
template <bool SUB>
__global__ void __launch_bounds__(kPlanThreads)
    k_p2p_plan(const int* __restrict__ tgt_list, const int* __restrict__ off, int rows, const int* __restrict__ t_count,
               const int* __restrict__ n_src, int goal, int na, int max_sums, int three, int gather,
               int4* __restrict__ items, int* __restrict__ n_items) {
  __shared__ unsigned long long tot[kPlanThreads / 32];
  __shared__ int2 sh[kPlanThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long work = 0;
  for (int r = threadIdx.x; r < rows; r += kPlanThreads) {
    const int tc = t_count[tgt_list[r]];
    int slots = 0;
    for (int t = 0, nt; t < tc; t += nt) {
      nt = next_tile<SUB>(tc - t);
      slots += tile_cost(nt, three != 0, gather);
    }
    work += (unsigned long long)slots * (unsigned)n_src[r];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) work += __shfl_xor_sync(kAll, work, o);
  if (lane == 0) tot[w] = work;
  __syncthreads();
  work = 0;
  for (int q = 0; q < kPlanThreads / 32; ++q) work += tot[q];
  const unsigned long long share = work / goal + 1;
  int2 run = make_int2(0, 0);  // items, sums of the rows before
  for (int r0 = 0; r0 < rows; r0 += kPlanThreads) {
    const int r = r0 + threadIdx.x;
    int tc = 0, ns = 0, a = 0, nl = 0;
    if (r < rows) {
      tc = t_count[tgt_list[r]];
      ns = n_src[r];
      a = off[r];
      nl = off[r + 1] - a;
    }
    auto cut = [&](int nt) {
      const unsigned long long cost = (unsigned long long)tile_cost(nt, three != 0, gather) * (unsigned)ns;
      const unsigned long long c = (cost + share - 1) / share;
      return (int)max(1ull, min(c, (unsigned long long)min(nl, ns / kItemSources)));
    };
    int2 v = make_int2(0, 0);
    for (int t = 0, nt; t < tc; t += nt) {
      nt = next_tile<SUB>(tc - t);
      const int c = cut(nt);
      v.x += c;
      if (c > 1) v.y += c * nt * na;
    }
    int2 in = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(kAll, in.x, o), y = __shfl_up_sync(kAll, in.y, o);
      if (lane >= o) in.x += x, in.y += y;
    }
    if (lane == 31) sh[w] = in;
    __syncthreads();
    int2 ex = make_int2(run.x + in.x - v.x, run.y + in.y - v.y);
    for (int q = 0; q < kPlanThreads / 32; ++q) {
      if (q < w) ex.x += sh[q].x, ex.y += sh[q].y;
      run.x += sh[q].x;
      run.y += sh[q].y;
    }
    __syncthreads();
    for (int t = 0, nt; t < tc; t += nt) {
      nt = next_tile<SUB>(tc - t);
      const int c = cut(nt);
      // (the bound on the items leaves room for every row's sums)
      const bool split = c > 1 && ex.y + c * nt * na <= max_sums;
      const int q = nl / c, more = nl - q * c;  // leaves per share, shares with one more
      for (int j = 0; j < c; ++j) {
        const int lo = split ? a + j * q + min(j, more) : a;
        const int hi = split ? lo + q + (j < more) : (j == 0 ? a + nl : a);
        items[2 * (ex.x + j)] = make_int4(r, t, lo, hi);
        items[2 * (ex.x + j) + 1] = make_int4(split ? ex.y + j * nt * na : -1, split && j == 0 ? c : 0, nt, 0);
      }
      ex.x += c;
      if (c > 1) ex.y += c * nt * na;
    }
  }
  if (threadIdx.x == 0) *n_items = run.x;
}

// the shares of every tile that was cut, added in order; those of a tile of few sums and many shares
// (rows of few targets and thousands of leaves) in several interleaved groups
constexpr int kSumThreads = 128, kSumManyShares = 32;
template <int KIND, bool PS, bool GS, int NA>
__global__ void __launch_bounds__(kSumThreads) k_p2p_sum(const int4* __restrict__ items,
                                                         const int* __restrict__ n_items,
                                                         const double* __restrict__ sums,
                                                         const int* __restrict__ tgt_list,
                                                         const int* __restrict__ t_start, double* __restrict__ acc13) {
  __shared__ double part[kSumThreads];
  if ((int)blockIdx.x >= *n_items) return;
  const int4 a = items[2 * blockIdx.x], b = items[2 * blockIdx.x + 1];
  if (b.y == 0) return;
  const int first = t_start[tgt_list[a.x]] + a.y, n = b.z * NA;
  // sum e of the shares from c0 in steps of dc
  auto add = [&](int e, int c0, int dc) {
    double v = 0.0;
#pragma unroll 8
    for (int c = c0; c < b.y; c += dc) v += sums[b.x + c * n + e];
    return v;
  };
  // atomic: under SelfTuning the rows of nested branches add to the same targets
  auto put = [&](int e, double v) {
    const int i = e / NA, ch = e - i * NA;
    if (KIND == FMM_POINT_SOURCE && ch == 0 && !PS) return;
    atomicAdd(acc13 + 13 * (int64_t)(first + i) + chan_row<KIND, GS>(ch), v * kOneOver4Pi);
  };
  const int groups = b.y >= kSumManyShares ? kSumThreads / n : 1;
  if (groups > 1) {
    const int g = threadIdx.x / n, e = threadIdx.x - g * n;
    if (g < groups) part[threadIdx.x] = add(e, g, groups);
    __syncthreads();
    if (g != 0) return;
    double v = part[e];
    for (int q = 1; q < groups; ++q) v += part[q * n + e];
    put(e, v);
    return;
  }
  for (int e = threadIdx.x; e < n; e += kSumThreads) put(e, add(e, 0, 1));
}

template <class R, int KIND, bool PS, bool GS, bool HS>
void run_p2p(const DevTree& tt, const DevTree& stt, DevLists& L, double* acc13, int exact_self, cudaStream_t st) {
  if (L.n_dir_targets == 0) return;
  constexpr size_t smem = p2p_smem_bytes<R, KIND, GS, HS>();
  const int rows = (int)L.n_dir_targets;
  note_launch();
  // target leaves of a few bodies (on average <= 8), packed FP32 kernel: one warp per row
  // (measured slower for the FP64 kernel, whose rows keep a CTA each)
  if constexpr (packed<R, KIND>()) {
    if (tt.n_bodies <= 8 * tt.n_leaves) {
      if (smem > 48 * 1024)
        FMM_CUDA_TRY(cudaFuncSetAttribute(k_p2p<R, KIND, PS, GS, HS, true, false>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      k_p2p<R, KIND, PS, GS, HS, true, false><<<(rows + kWarps - 1) / kWarps, kWarps * 32, smem, st>>>(
          L.dir_tgt.ptr, L.dir_off.ptr, rows, L.dir_s.ptr, tt.body_start.ptr, tt.body_count.ptr, tt.tcenter.ptr,
          stt.body_start.ptr, stt.body_count.ptr, tt.pos.ptr, stt.pos.ptr, stt.str.ptr, acc13, nullptr,
          nullptr, nullptr, exact_self);
      FMM_CUDA_TRY(cudaGetLastError());
      return;
    }
  }
  int dev = 0, n_sm = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  FMM_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  constexpr int NA = n_chan<KIND, GS, HS>();
  // body pairs (of a tuple's system: its part by the number of bodies)
  const double pairs = (double)L.n_pairs * ((double)stt.n_bodies / (double)L.n_source_bodies);
  if (rows <= kItemRowsPerSM * n_sm && pairs > kItemRowPairs * rows) {
    if (smem > 48 * 1024)
      FMM_CUDA_TRY(cudaFuncSetAttribute(k_p2p<R, KIND, PS, GS, HS, false, true>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    FMM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_p2p<R, KIND, PS, GS, HS, false, true>,
                                                               kWarps * 32, smem));
    const int goal = kItemWaves * std::max(1, per_sm) * n_sm;
    // a tile per 64 targets begun (up to three with sub-tiles), a share more per 1 / goal of the work;
    // at most twice the goal of them in tiles that are cut.  The targets of rows that are not leaves
    // (SelfTuning) can be those of other rows too, one of them per level
    const int64_t nest = L.rule_method == FMM_LIST_SELF_TUNING ? tt.n_levels : 1;
    const int64_t most = 3 * (int64_t)rows + nest * tt.n_bodies / (32 * kTPT) + goal + 1;
    // the sums: 64 targets of each of those, and (a share has kItemSources bodies or more) no more than the
    // pairs allow: 0.5 MB for 2,000 bodies instead of 10
    const int64_t sums = std::min((int64_t)2 * goal * 32 * kTPT, L.n_pairs / kItemSources + 1) * NA;
    L.p2p_items.grow(2 * (size_t)most);
    L.p2p_meta.grow((size_t)rows + 1);
    L.p2p_part.grow((size_t)sums);
    note_launch();
    const int64_t per_row = L.n_direct / rows;
    k_p2p_row_sources<<<rows, per_row <= 64 ? 32 : per_row <= 1024 ? 128 : 1024, 0, st>>>(
        L.dir_off.ptr, L.dir_s.ptr, stt.body_count.ptr, L.p2p_meta.ptr + 1);
    note_launch();
    constexpr int KT = max_targets_per_lane<R, KIND, HS>();
    k_p2p_plan<sub_tiles<R, KIND, true>() && KT == kTPT><<<1, kPlanThreads, 0, st>>>(
        L.dir_tgt.ptr, L.dir_off.ptr, rows, tt.body_count.ptr, L.p2p_meta.ptr + 1, goal, NA, (int)sums,
        KT == 3 ? 1 : 0, sizeof(R) == 4 ? kGatherSlotsF32 : kGatherSlotsF64, L.p2p_items.ptr, L.p2p_meta.ptr);
    note_launch();
    k_p2p<R, KIND, PS, GS, HS, false, true><<<(int)most, kWarps * 32, smem, st>>>(
        L.dir_tgt.ptr, L.dir_off.ptr, rows, L.dir_s.ptr, tt.body_start.ptr, tt.body_count.ptr, tt.tcenter.ptr,
        stt.body_start.ptr, stt.body_count.ptr, tt.pos.ptr, stt.pos.ptr, stt.str.ptr, acc13, L.p2p_items.ptr,
        L.p2p_meta.ptr, L.p2p_part.ptr, exact_self);
    note_launch();
    k_p2p_sum<KIND, PS, GS, NA><<<(int)most, kSumThreads, 0, st>>>(L.p2p_items.ptr, L.p2p_meta.ptr, L.p2p_part.ptr,
                                                          L.dir_tgt.ptr, tt.body_start.ptr, acc13);
  } else {
    if (smem > 48 * 1024)
      FMM_CUDA_TRY(cudaFuncSetAttribute(k_p2p<R, KIND, PS, GS, HS, false, false>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_p2p<R, KIND, PS, GS, HS, false, false><<<rows, kWarps * 32, smem, st>>>(
        L.dir_tgt.ptr, L.dir_off.ptr, rows, L.dir_s.ptr, tt.body_start.ptr, tt.body_count.ptr, tt.tcenter.ptr,
        stt.body_start.ptr, stt.body_count.ptr, tt.pos.ptr, stt.pos.ptr, stt.str.ptr, acc13, nullptr, nullptr, nullptr,
        exact_self);
  }
  FMM_CUDA_TRY(cudaGetLastError());
}

constexpr size_t kDirectPartMax = (size_t)64 << 20;  // bytes of the splits' sums

template <class R, int KIND, bool PS, bool GS, bool HS>
void run_direct(const double4* tpos, int64_t nt, const double4* spos, const double4* sstr, int64_t ns, double* acc13,
                DevBuf<double>* part, cudaStream_t st) {
  constexpr int T = tpt<KIND>(), NA = n_chan<KIND, GS, HS>();
  const int64_t tiles = (nt + kP2PThreads * T - 1) / (kP2PThreads * T);
  if (tiles == 0) return;
  const int64_t chunks = (ns + kP2PThreads - 1) / kP2PThreads;
  // splits of the sources: four waves of resident CTAs, at least four chunks each, sums of bounded size
  int64_t splits = 1;
  if (part) {
    int dev = 0, n_sm = 0, per_sm = 0;
    FMM_CUDA_TRY(cudaGetDevice(&dev));
    FMM_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    FMM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_direct<R, KIND, PS, GS, HS>, kP2PThreads, 0));
    splits = std::min<int64_t>((int64_t)4 * per_sm * n_sm / tiles, chunks / 4);
    splits = std::min<int64_t>(splits, (int64_t)(kDirectPartMax / (NA * sizeof(double))) / nt);
    splits = std::max<int64_t>(1, std::min<int64_t>(splits, 65535));
  }
  int64_t per = std::max<int64_t>(1, (chunks + splits - 1) / splits);
  splits = std::max<int64_t>(1, (chunks + per - 1) / per);
  double* sums = nullptr;
  if (splits > 1) {
    try {
      part->grow((size_t)splits * nt * NA);
      sums = part->ptr;
    } catch (const Error&) {  // no room for the sums: one pass over all the sources needs none
      cudaGetLastError();
      splits = 1;
      per = chunks;
    }
  }
  FMM_CHECK(per * kP2PThreads < INT_MAX && tiles < INT_MAX, FMM_ERR_MEMORY, "all-pairs sum exceeds the index range");
  note_launch();
  k_direct<R, KIND, PS, GS, HS><<<dim3((unsigned)tiles, (unsigned)splits), kP2PThreads, 0, st>>>(
      tpos, nt, spos, sstr, ns, (int)per, acc13, sums);
  FMM_CUDA_TRY(cudaGetLastError());
  if (sums) {
    note_launch();
    k_direct_sum<KIND, PS, GS, NA><<<(int)std::min<int64_t>((nt * NA + 255) / 256, 148 * 16), 256, 0, st>>>(
        sums, (int)splits, nt, acc13);
    FMM_CUDA_TRY(cudaGetLastError());
  }
}

template <class R, class F>
void dispatch(int kind, bool ps, bool gs, bool hs, F& f) {
  // Laplace: phi optional, gradient always (the reference's kernel ignores the switch)
  if (kind == FMM_POINT_SOURCE) {
    if (ps)
      f.template go<R, FMM_POINT_SOURCE, true, true, false>();
    else
      f.template go<R, FMM_POINT_SOURCE, false, true, false>();
  } else {
    if (gs && hs)
      f.template go<R, FMM_POINT_VORTEX, false, true, true>();
    else if (hs)
      f.template go<R, FMM_POINT_VORTEX, false, false, true>();
    else
      f.template go<R, FMM_POINT_VORTEX, false, true, false>();
  }
}

struct P2PLaunch {
  const DevTree& tt;
  const DevTree& stt;
  DevLists& L;
  double* acc13;
  int exact_self;
  cudaStream_t st;
  template <class R, int K, bool PS, bool GS, bool HS>
  void go() {
    run_p2p<R, K, PS, GS, HS>(tt, stt, L, acc13, exact_self, st);
  }
};

struct DirectLaunch {
  const double4* tpos;
  int64_t nt;
  const double4* spos;
  const double4* sstr;
  int64_t ns;
  double* acc13;
  DevBuf<double>* part;
  cudaStream_t st;
  template <class R, int K, bool PS, bool GS, bool HS>
  void go() {
    run_direct<R, K, PS, GS, HS>(tpos, nt, spos, sstr, ns, acc13, part, st);
  }
};

}  // namespace

void launch_p2p(const DevTree& tt, const DevTree& stt, DevLists& L, double* acc13, int kind, bool ps, bool gs,
                bool hs, int precision, cudaStream_t st, bool exact_self) {
  P2PLaunch f{tt, stt, L, acc13, exact_self ? 1 : 0, st};
  if (precision == FMM_PRECISION_MIXED)
    dispatch<float>(kind, ps, gs, hs, f);
  else
    dispatch<double>(kind, ps, gs, hs, f);
}

void launch_direct(const double4* tpos, int64_t nt, const double4* spos, const double4* sstr, int64_t ns, double* acc13,
                   int kind, bool gs, bool hs, int precision, cudaStream_t st, DevBuf<double>* part) {
  DirectLaunch f{tpos, nt, spos, sstr, ns, acc13, part, st};
  // direct! always evaluates the potential of point sources (src/direct.jl:66-70 + test/gravitational.jl:92)
  if (precision == FMM_PRECISION_MIXED)
    dispatch<float>(kind, true, gs, hs, f);
  else
    dispatch<double>(kind, true, gs, hs, f);
}

}  // namespace fmmb
