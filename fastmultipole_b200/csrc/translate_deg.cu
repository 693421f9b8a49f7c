// translate_deg.cu -- translations whose degrees are spread over the warps of a CTA.
//
// The rotation-based chain rotate_z -> rotate_y -> coaxial translation -> [Lamb-Helmholtz
// re-centring] -> rotate_y back -> rotate_z back (src/translate.jl:144-174, 519-550, 555-1412,
// 1896-1926) is independent from degree to degree except for the coaxial step, which mixes the
// degrees of one order.  Here the lanes of a warp hold pairs (or children) and the warps of a CTA
// take different degrees of the same pairs: every degree's rotation runs at the same time, the
// rotated degrees meet in shared memory, and the degrees of the result are formed side by side
// again.  The kernels before took a warp per output expansion, lanes over coefficients, one input
// after another with its Wigner matrices built per pair: a few hundred warps whose chains of
// dependent stages set the time.  Whole solves, before -> after: 150k clustered point sources,
// order 16, tolerance 1e-7: 98.4 -> 10.2 ms; 48k vortex particles, order 16, tolerance 1e-6: 18.0 ->
// 4.45 ms; 30k vortex ring, order 8: 2.17 -> 1.49 ms (M2M and L2L alone).  The M2L's shared memory
// lets an SM hold two CTAs up to order 16 and one above.  In FP32 (fixed orders of the mixed path)
// against a lane per pair: 300k clustered bodies, order 10, M2L 2.04 -> 1.02 ms; 200k vortex ring, order
// 12, 1.42 -> 0.67 ms.  Rows that are long and even are faster by lanes: m2l_lane.cu has the rule.
//
// Rotations about y are factorised as in m2l_lane.cu, with the magnitudes applied outside
// the two matrix products, so that one constant table of the Wigner matrix at pi/2 serves both
// magnitude sets and every order up to kMaxP.
#include <mutex>

#include "context.cuh"

namespace fmmb {

namespace {

constexpr unsigned kAll = 0xffffffffu;
__host__ __device__ constexpr int hi(int n, int m) { return n * (n + 1) / 2 + m; }
__host__ __device__ constexpr int lenT(int n) { return n < 0 ? 0 : (n + 1) * (n + 2) * (2 * n + 3) / 6; }

constexpr int kNh = hi(kMaxP + 1, 0);
constexpr int kLenH = lenT(kMaxP) + kMaxP + 1;  // padding: a column is read to the kernel's order
// H(a, nu) of degree n at lenT(n-1) + nu (n+1) + a; magnitudes A(m), B(a) of the zeta (multipole)
// and eta (local) sets; k!; the degree-power normalisations
__constant__ double c_H[kLenH];
__constant__ double c_Az[kNh], c_Bz[kNh], c_Ae[kNh], c_Be[kNh];
__constant__ double c_Mt[kNh], c_Lt[kNh];
// the same in global memory, for kernels whose lanes read different degrees (k_mm_ll)
__device__ double d_H[kLenH];
__device__ double d_mag[4][kNh];  // Az, Bz, Ae, Be
__constant__ double c_fact[2 * kMaxP + 2];
__constant__ double c_ifact[kMaxP + 1] = {FMM_INV_FACTORIALS};
// FP32 tables up to order 12 for the mixed path: B H over a, zeta and eta, the magnitude multiplied
// in before the one rounding; column (n, nu) at float4 kColQ hi(n, nu), zero past its degree, read
// four entries per constant load.  The same column gives the second product, whose outputs take
// A / B in FP64: factors rounded to FP32 by themselves would be the same for every pair and add up
// (ring far field 6.6e-9 -> 1.3e-8; with a second table of A H 6.6e-9 too, at 1.2 times the time)
constexpr int kMaxF = 12, kColQ = 4, kNhF = hi(kMaxF + 1, 0);
__constant__ float4 c_BzF[kNhF * kColQ], c_BeF[kNhF * kColQ];
__constant__ double c_ABz[kNhF], c_ABe[kNhF];
__constant__ float c_factF[2 * kMaxF + 2];

std::mutex g_mu;
bool g_done[64];

void ensure_tables(cudaStream_t st) {
  int dev = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_mu);
  if (dev < 64 && g_done[dev]) return;
  HostTables h;
  build_tables(h, kMaxP);
  std::vector<double> H(kLenH, 0.0), az(kNh), bz(kNh), ae(kNh), be(kNh), fact(2 * kMaxP + 2, 1.0);
  for (int n = 0; n <= kMaxP; ++n) {
    const double* Hn = h.Hs.data() + length_Hs(n - 1);
    const double* z = h.zeta.data() + length_Ts(n - 1);
    const double* e = h.eta.data() + length_Ts(n - 1);
    for (int a = 0; a <= n; ++a) {
      for (int nu = 0; nu <= n; ++nu) H[lenT(n - 1) + nu * (n + 1) + a] = Hn[H_index(std::min(a, nu), std::max(a, nu))];
      bz[hi(n, a)] = z[a];
      be[hi(n, a)] = e[a];
      az[hi(n, a)] = z[a * (n + 1)];
      ae[hi(n, a)] = e[a * (n + 1)];
    }
  }
  for (size_t k = 1; k < fact.size(); ++k) fact[k] = fact[k - 1] * (double)k;
  auto put = [&](const void* sym, const std::vector<double>& v) {
    FMM_CUDA_TRY(cudaMemcpyToSymbolAsync(sym, v.data(), v.size() * sizeof(double), 0, cudaMemcpyHostToDevice, st));
  };
  put(c_H, H);
  put(d_H, H);
  std::vector<double> mags(az);
  for (const auto* q : {&bz, &ae, &be}) mags.insert(mags.end(), q->begin(), q->end());
  put(d_mag, mags);
  put(c_Az, az);
  put(c_Bz, bz);
  put(c_Ae, ae);
  put(c_Be, be);
  put(c_fact, fact);
  put(c_Mt, std::vector<double>(h.Mt.begin(), h.Mt.begin() + kNh));
  put(c_Lt, std::vector<double>(h.Lt.begin(), h.Lt.begin() + kNh));
  auto put_f = [&](const void* sym, const std::vector<float>& v) {
    FMM_CUDA_TRY(cudaMemcpyToSymbolAsync(sym, v.data(), v.size() * sizeof(float), 0, cudaMemcpyHostToDevice, st));
  };
  std::vector<float> bzf((size_t)kNhF * kColQ * 4, 0.f), bef(bzf);
  std::vector<double> abz(kNhF), abe(kNhF);
  for (int n = 0; n <= kMaxF; ++n)
    for (int a = 0; a <= n; ++a) {
      abz[hi(n, a)] = az[hi(n, a)] / bz[hi(n, a)];
      abe[hi(n, a)] = ae[hi(n, a)] / be[hi(n, a)];
      for (int nu = 0; nu <= n; ++nu) {
        const double h0 = H[lenT(n - 1) + nu * (n + 1) + a];
        const size_t d = (size_t)hi(n, nu) * kColQ * 4 + a;
        bzf[d] = (float)(bz[hi(n, a)] * h0);
        bef[d] = (float)(be[hi(n, a)] * h0);
      }
    }
  put_f(c_BzF, bzf);
  put_f(c_BeF, bef);
  put(c_ABz, abz);
  put(c_ABe, abe);
  put_f(c_factF, std::vector<float>(fact.begin(), fact.begin() + 2 * kMaxF + 2));
  FMM_CUDA_TRY(cudaStreamSynchronize(st));
  if (dev < 64) g_done[dev] = true;
}

// cartesian_to_spherical (src/rotate.jl:9-21) in cos/sin form
struct Geo {
  double cph, sph, cth, sth, r;
};
__device__ __forceinline__ Geo geo_of(double x, double y, double z) {
  Geo g{1.0, 0.0, 1.0, 0.0, 0.0};
  const double x2y2 = x * x + y * y;
  const double r2 = x2y2 + z * z;
  g.r = (r2 == 0.0) ? r2 : sqrt(r2);
  if (x2y2 > 0) {
    const double rho = sqrt(x2y2);
    g.cph = x / rho;
    g.sph = y / rho;
    g.cth = z / g.r;
    g.sth = rho / g.r;
  } else {
    g.cth = (g.r > 0 && z < 0) ? -1.0 : 1.0;
  }
  return g;
}

// rotate_z of degree n of one set of an interleaved expansion, times sc, into padded registers
template <int PMAX, class V>
__device__ __forceinline__ void rotz_in(int n, const double2* __restrict__ e, int set, const Geo& g, double sc,
                                        V (&Xr)[PMAX + 1], V (&Xi)[PMAX + 1]) {
  double er = sc, ei = 0.0;
#pragma unroll
  for (int a = 0; a <= PMAX; ++a) {
    Xr[a] = Xi[a] = V(0);
    if (a > n) continue;
    const double2 u = e[2 * (hi(n, 0) + a) + set];
    Xr[a] = (V)(u.x * er - u.y * ei);
    Xi[a] = (V)(u.x * ei + u.y * er);
    const double t = er;
    er = er * g.cph - ei * g.sph;
    ei = t * g.sph + ei * g.cph;
  }
}

// one FP32 column in registers
template <int PMAX>
__device__ __forceinline__ void column(const float4* __restrict__ q, float (&h)[PMAX + 1]) {
#pragma unroll
  for (int i = 0; i <= PMAX / 4; ++i) {
    const float4 v = q[i];
    const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (4 * i + j <= PMAX) h[(4 * i + j) % (PMAX + 1)] = w[j];
  }
}

// rotate_y of degree n in place (entries past n: zero on entry, undefined on return).  LOCAL: eta
// magnitudes and e^{-+i nu beta}.  Column nu gives E, O, Z of the input, and P_nu +- Q_nu into every
// output (the derivation is in m2l_lane.cu); FP64 applies the magnitudes outside the nu loop, so that
// one table serves both products and both sets; FP32 see its tables.  Sums run to PMAX from one column base, so the
// tables are read at fixed offsets and no term is predicated.
// SH: the tables are sh (H, then A and B of the set, in shared memory), for warps whose lanes are at
// different degrees.
template <int PMAX, bool LOCAL, class V, bool SH = false>
__device__ __forceinline__ void rot_y(int n, V cth, V sth, V (&Xr)[PMAX + 1], V (&Xi)[PMAX + 1],
                                      const double* sh = nullptr, int sh_mag = 0, int sh_nh = 0) {
  constexpr bool F32 = sizeof(V) == 4;
  V Yr[PMAX + 1], Yi[PMAX + 1];
  const int b0 = hi(n, 0);
#pragma unroll
  for (int a = 0; a <= PMAX; ++a) {
    Yr[a] = Yi[a] = V(0);
    if (F32 || a > n) continue;
    const V b = (V)(SH ? sh[sh_mag + sh_nh + b0 + a] : LOCAL ? c_Be[b0 + a] : c_Bz[b0 + a]);
    Xr[a] *= b;
    Xi[a] *= b;
  }
  V c = V(1), s = V(0);  // cos, sin (nu beta) by the reference's recurrence
#pragma unroll 1
  for (int nu = 0; nu <= n; ++nu) {
    if (nu > 0) {
      const V cn = cth * c - sth * s;
      const V sn = sth * c + cth * s;
      c = cn;
      s = sn;
    }
    V h[F32 ? PMAX + 1 : 1];
    if constexpr (F32) column<PMAX>((LOCAL ? c_BeF : c_BzF) + (b0 + nu) * kColQ, h);
    const int col = lenT(n - 1) + nu * (n + 1);
    auto H = [&](int a) -> V {
      if constexpr (F32) return h[a];
      else if constexpr (SH) return sh[col + a];
      else return c_H[col + a];
    };
    V Er = 0, Ei = 0, Or = 0, Oi = 0;
#pragma unroll
    for (int a = 1; a <= PMAX; ++a) {
      if (a & 1) {
        Or += H(a) * Xr[a];
        Oi += H(a) * Xi[a];
      } else {
        Er += H(a) * Xr[a];
        Ei += H(a) * Xi[a];
      }
    }
    const V Zr = H(0) * Xr[0], Zi = H(0) * Xi[0];
    const V w = nu == 0 ? V(0.5) : V(1);  // weight w_nu / 2
    const V sg = ((n + nu) & 1) ? -w : w;
    const V S1r = Er - Or, S1i = Ei - Oi;
    const V S3r = Er + Or, S3i = Ei + Oi;
    const V S2r = Zr + S3r, S2i = -(Zi + S3i);
    const V S4r = Zr + S1r, S4i = -(Zi + S1i);
    const V A1r = w * S1r + sg * S2r, A1i = w * S1i + sg * S2i;
    const V A3r = w * S3r + sg * S4r, A3i = w * S3i + sg * S4i;
    const V ss = LOCAL ? -s : s;
    const V Pr = c * A1r - ss * A1i, Pi = c * A1i + ss * A1r;
    const V Qr = c * A3r + ss * A3i, Qi = c * A3i - ss * A3r;
    const V Rpr = Pr + Qr, Rpi = Pi + Qi, Rmr = Pr - Qr, Rmi = Pi - Qi;
#pragma unroll
    for (int m = 0; m <= PMAX; ++m) {
      Yr[m] += H(m) * ((m & 1) ? Rmr : Rpr);
      Yi[m] += H(m) * ((m & 1) ? Rmi : Rpi);
    }
  }
#pragma unroll
  for (int m = 0; m <= PMAX; ++m) {
    if (m > n) break;
    double a;
    if constexpr (F32) a = LOCAL ? c_ABe[b0 + m] : c_ABz[b0 + m];
    else if constexpr (SH) a = sh[sh_mag + b0 + m];
    else a = LOCAL ? c_Ae[b0 + m] : c_Az[b0 + m];
    Xr[m] = (V)(a * Yr[m]);
    Xi[m] = (V)(a * Yi[m]);
  }
}

// back_rotate_z of degree n in place
template <int PMAX, class V>
__device__ __forceinline__ void rotz_back(int n, V cph, V sph, V (&Yr)[PMAX + 1], V (&Yi)[PMAX + 1]) {
  V er = V(1), ei = V(0);
#pragma unroll
  for (int m = 0; m <= PMAX; ++m) {
    if (m > n) break;
    const V vr = Yr[m] * er + Yi[m] * ei;
    const V vi = Yi[m] * er - Yr[m] * ei;
    Yr[m] = vr;
    Yi[m] = vi;
    const V t = er;
    er = er * cph - ei * sph;
    ei = t * sph + ei * cph;
  }
}

// minimum_distance, src/error.jl:5-20
__device__ __forceinline__ double minabs(double x, double y) {
  return x * (fabs(x) <= fabs(y) ? 1.0 : 0.0) + y * (fabs(y) < fabs(x) ? 1.0 : 0.0);
}
__device__ __forceinline__ double min_dist_1d(double dx, double rm, double rp) {
  const double right = dx + rp, left = dx + rm;
  const double same = (right * left >= 0) ? 1.0 : 0.0;
  return same * minabs(right, left);
}

// algorithmic flops of one pair at order p, one set: 4 * [2 * sum_n (n+1)(2n+1) + sum_n sum_{m<=n} (p-m+1)]
__device__ __forceinline__ unsigned long long pair_flops(int p) {
  const unsigned long long rot = p * (p + 1) * (2 * p + 1) / 3 + 3 * p * (p + 1) / 2 + p + 1;
  const unsigned long long coax = (p + 1) * (p + 2) * (2 * p + 3) / 6;
  return 4ull * (2 * rot + coax);
}

// ---------------------------------------------------------------------------
// M2L.  One CTA of kW warps per target row, 32 pairs at a time (16 with LH: lanes 0-15 carry the
// phi set, lanes 16-31 the chi set of the same pairs); warp w takes the degrees n = w mod kW.
// Before the rotations phi of degree n is scaled by t^-n and chi by t^(1-n), so that the coaxial
// factors are (n+n')! alone, the local sets come out times t^(n+1) and t^(n+2), and the
// Lamb-Helmholtz coupling needs no power of t (m2l_lane.cu).
// Error control (src/translate.jl:555-1412): the reference tests degree after degree and stops at
// the first that passes; here a round rotates the next kW degrees, each warp tests its own, and
// the lowest that passed is taken.  The rotations past it are the price (under kW degrees).
constexpr int kW = 4;

template <int PMAX, bool LH>
__host__ __device__ constexpr int stage_entries() {  // one warp's staging of one plane of a degree (even)
  return LH ? 2 * (PMAX + 1) * 17 : ((PMAX + 1) * 33 + 1) & ~1;
}
// V: FP32 on the mixed path (fixed order up to 12, no error control), else FP64
template <int PMAX, bool LH, class V>
size_t m2l_deg_smem(int p, bool errc) {
  const size_t NH = nh(p);
  return ((LH ? 4 : 2) * NH + (errc ? (p + 1) * 32 : 0) + kW * 32) * sizeof(double) +
         (kW * stage_entries<PMAX, LH>() + 2 * NH * 32) * sizeof(V) + (errc ? kW * 32 * sizeof(int) : 0);
}

// sum_{np <= top} (n + np)! M'(np, m) for m <= mmax, source degrees outer
template <int PMAX, class V>
__device__ __forceinline__ void coax(int n, int mmax, int top, const V* Ms, int lane, V (&Xr)[PMAX + 1],
                                     V (&Xi)[PMAX + 1]) {
#pragma unroll
  for (int m = 0; m <= PMAX; ++m) Xr[m] = Xi[m] = V(0);
#pragma unroll 1
  for (int np = 0; np <= top; ++np) {
    V c;
    if constexpr (sizeof(V) == 4) c = c_factF[n + np];
    else c = c_fact[n + np];
    const V* s = Ms + 2 * hi(np, 0) * 32 + lane;
#pragma unroll
    for (int m = 0; m <= PMAX; ++m) {
      if (m > mmax || m > np) break;
      Xr[m] += c * s[(2 * m) * 32];
      Xi[m] += c * s[(2 * m + 1) * 32];
    }
  }
}

template <int PMAX, bool LH, class V>
__global__ void __launch_bounds__(32 * kW, sizeof(V) == 4 ? 4 : 2)
    k_m2l_deg(const int* __restrict__ tgt_list, const int* __restrict__ off, const int* __restrict__ src_of,
              double* __restrict__ local, const double* __restrict__ multipole, const double* __restrict__ tcen,
              const double* __restrict__ tbox, const double* __restrict__ trad, const double* __restrict__ maxinf,
              const double* __restrict__ scen, int p, int em, double eps_in, int be, int* __restrict__ st_pmax,
              int* __restrict__ st_fail, unsigned long long* __restrict__ st_flops) {
  constexpr int NP = LH ? 16 : 32;  // pairs at a time
  constexpr int SETS = LH ? 2 : 1;
  const int NH = hi(p + 1, 0);
  extern __shared__ double smem_d[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int set = LH ? lane >> 4 : 0, slot = LH ? lane & 15 : lane;
  double* acc = smem_d;                                 // [4 i + 2 set + c] (LH) or [2 i + c]
  double* pw = acc + 2 * SETS * NH;                     // degree powers of the lane's set [p+1][32]
  const bool errc = sizeof(V) == 8 && em != FMM_ERROR_NONE;
  double* tscs = pw + (errc ? (p + 1) * 32 : 0);
  double* tsc = tscs + w * 32;                          // this warp's t^-(n+1) (phi), t^-(n+2) (chi)
  V* stages = reinterpret_cast<V*>(tscs + kW * 32);
  V* stage = stages + w * stage_entries<PMAX, LH>();
  V* Ms = stages + kW * stage_entries<PMAX, LH>();      // [2 i + c][32]
  int* passed = reinterpret_cast<int*>(Ms + 2 * NH * 32);                     // [kW][32]
  const int b = blockIdx.x;
  const int t = tgt_list[b];
  const double tc0 = tcen[3 * t], tc1 = tcen[3 * t + 1], tc2 = tcen[3 * t + 2];
  const bool relative = (em == FMM_POWER_RELATIVE_GRADIENT || em == FMM_ROTATED_COEFFICIENTS_RELATIVE_GRADIENT ||
                         em == FMM_POWER_RELATIVE_POTENTIAL);
  const bool potential = em == FMM_POWER_ABSOLUTE_POTENTIAL || em == FMM_POWER_RELATIVE_POTENTIAL;
  const bool power = potential || em == FMM_POWER_ABSOLUTE_GRADIENT || em == FMM_POWER_RELATIVE_GRADIENT;
  const double thr = (relative ? maxinf[t] * eps_in : eps_in) * 4 * kPi;
  const double r_l = trad[t];
  for (int i = threadIdx.x; i < 2 * SETS * NH; i += 32 * kW) acc[i] = 0.0;
  int pmax = 0;
  bool fail = false;
  unsigned long long fl = 0;
  const int l0 = off[b], l1 = off[b + 1];
  for (int lb = l0; lb < l1; lb += NP) {
    const int l = lb + slot;
    const bool valid = l < l1;
    const double2* src = reinterpret_cast<const double2*>(multipole);
    Geo g{1.0, 0.0, 1.0, 0.0, 1.0};
    double r_mp = 1.0;
    if (valid) {
      const int s = src_of[l];
      src += (int64_t)2 * NH * s;
      const double x = tc0 - scen[3 * s], y = tc1 - scen[3 * s + 1], z = tc2 - scen[3 * s + 2];
      g = geo_of(x, y, z);
      if (errc) {
        const double tb0 = tbox[3 * t], tb1 = tbox[3 * t + 1], tb2 = tbox[3 * t + 2];
        const double mx = min_dist_1d(x, -tb0, tb0), my = min_dist_1d(y, -tb1, tb1), mz = min_dist_1d(z, -tb2, tb2);
        r_mp = sqrt(mx * mx + my * my + mz * mz);
      }
    }
    const double rinv = 1.0 / g.r;
    int P = p;
    bool ok = !errc;
    bool active = valid;
    // forward: this warp's degrees, scaled and rotated, into shared memory
    double sc = set ? g.r : 1.0;  // t^-n, chi t^(1-n)
    // error control at degree nt: r_mp^-(nt+2), 2 nt! (the reference's product), r_l^(nt-1), 1 / (nt-1)!
    const double r_mp_inv = 1.0 / r_mp;
    double mp_pow = r_mp_inv * r_mp_inv * r_mp_inv, np1_fact = 2.0, rl_pow = 1.0, nm1_inv = 1.0;
    int n_sc = 0, nt = 1;
#pragma unroll 1
    for (int n0 = 0; n0 <= p; n0 += kW) {
      if (!__any_sync(kAll, active)) break;  // the same in every warp
      const int n = n0 + w;
      if (n <= p && active) {
        for (; n_sc < n; ++n_sc) sc *= rinv;
        V Xr[PMAX + 1], Xi[PMAX + 1];
        rotz_in<PMAX, V>(n, src, set, g, sc, Xr, Xi);
        if (errc && power) {  // rotate_z_n_power! (src/rotate.jl:528-576), weight 1 for every order
          double a = 0.0;
#pragma unroll
          for (int m = 0; m <= PMAX; ++m) {
            if (m > n) break;
            const double2 u = src[2 * (hi(n, 0) + m) + set];
            const double Nt = c_Mt[hi(n, 0) + m];
            a += (u.x * u.x + u.y * u.y) * Nt * Nt;
          }
          pw[n * 32 + lane] = sqrt(a);
        }
        rot_y<PMAX, false, V>(n, (V)g.cth, (V)g.sth, Xr, Xi);
        V* o = Ms + 2 * hi(n, 0) * 32 + lane;
#pragma unroll
        for (int m = 0; m <= PMAX; ++m) {
          if (m > n) break;
          o[(2 * m) * 32] = Xr[m];
          o[(2 * m + 1) * 32] = Xi[m];
        }
      }
      if (!errc) continue;
      if constexpr (sizeof(V) == 8) {
        __syncthreads();
        bool pass = false;
        if (n >= 1 && n <= p) {  // the same for the whole warp: the exchanges below are uniform
          for (; nt < n; ++nt) {
            mp_pow *= r_mp_inv;
            np1_fact *= nt + 1;
            rl_pow *= r_l;
            nm1_inv /= nt;
          }
          const int in0 = hi(n, 0);
          double e_mp;
          if (power) {
            // phi: power of degree n - 1 (potential variants: n); chi: power of degree n
            const int np = (potential || (LH && set)) ? n : n - 1;
            const double Nn = (LH && set) ? c_Mt[in0] : c_Mt[hi(n - 1, 0)];
            e_mp = 1.7320508075688772 * pw[np * 32 + lane] * mp_pow * np1_fact / Nn;
            if (LH && set) e_mp *= n;
            if (potential) e_mp *= r_mp / (n + 1);
          } else {
            const double* s = Ms + 2 * in0 * 32 + lane;
            double un = 1.0;  // the stored degree is scaled by t^-n (chi t^(1-n))
            for (int k = set; k < n; ++k) un *= g.r;
            const double a1 = s[2 * 32], b1 = s[3 * 32];
            e_mp = un * (sqrt(a1 * a1 + b1 * b1) + ((LH && set) ? 0.0 : fabs(s[0]))) * np1_fact * mp_pow;
            if (LH && set) e_mp *= r_mp;
          }
          if (LH) e_mp += __shfl_xor_sync(kAll, e_mp, 16);
          const bool need = active && e_mp <= thr;
          if (__any_sync(kAll, need)) {
            double tn1 = rinv;  // t^-(n+1)
            for (int k = 0; k < n; ++k) tn1 *= rinv;
            double e_l;
            if (power) {
              // degree n of translate_multipole_to_local_z_n! and local_power (src/translate.jl:238-295, 455-502)
              double vr[PMAX + 1], vi[PMAX + 1];
              coax<PMAX, double>(n, n, n, Ms, lane, vr, vi);
              double a = 0.0;
#pragma unroll
              for (int m = 0; m <= PMAX; ++m) {
                if (m > n) break;
                double pr = vr[m], pi = vi[m];
                if (LH) {
                  const double qr = __shfl_xor_sync(kAll, vr[m], 16), qi = __shfl_xor_sync(kAll, vi[m], 16);
                  if (set == 0) {
                    pr -= qi * m / n;
                    pi += qr * m / n;
                  } else if (m < n) {
                    pr -= vr[(m + 1) % (PMAX + 1)] * g.r / (n + 1);
                    pi -= vi[(m + 1) % (PMAX + 1)] * g.r / (n + 1);
                  }
                }
                const double Nt = c_Lt[in0 + m];
                a += (pr * pr + pi * pi) * Nt * Nt;
              }
              e_l = 1.7320508075688772 * sqrt(a) * tn1 * rl_pow * nm1_inv / c_Lt[in0];
              if (LH && set)
                e_l *= rinv * r_l;
              else if (potential)
                e_l *= r_l / n;
            } else {
              // translate_multipole_to_local_z_m01_n (src/translate.jl:302-364)
              double a0 = 0.0, b1r = 0.0, b1i = 0.0;
              for (int np = 0; np <= n; ++np) {
                const double c = c_fact[n + np];
                const double* s = Ms + 2 * hi(np, 0) * 32 + lane;
                a0 += c * s[0];
                if (np > 0) {
                  b1r += c * s[2 * 32];
                  b1i += c * s[3 * 32];
                }
              }
              if (LH) {
                const double qr = __shfl_xor_sync(kAll, b1r, 16), qi = __shfl_xor_sync(kAll, b1i, 16);
                if (set == 0) {
                  b1r -= qi / n;
                  b1i += qr / n;
                }
              }
              e_l = (LH && set) ? sqrt(b1r * b1r + b1i * b1i) * rinv * r_l : fabs(b1r) + fabs(b1i) + fabs(a0);
              e_l *= tn1 * rl_pow * nm1_inv;
            }
            if (LH) e_l += __shfl_xor_sync(kAll, e_l, 16);
            pass = need && e_mp + e_l * 2.0 <= thr;
          }
        }
        passed[w * 32 + lane] = pass;
        __syncthreads();
        if (active) {
#pragma unroll
          for (int q = kW - 1; q >= 0; --q)
            if (passed[q * 32 + lane]) {
              P = n0 + q - 1 + (be ? 1 : 0);
              ok = true;
              active = false;
            }
        }
      }
    }
    __syncthreads();
    int top = valid ? P : -1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(kAll, top, o));
    // back: this warp's degrees of the local expansion
    double tn1 = rinv;  // t^-(n+1)
    int n_t = 0;
#pragma unroll 1
    for (int n = w; n <= top; n += kW) {
      for (; n_t < n; ++n_t) tn1 *= rinv;
      const bool on = valid && n <= P;
      V Xr[PMAX + 1], Xi[PMAX + 1];
      coax<PMAX, V>(n, n, on ? P : -1, Ms, lane, Xr, Xi);
      if constexpr (LH) {
        // transform_lamb_helmholtz_local! (src/translate.jl:98-142) on the scaled sets
        V Nr[PMAX + 1], Ni[PMAX + 1];
        coax<PMAX, V>(n + 1, n, (on && set && n < P) ? P : -1, Ms, lane, Nr, Ni);
        const V inv_n = n > 0 ? V(1) / (V)n : V(0), inv_n1 = V(1) / (V)(n + 1);
#pragma unroll
        for (int m = 0; m <= PMAX; ++m) {
          if (m > n) break;
          const V qr = __shfl_xor_sync(kAll, Xr[m], 16), qi = __shfl_xor_sync(kAll, Xi[m], 16);
          if (set == 0) {
            const V a = (V)m * inv_n;
            Xr[m] -= a * qi;
            Xi[m] += a * qr;
          } else {
            Xr[m] -= inv_n1 * Nr[m];
            Xi[m] -= inv_n1 * Ni[m];
          }
        }
      }
      rot_y<PMAX, true, V>(n, (V)g.cth, (V)g.sth, Xr, Xi);
      rotz_back<PMAX, V>(n, (V)g.cph, (V)g.sph, Xr, Xi);
      tsc[lane] = set ? tn1 * rinv : tn1;
      // sum over the pairs, value times power of t, one plane (re, im) at a time
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int m = 0; m <= PMAX; ++m) {
          if (m > n) break;
          const V v = c ? Xi[m] : Xr[m];
          stage[LH ? (2 * m + set) * 17 + slot : m * 33 + lane] = on ? v : V(0);
        }
        __syncwarp();
        for (int row = lane; row < SETS * (n + 1); row += 32) {
          const double* ts = tsc + ((LH && (row & 1)) ? 16 : 0);
          const V* sr = stage + row * (LH ? 17 : 33);
          double v = 0.0;
#pragma unroll 8
          for (int k = 0; k < NP; ++k) v += (double)sr[k] * ts[k];
          acc[2 * (SETS * hi(n, 0) + row) + c] += v;
        }
        __syncwarp();
      }
    }
    if (valid && set == 0) {
      pmax = max(pmax, P);
      fail = fail || !ok;
      fl += SETS * pair_flops(P);
    }
    __syncthreads();
  }
  double* dst = local + (int64_t)4 * NH * t;
  for (int i = threadIdx.x; i < 2 * SETS * NH; i += 32 * kW) dst[LH ? i : 4 * (i >> 1) + (i & 1)] += acc[i];
  if (w == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      pmax = max(pmax, __shfl_xor_sync(kAll, pmax, o));
      fl += __shfl_xor_sync(kAll, fl, o);
    }
    const bool any_fail = __any_sync(kAll, fail);
    if (lane == 0) {
      atomicMax(st_pmax, pmax);
      if (any_fail) atomicExch(st_fail, 1);
      atomicAdd(st_flops, fl);
    }
  }
}

// ---------------------------------------------------------------------------
// M2M and L2L (multipole_to_multipole!, src/translate.jl:144-174; local_to_local!,
// :1896-1926).  One CTA per parent: lane bits 0-2 are the child, bit 3 the set with LH, the
// others and the warp the degree, so every (child, set, degree) rotates at the same time; the
// rotated degrees meet in shared memory for the coaxial step.  Also for the orders up to 12 of point
// sources, in place of a lane per child that went through all degrees: 1e6 bodies, order 10, upward
// pass 1.2 -> 0.72 ms, L2L and L2P 1.08 -> 0.82 ms; 2e6 vortex ring, order 12, upward 8.1 -> 3.3 ms.
__host__ __device__ constexpr int mm_degrees(bool lh) { return lh ? 2 : 4; }  // degrees per warp
// rotated degrees, then the tables: H (a column is read to PMAX <= p + 3 entries), A, B
__host__ __device__ inline int mm_tab(int p) { return (lenT(p) + kMaxP + 2) & ~1; }
inline size_t mm_smem(int p, bool lh) {
  return ((size_t)(lh ? 2 : 1) * 2 * nh(p) * 8 + mm_tab(p) + 2 * nh(p)) * sizeof(double);
}

template <int PMAX, bool LH, bool LOCAL>
__global__ void __launch_bounds__(32 * ((PMAX + mm_degrees(LH)) / mm_degrees(LH)))
    k_mm_ll(int k0, const int* __restrict__ child_start, const int* __restrict__ n_children,
            const double* __restrict__ cen, double* __restrict__ E, int p) {
  const int NH = hi(p + 1, 0);
  extern __shared__ double smem_d[];
  const int k = k0 + blockIdx.x;
  const int nc = n_children[k];
  if (nc == 0) return;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = lane & 7, set = LH ? (lane >> 3) & 1 : 0;
  const int n = w * mm_degrees(LH) + (lane >> (LH ? 4 : 3));
  const bool on = j < nc && n <= p;
  const int c = child_start[k] + (j < nc ? j : 0);
  const double sgn = LOCAL ? 1.0 : -1.0;  // source centre to target centre: child to parent, or parent to child
  const Geo g = geo_of(sgn * (cen[3 * c] - cen[3 * k]), sgn * (cen[3 * c + 1] - cen[3 * k + 1]),
                       sgn * (cen[3 * c + 2] - cen[3 * k + 2]));
  const double2* src = reinterpret_cast<const double2*>(E) + (int64_t)2 * NH * (LOCAL ? k : c);
  double* Ms = smem_d + (size_t)set * 2 * NH * 8;  // the set's rotated degrees [2 i + c][8]
  // the lanes of a warp are at different degrees, whose columns the constant cache serves one after
  // the other: 150k bodies, order 16, upward pass 0.51 -> 0.42 ms, downward 0.41 -> 0.34 ms
  double* tab = smem_d + (size_t)(LH ? 2 : 1) * 2 * NH * 8;
  const int mag = mm_tab(p);
  for (int i = threadIdx.x; i < mag; i += blockDim.x) tab[i] = i < lenT(p) ? d_H[i] : 0.0;
  for (int i = threadIdx.x; i < NH; i += blockDim.x) {
    tab[mag + i] = d_mag[LOCAL ? 2 : 0][i];
    tab[mag + NH + i] = d_mag[LOCAL ? 3 : 1][i];
  }
  double Xr[PMAX + 1], Xi[PMAX + 1];
  if (on) rotz_in<PMAX, double>(n, src, set, g, 1.0, Xr, Xi);
  __syncthreads();
  if (on) {
    rot_y<PMAX, LOCAL, double, true>(n, g.cth, g.sth, Xr, Xi, tab, mag, NH);
#pragma unroll
    for (int m = 0; m <= PMAX; ++m) {
      if (m > n) break;
      Ms[(2 * (hi(n, 0) + m)) * 8 + j] = Xr[m];
      Ms[(2 * (hi(n, 0) + m) + 1) * 8 + j] = Xi[m];
    }
  }
  __syncthreads();
  // degree d of translate_multipole_z! (src/translate.jl:6-50): sum_{n'<=d} (-t)^(d-n') / (d-n')! M(n', m),
  // or of translate_local_z! (:1851-1891): sum_{n'>=d} (-t)^(n'-d) / (n'-d)! L(n', m); orders m <= mmax
  auto axis = [&](int d, int mmax, double (&Vr)[PMAX + 1], double (&Vi)[PMAX + 1]) {
#pragma unroll
    for (int m = 0; m <= PMAX; ++m) Vr[m] = Vi[m] = 0.0;
    double tp = 1.0;
#pragma unroll 1
    for (int s = 0; s <= (LOCAL ? p - d : d); ++s) {
      const int np = LOCAL ? d + s : d - s;
      const double cc = tp * c_ifact[s];
      const double* q = Ms + 2 * hi(np, 0) * 8 + j;
#pragma unroll
      for (int m = 0; m <= PMAX; ++m) {
        if (m > mmax || m > np) break;
        Vr[m] += cc * q[(2 * m) * 8];
        Vi[m] += cc * q[(2 * m + 1) * 8];
      }
      tp *= -g.r;
    }
  };
  if (on) {
    axis(n, n, Xr, Xi);
  } else {
#pragma unroll
    for (int m = 0; m <= PMAX; ++m) Xr[m] = Xi[m] = 0.0;
  }
  if constexpr (LH) {
    // transform_lamb_helmholtz_multipole! / _local! (src/translate.jl:52-142): phi takes chi of the same
    // degree, chi takes chi of the degree below (multipole) or above (local)
    double Nr[PMAX + 1], Ni[PMAX + 1];
    const int dn = LOCAL ? n + 1 : n - 1;
    if (on && set && dn >= 0 && dn <= p) {
      axis(dn, n, Nr, Ni);
    } else {
#pragma unroll
      for (int m = 0; m <= PMAX; ++m) Nr[m] = Ni[m] = 0.0;
    }
    const double fp = LOCAL ? (n > 0 ? -g.r / n : 0.0) : g.r / (n + 1);      // times m: chi into phi
    const double fc = LOCAL ? -g.r / (n + 1) : (n > 0 ? g.r / n : 0.0);      // neighbour degree into chi
#pragma unroll
    for (int m = 0; m <= PMAX; ++m) {
      const double qr = __shfl_xor_sync(kAll, Xr[m], 8), qi = __shfl_xor_sync(kAll, Xi[m], 8);
      if (set == 0) {
        Xr[m] += fp * m * qi;
        Xi[m] -= fp * m * qr;
      } else {
        Xr[m] += fc * Nr[m];
        Xi[m] += fc * Ni[m];
      }
      if (m > n) Xr[m] = Xi[m] = 0.0;
    }
  }
  if (on) {
    rot_y<PMAX, LOCAL, double, true>(n, g.cth, g.sth, Xr, Xi, tab, mag, NH);
    rotz_back<PMAX, double>(n, g.cph, g.sph, Xr, Xi);
  }
  double2* dst = reinterpret_cast<double2*>(E) + (int64_t)2 * NH * (LOCAL ? c : k);
  if constexpr (LOCAL) {
    if (on) {
#pragma unroll
      for (int m = 0; m <= PMAX; ++m) {
        if (m > n) break;
        double2 v = dst[2 * (hi(n, 0) + m) + set];
        v.x += Xr[m];
        v.y += Xi[m];
        dst[2 * (hi(n, 0) + m) + set] = v;
      }
    }
  } else {
    // sum over the children; the group's first lane owns the parent's entry
    __syncwarp();
    const int nmax = min(p, (w + 1) * mm_degrees(LH) - 1);
#pragma unroll
    for (int m = 0; m <= PMAX; ++m) {
      if (m > nmax) break;
      double vr = on ? Xr[m] : 0.0, vi = on ? Xi[m] : 0.0;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        vr += __shfl_xor_sync(kAll, vr, o);
        vi += __shfl_xor_sync(kAll, vi, o);
      }
      if (j == 0 && on && m <= n) {
        double2 v = dst[2 * (hi(n, 0) + m) + set];
        v.x += vr;
        v.y += vi;
        dst[2 * (hi(n, 0) + m) + set] = v;
      }
    }
  }
}

// call f.template go<PMAX>() for the smallest instantiated order >= p
template <class F>
void dispatch_pmax(int p, F&& f) {
  if (p <= 4)
    f.template go<4>();
  else if (p <= 6)
    f.template go<6>();
  else if (p <= 8)
    f.template go<8>();
  else if (p <= 10)
    f.template go<10>();
  else if (p <= 12)
    f.template go<12>();
  else if (p <= 16)
    f.template go<16>();
  else
    f.template go<kMaxP>();
}

template <class K>
void allow_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024)
    FMM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

template <bool LH, class V>
struct M2LDegGo {
  DevTree& t;
  const DevTree& s;
  const DevLists& L;
  int p, em, be;
  double eps;
  int* stats;
  cudaStream_t st;
  template <int PMAX>
  void go() {
    if constexpr (sizeof(V) == 8 || PMAX <= kMaxF) {
      const size_t sm = m2l_deg_smem<PMAX, LH, V>(p, em != FMM_ERROR_NONE);
      allow_smem(k_m2l_deg<PMAX, LH, V>, sm);
      note_launch();
      k_m2l_deg<PMAX, LH, V><<<(int)L.n_m2l_targets, 32 * kW, sm, st>>>(
          L.m2l_tgt.ptr, L.m2l_off.ptr, L.m2l_s.ptr, t.local.ptr, s.multipole.ptr, t.tcenter.ptr, t.tbox.ptr,
          t.tradius.ptr, t.max_influence.ptr, s.scenter.ptr, p, em, eps, be, stats, stats + 1,
          reinterpret_cast<unsigned long long*>(stats + 2));
      FMM_CUDA_TRY(cudaGetLastError());
    }
  }
};

template <bool LH, bool LOCAL>
struct MMLLGo {
  const DevTree& t;
  const double* cen;
  double* E;
  int p;
  cudaStream_t st;
  template <int PMAX>
  void go() {
    const size_t sm = mm_smem(p, LH);
    allow_smem(k_mm_ll<PMAX, LH, LOCAL>, sm);
    const int threads = 32 * ((p + mm_degrees(LH)) / mm_degrees(LH));
    for (int i = 0; i + 1 < t.n_levels; ++i) {
      const int l = LOCAL ? i : t.n_levels - 2 - i;
      const int k0 = (int)t.levels_start[l], k1 = (int)t.levels_end[l];
      note_launch();
      k_mm_ll<PMAX, LH, LOCAL><<<k1 - k0, threads, sm, st>>>(k0, t.child_start.ptr, t.n_children.ptr, cen, E, p);
    }
    FMM_CUDA_TRY(cudaGetLastError());
  }
};

}  // namespace

void launch_m2l_deg(DevTree& t, const DevTree& s, const DevLists& L, int p, bool lh, int em, double eps, int be,
                    int* stats, int precision, cudaStream_t st) {
  if (L.n_m2l_targets == 0) return;
  ensure_tables(st);
  // FP32 on the mixed path where the pairs' orders are fixed and its tables reach
  const bool f32 = precision == FMM_PRECISION_MIXED && em == FMM_ERROR_NONE && p <= kMaxF;
  if (lh && f32)
    dispatch_pmax(p, M2LDegGo<true, float>{t, s, L, p, em, be, eps, stats, st});
  else if (f32)
    dispatch_pmax(p, M2LDegGo<false, float>{t, s, L, p, em, be, eps, stats, st});
  else if (lh)
    dispatch_pmax(p, M2LDegGo<true, double>{t, s, L, p, em, be, eps, stats, st});
  else
    dispatch_pmax(p, M2LDegGo<false, double>{t, s, L, p, em, be, eps, stats, st});
}

void launch_m2m(DevTree& s, int p, bool lh, cudaStream_t st) {
  if (s.n_levels < 2) return;
  ensure_tables(st);
  if (lh)
    dispatch_pmax(p, MMLLGo<true, false>{s, s.scenter.ptr, s.multipole.ptr, p, st});
  else
    dispatch_pmax(p, MMLLGo<false, false>{s, s.scenter.ptr, s.multipole.ptr, p, st});
}

void launch_l2l(DevTree& t, int p, bool lh, cudaStream_t st) {
  if (t.n_levels < 2) return;
  ensure_tables(st);
  if (lh)
    dispatch_pmax(p, MMLLGo<true, true>{t, t.tcenter.ptr, t.local.ptr, p, st});
  else
    dispatch_pmax(p, MMLLGo<false, true>{t, t.tcenter.ptr, t.local.ptr, p, st});
}

}  // namespace fmmb
