// scgd0.cu -- the scGD0 plan: setup (src/scgd0.jl:127-245) and the iteration (src/scgd0.jl:246-346)
// on one GPU.
//
// HBM layout of a plan (column-major, reference index order):
//   Σ, Σ_new       [nω, ni, nT] double2        Σ_in [nω, ni] double2 (clamped, one T at a time)
//   ImΣ, ReΣ       [nω, ni] double             KK [nω, nω] double
//   DIRECT_FP64 :  g2_t, ωq_t [nm·nf, ni] double (the (ν f, i) layout of src/scgd0.jl:275-278)
//   GEMM paths  :  G [nc·nm, ni] coupling summed over each column set (a star, or one inner state)
//                  K_t [nω, nc·nm] the kernel tensor of one iteration and temperature
//   spectral    :  A [nωa, ni] double, D [nωa], column sums [ni]
#include "common.cuh"
#include "fp_pair.cuh"
#include "g2stream.cuh"
#include "scgd0.cuh"
#include "warmstart.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <array>
#include <chrono>
#include <limits>

namespace epsp {

// ---------------------------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------------------------

// kramers_kronig_matrix (src/frequency_grids.jl:5-44) on the padded nodes xs[0..n+1].
__device__ __forceinline__ double xlogx_d(double x) { return x == 0 ? 0.0 : x * log(fabs(x)); }

__global__ void kk_build_kernel(const double* __restrict__ xs, int n, double* __restrict__ K) {
  long idx = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= long(n) * n) return;
  int i = int(idx % n), j = int(idx / n);
  double x = xs[i + 1], x1 = xs[j], x2 = xs[j + 1], x3 = xs[j + 2];
  double v = xlogx_d(x1 - x) / (x2 - x1) - xlogx_d(x2 - x) * (x3 - x1) / (x2 - x1) / (x3 - x2) + xlogx_d(x3 - x) / (x3 - x2);
  K[idx] = v / 3.14159265358979323846;
}

void kk_matrix_to_device(Ctx* ctx, const std::vector<double>& w, DBuf<double>& K) {
  const long n = long(w.size());
  if (n < 2) fail(EPSP_EINVAL, "the Kramers-Kronig matrix needs at least two nodes");
  std::vector<double> xs(size_t(n + 2));
  xs[0] = w[0] - (w[1] - w[0]);
  for (long j = 0; j < n; ++j) xs[size_t(j + 1)] = w[size_t(j)];
  xs[size_t(n + 1)] = w[size_t(n - 1)] + (w[size_t(n - 1)] - w[size_t(n - 2)]);
  auto d_xs = to_device(ctx, xs);
  K.alloc(ctx, size_t(n * n));
  kk_build_kernel<<<div_up(size_t(n * n), 256), 256, 0, ctx->stream>>>(d_xs.p, int(n), K.p);
  EPSP_LAUNCHED(ctx);
  EPSP_CUDA(cudaStreamSynchronize(ctx->stream));
}

// g2 [nm, ni, nf] (any storage type) -> g2_t [nm, nf, ni] double (src/scgd0.jl:275-278), and
// ωq_t[ν, f, i] = ωph[ν, iq_kk[iks_i[i], iks_f[f]]] (gather_pair_table!, src/scgd0.jl:270).

template <class T>
__global__ void permute_g2_kernel(const T* __restrict__ g2, int nm, int ni, long nf, long f0, long nfc,
                                  double* __restrict__ g2t) {
  long idx = long(blockIdx.x) * blockDim.x + threadIdx.x;
  long total = long(nm) * nfc * ni;
  if (idx >= total) return;
  int nu = int(idx % nm);
  long f = (idx / nm) % nfc;
  int i = int(idx / (long(nm) * nfc));
  g2t[nu + nm * (f + nf * long(i))] = load_g2(g2, nu + nm * (long(i) + ni * (f0 + f)));
  (void)f0;
}

__global__ void gather_wq_kernel(const double* __restrict__ wph, const int32_t* __restrict__ iq_kk,
                                 const int32_t* __restrict__ iks_i, const int32_t* __restrict__ iks_f, int nm, int ni,
                                 long nf, long nk_i, double* __restrict__ wqt) {
  long idx = long(blockIdx.x) * blockDim.x + threadIdx.x;
  long total = long(nm) * nf * ni;
  if (idx >= total) return;
  int nu = int(idx % nm);
  long f = (idx / nm) % nf;
  int i = int(idx / (long(nm) * nf));
  long q = iq_kk[iks_i[i] + nk_i * long(iks_f[f])];
  wqt[idx] = wph[nu + long(nm) * q];
}

// Σ = Σ_new = -i η_init everywhere (the start without Σ_init, src/scgd0.jl:226).
__global__ void fill_start_kernel(double2* __restrict__ S, double2* __restrict__ Snew, long n, double eta_init) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n) return;
  S[k] = Snew[k] = make_double2(0.0, -eta_init);
}

// Σ_in = Re Σ + i min(Im Σ, -η_min) (src/scgd0.jl:256-260), for the active temperatures: slot a
// (blockIdx.y) reads Σ of temperature slots[a] and writes Sin + a n.
__global__ void clamp_kernel(const double2* __restrict__ S, double2* __restrict__ Sin, long n,
                             const int* __restrict__ slots, const TParams* __restrict__ tp,
                             unsigned long long* __restrict__ errbits_all) {
  pdl_wait();
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int a = blockIdx.y, t = slots[a];
  if (k == 0) errbits_all[t] = 0;  // the iteration's max |ΔΣ| starts at 0
  double2 z = S[long(t) * n + k];
  Sin[long(a) * n + k] = make_double2(z.x, fmin(z.y, -tp[t].eta_min));
}

// The reference's Fan-Migdal sum, term by term in FP64: for each (ω, i), the sum over νf of
// _fan_migdal_imsigma_term (src/scgd0_kernel.jl:27-39) in ascending νf, added to ImΣ
// (src/scgd0_kernel.jl:74-86). One thread per (ω, i); the block's νf tile (g2, ωq, n_B(ωq) and the
// per-state ε, w, i_f) is staged in shared memory. n_B is evaluated once per (νf, i), the same
// function on the same argument as the reference's per-term call.
constexpr int kFmTile = 128;

__global__ void __launch_bounds__(kFmTile) fm_direct_kernel(
    const double* __restrict__ ws, int nw, CellTableDev ct, const double2* __restrict__ Sin,
    const double* __restrict__ g2t, const double* __restrict__ wqt, long nvf, const double* __restrict__ eps_f,
    const double* __restrict__ w_f, const int32_t* __restrict__ f_to_i, int nm, long vf0, long vf1, double mu,
    double T, double w_ac, double* __restrict__ imsigma) {
  __shared__ double s_g2[kFmTile], s_wq[kFmTile], s_nq[kFmTile], s_eps[kFmTile], s_wf[kFmTile];
  __shared__ int s_col[kFmTile];
  const int i = blockIdx.y;
  const int iw = blockIdx.x * kFmTile + threadIdx.x;
  const double w = iw < nw ? ws[iw] : 0.0;
  double acc = 0.0;
  for (long t0 = vf0; t0 < vf1; t0 += kFmTile) {
    long vf = t0 + threadIdx.x;
    if (vf < vf1) {
      double wq = wqt[vf + nvf * i];
      long f = vf / nm;
      s_g2[threadIdx.x] = g2t[vf + nvf * i];
      s_wq[threadIdx.x] = wq;
      s_nq[threadIdx.x] = wq < w_ac ? 0.0 : occ_boson_d(wq, T);
      s_eps[threadIdx.x] = eps_f[f];
      s_wf[threadIdx.x] = w_f[f];
      s_col[threadIdx.x] = f_to_i[f];
    }
    __syncthreads();
    int nt = int(min(long(kFmTile), vf1 - t0));
    if (iw < nw) {
      for (int k = 0; k < nt; ++k) {
        double wq = s_wq[k];
        if (wq < w_ac) continue;
        const double2* col = Sin + long(nw) * s_col[k];
        double xa = w + wq, xe = w - wq;
        double2 sa = interp_grid_d(col, ct, xa);
        double2 se = interp_grid_d(col, ct, xe);
        double zar = xa - s_eps[k] - sa.x, zai = -sa.y;
        double zer = xe - s_eps[k] - se.x, zei = -se.y;
        double ga = -zai / (zar * zar + zai * zai);
        double ge = -zei / (zer * zer + zei * zei);
        double nq = s_nq[k];
        acc += s_wf[k] * s_g2[k] * (ga * (nq + occ_fermion_d(xa - mu, T)) + ge * (nq + 1 - occ_fermion_d(xe - mu, T)));
      }
    }
    __syncthreads();
  }
  if (iw < nw) imsigma[iw + long(nw) * i] += acc;
}

// The same sum with the FP64 operations of a term cut from about 160 to 27: FP64 instructions issue at
// 1/64 of the FP32 and integer rate here and bound the kernel (the term-by-term kernel above ran at that
// limit, on 30 of 152 SMs at 126 nodes and 30 states).
//  * Interpolation: Σ(x) = Σ_j + (x - ω_j) Σ'_j from a table per column, 4 doubles per cell: ω_j - ReΣ_j,
//    ImΣ_j, 1 - ReΣ'_j, ImΣ'_j (fm_cell_kernel), so that Re z = (U_j - ε) + (x - ω_j) E_j and Im Σ cost one
//    operation each beside x - ω_j; the flat continuation is an entry before and after the grid. The
//    cell is found without FP64: an FP32 bucket, lowered by a guard above its error, then two comparisons
//    on the values' ordered integers.
//  * Occupations: with E = exp((ω - μ)/T), e = exp(ωq/T): n + f(x_a - μ) = (1 + n)(1 + E)/(1 + E e) and
//    n + 1 - f(x_e - μ) = n (1 + E)/(1 + E/e) (detailed balance; no difference is taken), so a term
//    needs no exponential, and 1 + E leaves the sum. For E > 1 both sides are divided by E (p + q e with
//    (p, q) = (1/E, 1) in place of (1, E)). E and e carry the rounding of their arguments as a factor.
//  * One reciprocal per term: N_a/D_a + N_e/D_e = (N_a D_e + N_e D_a)/(D_a D_e), from an FP32 seed of the
//    mantissa (the exponent by integers) and one third-order Newton step (2^-23 -> 2^-69). A denominator that is
//    0, not finite or subnormal takes the plain formula.
// The sum over (ν, f) is split over blockIdx.z (partials summed in order by fm_add_kernel) until the SMs
// have work. Needs T > 0 with ωq/T <= 300 (e^300 squared times the denominators stays in range),
// ω_acoustic > 0 and a guard below half a bucket; other calls run the kernel above.
// Measured (126 nodes, 30 states, 5 modes x 375 inner states; and 401, 33, 1 x 64): 9.88 -> 0.433 ms,
// 0.355 -> 0.074 ms: about 36 operations' time a term with the staging, of the 27 it issues.
struct FmPair {
  double g1, g0, e, ie, wq, eps;  // w_f g2 (1 + n), w_f g2 n, exp(±ωq/T), ωq, ε
};

// Cell table of every column: entry j + 1 holds cell j, entry 0 the flat part below the grid.
__global__ void fm_cell_kernel(const double* __restrict__ ws, int nw, const double2* __restrict__ Sin, long ncol,
                               double4* __restrict__ tab) {
  pdl_wait();
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= (nw + 1l) * ncol) return;
  const int j = int(k % (nw + 1)) - 1;
  const double2* col = Sin + long(nw) * (k / (nw + 1));
  const int b = max(j, 0);
  const double2 lo = col[b];
  double4 o;
  o.x = ws[b] - lo.x;
  o.y = lo.y;
  o.z = 1.0;
  o.w = 0.0;
  if (j >= 0 && j < nw - 1) {
    const double inv = 1.0 / (ws[j + 1] - ws[j]);
    o.z = 1.0 - (col[j + 1].x - lo.x) * inv;
    o.w = (col[j + 1].y - lo.y) * inv;
  }
  tab[k] = o;
}

// A double as an integer of the same order.
__host__ __device__ __forceinline__ long long ordered(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffll); }

__device__ __forceinline__ double recip_seeded(double d) {
  const int hi = __double2hiint(d), lo = __double2loint(d);
  const float m = __uint_as_float(0x3f800000u | ((uint32_t(hi) & 0xfffffu) << 3) | (uint32_t(lo) >> 29));
  float s;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(m));  // in (1/2, 1]
  const uint32_t b = __float_as_uint(s);
  const int ex = int(b >> 23) + (1023 - 127) - (((hi >> 20) & 0x7ff) - 1023);
  const double r = __hiloint2double(int((uint32_t(ex) << 20) | ((b >> 3) & 0xfffffu)), int(b << 29));
  const double h = fma(-d, r, 1.0);
  return fma(r, fma(h, h, h), r);
}

constexpr int kFmFastTile = 128;  // staged (ν, f) pairs

__global__ void __launch_bounds__(512) fm_direct_fast_kernel(
    const double* __restrict__ ws, int nw, const long long* __restrict__ wkey, const int32_t* __restrict__ jtab, int ntab,
    float x0f, float inv_hf, float guard, const double4* __restrict__ tab, const double* __restrict__ g2t,
    const double* __restrict__ wqt, long nvf, const double* __restrict__ eps_f, const double* __restrict__ w_f,
    const int32_t* __restrict__ f_to_i, int nm, long vf0, long vf1, long per, double mu, double T, double invT, double w_ac,
    double* __restrict__ part) {
  pdl_wait();
  __shared__ FmPair sp[kFmFastTile];
  __shared__ int s_col[kFmFastTile];
  const int i = blockIdx.y;
  const int iw = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = iw < nw;
  const double w = in ? ws[iw] : ws[0];
  const float wf = float(w);
  const bool below = w <= mu;
  const double dv = below ? w - mu : mu - w;
  // exp(v / T) with the rounding of v / T put back as a factor
  const double av = dv * invT, E0 = exp(av), Ew = fma(E0, fma(-av, T, dv) * invT, E0);  // E, or 1/E above μ
  const double p = below ? 1.0 : Ew, q = below ? Ew : 1.0;
  const long t_end = min(vf1, vf0 + per * (long(blockIdx.z) + 1));
  double acc = 0.0;
  for (long t0 = vf0 + per * long(blockIdx.z); t0 < t_end; t0 += kFmFastTile) {
    const int nt = int(min(long(kFmFastTile), t_end - t0));
    __syncthreads();
    for (int k = threadIdx.x; k < nt; k += blockDim.x) {
      const long vf = t0 + k, f = vf / nm;
      const double wq = wqt[vf + nvf * i];
      s_col[k] = wq < w_ac ? -1 : f_to_i[f];
      if (!(wq < w_ac)) {
        const double g = w_f[f] * g2t[vf + nvf * i];
        const double a = wq * invT, m0 = expm1(a), m = fma(m0 + 1.0, fma(-a, T, wq) * invT, m0);  // exp(ωq/T) - 1
        const double e = m + 1.0, nq = recip_seeded(m);
        sp[k] = FmPair{g * (nq + 1.0), g * nq, e, recip_seeded(e), wq, eps_f[f]};
      }
    }
    __syncthreads();
    if (!in) continue;
    // the cell of x (as cell + 1: the table's entry) and x - ω_cell
    auto cell = [&](double x, float xf, int& e) -> double {
      const float v = fminf(fmaxf((xf - x0f) * inv_hf - guard, 0.f), float(ntab - 1));
      const int c = jtab[int(v)];
      const long long kx = ordered(__double_as_longlong(x));
      e = c + (kx >= wkey[c] ? 1 : 0) + (kx >= wkey[c + 1] ? 1 : 0);
      return x - ws[max(e - 1, 0)];
    };
#pragma unroll 2
    for (int k = 0; k < nt; ++k) {
      if (s_col[k] < 0) continue;
      const FmPair P = sp[k];
      const double4* col = tab + (nw + 1l) * s_col[k];
      const float wqf = float(P.wq);
      int ea, ee;
      const double da = cell(w + P.wq, wf + wqf, ea), de = cell(w - P.wq, wf - wqf, ee);
      const double4 A = col[ea], B = col[ee];
      const double zar = fma(da, A.z, A.x - P.eps), sia = fma(da, A.w, A.y);
      const double zer = fma(de, B.z, B.x - P.eps), sie = fma(de, B.w, B.y);
      const double dna = fma(zar, zar, sia * sia), dne = fma(zer, zer, sie * sie);
      const double oa = fma(q, P.e, p), oe = fma(q, P.ie, p);
      const double Da = dna * oa, De = dne * oe;
      const double Na = P.g1 * sia, Ne = P.g0 * sie;
      const double D = Da * De;
      const int E = (__double2hiint(D) >> 20) & 0x7ff;
      if (E > 0 && E < 0x7f0)
        acc = fma(fma(Na, De, Ne * Da), recip_seeded(D), acc);
      else
        acc += Na / dna / oa + Ne / dne / oe;
    }
  }
  if (in) part[iw + long(nw) * (i + long(gridDim.y) * blockIdx.z)] = acc * (p + q);
}

// ImΣ += Σ_s part[s]: 32 elements a block, eight runs of splits side by side, each in ascending s, added in order.
__global__ void __launch_bounds__(256) fm_add_kernel(const double* __restrict__ part, long n, int splits,
                                                     double* __restrict__ imsigma, bool set) {
  pdl_wait();
  __shared__ double sh[8][32];
  const int lane = threadIdx.x % 32, g = threadIdx.x / 32;
  const long k = long(blockIdx.x) * 32 + lane;
  const int per = (splits + 7) / 8;
  double v = 0.0;
  if (k < n)
#pragma unroll 4
    for (int s = g * per; s < min(splits, (g + 1) * per); ++s) v += part[k + n * s];
  sh[g][lane] = v;
  __syncthreads();
  if (g == 0 && k < n) {
#pragma unroll
    for (int r = 1; r < 8; ++r) v += sh[r][lane];
    imsigma[k] = set ? v : imsigma[k] + v;
  }
}

// The occupation factors of the recast sum, per (ω, ν): F_abs = n_ν + f(ω + ω_ν - μ) and
// F_emi = n_ν + 1 - f(ω - ω_ν - μ) (the two brackets of src/scgd0_kernel.jl:37-38); 0 for a mode
// below ω_acoustic. Blocks of 32, so that every SM's FP64 pipe has some (501 x 15: 9.8 us in blocks of 256, 6.2).
__global__ void occ_table_kernel(const double* __restrict__ ws, int nw, const double* __restrict__ wnu, int nm,
                                 double mu, double T, double w_ac, double* __restrict__ Fa, double* __restrict__ Fe) {
  pdl_wait();
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nw * nm) return;
  int iw = k % nw, nu = k / nw;
  double q = wnu[nu], w = ws[iw];
  if (q < w_ac) {
    Fa[k] = 0;
    Fe[k] = 0;
    return;
  }
  double nq = occ_boson_d(q, T);
  Fa[k] = nq + occ_fermion_d(w + q - mu, T);
  Fe[k] = nq + 1 - occ_fermion_d(w - q - mu, T);
}

// The kernel tensor of the recast sum (dispersionless modes): K_t[ω, (ν, c)] =
// Im G_c(ω + ω_ν) F_abs[ω, ν] + Im G_c(ω - ω_ν) F_emi[ω, ν], with Im G_c(x) = Im 1/(x - ε_c -
// Σ_in,col(c)(x)), for the column set c (a star of inner states sharing ε and the representative's
// Σ, or one inner state). Σ(x) from the columns' cell table (fm_cell_kernel) at the cells of ω ± ω_ν found at set-up
// (cell_e: the table's entry, cell_dx: x less its node), and one reciprocal for both sides: 20 FP64 operations an
// element, which bound the kernel, in place of about 90 with the search, two weights and two divisions
// (501 nodes x 1575: 130 -> 32 us).
__global__ void kbuild_f64_kernel(int nw, const double4* __restrict__ tab, const int32_t* __restrict__ cell_e,
                                  const double* __restrict__ cell_dx, const double* __restrict__ wnu, int nm,
                                  const double* __restrict__ eps_c, const int32_t* __restrict__ col_c,
                                  const double* __restrict__ Fa, const double* __restrict__ Fe, double w_ac,
                                  double* __restrict__ Kt) {
  pdl_wait();
  const int iw = blockIdx.x * blockDim.x + threadIdx.x;
  const long kc = blockIdx.y;  // (ν, c) with ν fastest
  if (iw >= nw) return;
  const int nu = int(kc % nm);
  const long c = kc / nm;
  double out = 0.0;
  if (!(wnu[nu] < w_ac)) {
    const double4* col = tab + (nw + 1l) * col_c[c];
    const long ka = iw + long(nw) * nu, ke = ka + long(nw) * nm;
    const double4 A = col[cell_e[ka]], B = col[cell_e[ke]];
    const double da = cell_dx[ka], de = cell_dx[ke], e = eps_c[c];
    const double zar = fma(da, A.z, A.x - e), sia = fma(da, A.w, A.y);
    const double zer = fma(de, B.z, B.x - e), sie = fma(de, B.w, B.y);
    const double dna = fma(zar, zar, sia * sia), dne = fma(zer, zer, sie * sie);
    const double Na = sia * Fa[ka], Ne = sie * Fe[ka];
    const double D = dna * dne;
    const int E = (__double2hiint(D) >> 20) & 0x7ff;
    out = E > 0 && E < 0x7f0 ? fma(Na, dne, Ne * dna) * recip_seeded(D) : Na / dna + Ne / dne;
  }
  Kt[iw + long(nw) * kc] = out;
}

// G[(ν, c), i] = Σ_{f in c} w_f g2[ν, i, f] over the inner states of column set c in star order,
// for the column sets [c0, c1) of one streamed chunk: g2c [nm, ni, p - p0] holds their members p.
// Rows of modes below ω_acoustic are 0 (they are skipped before g2 is read in the reference).
// Thread (ν, i) of column sets c0 + blockIdx.y, c0 + blockIdx.y + gridDim.y, ...: each set's sum is
// its own, so the sets run side by side.
template <class T>
__global__ void coupling_sum_chunk_kernel(const T* __restrict__ g2c, int nm, int ni, const int32_t* __restrict__ cptr,
                                          long c0, long c1, long p0, const int32_t* __restrict__ members, long nc,
                                          const double* __restrict__ w_f, const double* __restrict__ wnu, double w_ac,
                                          double* __restrict__ G) {
  const long idx = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= long(nm) * ni) return;
  const int nu = int(idx % nm), i = int(idx / nm);
  const bool skip = wnu[nu] < w_ac;
  for (long c = c0 + blockIdx.y; c < c1; c += gridDim.y) {
    double s = 0.0;
    if (!skip)
      for (int p = cptr[c]; p < cptr[c + 1]; ++p) {
        const long f = members[p];
        s += w_f[f] * load_g2(g2c, nu + long(nm) * (i + long(ni) * (p - p0)));
      }
    G[(nu + nm * c) + long(nm) * nc * i] = s;
  }
}

// max of |a - S[k]| over the block's elements into *errbits, and S[k] ← a (src/scgd0.jl:326-328). The maximum of
// non-negative doubles is taken on their bit patterns, which order the same way; NaN wins, as in Julia's maximum. It is
// taken of the squares, and one root a block: a hypot an element, which a block falls back to where a square leaves the
// middle of the range, was most of the kernel's time on the FP64 pipe (501 x 105: 6.0 -> 4.8 us).
__device__ __forceinline__ void err_copy(double2 a, bool on, double2* S, unsigned long long* errbits) {
  __shared__ unsigned long long sh[256];
  double x = 0, y = 0;
  if (on) {
    const double2 b = *S;
    x = a.x - b.x;
    y = a.y - b.y;
    *S = a;
  }
  double q = fma(x, x, y * y);
  const int ex = (__double2hiint(q) >> 20) & 0x7ff;
  const bool far = __syncthreads_or((ex < 0x100 || ex > 0x700) && (x != 0 || y != 0));
  if (far) q = hypot(x, y);
  sh[threadIdx.x] = (unsigned long long)__double_as_longlong(q);
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] = max(sh[threadIdx.x], sh[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double m = __longlong_as_double((long long)sh[0]);
    atomicMax(errbits, (unsigned long long)__double_as_longlong(far ? m : sqrt(m)));
  }
}

// Σ_new = re + i im (src/scgd0.jl:290-291) of one temperature; with S, which then is its Σ, also max |Σ_new - Σ| and Σ ← Σ_new. Hands the
// products' error flag on to the host's copy. 256 threads.
__global__ void __launch_bounds__(256) assemble_kernel(const double* __restrict__ re, const double* __restrict__ im,
                                                       double2* __restrict__ out, long n, double2* __restrict__ S,
                                                       unsigned long long* __restrict__ errbits,
                                                       const int* __restrict__ tcerr, int* __restrict__ tcerr_out) {
  pdl_wait();
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k == 0) *tcerr_out = *tcerr;
  const double2 a = k < n ? make_double2(re[k], im[k]) : make_double2(0.0, 0.0);
  if (k < n) out[k] = a;
  if (S) err_copy(a, k < n, S + k, errbits);
}

// The same where the multiplets' average comes between: max |Σ_new - Σ| and Σ ← Σ_new of every slot. 256 threads.
__global__ void __launch_bounds__(256) err_copy_kernel(const double2* __restrict__ Snew_all, double2* __restrict__ S_all, long n,
                                                       const int* __restrict__ slots,
                                                       unsigned long long* __restrict__ errbits_all) {
  pdl_wait();
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x, t = slots[blockIdx.y];
  err_copy(k < n ? Snew_all[t * n + k] : make_double2(0.0, 0.0), k < n, S_all + t * n + k, errbits_all + t);
}

// Average over degenerate multiplets (src/scgd0.jl:293-301): thread per (ω, multiplet), the sum
// over members in order divided by the count.
__global__ void multiplet_kernel(double2* __restrict__ Sall, int nw, long slab, const int* __restrict__ slots,
                                 const int32_t* __restrict__ mptr, const int32_t* __restrict__ midx, long nmult) {
  pdl_wait();
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= long(nw) * nmult) return;
  double2* S = Sall + slab * slots[blockIdx.y];
  int iw = int(k % nw);
  long g = k / nw;
  int p0 = mptr[g], p1 = mptr[g + 1];
  double sr = 0, si = 0;
  for (int p = p0; p < p1; ++p) {
    double2 z = S[iw + long(nw) * midx[p]];
    sr += z.x;
    si += z.y;
  }
  double len = double(p1 - p0);
  for (int p = p0; p < p1; ++p) S[iw + long(nw) * midx[p]] = make_double2(sr / len, si / len);
}

// Imaginary part of Julia's inv(z) (Smith's algorithm), as in `inv.(…)` of src/scgd0.jl:305.
__device__ __forceinline__ double imag_inv_d(double c, double d) {
  if (fabs(d) <= fabs(c)) {
    double r = d / c;
    double t = 1.0 / (c + d * r);
    return -r * t;
  }
  double r = c / d;
  double t = 1.0 / (d + c * r);
  return -t;
}

// Spectral functions on ωs_spectral (src/scgd0.jl:303-305): A[a, i] = -Im(1/(ωa - ε_i -
// Σ(ωa)))/π with Σ read by the table (j_sp, t_sp) (apply_interpolation_table!).

// FP64 paths (the tensor-core path has its own FP32 kernels below). The FP64 pipe bounds it (an instruction a warp in 16
// cycles): A = d / (π |z|²) with one refined reciprocal takes 15 of them an element, Smith's quotient and the division by
// π, which stay for |z|² near the ends of the range, 43 (3201 x 105: 25.4 -> 12.1 us).
__global__ void spectral_A_kernel(const double2* __restrict__ Sall, int nw, long slab, const int* __restrict__ slots,
                                  const double* __restrict__ wsa, int nwa, const int32_t* __restrict__ jsp,
                                  const double* __restrict__ tsp, const double* __restrict__ eps_i,
                                  double* __restrict__ Aall, int ni) {
  pdl_wait();
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y;
  if (a >= nwa) return;
  const double2* S = Sall + slab * slots[blockIdx.z];
  double* A = Aall + long(nwa) * ni * blockIdx.z;
  int j = jsp[a];
  double t = tsp[a];
  const double2* col = S + long(nw) * i;
  double2 lo = col[j], hi = col[j + 1];
  double sr = (1 - t) * lo.x + t * hi.x;
  double si = (1 - t) * lo.y + t * hi.y;
  const double c = wsa[a] - eps_i[i] - sr, d = -si, q = fma(c, c, d * d);
  const int e = (__double2hiint(q) >> 20) & 0x7ff;
  A[a + long(nwa) * i] = e > 0x100 && e < 0x700 ? d * recip_seeded(q) * 0.31830988618379067154
                                                : -imag_inv_d(c, d) / 3.14159265358979323846;
}

// Fixed-order block reduction helpers (deterministic for a fixed block size).
template <int NT>
__device__ __forceinline__ double block_sum(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
#pragma unroll
  for (int s = NT / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  double r = sh[0];
  __syncthreads();
  return r;
}

// colsum[i] = Σ_a A[a, i] Wa[a] (the ∫A_i of min_spectral_weight, src/scgd0.jl:308).
__global__ void __launch_bounds__(256) spectral_colsum_kernel(const double* __restrict__ Aall, int nwa, int ni,
                                                              const double* __restrict__ Wa, double* __restrict__ colsum_all) {
  pdl_wait();
  __shared__ double sh[256];
  int i = blockIdx.x;
  const double* A = Aall + long(nwa) * ni * blockIdx.y;
  double* colsum = colsum_all + long(ni) * blockIdx.y;
  double s = 0;
  for (int a = threadIdx.x; a < nwa; a += 256) s += A[a + long(nwa) * i] * Wa[a];
  double r = block_sum<256>(s, sh);
  if (threadIdx.x == 0) colsum[i] = r;
}

// The tensor-core path's spectral functions, in FP32 without FP64 arithmetic per (a, i) element.
// With ωa = ω_j + d_a (j = j_sp(a), t = t_sp(a)), the denominator's real part is
//   ωa - ε_i - [(1 - t) ReΣ_j + t ReΣ_{j+1}] = d_a - v_j - t δ_j,
//   v_j = ε_i - ω_j + ReΣ_j,  δ_j = ReΣ_{j+1} - ReΣ_j,
// where v_j and δ_j are formed on float pairs once per grid node (nω ni, not nωa ni) and rounded to FP32
// (P[i][j] = (v_j, δ_j, ImΣ_j, ImΣ_{j+1}), by kk_epilogue_kernel). Near a pole all three terms are of the size of the grid spacing, so the FP32 difference keeps an
// absolute error ~1e-7 h (~1e-10 eV). (Interpolating Σ in FP32 and subtracting it from ωa - ε_i
// instead leaves ~1e-8 eV, which near a pole puts ~1e-5 into A and, through μ, a floor of ~1e-7 eV
// under the iteration's convergence.)
// A[a, i] = -Im(1/(d_a - v_j - t δ_j + i((1-t) ImΣ_j + t ImΣ_{j+1})))/π, never stored: a block of
// 64 nodes a and one chunk of 32 states accumulates Σ_i A w_i per node (Dpart[slot][chunk][a]) and
// Σ_a A Wa per state (Cpart[slot][i][a-block], summed over the block's warps in warp order), both in
// FP32 over at most 32 resp. 64 terms. A warp keeps its 32 x 32 values A Wa in registers and sums them over the lanes
// by halving exchanges (31 shuffles for 32 states, where a tree per state took 160, each waited for), and loads eight
// states at a time: 3201 nodes x 105 states 22.4 -> 9.3 us, 8001 x 495 23.7 -> 10.4. Grid (nωa / 64, ni / 32, slots).
constexpr int kSpecChunk = 32;
constexpr int kSpecNodes = 64;
__global__ void __launch_bounds__(kSpecNodes) spectral_ad_f32_kernel(
    const float4* __restrict__ Pall, int nw, long slab, const int32_t* __restrict__ jsp, const float* __restrict__ dsp,
    const float* __restrict__ tsp, const float* __restrict__ Waf, const float* __restrict__ w_if, int nwa, int ni,
    float* __restrict__ Dpart, float* __restrict__ Cpart, const IterCtl* __restrict__ ctl) {
  pdl_wait();
  if (ctl && ctl->stop) return;
  __shared__ float sh[kSpecNodes / 32][kSpecChunk];
  const int a = blockIdx.x * kSpecNodes + threadIdx.x;
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  const int i0 = blockIdx.y * kSpecChunk, n = min(ni - i0, kSpecChunk);
  const int nab = gridDim.x, nch = gridDim.y;
  const bool ok = a < nwa;
  const int ac = min(a, nwa - 1), j = jsp[ac];
  const float d = dsp[ac], t = tsp[ac], wa = ok ? Waf[ac] : 0.f;
  const float4* P = Pall + slab * blockIdx.z + j + long(nw) * i0;
  float dsum = 0.f, cs[kSpecChunk];
#pragma unroll
  for (int u0 = 0; u0 < kSpecChunk; u0 += 8) {
    float4 p[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) p[u] = P[long(nw) * min(u0 + u, n - 1)];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float c = d - p[u].x - t * p[u].y;
      const float si = (1.f - t) * p[u].z + t * p[u].w;
      // -Im(1/(c + i si))/π = -si/(π (c² + si²)); Smith's form only where the square underflows
      const float den = fmaf(c, c, si * si);
      float A = (den > 1e-30f ? __fdividef(-si, den) : -imag_inv_f(c, -si)) * 0.318309886183790671538f;
      if (u0 + u >= n) A = 0.f;
      dsum += A * w_if[i0 + min(u0 + u, n - 1)];
      cs[u0 + u] = A * wa;
    }
  }
  if (ok) Dpart[(long(blockIdx.z) * nch + blockIdx.y) * nwa + a] = dsum;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {  // lane l ends with state l
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < o; ++k) {
      const float got = __shfl_xor_sync(0xffffffffu, up ? cs[k] : cs[k + o], o);
      cs[k] = (up ? cs[k + o] : cs[k]) + got;
    }
  }
  sh[wid][lane] = cs[0];
  __syncthreads();
  if (threadIdx.x < n) Cpart[(long(blockIdx.z) * ni + i0 + threadIdx.x) * nab + blockIdx.x] = sh[0][threadIdx.x] + sh[1][threadIdx.x];
}

__global__ void __launch_bounds__(256) min_kernel(const double* __restrict__ xall, int n, const int* __restrict__ slots,
                                                  double* __restrict__ out_all) {
  pdl_wait();
  __shared__ double sh[256];
  const double* x = xall + long(n) * blockIdx.x;
  double* out = out_all + slots[blockIdx.x];
  double m = INFINITY;
  for (int k = threadIdx.x; k < n; k += 256) m = fmin(m, x[k]);
  sh[threadIdx.x] = m;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] = fmin(sh[threadIdx.x], sh[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// Roots.jl's Bisection midpoint over floating-point values (Roots._middle).
__device__ __forceinline__ double float_middle_d(double x, double y) {
  if (!isfinite(x) || !isfinite(y)) return x + y;
  if (x != 0 && y != 0 && (signbit(x) != signbit(y))) return 0.0;
  bool negate = (x < 0) || (y < 0);
  unsigned long long ux = __double_as_longlong(fabs(x)), uy = __double_as_longlong(fabs(y));
  double m = __longlong_as_double((long long)((ux + uy) >> 1));
  return negate ? -m : m;
}

// The μ solve of one temperature (src/scgd0.jl:309-324): the root of n(μ) - n_target on the bracket,
// n(μ) = compute_ncarrier_spectral (src/scgd0.jl:361-366), FP64 throughout. The reference
// bisects to adjacent floats (Roots.find_zero on a bracket, ~64 evaluations); here a safeguarded
// Newton iteration on the same bracket finds the same root (n is increasing in μ, with
// dn/dμ = g Σ_a D_a f(1 - f)/T), falling back to Roots' floating-point midpoint whenever the
// Newton step leaves the bracket, and stops at a step below 2^-46 max(|μ|, 1) (the rounding noise of
// n(μ) moves the root by ~1e-15) or at adjacent floats.
// The first round's sums -- D_a f at both bracket ends (whose occupations do not change during a run: mu_ends_kernel),
// D_a f0, D_a f0 (1 - f0) at the start x0, D_a f at the probes x0 -+ 8 T -- are formed where D_a is (the kernels
// that end the spectral functions, mu_terms), as block sums, with E_a = exp((ωa - x0)/T): near x0 a later round's
// occupation costs one product and one reciprocal, exp((ωa - μ)/T) = E_a exp((x0 - μ)/T) (used while
// |μ - x0| <= 30 T; farther out, and at T ~ 0, exp is evaluated directly). When the probes put the root within
// x0 -+ 8 T, nodes with E_a outside [2^-69, 2^69) have, in every later round, occupation 1 to the last bit or, within
// 2^-57 of it, their occupation at x0 times exp(±(μ - x0)/T): D_a of the former and D_a f0 of the latter (all that a
// count of 1e-20 electrons is made of) are summed once, the seventh and eighth terms, and only the other nodes are
// evaluated -- at 300 K a sixth of ±8 eV, and FP64 evaluations (a dozen operations a node at 2 a cycle and SM) are
// what a round costs.
// One cluster of kMuCluster CTAs per temperature: groups of 64 nodes are dealt out to the CTAs in turn, the
// partials are combined through distributed shared memory in rank order, so every thread of the cluster holds the
// same totals and takes the same branches.
// status: 0 ok, 1 no sign change on the bracket.
// Measured at 3201 and 8001 nodes: 27.7 -> 16.6 us and 35.2 -> 21.5 us (before: with the kernel that prepared D at
// the nodes). spectral_fin_f32_kernel, which forms the first round's terms now, went from 3.6 to 8.3 us.
constexpr int kMuCluster = 8;
constexpr int kMuThreads = 128;
constexpr int kMuWarps = kMuThreads / 32;  // kMuCluster x kMuWarps partials: one per lane of the warp that sums them
constexpr int kMuTerms = 8;              // first-round terms per node
constexpr double kMuProbe = 8.0;         // the probes x0 -+ 8 T
constexpr double kMuProbeExp = 2980.957987041728;  // e^8

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Shared by mu_terms and mu_solve_kernel: the start x0 of slot's temperature on the bracket.
__device__ __forceinline__ double mu_start(double guess, double a, double b) {
  return (guess > a && guess < b) ? guess : float_middle_d(a, b);
}

// Occupation from y = exp((ωa - μ)/T) (electrons: 1/(1 + y); holes: y/(1 + y)), to an ulp or two: recip_seeded takes
// 1 + y up to 2^1000; beyond (693 T above μ) an electron's is below 1e-301 and a hole's is 1 to the last bit.
__device__ __forceinline__ double occ_from_y(double y, int holes) {
  if (y >= 0x1p1000) return holes ? 1.0 : 0.0;
  const double r = recip_seeded(1.0 + y);
  return holes ? y * r : r;
}

// The occupations at the bracket ends, per temperature of the run (ends[t][2][nωa]).
__global__ void mu_ends_kernel(const double* __restrict__ wsa, int nwa, const TParams* __restrict__ tp, double br0,
                               double br1, double* __restrict__ ends) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nwa) return;
  const TParams q = tp[blockIdx.y];
  auto occ = [&](double wa, double mu) { return occ_fermion_d(q.holes ? mu - wa : wa - mu, q.T); };
  ends[(2l * blockIdx.y) * nwa + k] = occ(wsa[k], br0);
  ends[(2l * blockIdx.y + 1) * nwa + k] = occ(wsa[k], br1);
}

// Where E lies: 0 within [2^-69, 2^69), -1 below, 1 above.
__device__ __forceinline__ int mu_band(double E) {
  const int hi = __double2hiint(E);
  return hi < ((1023 - 69) << 20) ? -1 : hi >= ((1023 + 69) << 20) ? 1 : 0;
}

// What the μ solve of a slot reads, and its first-round terms at one node.
struct MuIn {
  const double* ends = nullptr;  // null: no μ solve (μ fixed)
  const TParams* tp = nullptr;
  double br0 = 0, br1 = 0;
  double* E = nullptr;     // [slot][nωa]
  double* part = nullptr;  // [slot][blocks][kMuTerms]
};
__device__ __forceinline__ void mu_terms(const MuIn& M, int t, long slot, int k, int nwa, double wa, double d,
                                         double (&v)[kMuTerms]) {
  const TParams q = M.tp[t];
  const double T = q.T, x0 = mu_start(q.mu, M.br0, M.br1);
  const bool warm = T > 1.4901161193847656e-08;
  double f0, fl, fr, E = 0;
  int band = 0;
  if (warm) {
    E = exp((wa - x0) * q.inv_T);
    band = mu_band(E);
    f0 = occ_from_y(E, q.holes);
    fl = occ_from_y(E * kMuProbeExp, q.holes);  // at x0 - kMuProbe T: exp((ωa - x0)/T + kMuProbe)
    fr = occ_from_y(E * (1.0 / kMuProbeExp), q.holes);
  } else {
    f0 = occ_fermion_d(q.holes ? x0 - wa : wa - x0, T);
    fl = fr = f0;
  }
  M.E[slot * nwa + k] = E;
  v[0] = d * M.ends[(2l * t) * nwa + k];
  v[1] = d * M.ends[(2l * t + 1) * nwa + k];
  v[2] = d * f0;
  v[3] = d * (f0 * (1 - f0));
  v[4] = d * fl;
  v[5] = d * fr;
  v[6] = band == (q.holes ? 1 : -1) ? d : 0.0;
  v[7] = band == (q.holes ? -1 : 1) ? d * f0 : 0.0;
}
// A warp's sums of the eight terms into out[0 .. 8): halving exchanges leave sum q on lanes 4 q .. 4 q + 3 (9 FP64
// additions a lane, where a tree per term takes 35).
__device__ __forceinline__ void mu_warp_terms(const double (&v)[kMuTerms], double* out) {
  double x[8] = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
  const int lane = threadIdx.x % 32;
#pragma unroll
  for (int h = 4, o = 16; h > 0; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const double got = __shfl_xor_sync(0xffffffffu, up ? x[k] : x[k + h], o);
      x[k] = (up ? x[k + h] : x[k]) + got;
    }
  }
  x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
  x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
  if (lane % 4 == 0) out[lane / 4] = x[0];
}

// D[a] = Wa[a] Σ_chunk Dpart (FP64, chunk order) for blocks x < nab, and with it the μ solve's first round;
// the blocks after them give one warp to each state i: ∫A_i = Σ Cpart over the node blocks (FP64: lanes in strides of
// 32, then a shuffle tree), whose minimum over i goes to minA[slots[z]] by an atomic minimum of the bit
// patterns (∫A_i >= 0, so they order as the values; kk_epilogue_kernel sets +inf first). The first thread also copies
// the tensor-core wait flag into the iteration's results, and asks for a stop when its temperature has converged. Grid (nab + ni / 2, slots), 64 threads.
__global__ void __launch_bounds__(kSpecNodes) spectral_fin_f32_kernel(
    const float* __restrict__ Dpart, const float* __restrict__ Cpart, int nch, int nab, const double* __restrict__ Wa,
    const double* __restrict__ wsa, int nwa, int ni, const int* __restrict__ slots, double* __restrict__ Dall,
    double* __restrict__ minA_all, const MuIn M, const int* __restrict__ tc_err, int* __restrict__ tc_err_out,
    const unsigned long long* __restrict__ errbits, IterCtl* __restrict__ ctl) {
  pdl_wait();
  if (ctl && ctl->stop) return;
  __shared__ double sh[2][kMuTerms];
  const long z = blockIdx.y;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (z == 0) *tc_err_out = *tc_err;
    if (ctl && __longlong_as_double((long long)errbits[slots[z]]) < ctl->tol) ctl->stop_next = 1;
  }
  if (int(blockIdx.x) < nab) {
    const int a = blockIdx.x * kSpecNodes + threadIdx.x;
    double v[kMuTerms] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (a < nwa) {
      double s = 0;
#pragma unroll 8
      for (int c = 0; c < nch; ++c) s += double(Dpart[(z * nch + c) * nwa + a]);
      s *= Wa[a];
      Dall[z * nwa + a] = s;
      if (M.ends) mu_terms(M, slots[z], z, a, nwa, wsa[a], s, v);
    }
    if (!M.ends) return;
    mu_warp_terms(v, sh[threadIdx.x / 32]);
    __syncthreads();
    if (threadIdx.x < kMuTerms) M.part[(z * nab + blockIdx.x) * kMuTerms + threadIdx.x] = sh[0][threadIdx.x] + sh[1][threadIdx.x];
    return;
  }
  const int i = (int(blockIdx.x) - nab) * 2 + int(threadIdx.x) / 32, lane = threadIdx.x % 32;
  if (i >= ni) return;
  const float* c = Cpart + (z * ni + i) * nab;
  double s = 0;
#pragma unroll 4
  for (int b = lane; b < nab; b += 32) s += double(c[b]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) atomicMin(reinterpret_cast<unsigned long long*>(minA_all + slots[z]), (unsigned long long)__double_as_longlong(s));
}

// D[a] = (Σ_i A[a, i] w_i) Wa[a] (src/scgd0.jl:306-307). A block of 256 threads covers 32 nodes a
// (the lanes) and splits i over its 8 warps (i ≡ warp mod 8, ascending); the 8 partial sums are
// added in warp order, so the result is deterministic. With it, the μ solve's first round (FP64 paths).
__global__ void __launch_bounds__(256) spectral_D_kernel(const double* __restrict__ Aall, int nwa, int ni,
                                                         const double* __restrict__ w_i, const double* __restrict__ Wa,
                                                         const double* __restrict__ wsa, const int* __restrict__ slots,
                                                         double* __restrict__ Dall, const MuIn M) {
  pdl_wait();
  __shared__ double sh[8][32];
  const double* A = Aall + long(nwa) * ni * blockIdx.y;
  double* D = Dall + long(nwa) * blockIdx.y;
  const int lane = threadIdx.x % 32, g = threadIdx.x / 32;
  const int a = blockIdx.x * 32 + lane;
  double s = 0;
  if (a < nwa)
#pragma unroll 4
    for (int i = g; i < ni; i += 8) s += A[a + long(nwa) * i] * w_i[i];
  sh[g][lane] = s;
  __syncthreads();
  if (g == 0) {
    double v[kMuTerms] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (a < nwa) {
      double t = sh[0][lane];
#pragma unroll
      for (int k = 1; k < 8; ++k) t += sh[k][lane];
      t *= Wa[a];
      D[a] = t;
      mu_terms(M, slots[blockIdx.y], blockIdx.y, a, nwa, wsa[a], t, v);
    }
    mu_warp_terms(v, M.part + (long(blockIdx.y) * gridDim.x + blockIdx.x) * kMuTerms);
  }
}

// F / d for d > 0.
__device__ __forceinline__ double div_pos(double F, double d) {
  const int e = (__double2hiint(d) >> 20) & 0x7ff;
  return e > 0 && e < 0x7f0 ? F * recip_seeded(d) : F / d;
}

__global__ void __cluster_dims__(kMuCluster, 1, 1) __launch_bounds__(kMuThreads)
    mu_solve_kernel(const double* __restrict__ Dall, const double* __restrict__ wsa, int nwa, const int* __restrict__ slots,
                    TParams* __restrict__ tp, double W, double base, double gs, double br0, double br1,
                    const double* __restrict__ E_all, const double* __restrict__ part1, int npart, double* __restrict__ mu_all,
                    int* __restrict__ status_all, int* __restrict__ evals_all, const IterCtl* __restrict__ ctl) {
  pdl_wait();
  if (ctl && ctl->stop) return;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank();
  // one cluster per active temperature
  const int slot = blockIdx.x / kMuCluster, t = slots[slot];
  const double* D = Dall + long(nwa) * slot;
  const double* E = E_all + long(nwa) * slot;
  const double* P1 = part1 + long(kMuTerms) * npart * slot;
  const double T = tp[t].T, inv_T = tp[t].inv_T, n_target = tp[t].n_target, guess = tp[t].mu;
  const int holes = tp[t].holes;
  __shared__ double part[2][kMuWarps][2];
  __shared__ double tot[kMuTerms];
  const bool warm = T > 1.4901161193847656e-08;
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  // Totals of two per-thread sums over the cluster, on the threads of warp 0: every warp's sums go to its CTA's part
  // buffer (two buffers in turn, so one cluster barrier per round suffices: a CTA can only overwrite a buffer after
  // the next round's barrier, when every CTA has read it), and lane l of warp 0 reads those of CTA l / 4, warp l % 4.
  int round = 0;
  auto reduce = [&](double (&v)[2]) {
    v[0] = warp_sum_d(v[0]);
    v[1] = warp_sum_d(v[1]);
    double(*pb)[2] = part[round & 1];
    if (lane == 0) {
      pb[wid][0] = v[0];
      pb[wid][1] = v[1];
    }
    cluster.sync();
    if (wid == 0) {
      const double* r = cluster.map_shared_rank(&pb[0][0], unsigned(lane / kMuWarps)) + 2 * (lane % kMuWarps);
      v[0] = warp_sum_d(r[0]);
      v[1] = warp_sum_d(r[1]);
    }
    ++round;
  };
  auto occ = [&](double wa, double mu) { return occ_fermion_d(holes ? mu - wa : wa - mu, T); };
  auto total = [&](double t1) { return (holes ? (W - t1 + base) * gs : (t1 + base) * gs) - n_target; };
  // The bracket and the Newton step are scalar work: thread 0 of every CTA does it (each holds the
  // same totals, so all CTAs take the same steps) and publishes the next point through shared
  // memory, instead of every thread repeating it on the FP64 units.
  __shared__ double s_x, s_scale;
  __shared__ int s_fact, s_stop, s_win;
  double a = br0, b = br1, fa = 0, fb = 0, x = mu_start(guess, br0, br1), result = x;
  const double x0 = x;
  double x_sc = x0, scale0 = 1.0;  // scale0 = exp((x0 - x_sc)/T)
  int it = 0;
  bool failed = false;
  auto newton = [&](double F, double dF) -> int {  // 1: done (result set)
    result = x;
    if (F == 0) return 1;
    if (signbit(F) == signbit(fa)) {
      a = x;
      fa = F;
    } else {
      b = x;
      fb = F;
    }
    double xn = dF > 0 ? x - div_pos(F, dF) : x;
    // a converged Newton step ends the solve even when it rounds onto the end the bracket update
    // just moved to x (otherwise the safeguard below would bisect down to adjacent floats)
    if (dF > 0 && fabs(xn - x) <= 0x1p-46 * fmax(fabs(x), 1.0)) {
      result = xn;
      return 1;
    }
    if (!(dF > 0) || !(xn > a && xn < b)) xn = float_middle_d(a, b);
    if (xn == a || xn == b) {
      result = fabs(fa) <= fabs(fb) ? a : b;
      return 1;
    }
    x = xn;
    return ++it >= 400 ? 1 : 0;
  };
  auto publish = [&](int stop) {
    const double sx = (x0 - x) * inv_T;
    const bool fact = warm && fabs(sx) <= 30.0;
    if (fact && !stop) {  // exp((x0 - x)/T): by the series of the step where it is short (2^-45 / 9! relative)
      const double d = (x_sc - x) * inv_T;
      if (fabs(d) < 0.03125) {
        double p = fma(d, 1.0 / 40320, 1.0 / 5040);
        p = fma(d, p, 1.0 / 720);
        p = fma(d, p, 1.0 / 120);
        p = fma(d, p, 1.0 / 24);
        p = fma(d, p, 1.0 / 6);
        p = fma(d, p, 0.5);
        p = fma(d, p, 1.0);
        scale0 *= fma(d, p, 1.0);
      } else {
        scale0 = exp(sx);
      }
      x_sc = x;
    }
    s_x = x;
    s_scale = scale0;
    s_fact = fact ? 1 : 0;
    s_stop = stop;
  };
  // round 1: n(a), n(b), n(x0), n'(x0), n(x0 -+ 8T) and the sums of the nodes with E outside [2^-69, 2^69) from the
  // blocks' sums, by every CTA alike
  {
    for (int q = wid; q < kMuTerms; q += kMuWarps) {
      double t = 0;
#pragma unroll 4
      for (int k = lane; k < npart; k += 32) t += P1[k * kMuTerms + q];
      t = warp_sum_d(t);
      if (lane == 0) tot[q] = t;
    }
    if (threadIdx.x == 0) s_win = 0;
    __syncthreads();
    const double* v = tot;
    ++round;
    if (threadIdx.x == 0) {
      fa = total(v[0]);
      fb = total(v[1]);
      int stop = 1;
      if (fa * fb > 0) {
        failed = true;
      } else if (fa == 0) {
        result = a;
      } else if (fb == 0) {
        result = b;
      } else {
        // the probes narrow the bracket to the side (or the 16 T window) that holds the sign change
        const double xl = x0 - kMuProbe * T, xr = x0 + kMuProbe * T;
        const double fl = total(v[4]), fr = total(v[5]);
        const double F0 = total(v[2]), dF0 = warm ? gs * v[3] * inv_T : 0.0;
        if (warm && xl > a && xr < b && fl != 0 && fr != 0 && signbit(fl) == signbit(fr)) {
          // x0 lies outside the narrowed bracket: its Newton step (or the midpoint) starts round 2
          if (signbit(fl) != signbit(fa)) {
            b = xl;
            fb = fl;
          } else {
            a = xr;
            fa = fr;
          }
          double xn = x0 - F0 / dF0;
          if (!(dF0 > 0) || !(xn > a && xn < b)) xn = float_middle_d(a, b);
          x = xn;
          stop = 0;
        } else {
          if (warm && xl > a && xr < b && fl != 0 && fr != 0) {
            a = xl;
            fa = fl;
            b = xr;
            fb = fr;
            s_win = 1;  // every later point lies within x0 -+ 8 T
          }
          stop = newton(F0, dF0);
        }
      }
      publish(stop);
    }
    __syncthreads();
  }
  const bool win = s_win != 0;
  while (!s_stop) {
    const double xr = s_x, scale = s_scale;
    const bool fact = s_fact != 0;
    double v[2] = {0, 0};
#pragma unroll 4
    for (int k = (int(threadIdx.x) / 64 * kMuCluster + int(rank)) * 64 + int(threadIdx.x) % 64; k < nwa;
         k += kMuCluster * kMuThreads) {
      const double Ek = E[k], d = D[k];
      if (win && mu_band(Ek) != 0) continue;
      const double f = fact ? occ_from_y(Ek * scale, holes) : occ(wsa[k], xr);
      const double df = d * f;
      v[0] += df;
      v[1] += fma(-df, f, df);
    }
    reduce(v);
    if (threadIdx.x == 0) {
      const double tail = win ? tot[7] * (holes ? scale : recip_seeded(scale)) : 0.0;  // (f (1 - f) is f there)
      publish(newton(total(win ? tot[6] + tail + v[0] : v[0]), warm ? gs * (v[1] + tail) * inv_T : 0.0));
    }
    __syncthreads();
  }
  // no CTA leaves while another may still read its partials
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    evals_all[t] = round;
    if (failed) {
      status_all[t] = 1;
    } else {
      mu_all[t] = result;
      tp[t].mu = result;  // the next iteration's μ, without a round trip to the host
      status_all[t] = 0;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// setup
// ---------------------------------------------------------------------------------------------

static void check_model_common(const epsp_model* m) {
  if (!m) fail(EPSP_EINVAL, "model is NULL");
  if (m->nm < 1 || m->ni < 1 || m->nf < 1) fail(EPSP_EINVAL, "nm, ni and nf must be positive");
  if (!m->g2 || !m->omega_ph || !m->iq_kk || !m->iks_i || !m->iks_f || !m->eps_i || !m->w_i || !m->eps_f ||
      !m->w_f || !m->f_to_i)
    fail(EPSP_EINVAL, "a required model array is NULL");
  if (m->g2_dtype != EPSP_F64 && m->g2_dtype != EPSP_F32 && m->g2_dtype != EPSP_BF16)
    fail(EPSP_EINVAL, "g2_dtype must be EPSP_F64, EPSP_F32 or EPSP_BF16");
  if (m->nm > 1024) fail(EPSP_EINVAL, "at most 1024 modes");
  for (int64_t f = 0; f < m->nf; ++f) {
    if (m->f_to_i[f] < 0 || m->f_to_i[f] >= m->ni) fail(EPSP_EINVAL, "f_to_i out of range");
    if (m->iks_f[f] < 0 || m->iks_f[f] >= m->nk_f) fail(EPSP_EINVAL, "iks_f out of range");
  }
  for (int64_t i = 0; i < m->ni; ++i)
    if (m->iks_i[i] < 0 || m->iks_i[i] >= m->nk_i) fail(EPSP_EINVAL, "iks_i out of range");
  for (int64_t k = 0; k < m->nk_i * m->nk_f; ++k)
    if (m->iq_kk[k] < 0 || m->iq_kk[k] >= m->nq) fail(EPSP_EINVAL, "iq_kk out of range");
  if (m->nmult < 0 || (m->nmult > 0 && (!m->mult_ptr || !m->mult_idx))) fail(EPSP_EINVAL, "bad multiplet lists");
  std::vector<char> seen(size_t(m->ni), 0);
  for (int64_t g = 0; g < m->nmult; ++g) {
    if (m->mult_ptr[g + 1] < m->mult_ptr[g]) fail(EPSP_EINVAL, "multiplet pointers must not decrease");
    for (int32_t p = m->mult_ptr[g]; p < m->mult_ptr[g + 1]; ++p) {
      if (m->mult_idx[p] < 0 || m->mult_idx[p] >= m->ni) fail(EPSP_EINVAL, "multiplet member out of range");
      if (seen[size_t(m->mult_idx[p])]++) fail(EPSP_EINVAL, "a state belongs to two multiplets");
    }
  }
}

// Modes are dispersionless when every row of ωph is constant; then ωq[ν, f, i] = ω_ν for every pair.
static bool dispersionless(const epsp_model* m, std::vector<double>& wnu) {
  wnu.assign(size_t(m->nm), 0.0);
  for (int64_t nu = 0; nu < m->nm; ++nu) {
    double w0 = m->omega_ph[nu];
    for (int64_t q = 1; q < m->nq; ++q)
      if (!(m->omega_ph[nu + m->nm * q] == w0)) return false;
    wnu[size_t(nu)] = w0;
  }
  return true;
}

void upload_g2_permuted(Ctx* ctx, const epsp_model* m, DBuf<double>& g2t) {
  const size_t elem = m->g2_dtype == EPSP_F64 ? 8 : (m->g2_dtype == EPSP_F32 ? 4 : 2);
  const long nm = m->nm, ni = m->ni, nf = m->nf;
  g2t.alloc(ctx, size_t(nm * nf * ni));
  // Stage by slabs of inner states so the raw staging buffer stays bounded (~256 MB).
  long per_f = nm * ni;
  long fchunk = std::max<long>(1, long((size_t(256) << 20) / (elem * size_t(per_f))));
  DBuf<uint8_t> stage;
  stage.alloc(ctx, size_t(std::min(fchunk, nf) * per_f) * elem);
  for (long f0 = 0; f0 < nf; f0 += fchunk) {
    long nfc = std::min(fchunk, nf - f0);
    const uint8_t* src = static_cast<const uint8_t*>(m->g2) + size_t(f0 * per_f) * elem;
    EPSP_CUDA(cudaMemcpyAsync(stage.p, src, size_t(nfc * per_f) * elem, cudaMemcpyHostToDevice, ctx->stream));
    long total = nm * nfc * ni;
    unsigned grid = div_up(size_t(total), 256);
    // permute_g2_kernel reads slab-relative inner states and writes at absolute f0 + f.
    double* dst = g2t.p + nm * f0;
    if (m->g2_dtype == EPSP_F64)
      permute_g2_kernel<double><<<grid, 256, 0, ctx->stream>>>(reinterpret_cast<const double*>(stage.p), int(nm), int(ni), nf, 0, nfc, dst);
    else if (m->g2_dtype == EPSP_F32)
      permute_g2_kernel<float><<<grid, 256, 0, ctx->stream>>>(reinterpret_cast<const float*>(stage.p), int(nm), int(ni), nf, 0, nfc, dst);
    else
      permute_g2_kernel<uint16_t><<<grid, 256, 0, ctx->stream>>>(reinterpret_cast<const uint16_t*>(stage.p), int(nm), int(ni), nf, 0, nfc, dst);
    EPSP_LAUNCHED(ctx);
  }
  EPSP_CUDA(cudaStreamSynchronize(ctx->stream));
}

Scgd0Plan* scgd0_setup(Ctx* ctx, const epsp_model* m, const epsp_options* opts) {
  check_model_common(m);
  if (!opts) fail(EPSP_EINVAL, "options are NULL");
  if (opts->gpu_tile < 0) fail(EPSP_EINVAL, "gpu_tile must be nothing or a positive number of inner states");
  auto* P = new Scgd0Plan;
  std::unique_ptr<Scgd0Plan> guard(P);
  P->ctx = ctx;
  P->path = opts->path;
  if (P->path == EPSP_PATH_GEMM_TF32)
    fail(EPSP_EUNSUPPORTED, "GEMM_TF32 is a ladder path; scGD0 plans take DIRECT_FP64, GEMM_FP64 or GEMM_BF16");
  P->w_ac = opts->omega_acoustic;
  P->verbosity = opts->verbosity;
  P->nm = m->nm;
  P->ni = m->ni;
  P->nf = m->nf;
  P->ws = make_grid(m->omegas, "omegas");
  P->wsa = make_grid(m->omegas_spectral, "omegas_spectral");
  P->nw = P->ws.n;
  P->nwa = P->wsa.n;
  P->W = m->W;
  P->nstates_base = m->nstates_base;
  P->gpu_tile = opts->gpu_tile;
  PhaseLog plog(ctx, "scgd0", P->verbosity);
  cudaStream_t s = ctx->stream;
  // grid tables
  CellTableHost ct = make_cell_table(P->ws);
  P->d_jtab = to_device(ctx, ct.jtab);
  P->d_ws = to_device(ctx, P->ws.nodes);
  P->ct = CellTableDev{P->d_jtab.p, P->d_ws.p, ct.x0, ct.inv_h, int(P->nw)};
  P->d_wsa = to_device(ctx, P->wsa.nodes);
  std::vector<int32_t> jsp;
  std::vector<double> tsp;
  interp_table(P->ws.nodes, P->wsa.nodes, jsp, tsp);  // src/scgd0.jl:163
  P->d_jsp = to_device(ctx, jsp);
  P->d_tsp = to_device(ctx, tsp);
  P->d_Wa = to_device(ctx, trapezoid_weights(P->wsa.nodes));
  P->d_eps_i = to_device(ctx, m->eps_i, size_t(m->ni));
  P->d_w_i = to_device(ctx, m->w_i, size_t(m->ni));
  {
    std::vector<float> dspf(jsp.size()), tspf(jsp.size()), Waf(jsp.size()), w_if(static_cast<size_t>(m->ni));
    const std::vector<double> Wa = trapezoid_weights(P->wsa.nodes);
    for (size_t a = 0; a < jsp.size(); ++a) {
      dspf[a] = float(P->wsa.nodes[a] - P->ws.nodes[size_t(jsp[a])]);
      tspf[a] = float(tsp[a]);
      Waf[a] = float(Wa[a]);
    }
    for (size_t i = 0; i < w_if.size(); ++i) w_if[i] = float(m->w_i[i]);
    P->d_dspf = to_device(ctx, dspf);
    P->d_tspf = to_device(ctx, tspf);
    P->d_Waf = to_device(ctx, Waf);
    P->d_w_if = to_device(ctx, w_if);
  }
  if (m->nmult > 0) {
    P->nmult = m->nmult;
    P->d_mptr = to_device(ctx, m->mult_ptr, size_t(m->nmult + 1));
    P->d_midx = to_device(ctx, m->mult_idx, size_t(m->mult_ptr[m->nmult]));
  }
  {  // state groups of the tensor-core epilogue: the multiplets, then every state in none
    std::vector<int32_t> gptr{0}, gidx;
    std::vector<char> in_mult(size_t(m->ni), 0);
    for (int64_t g = 0; g < m->nmult; ++g) {
      for (int64_t p = m->mult_ptr[g]; p < m->mult_ptr[g + 1]; ++p) {
        gidx.push_back(int32_t(m->mult_idx[p]));
        in_mult[size_t(m->mult_idx[p])] = 1;
      }
      gptr.push_back(int32_t(gidx.size()));
    }
    for (int64_t i = 0; i < m->ni; ++i)
      if (!in_mult[size_t(i)]) {
        gidx.push_back(int32_t(i));
        gptr.push_back(int32_t(gidx.size()));
      }
    P->ngroups = long(gptr.size()) - 1;
    if (P->ngroups > 65535) fail(EPSP_EUNSUPPORTED, "at most 65535 state groups (multiplets and single states)");
    P->d_gptr = to_device(ctx, gptr);
    P->d_gidx = to_device(ctx, gidx);
  }
  plog.mark("grid tables");
  kk_matrix_to_device(ctx, P->ws.nodes, P->d_KK);
  const long nm = m->nm, ni = m->ni, nf = m->nf;
  if (P->path == EPSP_PATH_DIRECT_FP64) {
    // nf_chunk of src/scgd0.jl:201-202; the chunks fix the order of the f sum.
    const int64_t chunk_bytes = int64_t(1) << 30;
    P->nf_chunk = opts->gpu_tile <= 0 ? std::clamp<int64_t>(chunk_bytes / (8 * nm * ni), 1, nf) : std::min<int64_t>(opts->gpu_tile, nf);
    upload_g2_permuted(ctx, m, P->d_g2t);
    auto d_wph = to_device(ctx, m->omega_ph, size_t(nm * m->nq));
    auto d_iq = to_device(ctx, m->iq_kk, size_t(m->nk_i * m->nk_f));
    auto d_iksi = to_device(ctx, m->iks_i, size_t(ni));
    auto d_iksf = to_device(ctx, m->iks_f, size_t(nf));
    P->d_wqt.alloc(ctx, size_t(nm * nf * ni));
    gather_wq_kernel<<<div_up(size_t(nm * nf * ni), 256), 256, 0, s>>>(d_wph.p, d_iq.p, d_iksi.p, d_iksf.p, int(nm), int(ni), nf,
                                                                      m->nk_i, P->d_wqt.p);
    EPSP_LAUNCHED(ctx);
    P->d_eps_f = to_device(ctx, m->eps_f, size_t(nf));
    P->d_w_f = to_device(ctx, m->w_f, size_t(nf));
    P->d_f_to_i = to_device(ctx, m->f_to_i, size_t(nf));
    {  // fm_direct_fast_kernel: the nodes as ordered integers (one above all values after them), the largest ωq, and the
       // FP32 bucket's guard: x, x - x0 and the product round by 2^-24 of at most 9 max|ω| + 5 max ωq, over h, in all
      std::vector<long long> key(size_t(P->nw) + 1);
      double big = 0;
      for (long j = 0; j < P->nw; ++j) {
        long long b;
        std::memcpy(&b, &P->ws.nodes[size_t(j)], 8);
        key[size_t(j)] = ordered(b);
        big = std::max(big, std::fabs(P->ws.nodes[size_t(j)]));
      }
      key[size_t(P->nw)] = std::numeric_limits<long long>::max();
      P->d_wkey = to_device(ctx, key);
      for (int64_t k = 0; k < nm * m->nq; ++k) {
        if (!std::isfinite(m->omega_ph[k])) P->wq_max = std::numeric_limits<double>::infinity();
        P->wq_max = std::max(P->wq_max, m->omega_ph[k]);
      }
      const double guard = (12 * (big + std::min(P->wq_max, 1e30)) * P->ct.inv_h + 8) * 0x1p-24;
      P->fm_guard = float(guard);
      P->fm_fast = P->w_ac > 0 && guard < 0.4;
      EPSP_CUDA(cudaStreamSynchronize(s));  // key is a local
    }
  } else if (P->path == EPSP_PATH_GEMM_BF16 && [&] {
               std::vector<double> w;
               return !dispersionless(m, w);
             }()) {
    // dispersive modes on the tensor-core path: the Fan-Migdal sum term by term in FP32, the rest of
    // the iteration (Kramers-Kronig product and its epilogue, spectral functions, μ) as below
    tc_setup_dispersive(P, m);
    tc_setup(P);
    EPSP_CUDA(cudaStreamSynchronize(s));
  } else if (P->path == EPSP_PATH_GEMM_FP64 || P->path == EPSP_PATH_GEMM_BF16) {
    std::vector<double> wnu;
    if (!dispersionless(m, wnu))
      fail(EPSP_EUNSUPPORTED, "the GEMM paths need dispersionless modes (every row of omega_ph constant); use EPSP_PATH_DIRECT_FP64");
    // Column sets: the stars of the representatives when every inner state of a star has the same
    // energy (then the f sum of one star is one column); one inner state per column otherwise.
    std::vector<int32_t> order(static_cast<size_t>(nf));
    for (long f = 0; f < nf; ++f) order[size_t(f)] = int32_t(f);
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return m->f_to_i[a] < m->f_to_i[b]; });
    std::vector<int32_t> sptr(size_t(ni + 1), 0);
    for (long f = 0; f < nf; ++f) sptr[size_t(m->f_to_i[f] + 1)]++;
    for (long i = 0; i < ni; ++i) sptr[size_t(i + 1)] += sptr[size_t(i)];
    bool uniform = true;
    std::vector<double> eps_star(static_cast<size_t>(ni), 0.0);
    for (long i = 0; i < ni && uniform; ++i) {
      if (sptr[size_t(i + 1)] == sptr[size_t(i)]) continue;
      double e0 = m->eps_f[order[size_t(sptr[size_t(i)])]];
      eps_star[size_t(i)] = e0;
      for (int32_t p = sptr[size_t(i)]; p < sptr[size_t(i + 1)]; ++p)
        if (!(m->eps_f[order[size_t(p)]] == e0)) uniform = false;
    }
    std::vector<int32_t> cptr, members, colc;
    std::vector<double> epsc;
    if (uniform) {
      for (long i = 0; i < ni; ++i)
        if (sptr[size_t(i + 1)] > sptr[size_t(i)]) {
          cptr.push_back(sptr[size_t(i)]);
          colc.push_back(int32_t(i));
          epsc.push_back(eps_star[size_t(i)]);
        }
      cptr.push_back(int32_t(nf));
      members = order;
    } else {
      for (long f = 0; f < nf; ++f) {
        cptr.push_back(int32_t(f));
        members.push_back(int32_t(f));
        colc.push_back(m->f_to_i[f]);
        epsc.push_back(m->eps_f[f]);
      }
      cptr.push_back(int32_t(nf));
    }
    P->star_reduced = uniform;
    P->nc = long(colc.size());
    P->d_wnu = to_device(ctx, wnu);
    P->d_colc = to_device(ctx, colc);
    P->d_epsc = to_device(ctx, epsc);
    auto d_cptr = to_device(ctx, cptr);
    auto d_mem = to_device(ctx, members);
    auto d_wf = to_device(ctx, m->w_f, size_t(nf));
    plog.mark("KK matrix, column sets");
    // The coupling sums need g2 once: it streams through the device in star order, gpu_tile inner
    // states per chunk (or about 64 MiB of g2 per chunk), copies overlapped with the sums; g2
    // stays in the caller's host memory.
    P->d_G.alloc(ctx, size_t(nm * P->nc * ni));
    const size_t member_bytes = size_t(nm * ni) * g2_elem_bytes(m->g2_dtype);
    const long chunk_f = opts->gpu_tile > 0 ? long(opts->gpu_tile) : std::max<long>(1, long((size_t(64) << 20) / member_bytes));
    const unsigned grid = div_up(size_t(nm * ni), 128);
    stream_g2_by_columns(ctx, m, members, cptr, chunk_f, [&](const void* g2c, long c0, long c1, long p0) {
      if (m->g2_dtype == EPSP_F64)
        coupling_sum_chunk_kernel<double><<<dim3(grid, unsigned(std::min<long>(c1 - c0, 65535))), 128, 0, s>>>(static_cast<const double*>(g2c), int(nm), int(ni), d_cptr.p, c0,
                                                              c1, p0, d_mem.p, P->nc, d_wf.p, P->d_wnu.p, P->w_ac, P->d_G.p);
      else if (m->g2_dtype == EPSP_F32)
        coupling_sum_chunk_kernel<float><<<dim3(grid, unsigned(std::min<long>(c1 - c0, 65535))), 128, 0, s>>>(static_cast<const float*>(g2c), int(nm), int(ni), d_cptr.p, c0,
                                                             c1, p0, d_mem.p, P->nc, d_wf.p, P->d_wnu.p, P->w_ac, P->d_G.p);
      else
        coupling_sum_chunk_kernel<uint16_t><<<dim3(grid, unsigned(std::min<long>(c1 - c0, 65535))), 128, 0, s>>>(static_cast<const uint16_t*>(g2c), int(nm), int(ni), d_cptr.p,
                                                                c0, c1, p0, d_mem.p, P->nc, d_wf.p, P->d_wnu.p, P->w_ac,
                                                                P->d_G.p);
      EPSP_LAUNCHED(ctx);
    });
    plog.mark("g2 streamed, coupling sums");
    // The cells of ω ± ω_ν, by the lookup of _interp_linear_grid (src/frequency_grids.jl:207-219).
    {
      const auto& w = P->ws.nodes;
      const long n = P->nw;
      // (cell tables: cell j is entry j + 1, entry 0 the flat part below the grid.) FP32 records: a point that misses a
      // node from below by rounding alone, as where the modes are multiples of the grid's step, is taken from that node;
      // as the far end of the cell below it would carry 2^-24 of the values at that cell's start, which may be large
      // against those at the node.
      const double snap = P->path == EPSP_PATH_GEMM_BF16 ? 0x1p-44 * std::max(std::fabs(w.front()), std::fabs(w.back())) : 0.0;
      std::vector<int32_t> cj(size_t(2 * n * nm));
      std::vector<double> cdx(cj.size());
      for (long side = 0; side < 2; ++side)
        for (long nu = 0; nu < nm; ++nu)
          for (long iw = 0; iw < n; ++iw) {
            const double x = side == 0 ? w[size_t(iw)] + wnu[size_t(nu)] : w[size_t(iw)] - wnu[size_t(nu)];
            int32_t e;
            if (!(x > w[0])) {
              e = 0;
            } else if (x >= w[size_t(n - 1)]) {
              e = int32_t(n);
            } else {
              const int32_t c = ct.jtab[size_t(int64_t((x - ct.x0) * ct.inv_h))];
              e = c + (w[size_t(c)] <= x ? 1 : 0);
              if (w[size_t(e)] - x <= snap) ++e;
            }
            const size_t k = size_t(iw + n * (nu + nm * side));
            cj[k] = e;
            cdx[k] = x - w[size_t(std::max(e - 1, 0))];
          }
      P->d_cell_j = to_device(ctx, cj);
      P->d_cell_t = to_device(ctx, cdx);
    }
    P->d_Fa.alloc(ctx, size_t(P->nw * nm));
    P->d_Fe.alloc(ctx, size_t(P->nw * nm));
    if (P->path == EPSP_PATH_GEMM_FP64) {
      P->d_Kt.alloc(ctx, size_t(P->nw * nm * P->nc));
      P->ozG.keep(ctx, P->d_G.p, nm * P->nc, ni, nm * P->nc, true, oz_tile_n(ni));
    } else {
      tc_setup(P);
    }
    EPSP_CUDA(cudaStreamSynchronize(s));
  } else {
    fail(EPSP_EINVAL, "unknown path");
  }
  if (P->path != EPSP_PATH_GEMM_BF16) {
    P->ozKK.keep(ctx, P->d_KK.p, P->nw, P->nw, P->nw, false, kOzBoxM);
    EPSP_CUDA(cudaStreamSynchronize(s));
  }
  plog.mark("cells, tensor-core operands");
  // iteration buffers
  P->d_Sin.alloc(ctx, size_t(P->nw * ni));
  P->d_ImS.alloc(ctx, size_t(P->nw * ni));
  P->d_ReS.alloc(ctx, size_t(P->nw * ni));
  plog.mark("iteration buffers");
  return guard.release();
}

// ---------------------------------------------------------------------------------------------
// one Fan-Migdal sum at one temperature: ImΣ += Σ (src/scgd0_kernel.jl:59-86)
// ---------------------------------------------------------------------------------------------

// With `set`, for which d_ImS need not be zeroed, ImΣ = Σ (the FP64 paths).
void scgd0_imsigma(Scgd0Plan* P, const double2* d_Sin, double mu, double T, double* d_ImS, bool set = false) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  const long nm = P->nm, ni = P->ni, nf = P->nf, nw = P->nw;
  if (P->path == EPSP_PATH_DIRECT_FP64) {
    const long nvf = nm * nf;
    const bool fast = P->fm_fast && T > 1.4901161193847656e-08 && P->wq_max <= 300.0 * T;
    // blocks of up to 16 warps of 32 nodes, as even as they come (a block stages its pairs: about 50 operations each)
    const long nwarp = div_up(size_t(nw), 32);
    const int wpb = int(div_up(size_t(nwarp), div_up(size_t(nwarp), 16)));
    const dim3 tiles(fast ? div_up(size_t(nwarp), size_t(wpb)) : div_up(size_t(nw), kFmTile), unsigned(ni));
    if (fast) {
      const long n = (nw + 1) * ni;
      ensure(P->w_fmtab, ctx, size_t(n));
      launch_after(s, fm_cell_kernel, div_up(size_t(n), 128), 128, 0, P->d_ws.p, int(nw), d_Sin, ni, P->w_fmtab.p);
      EPSP_LAUNCHED(ctx);
    }
    for (long f0 = 0; f0 < nf; f0 += P->nf_chunk) {
      long f1 = std::min(nf, f0 + P->nf_chunk);
      long pi = prof_begin(ctx, "fan_migdal");
      if (fast) {
        // splits of the (ν, f) range: 64 warps a multiprocessor (the FP64 pipes take whole warps, so few of them share out
        // unevenly), 8 pairs a split at least (a thread's own exponential is worth two), 64 splits at most
        const long len = nm * (f1 - f0), want = std::min<long>(64, 64l * ctx->sm_count / (long(tiles.x) * ni * wpb) + 1);
        const long per = std::max<long>(8, (len + want - 1) / want);
        const int splits = int((len + per - 1) / per);
        ensure(P->w_fmpart, ctx, size_t(nw * ni * splits));
        launch_after(s, fm_direct_fast_kernel, dim3(tiles.x, tiles.y, unsigned(splits)), 32 * wpb, 0,
            P->d_ws.p, int(nw), P->d_wkey.p, P->d_jtab.p, int(P->d_jtab.n), float(P->ct.x0), float(P->ct.inv_h),
            P->fm_guard, P->w_fmtab.p, P->d_g2t.p, P->d_wqt.p, nvf, P->d_eps_f.p, P->d_w_f.p, P->d_f_to_i.p, int(nm),
            nm * f0, nm * f1, per, mu, T, 1.0 / T, P->w_ac, P->w_fmpart.p);
        EPSP_LAUNCHED(ctx);
        launch_after(s, fm_add_kernel, div_up(size_t(nw * ni), 32), 256, 0, P->w_fmpart.p, nw * ni, splits, d_ImS, set && f0 == 0);
      } else {
        if (set && f0 == 0) EPSP_CUDA(cudaMemsetAsync(d_ImS, 0, size_t(nw * ni) * sizeof(double), s));
        fm_direct_kernel<<<tiles, kFmTile, 0, s>>>(P->d_ws.p, int(nw), P->ct, d_Sin, P->d_g2t.p, P->d_wqt.p, nvf,
                                                   P->d_eps_f.p, P->d_w_f.p, P->d_f_to_i.p, int(nm), nm * f0, nm * f1, mu,
                                                   T, P->w_ac, d_ImS);
      }
      EPSP_LAUNCHED(ctx);
      prof_end(ctx, pi);
    }
    return;
  }
  if (P->disp) {
    tc_imsigma_disp(P, d_Sin, mu, T, d_ImS);
    return;
  }
  launch_after(s, occ_table_kernel, div_up(size_t(nw * nm), 32), 32, 0, P->d_ws.p, int(nw), P->d_wnu.p, int(nm), mu, T, P->w_ac,
                                                                 P->d_Fa.p, P->d_Fe.p);
  EPSP_LAUNCHED(ctx);
  const long nk = nm * P->nc;
  if (P->path == EPSP_PATH_GEMM_FP64) {
    long pk = prof_begin(ctx, "kbuild");
    ensure(P->w_fmtab, ctx, size_t((nw + 1) * ni));
    launch_after(s, fm_cell_kernel, div_up(size_t((nw + 1) * ni), 128), 128, 0, P->d_ws.p, int(nw), d_Sin, ni, P->w_fmtab.p);
    EPSP_LAUNCHED(ctx);
    launch_after(s, kbuild_f64_kernel, dim3(div_up(size_t(nw), 128), unsigned(nk)), 128, 0,
        int(nw), P->w_fmtab.p, P->d_cell_j.p, P->d_cell_t.p, P->d_wnu.p, int(nm), P->d_epsc.p, P->d_colc.p, P->d_Fa.p,
        P->d_Fe.p, P->w_ac, P->d_Kt.p);
    EPSP_LAUNCHED(ctx);
    prof_end(ctx, pk);
    long pg = prof_begin(ctx, "fm_gemm");
    // ImΣ[ω, i] += Σ_k K_t[ω, k] G[k, i]
    oz_gemm(ctx, P->oz, nw, ni, nk, P->d_Kt.p, nw, nullptr, P->d_G.p, nk, &P->ozG, set ? 0.0 : 1.0, d_ImS, nw);
    prof_end(ctx, pg);
    return;
  }
  tc_imsigma(P, d_Sin, d_ImS);
}

// ---------------------------------------------------------------------------------------------
// the iteration (src/scgd0.jl:246-346)
// ---------------------------------------------------------------------------------------------

// The iteration. With `warm`, the network corrects Σ of every still-active temperature after the
// first iteration (the G0D0 one), with coupling scale warm_scale[iT]; the iterations that follow
// compare against the corrected Σ, as a run started from Σ_init = G0D0 + correction would.
void scgd0_run(Scgd0Plan* P, const epsp_occ* occ, const double* eta_min, double eta_init, int32_t maxiter, double tol,
               int32_t fix_mu, const double* mu_start, const double* sigma_init, double* sigma_out, double* mu_out,
               uint8_t* converged, epsp_scgd0_history* hist, epsp_warmstart* warm = nullptr,
               const double* warm_scale = nullptr) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  if (!occ || !occ->Tlist || (!occ->nlist && !fix_mu)) fail(EPSP_EINVAL, "occ is incomplete");
  if (maxiter < 1) fail(EPSP_EINVAL, "maxiter must be at least 1, got " + std::to_string(maxiter));
  const int64_t nT = occ->nT;
  if (nT < 1) fail(EPSP_EINVAL, "at least one temperature");
  // sigma_out may be NULL: Σ then stays on the device (epsp_scgd0_sigma_device)
  if (!eta_min || !mu_start || !mu_out || !converged || !hist || !hist->err || !hist->mu ||
      !hist->min_spectral_weight || !hist->wall || !hist->iter_frozen)
    fail(EPSP_EINVAL, "an output or input array is NULL");
  for (int64_t iT = 0; iT < nT; ++iT)
    if (!(occ->Tlist[iT] >= 0)) fail(EPSP_EINVAL, "Temperature must be positive");
  const long nw = P->nw, ni = P->ni, nwa = P->nwa;
  const long slab = nw * ni;
  if (sigma_init)
    for (long k = 0; k < 2 * slab * nT; ++k)
      if (!std::isfinite(sigma_init[k])) fail(EPSP_EINVAL, "Sigma_init must be finite");
  // From here the plan's Σ is this run's: none until the run has succeeded. A run that fails waits for what it has
  // launched (an iteration may be in flight behind the one that failed), so that nothing writes after the call.
  P->sigma_nT = 0;
  struct Drain {
    cudaStream_t s;
    bool on = true;
    ~Drain() {
      if (on) cudaStreamSynchronize(s);
    }
  } drain{s};
  DBuf<double2>& S = P->w_S;
  DBuf<double2>& Snew = P->w_Snew;
  if (ensure(S, ctx, size_t(slab * nT))) ++P->w_gen;
  if (ensure(Snew, ctx, size_t(slab * nT))) ++P->w_gen;
  if (sigma_init) {
    long pu = prof_begin(ctx, "scgd0_io");
    S.upload(reinterpret_cast<const double2*>(sigma_init), size_t(slab * nT), s);
    prof_end(ctx, pu);
    EPSP_CUDA(cudaMemcpyAsync(Snew.p, S.p, size_t(slab * nT) * sizeof(double2), cudaMemcpyDeviceToDevice, s));
  } else {
    fill_start_kernel<<<div_up(size_t(slab * nT), 256), 256, 0, s>>>(S.p, Snew.p, slab * nT, eta_init);
    EPSP_LAUNCHED(ctx);
  }
  std::vector<double> mu(mu_start, mu_start + nT);
  std::vector<char> active(static_cast<size_t>(nT), 1);
  const double nan = std::numeric_limits<double>::quiet_NaN();
  for (int64_t k = 0; k < nT * maxiter; ++k) hist->err[k] = hist->mu[k] = hist->min_spectral_weight[k] = nan;
  for (int32_t k = 0; k < maxiter; ++k) hist->wall[k] = 0;
  for (int64_t k = 0; k < nT; ++k) hist->iter_frozen[k] = 0;
  const double br0 = P->wsa.nodes.front() - 0.1, br1 = P->wsa.nodes.back() + 0.1;  // src/scgd0.jl:197
  // the per-iteration results in one buffer (one copy back per iteration): err bits [nT], μ [nT],
  // min ∫A [nT], μ status [nT] and evaluations [nT] (ints, in nT doubles), the tensor-core wait flag
  const size_t npack = size_t(4 * nT + 1);
  DBuf<double>& d_pack = P->w_pack;
  if (ensure(d_pack, ctx, npack)) ++P->w_gen;
  d_pack.zero(s);
  auto* d_err = reinterpret_cast<unsigned long long*>(d_pack.p);
  double* d_mu = d_pack.p + nT;
  double* d_minA = d_pack.p + 2 * nT;
  int* d_status = reinterpret_cast<int*>(d_pack.p + 3 * nT);
  int* d_evals = d_status + nT;
  int* d_tcerr = reinterpret_cast<int*>(d_pack.p + 4 * nT);
  // host side of the readback and of the slot list: pinned
  P->h_pin.ensure(2 * npack * sizeof(double) + size_t(nT) * sizeof(int));
  double* h_packs[2] = {static_cast<double*>(P->h_pin.p), static_cast<double*>(P->h_pin.p) + npack};
  int* h_slots = reinterpret_cast<int*>(h_packs[1] + npack);
  for (auto& e : P->read_ev)
    if (!e) EPSP_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  std::vector<int> up_slots;  // the slot list on the device (uploaded when it changes)
  int32_t niter = 0;
  const unsigned eb = div_up(size_t(slab), 256);
  // Every active temperature of an iteration is processed by the same launches (slot a ->
  // temperature slots[a]); per-temperature T, μ, η_min, target and branch live on the device.
  DBuf<int>& d_slots = P->w_slots;
  DBuf<TParams>& d_tp = P->w_tp;
  DBuf<double2>& Sin_b = P->w_Sin;
  DBuf<double>& A_b = P->w_A;
  DBuf<double>& colsum_b = P->w_colsum;
  DBuf<double>& D_b = P->w_D;
  bool grown = false;
  grown |= ensure(d_slots, ctx, size_t(nT));
  grown |= ensure(P->w_ctl, ctx, 1);
  grown |= ensure(d_tp, ctx, size_t(nT));
  if (P->path != EPSP_PATH_GEMM_BF16) grown |= ensure(Sin_b, ctx, size_t(slab * nT));  // the tensor-core path clamps into FP32
  const bool f32_spec = P->path == EPSP_PATH_GEMM_BF16;
  const int spec_nab = int(div_up(size_t(nwa), f32_spec ? kSpecNodes : 32)), spec_nch = int(div_up(size_t(ni), size_t(kSpecChunk)));
  if (f32_spec) {
    grown |= ensure(P->w_Pf, ctx, size_t(slab * nT));
    grown |= ensure(P->w_Dpart, ctx, size_t(long(spec_nch) * nwa * nT));
    grown |= ensure(P->w_Cpart, ctx, size_t(long(spec_nab) * ni * nT));
  } else {
    grown |= ensure(A_b, ctx, size_t(nwa * ni * nT));
    grown |= ensure(colsum_b, ctx, size_t(ni * nT));
  }
  grown |= ensure(D_b, ctx, size_t(nwa * nT));
  grown |= ensure(P->w_E, ctx, size_t(nwa * nT));
  grown |= ensure(P->w_R1, ctx, size_t(kMuTerms * spec_nab * nT));
  grown |= ensure(P->w_ends, ctx, size_t(2 * nwa * nT));
  if (P->path == EPSP_PATH_GEMM_BF16) {
    const long cap0 = tc_capacity(P);
    tc_reserve(P, nT);
    grown |= tc_capacity(P) != cap0;
    tc_disp_choose(P, occ->Tlist, nT);
  }
  if (grown) ++P->w_gen;
  std::vector<TParams> h_tp(static_cast<size_t>(nT));
  std::vector<int> slots;
  // CUDA graph of the iteration body (tensor-core path; not while one of its kernels is profiled)
  static const char* kBodyProfiles[] = {"kprep", "kbuild", "tc_fm", "tc_kk", "finalize", "kk_epilogue", "spectral", "mu", "fm_disp"};
  bool use_graph = P->path == EPSP_PATH_GEMM_BF16;
  for (const char* nm : kBodyProfiles)
    if (ctx->prof_name == nm) use_graph = false;
  // a replayed graph bakes in the buffers, nT, fix_mu, the spin degeneracy, the active count and the choice of the
  // dispersive kernel
  auto graph_key = [&](int nA) {
    return std::array<long, 6>{long(nA), long(nT), long(fix_mu), P->w_gen,
                               long(std::llround(occ->spin_degeneracy * 1e6)), long(P->path) + 16 * long(P->fd_fast)};
  };
  // An iteration is launched before the host has read the one before it (IterCtl; the tensor-core path without
  // dispersive modes, whose iterations take about as long as the round trip): the round trips run beside the iterations,
  // and only the last one of a set of active temperatures waits, with one iteration after it that does nothing.
  IterCtl* ctl = P->path == EPSP_PATH_GEMM_BF16 && !P->disp ? P->w_ctl.p : nullptr;
  auto reset_ctl = [&] {
    const IterCtl c{tol, 0, 0};
    P->w_ctl.upload(&c, 1, s);
  };
  auto launch_iteration = [&](int32_t iter) {
    slots.clear();
    for (int64_t iT = 0; iT < nT; ++iT) {
      if (!active[size_t(iT)]) continue;
      slots.push_back(int(iT));
      TParams& q = h_tp[size_t(iT)];
      q.T = occ->Tlist[iT];
      q.inv_T = 1.0 / q.T;
      q.mu = mu[size_t(iT)];
      q.eta_min = eta_min[iT];
      q.holes = (!fix_mu && occ->type == EPSP_SEMICONDUCTOR && occ->nlist[iT] < 0) ? 1 : 0;
      q.n_target = fix_mu ? 0.0 : occ->nlist[iT] + occ->nelec;
      q.pad = 0;
    }
    const int nA = int(slots.size());
    if (slots != up_slots) {
      std::copy(slots.begin(), slots.end(), h_slots);
      EPSP_CUDA(cudaMemcpyAsync(d_slots.p, h_slots, slots.size() * sizeof(int), cudaMemcpyHostToDevice, s));
      up_slots = slots;
      if (ctl) reset_ctl();
    }
    // T, η_min, target and branch are fixed for the run; μ is written on the device by the μ solve
    if (iter == 1) {
      d_tp.upload(h_tp.data(), h_tp.size(), s);
      if (!fix_mu) {
        mu_ends_kernel<<<dim3(div_up(size_t(nwa), 64), unsigned(nT)), 64, 0, s>>>(P->d_wsa.p, int(nwa), d_tp.p, br0, br1,
                                                                              P->w_ends.p);
        EPSP_LAUNCHED(ctx);
      }
    }
    // the tensor-core path's form of the clamped Σ: made here for the first iteration and after the network's
    // correction, by each iteration's last pass for the next
    if (P->path == EPSP_PATH_GEMM_BF16) {
      if (iter == 1) tc_start(P, nT, d_tp.p);
      if (iter == 1 || (warm && iter == 2)) tc_take_sigma(P, nA, d_slots.p, d_tp.p, S.p);
    }
    // the launches of one iteration; on the tensor-core path they are captured once per active set
    // into a CUDA graph and replayed (μ, T come from the device, so a replay sees the current ones)
    auto body = [&] {
      MuIn mu_in;
      mu_in.ends = fix_mu ? nullptr : P->w_ends.p;
      mu_in.tp = d_tp.p;
      mu_in.br0 = br0;
      mu_in.br1 = br1;
      mu_in.E = P->w_E.p;
      mu_in.part = P->w_R1.p;
      if (P->path == EPSP_PATH_GEMM_BF16 && P->disp) EPSP_CUDA(cudaMemsetAsync(d_err, 0, size_t(nT) * 8, s));
      if (P->path != EPSP_PATH_GEMM_BF16) {
        launch_after(s, clamp_kernel, dim3(eb, unsigned(nA)), 256, 0, S.p, Sin_b.p, slab, d_slots.p, d_tp.p, d_err);
        EPSP_LAUNCHED(ctx);
      }
      if (P->path == EPSP_PATH_GEMM_BF16) {
        // Σ_new, its multiplet average, max|ΔΣ|, Σ ← Σ_new and the spectral terms from the
        // Kramers-Kronig product's epilogue (so no multiplet, spectral-prep or err/copy pass below)
        tc_iterate(P, nA, d_slots.p, d_tp.p, S.p, P->w_Pf.p, d_err, d_minA, ctl);
      } else {
        for (int a = 0; a < nA; ++a) {
          const int64_t iT = slots[size_t(a)];
          scgd0_imsigma(P, Sin_b.p + slab * a, mu[size_t(iT)], occ->Tlist[iT], P->d_ImS.p, true);
          long pk = prof_begin(ctx, "kk");
          oz_gemm(ctx, P->oz, nw, ni, nw, P->d_KK.p, nw, &P->ozKK, P->d_ImS.p, nw, nullptr, 0.0, P->d_ReS.p, nw);
          const bool last = P->nmult == 0;  // no multiplet average to come: max |ΔΣ| and Σ ← Σ_new in the same pass
          launch_after(s, assemble_kernel, eb, 256, 0, P->d_ReS.p, P->d_ImS.p, Snew.p + slab * iT, slab,
                                             last ? S.p + slab * iT : nullptr, d_err + iT, P->oz.err.p, d_tcerr);
          EPSP_LAUNCHED(ctx);
          prof_end(ctx, pk);
        }
      }
      if (P->nmult > 0 && !f32_spec) {
        launch_after(s, multiplet_kernel, dim3(div_up(size_t(nw * P->nmult), 256), unsigned(nA)), 256, 0,
            Snew.p, int(nw), slab, d_slots.p, P->d_mptr.p, P->d_midx.p, P->nmult);
        EPSP_LAUNCHED(ctx);
      }
      long psp = prof_begin(ctx, "spectral");
      if (f32_spec) {  // the per-node terms came from the Kramers-Kronig epilogue
        launch_after(s, spectral_ad_f32_kernel, dim3(unsigned(spec_nab), unsigned(spec_nch), unsigned(nA)), kSpecNodes, 0,
                     P->w_Pf.p, int(nw), slab, P->d_jsp.p, P->d_dspf.p, P->d_tspf.p, P->d_Waf.p, P->d_w_if.p, int(nwa),
                     int(ni), P->w_Dpart.p, P->w_Cpart.p, ctl);
        EPSP_LAUNCHED(ctx);
        launch_after(s, spectral_fin_f32_kernel, dim3(unsigned(spec_nab + div_up(size_t(ni), 2)), unsigned(nA)), kSpecNodes,
                     0, P->w_Dpart.p, P->w_Cpart.p, spec_nch, spec_nab, P->d_Wa.p, P->d_wsa.p, int(nwa), int(ni), d_slots.p,
                     D_b.p, d_minA, mu_in, tc_err_ptr(P), d_tcerr, d_err, ctl);
        EPSP_LAUNCHED(ctx);
      } else {
        launch_after(s, spectral_A_kernel, dim3(div_up(size_t(nwa), 256), unsigned(ni), unsigned(nA)), 256, 0,
            Snew.p, int(nw), slab, d_slots.p, P->d_wsa.p, int(nwa), P->d_jsp.p, P->d_tsp.p, P->d_eps_i.p, A_b.p, int(ni));
        EPSP_LAUNCHED(ctx);
        launch_after(s, spectral_colsum_kernel, dim3(unsigned(ni), unsigned(nA)), 256, 0, A_b.p, int(nwa), int(ni), P->d_Wa.p,
                                                                              colsum_b.p);
        EPSP_LAUNCHED(ctx);
        launch_after(s, min_kernel, unsigned(nA), 256, 0, colsum_b.p, int(ni), d_slots.p, d_minA);
        EPSP_LAUNCHED(ctx);
        if (!fix_mu) {
          launch_after(s, spectral_D_kernel, dim3(unsigned(spec_nab), unsigned(nA)), 256, 0,
              A_b.p, int(nwa), int(ni), P->d_w_i.p, P->d_Wa.p, P->d_wsa.p, d_slots.p, D_b.p, mu_in);
          EPSP_LAUNCHED(ctx);
        }
      }
      prof_end(ctx, psp);
      if (!fix_mu) {
        long pm = prof_begin(ctx, "mu");
        launch_after(s, mu_solve_kernel, unsigned(kMuCluster * nA), kMuThreads, 0, D_b.p, P->d_wsa.p, int(nwa), d_slots.p,
                     d_tp.p, P->W, P->nstates_base, occ->spin_degeneracy, br0, br1, P->w_E.p, P->w_R1.p, spec_nab, d_mu,
                     d_status, d_evals, ctl);
        EPSP_LAUNCHED(ctx);
        prof_end(ctx, pm);
      }
      if (P->path != EPSP_PATH_GEMM_BF16 && P->nmult > 0) {  // (the tensor-core epilogue took err and the copy)
        launch_after(s, err_copy_kernel, dim3(eb, unsigned(nA)), 256, 0, Snew.p, S.p, slab, d_slots.p, d_err);
        EPSP_LAUNCHED(ctx);
      }
    };
    // iteration 1 replays a graph a previous run captured with the same key; otherwise it runs
    // eagerly (first launches set kernel attributes) and iteration 2 captures
    const auto key = graph_key(nA);
    auto have = std::find_if(P->graphs.begin(), P->graphs.end(), [&](const auto& g) { return g.key == key; });
    if (use_graph && (iter > 1 || have != P->graphs.end())) {
      if (have == P->graphs.end()) {
        const int64_t l0 = ctx->launches;
        cudaGraph_t g = nullptr;
        EPSP_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        try {
          body();
        } catch (...) {
          cudaStreamEndCapture(s, &g);
          if (g) cudaGraphDestroy(g);
          throw;
        }
        EPSP_CUDA(cudaStreamEndCapture(s, &g));
        cudaGraphExec_t exec = nullptr;
        cudaError_t ie = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
        EPSP_CUDA(ie);
        while (P->graphs.size() >= Scgd0Plan::kGraphs) {
          cudaGraphExecDestroy(P->graphs.back().exec);
          P->graphs.pop_back();
        }
        P->graphs.insert(P->graphs.begin(), {key, exec, long(ctx->launches - l0)});
        ctx->launches = l0;
      } else if (have != P->graphs.begin()) {
        std::rotate(P->graphs.begin(), have, have + 1);
      }
      EPSP_CUDA(cudaGraphLaunch(P->graphs.front().exec, s));
      ctx->launches += P->graphs.front().launches;
    } else {
      body();
    }
    EPSP_CUDA(cudaMemcpyAsync(h_packs[iter & 1], d_pack.p, npack * sizeof(double), cudaMemcpyDeviceToHost, s));
    EPSP_CUDA(cudaEventRecord(P->read_ev[iter & 1], s));
  };
  int32_t launched = 0;
  auto t0 = std::chrono::steady_clock::now();
  for (int32_t iter = 1; iter <= maxiter; ++iter) {
    if (launched < iter) launch_iteration(iter);
    launched = iter;
    if (ctl && iter < maxiter && !(warm && iter == 1)) {
      launch_iteration(iter + 1);
      launched = iter + 1;
    }
    EPSP_CUDA(cudaEventSynchronize(P->read_ev[iter & 1]));
    const double* h_pack = h_packs[iter & 1];
    {
      int tcerr = 0;
      std::memcpy(&tcerr, &h_pack[size_t(4 * nT)], sizeof(int));
      if (tcerr) {
        int* flag = P->path == EPSP_PATH_GEMM_BF16 ? tc_err_ptr(P) : P->oz.err.p;
        EPSP_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), s));  // the plan's next run starts clean
        fail(EPSP_EDEVICE_TIMEOUT, "a tensor-core GEMM wait ran out (bounded device wait)");
      }
    }
    const auto* h_err = reinterpret_cast<const unsigned long long*>(h_pack);
    const double* h_mu = h_pack + nT;
    const double* h_minA = h_pack + 2 * nT;
    const auto* h_status = reinterpret_cast<const int*>(h_pack + 3 * nT);
    for (int64_t iT = 0; iT < nT; ++iT) {
      if (!active[size_t(iT)]) continue;
      hist->min_spectral_weight[iT + nT * (iter - 1)] = h_minA[size_t(iT)];
      if (!fix_mu) {
        if (h_status[size_t(iT)] != 0) {
          char buf[400];
          std::snprintf(buf, sizeof buf,
                        "no chemical potential in (%g, %g) gives %g electrons per cell at T = %g: the window holds too "
                        "few states on one side of the gap, or the spectral weight it loses outside omegas_spectral "
                        "moves the count past the target. Pass mu_start with fix_mu, or widen the window or omegas.",
                        br0, br1, occ->nlist[iT] + occ->nelec, occ->Tlist[iT]);
          fail(EPSP_ENOROOT_MU, buf);
        }
        mu[size_t(iT)] = h_mu[size_t(iT)];
      }
      double err;
      std::memcpy(&err, &h_err[size_t(iT)], 8);
      hist->err[iT + nT * (iter - 1)] = err;
      hist->mu[iT + nT * (iter - 1)] = mu[size_t(iT)];
      if (err < tol) {
        active[size_t(iT)] = 0;
        hist->iter_frozen[iT] = iter;
        launched = iter;  // the next iteration, if it was launched, stops itself
      }
      if (P->verbosity >= 2)
        std::fprintf(stderr, "scgd0 iteration %d, T = %.6g: err = %.3e, mu = %.15g, mu evaluations %d\n", int(iter),
                     occ->Tlist[iT], err, mu[size_t(iT)], fix_mu ? 0 : h_status[size_t(nT + iT)]);
    }
    if (warm && iter == 1 && iter < maxiter)
      for (int64_t iT = 0; iT < nT; ++iT)
        if (active[size_t(iT)])
          warmstart_correct(warm, ctx, S.p + slab * iT, nw, ni, P->d_eps_i.p, occ->Tlist[iT], mu[size_t(iT)],
                            warm_scale[iT], P->path == EPSP_PATH_GEMM_BF16 ? tc_err_ptr(P) : nullptr);
    const auto now = std::chrono::steady_clock::now();
    hist->wall[iter - 1] = std::chrono::duration<double>(now - t0).count();
    t0 = now;
    niter = iter;
    if (std::none_of(active.begin(), active.end(), [](char a) { return a != 0; })) break;
  }
  hist->niter = niter;
  long pd = prof_begin(ctx, "scgd0_io");
  if (sigma_out) S.download(reinterpret_cast<double2*>(sigma_out), size_t(slab * nT), s);
  prof_end(ctx, pd);
  EPSP_CUDA(cudaStreamSynchronize(s));
  drain.on = false;
  P->sigma_nT = nT;
  for (int64_t iT = 0; iT < nT; ++iT) {
    mu_out[iT] = mu[size_t(iT)];
    converged[iT] = active[size_t(iT)] ? 0 : 1;
  }
}

}  // namespace epsp

using namespace epsp;

template <class F>
static epsp_status guarded(Ctx* c, F&& f) {
  try {
    EPSP_CUDA(cudaSetDevice(c->device));
    f();
    c->last_error.clear();
    return EPSP_OK;
  } catch (const Error& e) {
    c->last_error = e.msg;
    return epsp_status(e.code);
  } catch (const std::bad_alloc&) {
    c->last_error = "host allocation failed";
    return EPSP_ENOMEM;
  } catch (const std::exception& e) {
    c->last_error = e.what();
    return EPSP_EINVAL;
  }
}

extern "C" {

epsp_status epsp_scgd0_setup(epsp_ctx* ctx, const epsp_model* model, const epsp_options* opts, epsp_scgd0_plan** plan) {
  if (!ctx || !plan) return EPSP_EINVAL;
  *plan = nullptr;
  return guarded(&ctx->c, [&] { *plan = reinterpret_cast<epsp_scgd0_plan*>(scgd0_setup(&ctx->c, model, opts)); });
}

void epsp_scgd0_plan_destroy(epsp_scgd0_plan* plan) {
  if (!plan) return;
  auto* P = reinterpret_cast<Scgd0Plan*>(plan);
  cudaSetDevice(P->ctx->device);
  delete P;
}

epsp_status epsp_scgd0_run(epsp_scgd0_plan* plan, const epsp_occ* occ, const double* eta_min, double eta_init,
                           int32_t maxiter, double tol, int32_t fix_mu, const double* mu_start, const double* sigma_init,
                           double* sigma_out, double* mu_out, uint8_t* converged, epsp_scgd0_history* hist) {
  if (!plan) return EPSP_EINVAL;
  auto* P = reinterpret_cast<Scgd0Plan*>(plan);
  return guarded(P->ctx, [&] {
    scgd0_run(P, occ, eta_min, eta_init, maxiter, tol, fix_mu, mu_start, sigma_init, sigma_out, mu_out, converged, hist);
  });
}

epsp_status epsp_scgd0_run_warm(epsp_scgd0_plan* plan, epsp_warmstart* net, const double* coupling_scale,
                                const epsp_occ* occ, const double* eta_min, double eta_init, int32_t maxiter, double tol,
                                int32_t fix_mu, const double* mu_start, double* sigma_out, double* mu_out,
                                uint8_t* converged, epsp_scgd0_history* hist, int32_t* iters_total, int32_t* fallback) {
  if (!plan || !net || !coupling_scale || !iters_total || !fallback) return EPSP_EINVAL;
  auto* P = reinterpret_cast<Scgd0Plan*>(plan);
  return guarded(P->ctx, [&] {
    scgd0_run(P, occ, eta_min, eta_init, maxiter, tol, fix_mu, mu_start, nullptr, sigma_out, mu_out, converged, hist,
              net, coupling_scale);
    *iters_total = hist->niter;
    *fallback = 0;
    bool all = true;
    for (int64_t iT = 0; iT < occ->nT; ++iT) all = all && converged[iT];
    if (!all) {  // the plain start decides
      const int32_t used = hist->niter;
      scgd0_run(P, occ, eta_min, eta_init, maxiter, tol, fix_mu, mu_start, nullptr, sigma_out, mu_out, converged, hist);
      *iters_total = used + hist->niter;
      *fallback = 1;
    }
  });
}

epsp_status epsp_scgd0_sigma_device(const epsp_scgd0_plan* plan, const double** sigma_dev, int64_t* nT) {
  if (!plan || !sigma_dev) return EPSP_EINVAL;
  auto* P = reinterpret_cast<const Scgd0Plan*>(plan);
  if (P->sigma_nT < 1) return EPSP_EINVAL;  // no run yet
  *sigma_dev = reinterpret_cast<const double*>(P->w_S.p);
  if (nT) *nT = P->sigma_nT;
  return EPSP_OK;
}

epsp_status epsp_scgd0_imsigma(epsp_scgd0_plan* plan, const double* sigma_in, double mu, double T, double* imsigma) {
  if (!plan || !sigma_in || !imsigma) return EPSP_EINVAL;
  auto* P = reinterpret_cast<Scgd0Plan*>(plan);
  return guarded(P->ctx, [&] {
    if (!(T >= 0)) fail(EPSP_EINVAL, "Temperature must be positive");
    cudaStream_t s = P->ctx->stream;
    const size_t n = size_t(P->nw * P->ni);
    P->d_Sin.upload(reinterpret_cast<const double2*>(sigma_in), n, s);
    P->d_ImS.upload(imsigma, n, s);
    scgd0_imsigma(P, P->d_Sin.p, mu, T, P->d_ImS.p);
    oz_check(P->ctx, P->oz);
    P->d_ImS.download(imsigma, n, s);
    EPSP_CUDA(cudaStreamSynchronize(s));
  });
}

}  // extern "C"
