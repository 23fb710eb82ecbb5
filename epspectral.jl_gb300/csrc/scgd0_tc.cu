// scgd0_tc.cu -- the GEMM_BF16 path of the scGD0 iteration: the kernel tensor written directly as
// BF16 split operands, the Fan-Migdal contraction and the Kramers-Kronig map on the tcgen05 tensor
// cores (tc_gemm.cuh), split-K partials summed in fixed order.
//
//   ImΣ[ω, i] = Σ_k K_t[ω, k] G[k, i]      A = K_t  [nω][Kp]  (K-major),  B = G^T [ni][Kp]
//   ReΣ[ω, i] = Σ_ω' KK[ω, ω'] ImΣ[ω', i]   A = KK   [nω][Kp2],           B = ImΣ^T [ni][Kp2]
//
// Both contractions use the three-way split (x = hi + mid + lo, six products, ~2^-23 relative): the
// iteration's own convergence test compares successive Σ to tol (1e-6 eV for the benchmark), and a
// two-way split's ~2^-16 rounding of the map (~2e-6 eV here) would stall it above that.
#include "scgd0.cuh"
#include "fp_pair.cuh"
#include "tc_gemm.cuh"

#include <algorithm>
#include <limits>
#include <numeric>

namespace epsp {

constexpr int kNs = 3;
// K-blocks of 64 summed by one FP32 accumulator at most: the Fan-Migdal sums are long and of one
// sign, and their FP32 rounding must stay well below the iteration's tol (1e-6 eV)
constexpr int kKbCap = 16;
// The Kramers-Kronig product's bound: its terms cancel (principal value), so the FP32 rounding of
// a long accumulation is large against the result (at 4101 nodes and 800 K, 16 K blocks per
// accumulator left |ΔReΣ| ~1e-5 eV against FP64, 4 K blocks ~3x less).
constexpr int kKbCapKK = 4;
// Split limit of a product of depth K: enough splits that no FP32 accumulator sums more than cap
// K blocks (the Fan-Migdal product of a 32^3 model has ~680), and at least 16.
static int max_splits_for(long K, int cap = kKbCap) {
  const long kb = (K + kTcBK - 1) / kTcBK;
  return int(std::max<long>(16, (kb + cap - 1) / cap));
}

struct Scgd0Plan::Tc {
  long Kp = 0, Kp2 = 0;
  int splits1 = 1, splits2 = 1, bn1 = 128, bn2 = 128;
  DBuf<__nv_bfloat16> Kt[kNs], G[kNs], KK[kNs], Im[kNs];
  DBuf<float> part;
  DBuf<int> err;
  TcOperand opK, opG, opKK, opIm;
  // FP32 forms of the K-tensor inputs: distances from the cells' nodes, the cell energies as pairs, the occupation
  // tables; per temperature the columns' cell records (rec, dim; kbuild_bf16_kernel) or, with dispersive modes, Σ_in as
  // {Re hi, Re lo, Im, 0}; ε_i as pairs, and the modes' exp(ω_ν/T) and n of the run's temperatures
  DBuf<float2> ef, epair, tf;
  DBuf<float> Ff, dim;
  DBuf<float4> Sf, rec;
  DBuf<double2> modes;
  // dispersive modes: cell records and Im slopes of every column and slot, partial sums of the splits
  DBuf<float4> fdrec;
  DBuf<float> fddim;
  DBuf<double> fdpart;
  // 1 for modes below the acoustic cutoff (left out of the sum)
  DBuf<uint8_t> skip;
  // batched iteration: capacity in temperatures, ImΣ of every slot
  long capT = 1;
  DBuf<double> ImS_b;
};

__global__ void split_df_kernel(const double* __restrict__ x, long n, float2* __restrict__ out) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) out[k] = split_df(x[k]);
}

// gw[vf + nvf i] = w_f[f] g2t[vf + nvf i] rounded to FP32 (vf = ν + nm f).
__global__ void gw_f32_kernel(const double* __restrict__ g2t, const double* __restrict__ w_f, int nm, long nvf, long ni,
                              float* __restrict__ gw) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= nvf * ni) return;
  gw[k] = float(w_f[(k % nvf) / nm] * g2t[k]);
}

// Pairs with high parts on the plan's quantum (split_q).
__global__ void split_q_kernel(const double* __restrict__ x, long n, double qm, float2* __restrict__ out) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) out[k] = split_q(x[k], qm);
}

__global__ void to_f32_kernel(const double* __restrict__ x, long n, float* __restrict__ out) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) out[k] = float(x[k]);
}

// Σ_s part[s stride] in ascending s.
__device__ __forceinline__ float sum_splits(const float* __restrict__ part, int splits, long stride) {
  float acc = 0.f;
#pragma unroll 4
  for (int p = 0; p < splits; ++p) acc += part[stride * p];
  return acc;
}

// One node's Σ as FP32: Re as a pair, Im. Cell j of a column from its nodes' values z (node j) and zn (node j + 1):
// {ω_j - ReΣ_j as a pair (U), -ReΣ', ImΣ_j} and ImΣ' (Im clamped at -η_min = etam), so that at x = ω_j + dx
//   Re z = ((U_hi - ε_hi) + dx_hi) + ((U_lo - ε_lo) + dx_lo - dx ReΣ'),  Im Σ = ImΣ_j + dx ImΣ'.
// The high parts are multiples of one quantum (split_q; qm = 1.5 2^23 times it), so the first bracket is exact and Re z
// keeps its distance to a pole wherever in a cell it lies (dx as one FP32 number, times 1 - ReΣ', moved elements by up to
// 2^-26 dx over the pole's width: 1e-6 relative for 0.1 eV and 1e-3 eV). wj: {ω_j hi, lo, 1 / (ω_{j+1} - ω_j) (0 at the
// last node, whose cell is the flat part above the grid), ..}.
__device__ __forceinline__ float4 cell_record(float4 z, float4 zn, float4 wj, float etam, float qm, float& dim) {
  float e;
  const float s = two_sum(wj.x, -z.x, e);
  const float h = (s + qm) - qm;
  const float im = fminf(z.z, etam);
  dim = (fminf(zn.z, etam) - im) * wj.z;
  return make_float4(h, (s - h) + (e + (wj.y - z.y)), ((z.x - zn.x) + (z.y - zn.y)) * wj.z, im);
}
__device__ __forceinline__ float4 sigma_f32(double2 z) {
  const float2 r = split_df(z.x);
  return make_float4(r.x, r.y, float(z.y), 0.f);
}

// The records of the columns of temperature slots[blockIdx.y] from Σ there, clamped at -η_min: [ni][nω + 1] entries a
// temperature, entry j + 1 cell j, entry 0 the flat part below the grid. Without slots: of one Σ, as it is.
__global__ void cell_records_kernel(const double2* __restrict__ S_all, const int* __restrict__ slots,
                                    const TParams* __restrict__ tp, const float4* __restrict__ wtab, float qm, int nw,
                                    long slab, float4* __restrict__ rec_all, float* __restrict__ dim_all) {
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= slab) return;
  const int t = slots ? slots[blockIdx.y] : 0, j = int(k % nw);
  const double2* S = S_all + slab * t;
  const float etam = slots ? float(-tp[t].eta_min) : INFINITY;
  const float4 z = sigma_f32(S[k]), zn = j + 1 < nw ? sigma_f32(S[k + 1]) : z, wj = wtab[j];
  const long at = (k / nw + slab / nw * t) * (nw + 1l) + j + 1;
  float d;
  rec_all[at] = cell_record(z, zn, wj, etam, qm, d);
  dim_all[at] = d;
  if (j == 0) {
    rec_all[at - 1] = cell_record(z, z, wj, etam, qm, d);
    dim_all[at - 1] = 0.f;
  }
}

// clamp_kernel's Σ_in in FP32 {Re Σ as a float pair, Im Σ, 0} (temperature t at Sf + t n), for the dispersive sum.
__global__ void clamp_f32_kernel(const double2* __restrict__ S, float4* __restrict__ Sf, long n,
                                 const int* __restrict__ slots, const TParams* __restrict__ tp) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int a = blockIdx.y, t = slots[a];
  const double2 z = S[long(t) * n + k];
  const float2 r = split_df(z.x);
  Sf[long(t) * n + k] = make_float4(r.x, r.y, float(fmin(z.y, -tp[t].eta_min)), 0.f);
}

__global__ void sigma_f32_kernel(const double2* __restrict__ S, long n, float4* __restrict__ out) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double2 z = S[k];
  const float2 r = split_df(z.x);
  out[k] = make_float4(r.x, r.y, float(z.y), 0.f);
}

// Kernel tensor of the recast Fan-Migdal sum (see kbuild_f64_kernel in scgd0.cu), written as BF16
// split rows K_t[ω][k], k = c nm + ν, through a shared-memory transpose. Σ(ω ± ω_ν) comes from the columns' cell
// records (cell_record above; the cells and distances from set-up), the reciprocal and the occupation products are
// FP32: the kernel runs on the FP32 units only. Instructions and the latency of its gathers bound it: a side of an element
// is 20 bytes and about 15 instructions, the BF16 parts are formed two elements at a time, and eight blocks are kept on an
// SM (with four 16-byte gathers, two weights and two two-sums a side 54 us at 1251 x 7425; now 38.4, 10.5 at 501 x 1575.
// Two columns in flight spill at eight blocks' 32 registers: 42.5 and 10.0; with seven blocks 42.3, six 46.3; four columns
// and six blocks 40.2 and 10.5).
// Grid (nω / 16, Kp / (kKbCols nm), slots), 256 threads: thread (node ω0 + t % 16, modes t / 16,
// t / 16 + 16, ..) loads the cells and occupations of its (ω, ν) once and runs over the block's
// kKbCols columns c (their records' offset and energy from shared memory). Dynamic shared memory: the tile
// [kKbCols nm][17] floats. kKbCols nm must be a multiple of 8, so that the write-out's 16-byte chunks never
// straddle two blocks (nor Kp, a multiple of 64).
constexpr int kKbCols = 8;
constexpr int kKbW = 16;

__device__ __forceinline__ float rcp_f(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// split_bf16_n of a and b in three parts, each part's two values packed (a in the low half): the packed conversion takes
// both, and a part's value as FP32 is its 16 bits moved up.
__device__ __forceinline__ void split_bf16_pair(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  auto pack = [](float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
  };
  p0 = pack(a, b);
  a -= __uint_as_float(p0 << 16);
  b -= __uint_as_float(p0 & 0xffff0000u);
  p1 = pack(a, b);
  a -= __uint_as_float(p1 << 16);
  b -= __uint_as_float(p1 & 0xffff0000u);
  p2 = pack(a, b);
}

__global__ void __launch_bounds__(256, 8) kbuild_bf16_kernel(int nw, int ni, const float4* __restrict__ rec_all,
                                                          const float* __restrict__ dim_all,
                                                          const int* __restrict__ slots,
                                                          const int32_t* __restrict__ cell_e,
                                                          const float2* __restrict__ cell_dx,
                                                          const uint8_t* __restrict__ skip, int nm,
                                                          const float2* __restrict__ eps_c,
                                                          const int32_t* __restrict__ col_c, int nc,
                                                          const float* __restrict__ F_all,
                                                          __nv_bfloat16* __restrict__ K0, __nv_bfloat16* __restrict__ K1,
                                                          __nv_bfloat16* __restrict__ K2, long Kp,
                                                          const IterCtl* __restrict__ ctl) {
  pdl_wait();
  if (ctl && ctl->stop) return;
  extern __shared__ float kb_tile[];  // [kKbCols nm][kKbW + 1]
  __shared__ float4 s_col[kKbCols];  // ε as a float pair, the records' offset (integer bits)
  const int w0 = blockIdx.x * kKbW;
  const int cbeg = blockIdx.y * kKbCols;
  const int tw = threadIdx.x % kKbW, tm = threadIdx.x / kKbW;
  const int iw = w0 + tw;
  const int nwm = nw * nm;
  const long tab = (nw + 1l) * ni * (slots ? slots[blockIdx.z] : 0);
  const float4* rec = rec_all + tab;
  const float* dim = dim_all + tab;
  const float* F = F_all + 2l * nwm * blockIdx.z;
  if (threadIdx.x < kKbCols) {
    const int c = cbeg + threadIdx.x;
    // (past the last column: |z|² overflows, its reciprocal and the element are 0)
    const float2 e = c < nc ? eps_c[c] : make_float2(-1e25f, 0.f);
    s_col[threadIdx.x] = make_float4(e.x, e.y, __int_as_float(c < nc ? (nw + 1) * col_c[c] : 0), 0.f);
  }
  __syncthreads();
  for (int nu = tm; nu < nm; nu += 256 / kKbW) {
    const bool on = iw < nw && !skip[nu];
    int ea = 0, ee = 0;
    float2 da = make_float2(0.f, 0.f), de = da;
    float Fa = 0.f, Fe = 0.f;
    if (on) {
      const int ia = iw + nw * nu, ie = ia + nwm;
      ea = cell_e[ia];
      ee = cell_e[ie];
      da = cell_dx[ia];
      de = cell_dx[ie];
      Fa = F[ia];
      Fe = F[ie];
    }
#pragma unroll 1
    for (int cl = 0; cl < kKbCols; ++cl) {
      const float4 e = s_col[cl];
      const int ia = __float_as_int(e.z) + ea, ie = __float_as_int(e.z) + ee;
      const float4 A = rec[ia], B = rec[ie];
      const float xa = da.x + da.y, xe = de.x + de.y;
      const float zar = ((A.x - e.x) + da.x) + fmaf(xa, A.z, (A.y - e.y) + da.y), sia = fmaf(xa, dim[ia], A.w);
      const float zer = ((B.x - e.x) + de.x) + fmaf(xe, B.z, (B.y - e.y) + de.y), sie = fmaf(xe, dim[ie], B.w);
      // Im 1/z with Im z = -Im Σ, by an approximate reciprocal (1 ulp): the K tensor carries FP32 precision
      const float ga = sia * rcp_f(fmaf(zar, zar, sia * sia));
      const float ge = sie * rcp_f(fmaf(zer, zer, sie * sie));
      const float v = on ? ga * Fa + ge * Fe : 0.f;
      kb_tile[(cl * nm + nu) * (kKbW + 1) + tw] = v;
    }
  }
  __syncthreads();
  // write-out: the block's columns [cbeg nm, (cbeg + kKbCols) nm) of rows ω0.., 8 BF16 per store; a
  // half-warp writes one row's chunks (contiguous)
  const long kbeg = long(cbeg) * nm;
  const int nchunk = kKbCols * nm / 8;
  const long krow0 = long(nw) * blockIdx.z;
  for (int wr = threadIdx.x / 16; wr < kKbW; wr += 16) {
    for (int ch = threadIdx.x % 16; ch < nchunk; ch += 16) {
      const int ow = w0 + wr;
      const long k = kbeg + 8 * ch;
      if (ow >= nw || k >= Kp) continue;
      uint32_t p[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        split_bf16_pair(kb_tile[(8 * ch + 2 * j) * (kKbW + 1) + wr], kb_tile[(8 * ch + 2 * j + 1) * (kKbW + 1) + wr],
                        p[0][j], p[1][j], p[2][j]);
      const long off = (krow0 + ow) * Kp + k;
      *reinterpret_cast<uint4*>(K0 + off) = make_uint4(p[0][0], p[0][1], p[0][2], p[0][3]);
      *reinterpret_cast<uint4*>(K1 + off) = make_uint4(p[1][0], p[1][1], p[1][2], p[1][3]);
      *reinterpret_cast<uint4*>(K2 + off) = make_uint4(p[2][0], p[2][1], p[2][2], p[2][3]);
    }
  }
}

static size_t kbuild_smem_bytes(long nm) { return size_t(kKbCols * nm * (kKbW + 1)) * sizeof(float); }

// ---- dispersive phonons: the Fan-Migdal sum term by term in FP32 ----
// The reference's element sum (src/scgd0_kernel.jl:27-39, 59-86) with ωq gathered per pair
// (ωq[ν, f, i] = ωph[ν, iq_kk[iks_i[i], iks_f[f]]], src/scgd0.jl:270): for each (ω, i) and every
// (ν, f) with ωq >= ω_acoustic, w_f g2 {Im[1/(x_a - ε_f - Σ_in(x_a))] (n + f(x_a - μ)) +
// Im[1/(x_e - ε_f - Σ_in(x_e))] (n + 1 - f(x_e - μ))}, x_a,e = ω ± ωq. FP32 arithmetic with float
// pairs where the value cancels: x = ω ± ωq, ε_f and Re Σ are float pairs and Re z = (x - ε) - Re Σ(x)
// is formed exactly on them (re_z), as in kbuild_bf16_kernel; the cell of x (the O(1) bucket table of
// _interp_linear_grid, flat outside the grid: a bucket, then one node entry that carries the inverse
// widths of both its cells, so the weight needs no division) is found on the pair; the weight, Im Σ,
// the reciprocal and the occupations are FP32, the Fermi factors from exp((ω - μ)/T) exp(±ωq/T)
// (one exponential per thread and one per staged mode instead of two per term; evaluated directly
// where a factor leaves FP32's range), and each thread sums its terms in FP32 runs of one tile
// (256 pairs (ν, f)) added into FP64. The (ν, f) tile of the block's outer state -- w_f g2, ωq,
// n(ωq), exp(±ωq/T), ε_f, the Σ column -- is staged in shared memory by the block; the node table
// and the bucket table too, when they fit.
// Grid (nω / 256, ni, slots), 256 threads, thread = node ω. Slot a reads Σ_in from Sf_all + slots[a] nω ni
// and T, μ from tp[slots[a]]. Output: with ImS_b, ImΣ of the slot (ImS_b + a nω ni) and its BF16
// split as the Kramers-Kronig product's B operand (rows a ni + i, columns ω, stride Kp2), as
// finalize_fm_batch_kernel writes them; else ImΣ added into add_out [nω, ni] (slot 0).
constexpr int kFdTile = 256;

__device__ __forceinline__ float occ_boson_f(float e, float T) {  // occ_boson, src/utils.jl:24-38
  if (T > 1.4901161193847656e-08f) return e == 0.f ? -0.5f : 1.f / expm1f(e / T);
  return e > 0.f ? 0.f : (e == 0.f ? -0.5f : -1.f);
}

template <bool kSmemTab>
__global__ void __launch_bounds__(kFdTile) fm_disp_f32_kernel(
    int nw, long slab, const float4* __restrict__ Sf_all, const float4* __restrict__ wtab_g,
    const int32_t* __restrict__ jtab_g, float x0, float inv_h, long ntab, const float* __restrict__ gw,
    const double* __restrict__ wph, const int32_t* __restrict__ iq_kk, const int32_t* __restrict__ iks_i,
    const int32_t* __restrict__ iks_f, long nk_i, const double* __restrict__ eps_f, const int32_t* __restrict__ f_to_i,
    int nm, long nvf, int ni, double w_ac, const int* __restrict__ slots, const TParams* __restrict__ tp,
    double* __restrict__ ImS_b, __nv_bfloat16* __restrict__ Im0, __nv_bfloat16* __restrict__ Im1,
    __nv_bfloat16* __restrict__ Im2, long Kp2, double* __restrict__ add_out) {
  extern __shared__ __align__(16) unsigned char fd_tab[];  // kSmemTab: node table [nw] float4, then the buckets
  // the staged (ν, f) pairs: {w_f g2, n(ωq), exp(ωq/T), exp(-ωq/T)}, {ε - ωq, ε + ωq} as float pairs,
  // {ωq as a float pair, the Σ column's offset, 0}
  __shared__ float4 s_a[kFdTile], s_e[kFdTile], s_q[kFdTile];
  const float4* wtab = wtab_g;
  const int32_t* jtab = jtab_g;
  if constexpr (kSmemTab) {
    float4* sw = reinterpret_cast<float4*>(fd_tab);
    int32_t* sj = reinterpret_cast<int32_t*>(fd_tab + sizeof(float4) * size_t(nw));
    for (int k = threadIdx.x; k < nw; k += kFdTile) sw[k] = wtab_g[k];
    for (long k = threadIdx.x; k < ntab; k += kFdTile) sj[k] = jtab_g[k];
    wtab = sw;
    jtab = sj;
  }
  const int i = blockIdx.y, a = blockIdx.z;
  const int iw = blockIdx.x * kFdTile + threadIdx.x;
  const bool on = iw < nw;
  const TParams q = tp[slots[a]];
  const float T = float(q.T);
  const bool warm = T > 1.4901161193847656e-08f;
  const float invT = warm ? 1.f / T : 0.f;
  const float2 mu = split_df(q.mu);
  const float4* Sf = Sf_all + slab * slots[a];
  const float4 wn = wtab_g[on ? iw : 0];
  const float2 w = make_float2(wn.x, wn.y);
  // exp((ω - μ)/T) of the thread's node: f(ω ± ωq - μ) = 1 / (E exp(±ωq/T) + 1); a node whose E
  // leaves FP32's range takes the exponential of each term directly
  const float wm = (w.x - mu.x) + (w.y - mu.y);
  const float E = warm ? __expf(wm * invT) : 0.f;
  const bool Eok = warm && E > 0.f && E < INFINITY;
  const int ntab_i = int(ntab), jmax = nw - 2;
  const int ki = iks_i[i];
  // one side of a term, x = ω + sg ωq (sg = ±1), with em = ε - sg ωq: Im 1/(x - ε - Σ(x)) times its
  // occupation bracket
  auto side = [&](const float4* col, float sgwq_hi, float sgwq_lo, float2 em, float nq, float eq, bool absorb) -> float {
    const float xh = w.x + sgwq_hi;
    const float v = fminf(fmaxf((xh - x0) * inv_h, -1.f), float(ntab_i)) - 0.5f;
    // the bucket floor((x - x0) / h) in 32-bit integer arithmetic (1.5 2^23 added: the integer part
    // lands in the mantissa; |v| < 2^22); an off-by-one bucket at a bucket edge still picks the
    // cell whose value is continuous there
    int b = __float_as_int(v + 12582912.f) - 0x4B400000;
    b = min(max(b, 0), ntab_i - 1);
    const int c = jtab[b];
    const float4 wc = wtab[c];  // node c: (hi, lo, 1 / (w[c+1] - w[c]), 1 / (w[c] - w[c-1]))
    const float dx = ((w.x - wc.x) + sgwq_hi) + ((w.y - wc.y) + sgwq_lo);
    const bool below = dx < 0.f;
    int j = below ? c - 1 : c;
    float t = below ? fmaf(dx, wc.w, 1.f) : dx * wc.z;
    if (j < 0 || j > jmax) {  // outside the grid the value is flat (the first or the last node)
      t = j < 0 ? 0.f : 1.f;
      j = j < 0 ? 0 : jmax;
    }
    const float4 lo = col[j], hi = col[j + 1];
    // Re z = (x - ε) - Re Σ(x) = (ω - em) - Re Σ(x), exact on the float pairs
    const float zr = re_z(w, em, lo, hi, t);
    const float si = fmaf(t, hi.z - lo.z, lo.z);  // Im Σ(x)
    const float g = __fdividef(si, fmaf(zr, zr, si * si));
    float y = E * eq;
    if (!Eok || y != y) {  // a factor out of range (stored as NaN), or T -> 0
      const float xm = (xh - mu.x) + ((w.y + sgwq_lo) - mu.y);
      y = warm ? __expf(xm * invT) : (xm > 0.f ? INFINITY : (xm < 0.f ? 0.f : 1.f));
    }
    const float f = __fdividef(1.f, y + 1.f);
    return g * (absorb ? nq + f : nq + 1.f - f);
  };
  double acc = 0.0;
  for (long t0 = 0; t0 < nvf; t0 += kFdTile) {
    const long vf = t0 + threadIdx.x;
    __syncthreads();  // the previous tile's readers are done (and, first, the tables are staged)
    // below ω_acoustic (and past the end) no term: zero coupling, the first column as a stand-in and
    // ε - ωq = -1e30, so that Re z^2 overflows and Im 1/z is exactly 0 whatever the column holds
    float4 sa = make_float4(0.f, 0.f, 0.f, 0.f), se = make_float4(-1e30f, 0.f, -1e30f, 0.f), sq = sa;
    if (vf < nvf) {
      const int nu = int(vf % nm);
      const long f = vf / nm;
      const double wq = wph[nu + long(nm) * iq_kk[ki + nk_i * long(iks_f[f])]];
      if (!(wq < w_ac)) {
        const double e = eps_f[f];
        const float wqf = float(wq);
        const float2 ea = split_df(e - wq), ee = split_df(e + wq), wqp = split_df(wq);
        float eq = warm ? __expf(wqf * invT) : 0.f, ieq = warm ? __expf(-wqf * invT) : 0.f;
        if (!(eq < INFINITY) || !(ieq > 0.f)) eq = ieq = __int_as_float(0x7fc00000);  // out of range: NaN
        sa = make_float4(gw[vf + nvf * i], occ_boson_f(wqf, T), eq, ieq);
        se = make_float4(ea.x, ea.y, ee.x, ee.y);
        sq = make_float4(wqp.x, wqp.y, __int_as_float(nw * f_to_i[f]), 0.f);
      }
    }
    s_a[threadIdx.x] = sa;
    s_e[threadIdx.x] = se;
    s_q[threadIdx.x] = sq;
    __syncthreads();
    float run0 = 0.f, run1 = 0.f;
    if (on) {
      const int nt = int(min(long(kFdTile), nvf - t0));
#pragma unroll 2
      for (int k = 0; k < nt; ++k) {
        const float4 A = s_a[k], Ee = s_e[k], Q = s_q[k];
        const float4* col = Sf + __float_as_int(Q.z);
        const float va = side(col, Q.x, Q.y, make_float2(Ee.x, Ee.y), A.y, A.z, true);
        const float ve = side(col, -Q.x, -Q.y, make_float2(Ee.z, Ee.w), A.y, A.w, false);
        const float v = A.x * (va + ve);
        if (k & 1)
          run1 += v;
        else
          run0 += v;
      }
    }
    acc += double(run0) + double(run1);
  }
  if (!on) return;
  const long k = iw + long(nw) * i;
  if (ImS_b) {
    ImS_b[slab * a + k] = acc;
    __nv_bfloat16 p[3];
    split_bf16_n(float(acc), 3, p);
    const long o = (long(a) * ni + i) * Kp2 + iw;
    Im0[o] = p[0];
    Im1[o] = p[1];
    Im2[o] = p[2];
  } else {
    add_out[k] += acc;
  }
}

// The same sum in about 47 instructions a term (the L1 data pipe bounds it; fm_disp_f32_kernel above takes about 180),
// for temperatures above ωq / 40:
//  * Frequencies in grid units u (the nodes are origin + offset u, whole offsets): x = ω ± ωq is a whole number b,
//    ωq's being the same for all nodes, and a fraction that all nodes share. A table over b gives the cell that x is in
//    and b's distance from the cell's lower node; padded by ωq's largest number, it needs no clamp.
//  * A record a cell and column describes Σ from the cell's lower node c: U = ω_c - ReΣ_c as a float pair, u_lo - u ReΣ',
//    ImΣ_c, u ImΣ', with u = u_hi + u_lo. x is b whole units and a fraction f from ω_c; the fraction's f u_hi is taken off
//    ε (ε' = ε - f u_hi, a pair a side), so Re z = ((U_hi - ε'_hi) + b u_hi) + ((U_lo - ε'_lo) + (b + f) (u_lo - u ReΣ')).
//    High parts are multiples of one quantum (split_q): the first bracket is exact, and Re z keeps its distance to a
//    pole anywhere in a wide cell (as (b + f) times u (1 - ReΣ') in FP32, terms near poles 0.2 meV wide were off by
//    1e-5 in cells of 0.25 eV). The cells below and above the grid have slopes 0 (fd_cell_kernel). Where ωq is a whole
//    number to rounding, x is that node on both sides (not the far end of the cell below, 2^-24 of whose start's ImΣ may
//    be large against the node's).
//  * n + f(x_a - μ) = (1 + n)(1 + E)/(1 + E e) and n + 1 - f(x_e - μ) = n (1 + E)/(1 + E/e), E = exp((ω - μ)/T),
//    e = exp(ωq/T): one FMA a side, the bracket's reciprocal shared with 1/|z|², and 1 + E outside the sum
//    (both sides over E above μ, so that every factor stays below e^40).
// A column's records are contiguous over the cells (four wavefronts of L1 a load) and a staged pair is read once for
// NPT nodes of a thread. Grid (nω / (256 NPT), ni, slots x splits): the (ν, f) range is split, in whole tiles, until the
// last of the waves of resident blocks weighs little (partials summed in order by fd_finish_kernel); at 501 nodes and
// 105 states the unsplit grid of 210 blocks left a third of the SMs half empty.
// Measured: 1.2e9 terms (501 nodes, 105 states, 15 modes, 1536 inner states) 13.0 ms by the kernel above, 3.25 with a
// search for the nearest node and a record for either side of it, 2.31 with (b + f) u as one FP32 number (7.7 wavefronts a
// side and warp, 4.7 of them the records' 20 bytes a lane, kept the L1 data pipe 90 % busy and the issue slots 71 %), 2.48
// with it exact, 2.32 now, a term's two sides in one instruction where their operands lie side by side. Three blocks an SM
// and two pairs in flight (us there, at 416 nodes x 60 states x 2 temperatures, 312 x 30 with two nodes a thread, 201 x
// 105 and 208 x 30 with one): 2320, 551, 148, 1237, 103, and 230 ms at 1251 x 495; four and two 2286, 575, 162, 1223, 99, and
// 245 ms; three and one 2355, 557, 163, 1228, 119; two and four 2401, 559, 136, 1363, 92.
constexpr float kFdMaxArg = 40.f;
// Terms of an FP32 run (added into FP64). Error of one sum against the FP64 kernel, relative (30 states x 251 nodes x 6
// modes, 105 x 501 x 15): 7.6e-8, 2.7e-8 with runs of a tile's 256, 3.9e-8, 1.5e-8 with 64, 3.4e-8, 1.4e-8 with 32; the
// kernel above 5.6e-8, 2.1e-8. Shorter runs take the FP64 pipe's time: 28.3, 28.6, 28.9 ms a run.
constexpr int kFdRun = 64;
constexpr long kFdMaxTable = 1l << 24;  // entries; those that fit 96 KB are kept in shared memory
constexpr long kFdMaxCell = 32767;      // grid units of a cell or ωq: distances are 16 bits

// Two FP32 values in a register pair, and operations on both (each rounded as alone).
using F2 = unsigned long long;
__device__ __forceinline__ F2 pk(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 upk(F2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ float exp_comp(float v, float T) {  // exp(v / T), v / T's rounding put back
  const float a = v / T, E = expf(a);
  return fmaf(E, fmaf(-a, T, v) / T, E);
}

// Records [column][nω + 1] of slot blockIdx.y: cell 0 is below the grid, cell c from node c - 1 to node c, cell nω above.
// Slopes in FP64 and rounded once: far inside a wide cell they are what is left of the error.
__global__ void fd_cell_kernel(const float4* __restrict__ Sf_all, const int* __restrict__ slots,
                               const double* __restrict__ ws, int nw, long slab, double unit, double u_hi, double qm,
                               float4* __restrict__ rec, float* __restrict__ dim) {
  const long ncell = slab / nw * (nw + 1);
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= ncell) return;
  const int c = int(k % (nw + 1)), j = max(c - 1, 0), o = min(c, nw - 1);
  const float4* Sf = Sf_all + slab * slots[blockIdx.y] + k / (nw + 1) * nw;
  const float4 s = Sf[j], t = Sf[o];
  const double re = double(s.x) + double(s.y);
  const float2 u = split_q(ws[j] - re, qm);
  const double per = o > j ? unit / (ws[o] - ws[j]) : 0.0;  // (0 below and above the grid)
  rec[ncell * blockIdx.y + k] =
      make_float4(u.x, u.y, float((unit - u_hi) - per * ((double(t.x) + double(t.y)) - re)), s.z);
  dim[ncell * blockIdx.y + k] = float(per * (double(t.z) - double(s.z)));
}

template <int NPT, bool kSmemTab>
__global__ void __launch_bounds__(kFdTile, 3) fm_disp_fast_kernel(
    int nw, long slab, const float4* __restrict__ rec_all, const float* __restrict__ dim_all,
    const float4* __restrict__ wtab_g, const int32_t* __restrict__ offs, const uint32_t* __restrict__ tab_g, int ntab, int pad,
    double unit, double inv_unit, double qm, double u_hi, const float* __restrict__ gw, const double* __restrict__ wph,
    const int32_t* __restrict__ iq_kk,
    const int32_t* __restrict__ iks_i, const int32_t* __restrict__ iks_f, long nk_i, const double* __restrict__ eps_f,
    const int32_t* __restrict__ f_to_i, int nm, long nvf, long per, int nsplit, double w_ac, const int* __restrict__ slots,
    const TParams* __restrict__ tp, double* __restrict__ part) {
  extern __shared__ __align__(16) uint32_t fd_cells[];  // kSmemTab: the cell table
  // the staged (ν, f) pairs: {w_f g2 (1 + n), w_f g2 n, exp(ωq/T), exp(-ωq/T)}, {-ε' of the absorption and of the emission
  // as pairs}, {the column, ωq's whole numbers of the absorption and (<< 16) of the emission, what they leave (float bits)}
  __shared__ float4 s_a[kFdTile], s_e[kFdTile];
  __shared__ int4 s_c[kFdTile];
  if constexpr (kSmemTab)
    for (int k = threadIdx.x; k < ntab; k += kFdTile) fd_cells[k] = tab_g[k];
  const uint32_t* tab = kSmemTab ? fd_cells : tab_g;
  const int i = blockIdx.y, a = blockIdx.z / nsplit, sp = blockIdx.z % nsplit;
  const int iw0 = blockIdx.x * (kFdTile * NPT) + threadIdx.x;  // the nodes iw0 + 256 n
  const TParams tq = tp[slots[a]];
  const float T = float(tq.T);
  const long ncell = slab / nw * (nw + 1);
  const float4* rec = rec_all + ncell * a;
  const float* dim = dim_all + ncell * a;
  const float2 mu = split_df(tq.mu);
  float p[NPT], qe[NPT];
  int off[NPT];
#pragma unroll
  for (int n = 0; n < NPT; ++n) {
    const int iw = min(iw0 + kFdTile * n, nw - 1);
    const float4 wn = wtab_g[iw];
    const float wm = (wn.x - mu.x) + (wn.y - mu.y);
    const float Ew = exp_comp(-fabsf(wm), T);  // E, or 1/E above μ
    p[n] = wm <= 0.f ? 1.f : Ew;
    qe[n] = wm <= 0.f ? Ew : 1.f;
    off[n] = offs[iw] + pad;
  }
  const int ki = iks_i[i];
  const float uf = float(u_hi);
  // both sides of a term at one node, two FP32 operations an instruction: the record's differences, then (absorption,
  // emission) side by side
  const F2 magic = pk(-8421376.f, -8421376.f);
  auto sides = [&](int ba, int be, F2 frac, F2 ea, F2 ee, int col, F2 o, F2 g, F2& run) {
    const uint32_t ta = tab[ba], te = tab[be];  // the cell, and b's distance from its lower node + 32768
    const F2 n = add2(pk(__uint_as_float(__byte_perm(ta, 0x4B000000u, 0x7610)), __uint_as_float(__byte_perm(te, 0x4B000000u, 0x7610))), magic);
    const F2 dx = add2(n, frac);
    const int aa = col + int(ta >> 16), ae = col + int(te >> 16);
    const float4 ra = rec[aa], re = rec[ae];
    const F2 ua = add2(pk(ra.x, ra.y), ea), ue = add2(pk(re.x, re.y), ee);
    const float2 nn = upk(n), dd = upk(dx), va = upk(ua), ve = upk(ue);
    const F2 zr = pk(fmaf(nn.x, uf, va.x) + fmaf(dd.x, ra.z, va.y), fmaf(nn.y, uf, ve.x) + fmaf(dd.y, re.z, ve.y));
    const F2 si = pk(fmaf(dd.x, dim[aa], ra.w), fmaf(dd.y, dim[ae], re.w));
    const float2 d = upk(mul2(fma2(zr, zr, mul2(si, si)), o));
    run = fma2(mul2(g, si), pk(rcp_f(d.x), rcp_f(d.y)), run);
  };
  double acc[NPT];
#pragma unroll
  for (int n = 0; n < NPT; ++n) acc[n] = 0.0;
  const long t_end = min(nvf, per * (sp + 1l));
  for (long t0 = per * sp; t0 < t_end; t0 += kFdTile) {
    const long vf = t0 + threadIdx.x;
    __syncthreads();  // the previous tile's readers are done (and, first, the table is staged)
    // below ω_acoustic no term: zero coupling, and ε = -1e25, so that |z|² overflows and the reciprocal is 0
    float4 sa = make_float4(0.f, 0.f, 1.f, 1.f), se = make_float4(1e25f, 0.f, 1e25f, 0.f);
    int4 sc = make_int4(0, 0, 0, 0);
    if (vf < t_end) {
      const int nu = int(vf % nm);
      const long f = vf / nm;
      const double wq = wph[nu + long(nm) * iq_kk[ki + nk_i * long(iks_f[f])]];
      if (!(wq < w_ac)) {
        const float wp = float(wq), n = occ_boson_f(wp, T), g = gw[vf + nvf * i];
        // x = ω + ωq = b + wb and fr, ω - ωq = b - wb - up and fe, in units; fr within 2^-32 of a whole number is next to it
        const double wb = fmin(floor(fma(wq, inv_unit, 0x1p-32)), double(pad - 1)), fr = fma(-wb, unit, wq) * inv_unit;
        const int up = fr > 0x1p-32 ? 1 : 0;
        const double fe = double(up) - fr, ef = eps_f[f];
        const float2 ea = split_q(fma(-fr, u_hi, ef), qm), ee = split_q(fma(-fe, u_hi, ef), qm);
        sa = make_float4(g * (n + 1.f), g * n, exp_comp(wp, T), exp_comp(-wp, T));
        se = make_float4(-ea.x, -ea.y, -ee.x, -ee.y);
        sc = make_int4((nw + 1) * f_to_i[f], int(wb) | (int(wb) + up) << 16, __float_as_int(float(fr)), __float_as_int(float(fe)));
      }
    }
    s_a[threadIdx.x] = sa;
    s_e[threadIdx.x] = se;
    s_c[threadIdx.x] = sc;
    __syncthreads();
    const int nt = int(min(long(kFdTile), t_end - t0));
    // (a warp past the last node, or whose second nodes are, does that part of the work no more than it must)
    if (iw0 - int(threadIdx.x % 32) >= nw) continue;
    const bool both = NPT == 1 || iw0 - int(threadIdx.x % 32) + kFdTile < nw;
    auto terms = [&](auto nodes) {
      for (int k0 = 0; k0 < nt; k0 += kFdRun) {
        F2 run[NPT];
#pragma unroll
        for (int n = 0; n < NPT; ++n) run[n] = pk(0.f, 0.f);
        const int k1 = min(nt, k0 + kFdRun);
#pragma unroll 2
        for (int k = k0; k < k1; ++k) {
          const float4 A = s_a[k], E = s_e[k];
          const int4 C = s_c[k];
          const int wa = C.y & 0xffff, we = C.y >> 16;
#pragma unroll
          for (int n = 0; n < decltype(nodes)::value; ++n) {
            sides(off[n] + wa, off[n] - we, pk(__int_as_float(C.z), __int_as_float(C.w)), pk(E.x, E.y), pk(E.z, E.w), C.x,
                  fma2(pk(qe[n], qe[n]), pk(A.z, A.w), pk(p[n], p[n])), pk(A.x, A.y), run[n]);
          }
        }
#pragma unroll
        for (int n = 0; n < decltype(nodes)::value; ++n) acc[n] += double(upk(run[n]).x) + double(upk(run[n]).y);
      }
    };
    if (both)
      terms(std::integral_constant<int, NPT>{});
    else
      terms(std::integral_constant<int, 1>{});
  }
#pragma unroll
  for (int n = 0; n < NPT; ++n) {
    const int iw = iw0 + kFdTile * n;
    if (iw < nw) part[iw + long(nw) * i + slab * blockIdx.z] = acc[n] * (double(p[n]) + double(qe[n]));
  }
}

// ImΣ of slot a = the sum of its partials in order: into ImS_b and the Kramers-Kronig operand, or added to add_out.
__global__ void fd_finish_kernel(const double* __restrict__ part, int nw, long slab, int nsplit, double* __restrict__ ImS_b,
                                 __nv_bfloat16* __restrict__ Im0, __nv_bfloat16* __restrict__ Im1,
                                 __nv_bfloat16* __restrict__ Im2, long Kp2, double* __restrict__ add_out) {
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= slab) return;
  const long a = blockIdx.y;
  double v = 0.0;
  for (int s = 0; s < nsplit; ++s) v += part[k + slab * (a * nsplit + s)];
  if (!ImS_b) {
    add_out[k] += v;
    return;
  }
  ImS_b[slab * a + k] = v;
  __nv_bfloat16 p[3];
  split_bf16_n(float(v), 3, p);
  const long o = (slab / nw * a + k / nw) * Kp2 + k % nw;
  Im0[o] = p[0];
  Im1[o] = p[1];
  Im2[o] = p[2];
}

// The node table of fm_disp_f32_kernel: node j as (hi, lo, 1 / (w[j+1] - w[j]), 1 / (w[j] - w[j-1]))
// (0 past the ends).
__global__ void fd_node_table_kernel(const double* __restrict__ ws, int nw, float4* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nw) return;
  const float2 p = split_df(ws[j]);
  const float up = j + 1 < nw ? float(1.0 / (ws[j + 1] - ws[j])) : 0.f;
  const float dn = j > 0 ? float(1.0 / (ws[j] - ws[j - 1])) : 0.f;
  out[j] = make_float4(p.x, p.y, up, dn);
}


// out_p[r * ld + c] = part p of S(r, c) for c < cols, 0 for cols <= c < ld, with S(r, c) =
// S[c + ldc r] (transposed = false: rows of the output are columns of the column-major S) or
// S[r + ldc c] (transposed = true).
__global__ void split3_rows_kernel(const double* __restrict__ S, long ldc, long rows, long cols, long ld, bool transposed,
                                   __nv_bfloat16* __restrict__ o0, __nv_bfloat16* __restrict__ o1,
                                   __nv_bfloat16* __restrict__ o2) {
  long idx = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= rows * ld) return;
  long r = idx / ld, c = idx % ld;
  float x = 0.f;
  if (c < cols) x = float(transposed ? S[r + ldc * c] : S[c + ldc * r]);
  __nv_bfloat16 q[3];
  split_bf16_n(x, 3, q);
  o0[idx] = q[0];
  o1[idx] = q[1];
  o2[idx] = q[2];
}

// ImΣ (FP64) += Σ_s part[s] in ascending s.
__global__ void finalize_add_kernel(const float* __restrict__ part, long n, int splits, long stride, double* __restrict__ out) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n) return;
  float s = 0.f;
  for (int p = 0; p < splits; ++p) s += part[k + stride * p];
  out[k] += double(s);
}

// exp(ω_ν/T) and n(ω_ν) of every temperature and mode of a run (the quotient's rounding put back); 0 where the
// occupation table takes the plain formula: ω_ν > 300 T, T ~ 0, a mode left out or at 0.
__global__ void mode_table_kernel(const double* __restrict__ wnu, int nm, const TParams* __restrict__ tp, double w_ac,
                                  double2* __restrict__ modes) {
  const int nu = threadIdx.x + blockIdx.x * blockDim.x, t = blockIdx.y;
  if (nu >= nm) return;
  const double wq = wnu[nu], T = tp[t].T;
  double2 o = make_double2(0.0, 0.0);
  if (T > 1.4901161193847656e-08 && !(wq < w_ac) && wq > 0.0 && wq <= 300.0 * T) {
    const double a = wq / T, m0 = expm1(a), m = fma(m0 + 1.0, fma(-a, T, wq) / T, m0);
    o = make_double2(m + 1.0, 1.0 / m);
  }
  modes[nu + nm * t] = o;
}

// The occupation tables of the active temperatures as FP32, computed in FP64: F[a][0 .. nω nm) absorption
// n + f(ω + ω_ν - μ), F[a][nω nm .. 2 nω nm) emission n + 1 - f(ω - ω_ν - μ). By detailed balance these are
// (1 + n)(1 + E)/(1 + E e) and n (1 + E)/(1 + E/e) with E = exp((ω - μ)/T), e = exp(ω_ν/T) (both over E above μ): one
// exponential a node and a dozen operations an element, in blocks of four nodes over all SMs (FP64 instructions issue
// at one per 16 cycles and SM; two exponentials and divisions an element before: 501 x 15 6.5 -> 5.3 us). Also resets
// the iteration's max|ΔΣ|. Grid (nω / 4, slots).
constexpr int kOccW = 4;
__global__ void __launch_bounds__(64) occ_table_f32_kernel(const double* __restrict__ ws, int nw,
                                                           const double* __restrict__ wnu, int nm,
                                                           const int* __restrict__ slots, const TParams* __restrict__ tp,
                                                           const double2* __restrict__ modes, double w_ac,
                                                           float* __restrict__ F_all,
                                                           unsigned long long* __restrict__ errbits,
                                                           IterCtl* __restrict__ ctl) {
  pdl_wait();
  __shared__ double s_p[kOccW], s_q[kOccW];
  const int a = blockIdx.y, t = slots[a];
  const int stop = ctl->stop_next;  // set by the iteration before, unchanged during this one's first kernels
  if (blockIdx.x == 0 && a == 0 && threadIdx.x == 0) ctl->stop = stop;
  if (stop) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) errbits[t] = 0;
  const long nwm = long(nw) * nm;
  const TParams q = tp[t];
  float* F = F_all + 2 * nwm * a;
  const int wl = threadIdx.x % kOccW, iw = blockIdx.x * kOccW + wl;
  if (threadIdx.x < kOccW && iw < nw && q.T > 1.4901161193847656e-08) {
    const double v = ws[iw] - q.mu, m = -fabs(v), av = m * q.inv_T, E0 = exp(av), E = fma(E0, fma(-av, q.T, m) * q.inv_T, E0);
    s_p[wl] = v <= 0.0 ? 1.0 : E;
    s_q[wl] = v <= 0.0 ? E : 1.0;
  }
  __syncthreads();
  if (iw >= nw) return;
  for (int nu = threadIdx.x / kOccW; nu < nm; nu += 64 / kOccW) {
    const long k = iw + long(nw) * nu;
    const double wq = wnu[nu];
    const double2 en = modes[nu + nm * t];
    float fa = 0.f, fe = 0.f;
    if (en.x > 0.0) {
      const double c = s_p[wl] + s_q[wl];
      // 1 / (p + q e) and 1 / (p + q / e) = e / (p e + q) from one division
      const double da = fma(s_q[wl], en.x, s_p[wl]), de = fma(s_p[wl], en.x, s_q[wl]), r = c / (da * de);
      fa = float((en.y + 1.0) * r * de);
      fe = float(en.y * en.x * r * da);
    } else if (!(wq < w_ac)) {
      const double nq = occ_boson_d(wq, q.T), w = ws[iw];
      fa = float(nq + occ_fermion_d(w + wq - q.mu, q.T));
      fe = float(nq + 1 - occ_fermion_d(w - wq - q.mu, q.T));
    }
    F[k] = fa;
    F[k + nwm] = fe;
  }
}

// ImΣ of slot a: ImS[a][ω + nω i] = Σ_s part[s][(a nω + ω) + M i], M = nA nω (the stacked rows).
// With Im0 (the batched iteration), it also writes ImΣ split into the KK product's B operand (whose
// padding columns nω.. Kp2 stay zero from the reservation).
__global__ void finalize_fm_batch_kernel(const float* __restrict__ part, int nw, long slab, int nA, int splits,
                                         long stride, double* __restrict__ ImS, __nv_bfloat16* __restrict__ Im0 = nullptr,
                                         __nv_bfloat16* __restrict__ Im1 = nullptr, __nv_bfloat16* __restrict__ Im2 = nullptr,
                                         long Kp2 = 0, const IterCtl* __restrict__ ctl = nullptr) {
  pdl_wait();
  if (ctl && ctl->stop) return;
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= slab) return;
  const int a = blockIdx.y;
  const long w = k % nw, i = k / nw;
  const long src = (long(a) * nw + w) + long(nA) * nw * i;
  const float acc = sum_splits(part + src, splits, stride);
  ImS[slab * a + k] = double(acc);
  if (Im0) {  // and the B operand of the Kramers-Kronig product: row a ni + i, column ω, three parts
    __nv_bfloat16 q[3];
    split_bf16_n(acc, 3, q);
    const long o = (long(a) * (slab / nw) + i) * Kp2 + w;
    Im0[o] = q[0];
    Im1[o] = q[1];
    Im2[o] = q[2];
  }
}

// The Kramers-Kronig product's epilogue and the rest of the iteration's tail, in one pass over its
// split-K partials (src/scgd0.jl:287-301, 326-328): per state group of slot a -- a degenerate
// multiplet, or a single state -- Σ_new(ω_j) = Σ_s part[s] + i ImΣ of every member (the partials in
// ascending order), averaged over the members of a multiplet (their sum in member order divided by
// the count); then per member: err = max |Σ_new - Σ| over the slot's temperature (FP64 differences,
// FP32 magnitude, the maximum taken on the bit patterns as err_copy does), Σ ← Σ_new, its clamped form for the
// next iteration -- the columns' cell records (rec, dim), or Sf with dispersive modes (rec null) -- and the
// spectral functions' per-node terms P[i][j] = (ε_i - ω_j + ReΣ_j, ReΣ_{j+1} - ReΣ_j, ImΣ_j, ImΣ_{j+1})
// (ImΣ_{j+1}, ReΣ_{j+1} = those of j at the last node). Everything but Σ itself and its change is formed on float pairs
// (a single state's ReΣ is an FP32 sum): six instructions on the FP64 pipe a state and node, where about 25 bound the
// kernel (1251 x 495: 26 -> 24.3 us, 8 x 626 x 168: 32 -> 28.9 us, with the next iteration's clamp, 10 us, included).
// Groups: CSR (gptr, gidx), members in order. Grid (nω / 255,
// groups, slots), 256 threads: thread t takes node j = 255 blockIdx.x + t; the last thread's node
// is the next block's first, formed again to give node 254 its neighbour.
__global__ void __launch_bounds__(256) kk_epilogue_kernel(const float* __restrict__ part, int splits, long stride,
                                                          const double* __restrict__ ImS_b, int nw, long slab,
                                                          const int* __restrict__ slots, const int32_t* __restrict__ gptr,
                                                          const int32_t* __restrict__ gidx, const float4* __restrict__ wtab,
                                                          float qm, const float2* __restrict__ epair,
                                                          const TParams* __restrict__ tp, double2* __restrict__ S_all,
                                                          float4* __restrict__ Sf_all, float4* __restrict__ rec_all,
                                                          float* __restrict__ dim_all, float4* __restrict__ Pall,
                                                          unsigned long long* __restrict__ errbits_all,
                                                          double* __restrict__ minA_all,
                                                          const IterCtl* __restrict__ ctl) {
  pdl_wait();
  if (ctl && ctl->stop) return;
  __shared__ float4 sh[256];
  __shared__ uint32_t she[8];
  const int a = blockIdx.z, t = slots[a];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)  // the minimum of spectral_fin starts at +inf
    minA_all[t] = INFINITY;
  const int j = blockIdx.x * 255 + threadIdx.x;
  const bool in = j < nw;
  const int p0 = gptr[blockIdx.y], p1 = gptr[blockIdx.y + 1];
  double2 z = make_double2(0.0, 0.0);
  float4 zf = make_float4(0.f, 0.f, 0.f, 0.f);  // {Re hi, Re lo, Im}
  if (in) {
    if (p1 - p0 == 1) {
      const long src = slab * a + j + long(nw) * gidx[p0];
      const float acc = sum_splits(part + src, splits, stride);
      z = make_double2(double(acc), ImS_b[src]);
      zf = make_float4(acc, 0.f, float(z.y), 0.f);
    } else {
      for (int p = p0; p < p1; ++p) {
        const long src = slab * a + j + long(nw) * gidx[p];
        z.x += double(sum_splits(part + src, splits, stride));
        z.y += ImS_b[src];
      }
      const double len = double(p1 - p0);
      z.x /= len;
      z.y /= len;
      zf = sigma_f32(z);
    }
  }
  sh[threadIdx.x] = zf;
  __syncthreads();
  uint32_t e = 0;  // the largest magnitude's bits: non-negative floats order as integers, and NaN above all
  if (in && threadIdx.x < 255) {
    const float4 zn = j + 1 < nw ? sh[threadIdx.x + 1] : zf, wj = wtab[j];
    const float etam = float(-tp[t].eta_min);
    float dim, d0;
    const float4 rec = cell_record(zf, zn, wj, etam, qm, dim);
    const float dre = (zn.x - zf.x) + (zn.y - zf.y);
    double2* S = S_all + slab * t;
    const long ni = slab / nw;
    for (int p = p0; p < p1; ++p) {
      const int i = gidx[p];
      const long k = j + long(nw) * i;
      const double2 b = S[k];
      e = max(e, __float_as_uint(hypotf(float(z.x - b.x), float(z.y - b.y))));
      S[k] = z;
      if (rec_all) {
        const long at = (ni * t + i) * (nw + 1l) + j + 1;
        rec_all[at] = rec;
        dim_all[at] = dim;
        if (j == 0) {
          rec_all[at - 1] = cell_record(zf, zf, wj, etam, qm, d0);
          dim_all[at - 1] = 0.f;
        }
      } else {
        Sf_all[slab * t + k] = make_float4(zf.x, zf.y, fminf(zf.z, etam), 0.f);
      }
      // ε_i - ω_j + ReΣ_j with its cancelling parts exact
      const float2 ep = epair[i];
      float e1, e2;
      const float s1 = two_sum(ep.x, -wj.x, e1), s2 = two_sum(s1, zf.x, e2);
      Pall[slab * a + k] = make_float4(s2 + ((e1 + e2) + ((ep.y - wj.y) + zf.y)), dre, zf.z, zn.z);
    }
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if (threadIdx.x % 32 == 0) she[threadIdx.x / 32] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) e = max(e, she[w]);
    atomicMax(errbits_all + t, (unsigned long long)__double_as_longlong(double(__uint_as_float(e))));
  }
}

static long pad64(long x) { return (x + 63) / 64 * 64; }

// K block of the three-part products' operand maps (64: two 96 KB pipeline stages; 32: four of
// 48 KB, measured no faster on these short products).
constexpr int kScgd0Bk = 64;

static TcOperand operand(DBuf<__nv_bfloat16>* parts, long rows, long cols, long ld, int box_rows) {
  TcOperand op;
  op.ns = kNs;
  op.bk = kScgd0Bk;
  for (int p = 0; p < kNs; ++p) op.m[p] = make_tmap_bf16(parts[p].p, rows, cols, ld, box_rows, kScgd0Bk);
  return op;
}

void tc_setup(Scgd0Plan* P) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  auto* T = new Scgd0Plan::Tc;
  P->tc = std::unique_ptr<Scgd0Plan::Tc, void (*)(Scgd0Plan::Tc*)>(T, [](Scgd0Plan::Tc* t) { delete t; });
  const long nw = P->nw, ni = P->ni, nk = P->nm * P->nc;
  T->Kp = pad64(nk);
  T->Kp2 = pad64(nw);
  // the quantum of high parts: 2^20 of it reach beyond the grid's nodes, so that sums of nodes, energies, distances and
  // Σ within four times that stay below the 2^24 that FP32 adds exactly
  P->re_q = std::ldexp(1.0, std::ilogb(std::max(std::fabs(P->ws.nodes.front()), std::fabs(P->ws.nodes.back()))) + 1 - 20);
  P->re_qm = float(1.5 * 0x1p23 * P->re_q);
  P->re_qmd = 1.5 * 0x1p52 * P->re_q;
  if (nw > (1l << 30) || ni > (1l << 30) || nk > (1l << 30)) fail(EPSP_EINVAL, "sizes beyond the 32-bit tile grid");
  T->epair.alloc(ctx, size_t(ni));
  split_df_kernel<<<div_up(size_t(ni), 256), 256, 0, s>>>(P->d_eps_i.p, ni, T->epair.p);
  EPSP_LAUNCHED(ctx);
  if (!P->disp) {
    P->d_wtab.alloc(ctx, size_t(nw));
    fd_node_table_kernel<<<div_up(size_t(nw), 256), 256, 0, s>>>(P->d_ws.p, int(nw), P->d_wtab.p);
    EPSP_LAUNCHED(ctx);
  }
  if (P->disp) {  // the Kramers-Kronig map's operands only: the Fan-Migdal sum goes term by term (launch_fm_disp)
    for (int p = 0; p < kNs; ++p) {
      T->KK[p].alloc(ctx, size_t(nw * T->Kp2));
      T->Im[p].alloc(ctx, size_t(ni * T->Kp2));
    }
    T->err.alloc(ctx, 1);
    T->err.zero(s);
    split3_rows_kernel<<<div_up(size_t(nw * T->Kp2), 256), 256, 0, s>>>(P->d_KK.p, nw, nw, nw, T->Kp2, true, T->KK[0].p,
                                                                        T->KK[1].p, T->KK[2].p);
    EPSP_LAUNCHED(ctx);
    tc_gemm_shape(ctx, int(nw), int(ni), int(nw), max_splits_for(nw, kKbCapKK), kNs, &T->bn2, &T->splits2, kKbCapKK);
    T->part.alloc(ctx, size_t(T->splits2) * size_t(nw * ni));
    T->Sf.alloc(ctx, size_t(nw * ni));
    T->opKK = operand(T->KK, nw, nw, T->Kp2, kTcBM);
    T->opIm = operand(T->Im, ni, nw, T->Kp2, T->bn2);
    return;
  }
  if (kbuild_smem_bytes(P->nm) > size_t(227 * 1024))
    fail(EPSP_EUNSUPPORTED, "the BF16 scGD0 path takes at most 427 modes; use EPSP_PATH_GEMM_FP64");
  if (kbuild_smem_bytes(P->nm) > size_t(48 * 1024))
    EPSP_CUDA(cudaFuncSetAttribute(kbuild_bf16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(kbuild_smem_bytes(P->nm))));
  for (int p = 0; p < kNs; ++p) {
    T->Kt[p].alloc(ctx, size_t(nw * T->Kp));
    T->G[p].alloc(ctx, size_t(ni * T->Kp));
    T->KK[p].alloc(ctx, size_t(nw * T->Kp2));
    T->Im[p].alloc(ctx, size_t(ni * T->Kp2));
  }
  T->err.alloc(ctx, 1);
  T->err.zero(s);
  {
    std::vector<double> wnu(static_cast<size_t>(P->nm));
    P->d_wnu.download(wnu.data(), wnu.size(), s);
    EPSP_CUDA(cudaStreamSynchronize(s));
    std::vector<uint8_t> skip(wnu.size());
    for (size_t nu = 0; nu < wnu.size(); ++nu) skip[nu] = wnu[nu] < P->w_ac ? 1 : 0;
    T->skip = to_device(ctx, skip);
  }
  // B of the contraction: G [nk, ni] column-major is G^T row-major [ni][nk].
  split3_rows_kernel<<<div_up(size_t(ni * T->Kp), 256), 256, 0, s>>>(P->d_G.p, nk, ni, nk, T->Kp, false, T->G[0].p,
                                                                     T->G[1].p, T->G[2].p);
  EPSP_LAUNCHED(ctx);
  // A of the Kramers-Kronig map: A[ω][ω'] = KK[ω + nω ω'].
  split3_rows_kernel<<<div_up(size_t(nw * T->Kp2), 256), 256, 0, s>>>(P->d_KK.p, nw, nw, nw, T->Kp2, true, T->KK[0].p,
                                                                      T->KK[1].p, T->KK[2].p);
  EPSP_LAUNCHED(ctx);
  tc_gemm_shape(ctx, int(nw), int(ni), int(nk), max_splits_for(nk), kNs, &T->bn1, &T->splits1, kKbCap);
  tc_gemm_shape(ctx, int(nw), int(ni), int(nw), max_splits_for(nw, kKbCapKK), kNs, &T->bn2, &T->splits2, kKbCapKK);
  T->part.alloc(ctx, size_t(std::max(T->splits1, T->splits2)) * size_t(nw * ni));
  const long nwm = nw * P->nm;
  T->tf.alloc(ctx, size_t(2 * nwm));
  T->Ff.alloc(ctx, size_t(2 * nwm));
  T->ef.alloc(ctx, size_t(P->nc));
  T->rec.alloc(ctx, size_t((nw + 1) * ni));
  T->dim.alloc(ctx, size_t((nw + 1) * ni));
  T->modes.alloc(ctx, size_t(P->nm));
  split_q_kernel<<<div_up(size_t(2 * nwm), 256), 256, 0, s>>>(P->d_cell_t.p, 2 * nwm, P->re_qmd, T->tf.p);
  EPSP_LAUNCHED(ctx);
  split_q_kernel<<<div_up(size_t(P->nc), 256), 256, 0, s>>>(P->d_epsc.p, P->nc, P->re_qmd, T->ef.p);
  EPSP_LAUNCHED(ctx);
  T->opK = operand(T->Kt, nw, nk, T->Kp, kTcBM);
  T->opG = operand(T->G, ni, nk, T->Kp, T->bn1);
  T->opKK = operand(T->KK, nw, nw, T->Kp2, kTcBM);
  T->opIm = operand(T->Im, ni, nw, T->Kp2, T->bn2);
}

static void check_err(Scgd0Plan* P) {
  int e = 0;
  P->tc->err.download(&e, 1, P->ctx->stream);
  EPSP_CUDA(cudaStreamSynchronize(P->ctx->stream));
  if (e) {
    P->tc->err.zero(P->ctx->stream);  // cleared, so that the plan's next call starts clean
    fail(EPSP_EDEVICE_TIMEOUT, "a tensor-core GEMM wait ran out (bounded device wait)");
  }
}

// Nodes of a thread: two as soon as one tile does not hold them all (a dispersive run at 501 nodes: 28.4 ms, with one
// 32.1; the second node's work is skipped by the warps that have none).
static int fd_nodes(const Scgd0Plan* P) { return P->nw > kFdTile ? 2 : 1; }

// Splits of the (ν, f) range for nA slots: about 40 blocks a multiprocessor (three are resident, so the last wave is a
// small part of the time), two tiles of pairs a split at least (a block's tables and tail; with eight, which left SMs
// idle, 416 nodes x 60 states x 2 temperatures took 1.5 times as long, 208 x 30 2.5 times, 501 x 105 as long).
static int fd_splits(const Scgd0Plan* P, long nA) {
  const long tiles = div_up(size_t(P->nm * P->nf), kFdTile);
  const long blocks = long(div_up(size_t(P->nw), size_t(kFdTile * fd_nodes(P)))) * P->ni * nA;
  const long want = std::max<long>(1, (40l * P->ctx->sm_count + blocks - 1) / blocks);
  const long n = std::min(want, std::max<long>(1, tiles / 2));
  return int(div_up(size_t(tiles), div_up(size_t(tiles), size_t(n))));  // no empty split
}

// The Fan-Migdal sum term by term over nA slots (Σ_in in T->Sf): into ImS_b and the Kramers-Kronig operand, or
// added into add_out (one slot).
static void launch_fm_disp(Scgd0Plan* P, int nA, const int* d_slots, const TParams* d_tp, double* ImS_b,
                           double* add_out) {
  Ctx* ctx = P->ctx;
  auto* T = P->tc.get();
  const long nw = P->nw, ni = P->ni;
  if (P->fd_fast) {
    const long slab = nw * ni, ncell = (nw + 1) * ni, nvf = P->nm * P->nf;
    ensure(T->fdrec, ctx, size_t(ncell * nA));
    ensure(T->fddim, ctx, size_t(ncell * nA));
    const double u_hi = std::rint(P->fd_unit / P->re_q) * P->re_q;
    fd_cell_kernel<<<dim3(div_up(size_t(ncell), 256), unsigned(nA)), 256, 0, ctx->stream>>>(
        T->Sf.p, d_slots, P->d_ws.p, int(nw), slab, P->fd_unit, u_hi, P->re_qmd, T->fdrec.p, T->fddim.p);
    EPSP_LAUNCHED(ctx);
    const size_t tab = sizeof(uint32_t) * P->d_fdtab.n;
    const int nsplit = fd_splits(P, nA), npt = fd_nodes(P);
    const long per = (div_up(size_t(nvf), kFdTile) + nsplit - 1) / nsplit * kFdTile;
    ensure(T->fdpart, ctx, size_t(slab * nA) * size_t(nsplit));
    const dim3 grid(div_up(size_t(nw), size_t(kFdTile * npt)), unsigned(ni), unsigned(nA * nsplit));
    auto go = [&](auto kern, size_t bytes) {
      EPSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
      kern<<<grid, kFdTile, bytes, ctx->stream>>>(int(nw), slab, T->fdrec.p, T->fddim.p, P->d_wtab.p, P->d_fdoff.p,
                                                  P->d_fdtab.p, int(P->d_fdtab.n), P->fd_pad, P->fd_unit, 1.0 / P->fd_unit, P->re_qmd, u_hi, P->d_gwf.p, P->d_wph.p, P->d_iq.p, P->d_iksi.p, P->d_iksf.p, P->nk_i, P->d_epsf.p,
                                                  P->d_fti.p, int(P->nm), nvf, per, nsplit, P->w_ac, d_slots, d_tp,
                                                  T->fdpart.p);
    };
    const bool smem = tab <= (size_t(96) << 10);
    if (npt == 2)
      smem ? go(fm_disp_fast_kernel<2, true>, tab) : go(fm_disp_fast_kernel<2, false>, size_t(0));
    else
      smem ? go(fm_disp_fast_kernel<1, true>, tab) : go(fm_disp_fast_kernel<1, false>, size_t(0));
    EPSP_LAUNCHED(ctx);
    fd_finish_kernel<<<dim3(div_up(size_t(slab), 256), unsigned(nA)), 256, 0, ctx->stream>>>(
        T->fdpart.p, int(nw), slab, nsplit, ImS_b, T->Im[0].p, T->Im[1].p, T->Im[2].p, T->Kp2, add_out);
    EPSP_LAUNCHED(ctx);
    return;
  }
  // the grid nodes and the bucket table in shared memory when they fit 96 KB
  const size_t tab = sizeof(float4) * size_t(nw) + sizeof(int32_t) * size_t(P->ntab);
  const bool smem = tab <= (size_t(96) << 10);
  const dim3 grid(div_up(size_t(nw), kFdTile), unsigned(ni), unsigned(nA));
  static size_t smem_set = 0;
  if (smem && tab > smem_set) {
    EPSP_CUDA(cudaFuncSetAttribute(fm_disp_f32_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tab)));
    smem_set = tab;
  }
  auto args = [&](auto kern, size_t bytes) {
    kern<<<grid, kFdTile, bytes, ctx->stream>>>(
        int(nw), nw * ni, T->Sf.p, P->d_wtab.p, P->d_jtab.p, P->x0f, P->inv_hf, P->ntab, P->d_gwf.p, P->d_wph.p,
        P->d_iq.p, P->d_iksi.p, P->d_iksf.p, P->nk_i, P->d_epsf.p, P->d_fti.p, int(P->nm), P->nm * P->nf, int(ni),
        P->w_ac, d_slots, d_tp, ImS_b, T->Im[0].p, T->Im[1].p, T->Im[2].p, T->Kp2, add_out);
  };
  if (smem)
    args(fm_disp_f32_kernel<true>, tab);
  else
    args(fm_disp_f32_kernel<false>, size_t(0));
  EPSP_LAUNCHED(ctx);
}

// Whether the plan has the table of fm_disp_fast_kernel and the temperatures of a call allow it (every exp(ωq/T) within
// e^40; ω_acoustic above 0, so that n(ωq) is finite). Reserves its buffers for nT slots, so that none is allocated while a graph is captured.
void tc_disp_choose(Scgd0Plan* P, const double* Tlist, long nT) {
  if (!P->disp) return;
  P->fd_fast = P->w_ac > 0 && P->d_fdtab.n > 0;
  for (long t = 0; t < nT; ++t) P->fd_fast = P->fd_fast && Tlist[t] > 1.4901161193847656e-08 && P->wq_max <= kFdMaxArg * Tlist[t];
  if (!P->fd_fast) return;
  auto* T = P->tc.get();
  const size_t n = size_t((P->nw + 1) * P->ni) * size_t(nT);
  bool grown = ensure(T->fdrec, P->ctx, n);
  grown |= ensure(T->fddim, P->ctx, n);
  size_t part = 0;
  for (long a = 1; a <= nT; ++a) part = std::max(part, size_t(P->nw * P->ni) * size_t(a) * size_t(fd_splits(P, a)));
  grown |= ensure(T->fdpart, P->ctx, part);
  if (grown) ++P->w_gen;
}

// One Fan-Migdal sum at (μ, T) for a model with dispersive modes, added into d_ImS.
void tc_imsigma_disp(Scgd0Plan* P, const double2* d_Sin, double mu, double T, double* d_ImS) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  auto* T_ = P->tc.get();
  const long nw = P->nw, ni = P->ni;
  sigma_f32_kernel<<<div_up(size_t(nw * ni), 256), 256, 0, s>>>(d_Sin, nw * ni, T_->Sf.p);
  EPSP_LAUNCHED(ctx);
  tc_disp_choose(P, &T, 1);
  TParams q{};
  q.T = T;
  q.inv_T = 1.0 / T;
  q.mu = mu;
  DBuf<TParams> d_q = to_device(ctx, &q, 1);
  DBuf<int> d_slot0;
  d_slot0.alloc(ctx, 1);
  d_slot0.zero(s);
  long pk = prof_begin(ctx, "fm_disp");
  launch_fm_disp(P, 1, d_slot0.p, d_q.p, nullptr, d_ImS);
  prof_end(ctx, pk);
  EPSP_CUDA(cudaStreamSynchronize(s));  // the parameter buffers are locals
}

// fm_disp_fast_kernel's nodes and cell table in units of the offsets' common divisor. None where ωq or a cell is too wide
// in them, the table too long, or the records' offsets pass 32 bits: those plans keep fm_disp_f32_kernel.
static void fd_table(Scgd0Plan* P) {
  const GridHost& g = P->ws;
  const long nw = P->nw;
  long div = 0, widest = 0;
  for (long j = 1; j < nw; ++j) {
    const long d = g.offsets[size_t(j)] - g.offsets[size_t(j - 1)];
    div = std::gcd(div, d);
    widest = std::max(widest, d);
  }
  div = std::max(1l, div);
  const double unit = g.unit * double(div), wq = P->wq_max / unit;
  if (!(wq < double(kFdMaxCell - 1)) || widest / div > kFdMaxCell || nw > 65534 || (nw + 1) * P->ni >= (1l << 31)) return;
  const long pad = long(std::floor(std::max(0.0, wq))) + 2;  // the whole numbers are 0 .. pad - 1 (rounded up at most)
  const long range = (g.offsets[size_t(nw - 1)] - g.offsets[0]) / div, n = range + 2 * pad;
  if (n > kFdMaxTable) return;
  std::vector<int32_t> off(static_cast<size_t>(nw));
  for (long j = 0; j < nw; ++j) off[size_t(j)] = int32_t((g.offsets[size_t(j)] - g.offsets[0]) / div);
  std::vector<uint32_t> tab(static_cast<size_t>(n));
  long c = 0;  // the cell of b: the nodes at or below it
  for (long e = 0; e < n; ++e) {
    const long b = e - pad;
    while (c < nw && off[size_t(c)] <= b) ++c;
    tab[size_t(e)] = uint32_t(c) << 16 | uint32_t(b - off[size_t(std::max(0l, c - 1))] + 32768);
  }
  P->fd_unit = unit;
  P->fd_pad = int(pad);
  P->d_fdoff = to_device(P->ctx, off);
  P->d_fdtab = to_device(P->ctx, tab);
  EPSP_CUDA(cudaStreamSynchronize(P->ctx->stream));  // off and tab are locals
}

// The tables of fm_disp_f32_kernel (see Scgd0Plan): w_f g2 permuted to [ν f, i] and rounded to
// FP32, ωph, iq_kk, iks_i, iks_f, f_to_i, ε_f and the grid nodes as float pairs, the bucket table's
// origin and scale. ωq itself is gathered per term, never stored.
void tc_setup_dispersive(Scgd0Plan* P, const epsp_model* m) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  P->disp = true;
  const long nm = m->nm, ni = m->ni, nf = m->nf, nvf = nm * nf;
  {
    DBuf<double> g2t;
    upload_g2_permuted(ctx, m, g2t);
    auto d_wf = to_device(ctx, m->w_f, size_t(nf));
    auto d_fti = to_device(ctx, m->f_to_i, size_t(nf));
    P->d_gwf.alloc(ctx, size_t(nvf * ni));
    gw_f32_kernel<<<div_up(size_t(nvf * ni), 256), 256, 0, s>>>(g2t.p, d_wf.p, int(nm), nvf, ni, P->d_gwf.p);
    EPSP_LAUNCHED(ctx);
    EPSP_CUDA(cudaStreamSynchronize(s));
  }
  for (int64_t k = 0; k < nm * m->nq; ++k)
    P->wq_max = std::isfinite(m->omega_ph[k]) ? std::max(P->wq_max, m->omega_ph[k]) : std::numeric_limits<double>::infinity();
  P->d_wph = to_device(ctx, m->omega_ph, size_t(nm * m->nq));
  P->d_iq = to_device(ctx, m->iq_kk, size_t(m->nk_i * m->nk_f));
  P->d_iksi = to_device(ctx, m->iks_i, size_t(ni));
  P->d_iksf = to_device(ctx, m->iks_f, size_t(nf));
  P->d_fti = to_device(ctx, m->f_to_i, size_t(nf));
  P->nk_i = m->nk_i;
  P->d_epsf = to_device(ctx, m->eps_f, size_t(nf));
  P->d_wtab.alloc(ctx, size_t(P->nw));
  fd_node_table_kernel<<<div_up(size_t(P->nw), 256), 256, 0, s>>>(P->d_ws.p, int(P->nw), P->d_wtab.p);
  EPSP_LAUNCHED(ctx);
  fd_table(P);
  P->x0f = float(P->ct.x0);
  P->inv_hf = float(P->ct.inv_h);
  P->ntab = long(P->d_jtab.n);
  if (P->ntab >= (long(1) << 21))
    fail(EPSP_EUNSUPPORTED, "the grid's cell-search table is too long for the FP32 dispersive path (2^21 buckets at "
                            "most); use EPSP_PATH_DIRECT_FP64");
  EPSP_CUDA(cudaStreamSynchronize(s));
}

void tc_imsigma(Scgd0Plan* P, const double2* d_Sin, double* d_ImS) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  auto* T = P->tc.get();
  const long nw = P->nw, ni = P->ni, nk = P->nm * P->nc;
  long pk = prof_begin(ctx, "kbuild");
  const long nwm = nw * P->nm;
  cell_records_kernel<<<div_up(size_t(nw * ni), 256), 256, 0, s>>>(d_Sin, nullptr, nullptr, P->d_wtab.p, P->re_qm, int(nw), nw * ni,
                                                                   T->rec.p, T->dim.p);
  EPSP_LAUNCHED(ctx);
  to_f32_kernel<<<div_up(size_t(nwm), 256), 256, 0, s>>>(P->d_Fa.p, nwm, T->Ff.p);
  EPSP_LAUNCHED(ctx);
  to_f32_kernel<<<div_up(size_t(nwm), 256), 256, 0, s>>>(P->d_Fe.p, nwm, T->Ff.p + nwm);
  EPSP_LAUNCHED(ctx);
  kbuild_bf16_kernel<<<dim3(div_up(size_t(nw), kKbW), unsigned(div_up(size_t(T->Kp), size_t(kKbCols * P->nm))), 1), 256,
                       kbuild_smem_bytes(P->nm), s>>>(int(nw), int(ni), T->rec.p, T->dim.p, nullptr, P->d_cell_j.p, T->tf.p,
                                                      T->skip.p, int(P->nm), T->ef.p, P->d_colc.p, int(P->nc), T->Ff.p,
                                                      T->Kt[0].p, T->Kt[1].p, T->Kt[2].p, T->Kp, nullptr);
  EPSP_LAUNCHED(ctx);
  prof_end(ctx, pk);
  const long slab = nw * ni;
  int sp = tc_gemm_launch(ctx, T->opK, T->opG, int(nw), int(ni), int(nk), T->part.p, nw, slab, max_splits_for(nk),
                          T->err.p, "tc_fm", kKbCap);
  finalize_add_kernel<<<div_up(size_t(slab), 256), 256, 0, s>>>(T->part.p, slab, sp, slab, d_ImS);
  EPSP_LAUNCHED(ctx);
  check_err(P);
}

void tc_reserve(Scgd0Plan* P, long nT) {
  auto* T = P->tc.get();
  if (nT <= T->capT && T->ImS_b.p) return;
  Ctx* ctx = P->ctx;
  const long nw = P->nw, ni = P->ni, nk = P->nm * P->nc, nwm = nw * P->nm, slab = nw * ni;
  nT = std::max(nT, T->capT);
  if (nT * nw > (1l << 30) || nT * ni > (1l << 30)) fail(EPSP_EINVAL, "too many temperatures for the 32-bit tile grid");
  for (int p = 0; p < kNs; ++p) {
    if (!P->disp) T->Kt[p].alloc(ctx, size_t(nT * nw * T->Kp));
    T->Im[p].alloc(ctx, size_t(nT * ni * T->Kp2));
    T->Im[p].zero(ctx->stream);  // the padding columns nω.. Kp2 of the KK operand stay zero
  }
  if (P->disp) {
    T->Sf.alloc(ctx, size_t(nT * slab));
  } else {
    T->rec.alloc(ctx, size_t(nT * (nw + 1) * ni));
    T->dim.alloc(ctx, size_t(nT * (nw + 1) * ni));
    T->modes.alloc(ctx, size_t(nT * P->nm));
    T->Ff.alloc(ctx, size_t(nT * 2 * nwm));
  }
  T->ImS_b.alloc(ctx, size_t(nT * slab));
  size_t part = 0;
  for (long a = 1; a <= nT; ++a) {
    int bn, sp1 = 1, sp2;
    if (!P->disp) tc_gemm_shape(ctx, int(a * nw), int(ni), int(nk), max_splits_for(nk), kNs, &bn, &sp1, kKbCap);
    tc_gemm_shape(ctx, int(nw), int(a * ni), int(nw), max_splits_for(nw, kKbCapKK), kNs, &bn, &sp2, kKbCapKK);
    part = std::max(part, size_t(std::max(sp1, sp2)) * size_t(a * slab));
  }
  T->part.alloc(ctx, part);
  if (!P->disp) T->opK = operand(T->Kt, nT * nw, nk, T->Kp, kTcBM);
  T->opIm = operand(T->Im, nT * ni, nw, T->Kp2, T->bn2);
  T->capT = nT;
}


int* tc_err_ptr(Scgd0Plan* P) { return P->tc->err.p; }

long tc_capacity(Scgd0Plan* P) { return P->tc->ImS_b.p ? P->tc->capT : 0; }

void tc_start(Scgd0Plan* P, long nT, const TParams* d_tp) {
  if (P->disp) return;
  mode_table_kernel<<<dim3(div_up(size_t(P->nm), 32), unsigned(nT)), 32, 0, P->ctx->stream>>>(P->d_wnu.p, int(P->nm), d_tp,
                                                                                            P->w_ac, P->tc->modes.p);
  EPSP_LAUNCHED(P->ctx);
}

void tc_take_sigma(Scgd0Plan* P, int nA, const int* d_slots, const TParams* d_tp, const double2* d_S_all) {
  auto* T = P->tc.get();
  const long slab = P->nw * P->ni;
  const dim3 grid(div_up(size_t(slab), 256), unsigned(nA));
  if (P->disp)
    clamp_f32_kernel<<<grid, 256, 0, P->ctx->stream>>>(d_S_all, T->Sf.p, slab, d_slots, d_tp);
  else
    cell_records_kernel<<<grid, 256, 0, P->ctx->stream>>>(d_S_all, d_slots, d_tp, P->d_wtab.p, P->re_qm, int(P->nw), slab, T->rec.p,
                                                          T->dim.p);
  EPSP_LAUNCHED(P->ctx);
}

static void tc_kk_tail(Scgd0Plan* P, int nA, const int* d_slots, const TParams* d_tp, double2* d_S_all, float4* d_P,
                       unsigned long long* d_errbits, double* d_minA, const IterCtl* ctl);

void tc_iterate(Scgd0Plan* P, int nA, const int* d_slots, const TParams* d_tp, double2* d_S_all, float4* d_P,
                unsigned long long* d_errbits, double* d_minA, IterCtl* ctl) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  auto* T = P->tc.get();
  if (nA > T->capT) fail(EPSP_EINVAL, "more active temperatures than reserved");
  const long nw = P->nw, ni = P->ni, nk = P->nm * P->nc, slab = nw * ni;
  const unsigned eb = div_up(size_t(slab), 256);
  if (P->disp) {  // dispersive modes: ImΣ of every slot term by term, then the same Kramers-Kronig tail
    long pk = prof_begin(ctx, "fm_disp");
    launch_fm_disp(P, nA, d_slots, d_tp, T->ImS_b.p, nullptr);
    prof_end(ctx, pk);
    tc_kk_tail(P, nA, d_slots, d_tp, d_S_all, d_P, d_errbits, d_minA, nullptr);
    return;
  }
  long pp = prof_begin(ctx, "kprep");
  occ_table_f32_kernel<<<dim3(div_up(size_t(nw), kOccW), unsigned(nA)), 64, 0, s>>>(
      P->d_ws.p, int(nw), P->d_wnu.p, int(P->nm), d_slots, d_tp, T->modes.p, P->w_ac, T->Ff.p, d_errbits, ctl);
  EPSP_LAUNCHED(ctx);
  prof_end(ctx, pp);
  long pk = prof_begin(ctx, "kbuild");
  launch_after(s, kbuild_bf16_kernel,
               dim3(div_up(size_t(nw), kKbW), unsigned(div_up(size_t(T->Kp), size_t(kKbCols * P->nm))), unsigned(nA)), 256,
               kbuild_smem_bytes(P->nm), int(nw), int(ni), T->rec.p, T->dim.p, d_slots, P->d_cell_j.p, T->tf.p, T->skip.p,
               int(P->nm), T->ef.p, P->d_colc.p, int(P->nc), T->Ff.p, T->Kt[0].p, T->Kt[1].p, T->Kt[2].p, T->Kp, ctl);
  EPSP_LAUNCHED(ctx);
  prof_end(ctx, pk);
  // ImΣ of every slot: the stacked K_t rows times G
  const long M = long(nA) * nw;
  int sp = tc_gemm_launch(ctx, T->opK, T->opG, int(M), int(ni), int(nk), T->part.p, M, M * ni, max_splits_for(nk),
                          T->err.p, "tc_fm", kKbCap, ctl ? &ctl->stop : nullptr);
  // ImΣ of every slot, and its BF16 split as the B operand of ReΣ = KK ImΣ (columns: the slots'
  // states in order)
  long pf = prof_begin(ctx, "finalize");
  launch_after(s, finalize_fm_batch_kernel, dim3(eb, unsigned(nA)), 256, 0, T->part.p, int(nw), slab, nA, sp, M * ni,
               T->ImS_b.p, T->Im[0].p, T->Im[1].p, T->Im[2].p, T->Kp2, ctl);
  EPSP_LAUNCHED(ctx);
  prof_end(ctx, pf);
  tc_kk_tail(P, nA, d_slots, d_tp, d_S_all, d_P, d_errbits, d_minA, ctl);
}

// ReΣ = KK ImΣ for every slot (the split ImΣ rows already in T->Im) and the fused epilogue.
static void tc_kk_tail(Scgd0Plan* P, int nA, const int* d_slots, const TParams* d_tp, double2* d_S_all, float4* d_P,
                       unsigned long long* d_errbits, double* d_minA, const IterCtl* ctl) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  auto* T = P->tc.get();
  const long nw = P->nw, ni = P->ni, slab = nw * ni;
  const long N2 = long(nA) * ni;
  int sp2 = tc_gemm_launch(ctx, T->opKK, T->opIm, int(nw), int(N2), int(nw), T->part.p, nw, nw * N2,
                           max_splits_for(nw, kKbCapKK), T->err.p, "tc_kk", kKbCapKK, ctl ? &ctl->stop : nullptr);
  long pf = prof_begin(ctx, "kk_epilogue");
  launch_after(s, kk_epilogue_kernel, dim3(div_up(size_t(nw), 255), unsigned(P->ngroups), unsigned(nA)), 256, 0, T->part.p,
               sp2, nw * N2, T->ImS_b.p, int(nw), slab, d_slots, P->d_gptr.p, P->d_gidx.p, P->d_wtab.p, P->re_qm, T->epair.p, d_tp,
               d_S_all, T->Sf.p, T->rec.p, T->dim.p, d_P, d_errbits, d_minA, ctl);
  EPSP_LAUNCHED(ctx);
  prof_end(ctx, pf);
}

}  // namespace epsp
