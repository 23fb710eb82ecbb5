// tc_gemm.cu -- host side of the tcgen05 GEMMs (BF16x3, TF32): tensor maps, tile shape, split-K choice.
#include "tc_gemm.cuh"

#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <set>

namespace epsp {

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  if (!fn) fail(EPSP_ECUDA, "cuTensorMapEncodeTiled is not available from the driver");
  return fn;
}

CUtensorMap make_tmap_bf16(const void* base, long rows, long cols, long ld, int box_rows, int bk) {
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld * 2) % 16 != 0)
    fail(EPSP_EINVAL, "tensor map base and row stride must be 16-byte aligned");
  if (bk != 64 && bk != 32) fail(EPSP_EINVAL, "tensor map K box must be 64 or 32 columns");
  CUtensorMap m;
  cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows)};
  cuuint64_t strides[1] = {cuuint64_t(ld * 2)};
  cuuint32_t box[2] = {cuuint32_t(bk), cuuint32_t(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(EPSP_ECUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return m;
}

CUtensorMap make_tmap_f32(const void* base, long rows, long cols, long ld, int box_rows, int bk) {
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld * 4) % 16 != 0)
    fail(EPSP_EINVAL, "tensor map base and row stride must be 16-byte aligned");
  if (bk != 32 && bk != 16) fail(EPSP_EINVAL, "FP32 tensor map K box must be 32 or 16 columns");
  CUtensorMap m;
  cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows)};
  cuuint64_t strides[1] = {cuuint64_t(ld * 4)};
  cuuint32_t box[2] = {cuuint32_t(bk), cuuint32_t(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, bk == 32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(EPSP_ECUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return m;
}

void tc_gemm_shape(Ctx* ctx, int M, int N, int K, int max_splits, int ns, int* bn, int* splits, int kb_cap) {
  const int BN = (ns == 2 && N > 128) ? 256 : 128;
  const int tiles = ((M + kTcBM - 1) / kTcBM) * ((N + BN - 1) / BN);
  const int kblocks = (K + kTcBK - 1) / kTcBK;
  const int cap = std::min(std::max(1, max_splits), std::max(1, kblocks));
  if (kb_cap <= 0) {  // fill the SMs once; no accumulation bound
    int sp = std::min(std::max(1, (ctx->sm_count + tiles - 1) / tiles), cap);
    const int per = (kblocks + sp - 1) / sp;
    *bn = BN;
    *splits = std::max(1, (kblocks + per - 1) / per);
    return;
  }
  int lo = std::min(std::max(1, (kblocks + kb_cap - 1) / kb_cap), cap);
  // With an accumulation bound (the scGD0 products): one CTA per SM (the operand stages fill shared
  // memory), so a launch takes ceil(CTAs / SMs) rounds of ceil(kblocks / splits) K blocks each,
  // plus a CTA's fixed cost (pipeline fill, TMEM, the epilogue's partial slab) of about three K
  // blocks. Take the split count with the shortest such critical path (ties: fewer splits, whose
  // partial sums cost less), from the smallest the accumulation bound allows up to a little past
  // the one that first fills every SM.
  const int hi = std::min(cap, std::max(lo, 2 * ((ctx->sm_count + tiles - 1) / tiles) + 8));
  int best = lo;
  long best_cost = -1;
  for (int sp = lo; sp <= hi; ++sp) {
    const int per = (kblocks + sp - 1) / sp;
    const int used = (kblocks + per - 1) / per;
    const long rounds = (long(tiles) * used + ctx->sm_count - 1) / ctx->sm_count;
    const long cost = rounds * (per + 3);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = used;
    }
  }
  *bn = BN;
  *splits = best;
}

template <int BN, int STAGES, int NS, int BK = kTcBK, bool TF32 = false>
static void launch(Ctx* ctx, const TcOperand& A, const TcOperand& B, int M, int N, int kblocks, int per, int splits,
                   float* out, long ld_out, long split_stride, int* d_err, int gm = 1) {
  using L = TcSmem<BN, STAGES, NS, BK, TF32>;
  if (A.bk != BK || B.bk != BK) fail(EPSP_EINVAL, "operand tensor maps were built for another K block");
  if (A.tf32 != TF32 || B.tf32 != TF32) fail(EPSP_EINVAL, "operand tensor maps were built for another element type");
  static bool configured = false;  // one process, one attribute setting per instantiation
  if (!configured) {
    EPSP_CUDA(cudaFuncSetAttribute(tc_gemm_split_kernel<BN, STAGES, NS, BK, TF32>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
    configured = true;
  }
  TcMaps maps;
  for (int p = 0; p < 3; ++p) {
    maps.a[p] = A.m[p < NS ? p : 0];
    maps.b[p] = B.m[p < NS ? p : 0];
  }
  dim3 grid((N + BN - 1) / BN, (M + kTcBM - 1) / kTcBM, splits);
  tc_gemm_split_kernel<BN, STAGES, NS, BK, TF32><<<grid, 128, L::kBytes, ctx->stream>>>(
      maps, M, N, kblocks, per, out, ld_out, split_stride, d_err, gm, ctx->stall_kb,
      ctx->stall_wait_limit ? ctx->stall_wait_limit : kWaitLimit);
  EPSP_LAUNCHED(ctx);
}

// Part p of an operand mapped again with boxes of box_rows rows (from the matrix behind its maps).
static CUtensorMap remap(const TcOperand& op, int p, int box_rows) {
  if (!op.base[p]) fail(EPSP_EINVAL, "internal: operand without its matrix description");
  return op.tf32 ? make_tmap_f32(op.base[p], op.rows, op.cols, op.ld, box_rows, op.bk)
                 : make_tmap_bf16(op.base[p], op.rows, op.cols, op.ld, box_rows, op.bk);
}

template <int BN, int STAGES, int NS, int BK, bool TF32 = false, int NA = NS>
static void launch_persist(Ctx* ctx, const TcOperand& A, const TcOperand& B, int M, int N, int kblocks, int per,
                           int splits, float* out, long ld_out, long split_stride, int* d_err, int gm = 1, const int* skip = nullptr) {
  using L = TcPSmem<BN, STAGES, NS, BK, TF32, NA>;
  if (A.bk != BK || B.bk != BK) fail(EPSP_EINVAL, "operand tensor maps were built for another K block");
  if (A.tf32 != TF32 || B.tf32 != TF32) fail(EPSP_EINVAL, "operand tensor maps were built for another element type");
  auto* kern = tc_gemm_persist_kernel<BN, STAGES, NS, BK, TF32, NA>;
  static bool configured = false;  // one process, one attribute setting per instantiation
  if (!configured) {
    EPSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
    configured = true;
  }
  TcMaps maps;
  for (int p = 0; p < 3; ++p) {
    maps.a[p] = A.m[p < NA ? p : 0];
    maps.b[p] = B.m[p < NS ? p : 0];
  }
  const int nN = (N + BN - 1) / BN, nM = (M + kTcBM - 1) / kTcBM;
  const int nitems = nN * nM * splits;  // (N tile, M tile, split)
  const int grid = std::min(nitems, ctx->sm_count);
  launch_after(ctx->stream, kern, grid, 192, L::kBytes, maps, M, N, kblocks, per, nN, nM, nitems, out, ld_out, split_stride,
               d_err, gm, skip);
  EPSP_LAUNCHED(ctx);
}

// The CTA-pair kernel: clusters of two CTAs, each pair one 256 x BN tile (B halves of BN / 2 rows).
template <int BN, int STAGES, int NS, int BK, bool TF32>
static void launch_pair(Ctx* ctx, const TcOperand& A, const TcOperand& B, int M, int N, int kblocks, int per,
                        int splits, float* out, long ld_out, long split_stride, int* d_err, int gm = 1) {
  using L = TcPairSmem<BN, STAGES, NS, BK, TF32>;
  if (A.bk != BK || B.bk != BK) fail(EPSP_EINVAL, "operand tensor maps were built for another K block");
  if (A.tf32 != TF32 || B.tf32 != TF32) fail(EPSP_EINVAL, "operand tensor maps were built for another element type");
  auto* kern = tc_gemm_pair_kernel<BN, STAGES, NS, BK, TF32>;
  static bool configured = false;  // one process, one attribute setting per instantiation
  if (!configured) {
    EPSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
    configured = true;
  }
  TcMaps maps;
  for (int p = 0; p < 3; ++p) {
    maps.a[p] = A.m[p < NS ? p : 0];
    maps.b[p] = p < NS ? remap(B, p, BN / 2) : maps.b[0];  // B halves of BN / 2 rows, each part encoded once
  }
  cudaLaunchAttribute cl;
  cl.id = cudaLaunchAttributeClusterDimension;
  cl.val.clusterDim.x = 2;
  cl.val.clusterDim.y = 1;
  cl.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(2 * ((N + BN - 1) / BN)), unsigned((M + 2 * kTcBM - 1) / (2 * kTcBM)), unsigned(splits));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = L::kBytes;
  cfg.stream = ctx->stream;
  cfg.attrs = &cl;
  cfg.numAttrs = 1;
  EPSP_CUDA(cudaLaunchKernelEx(&cfg, kern, maps, M, N, kblocks, per, out, ld_out, split_stride, d_err, gm));
  EPSP_LAUNCHED(ctx);
}

// The persistent CTA-pair kernel: one cluster of two CTAs per SM pair over all items.
template <int BN, int STAGES, int NS, int BK, bool TF32>
static void launch_pair_persist(Ctx* ctx, const TcOperand& A, const TcOperand& B, int M, int N, int kblocks, int per,
                                int splits, float* out, long ld_out, long split_stride, int* d_err, int gm = 1) {
  using L = TcPairPSmem<BN, STAGES, NS, BK, TF32>;
  if (A.bk != BK || B.bk != BK) fail(EPSP_EINVAL, "operand tensor maps were built for another K block");
  if (A.tf32 != TF32 || B.tf32 != TF32) fail(EPSP_EINVAL, "operand tensor maps were built for another element type");
  auto* kern = tc_gemm_pair_persist_kernel<BN, STAGES, NS, BK, TF32>;
  static bool configured = false;  // one process, one attribute setting per instantiation
  if (!configured) {
    EPSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
    configured = true;
  }
  TcMaps maps;
  for (int p = 0; p < 3; ++p) {
    maps.a[p] = A.m[p < NS ? p : 0];
    maps.b[p] = p < NS ? remap(B, p, BN / 2) : maps.b[0];  // B halves of BN / 2 rows, each part encoded once
  }
  const int nN = (N + BN - 1) / BN, nM2 = (M + 2 * kTcBM - 1) / (2 * kTcBM);
  const long items = long(nN) * nM2 * splits;
  if (items > (1l << 30)) fail(EPSP_EINVAL, "too many tiles for the persistent kernel");
  const int npairs = int(std::min<long>(std::max(1, ctx->sm_count / 2), items));
  cudaLaunchAttribute cl[2];
  cl[0].id = cudaLaunchAttributeClusterDimension;
  cl[0].val.clusterDim.x = 2;
  cl[0].val.clusterDim.y = 1;
  cl[0].val.clusterDim.z = 1;
  cl[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (as launch_after: the kernel waits in pdl_wait)
  cl[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(2 * npairs), 1, 1);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = L::kBytes;
  cfg.stream = ctx->stream;
  cfg.attrs = cl;
  cfg.numAttrs = 2;
  EPSP_CUDA(cudaLaunchKernelEx(&cfg, kern, maps, M, N, kblocks, per, nN, nM2, int(items), out, ld_out, split_stride,
                               d_err, gm));
  EPSP_LAUNCHED(ctx);
}

int tc_gemm_launch(Ctx* ctx, const TcOperand& A, const TcOperand& B, int M, int N, int K, float* out, long ld_out,
                   long split_stride, int max_splits, int* d_err, const char* prof_name, int kb_cap, const int* skip) {
  if (A.tf32 || B.tf32) fail(EPSP_EINVAL, "TF32 operands take tc_gemm_launch_with");
  if (skip && (A.ns != 3 || A.bk != kTcBK)) fail(EPSP_EINVAL, "internal: the skip flag is for three-part operands");
  const bool one = A.ns == 1 && B.ns == 3;  // A exact in BF16
  if (!one && (A.ns != B.ns || (A.ns != 2 && A.ns != 3))) fail(EPSP_EINVAL, "operands must be split into 2 or 3 parts alike");
  if (A.bk != B.bk) fail(EPSP_EINVAL, "operands built for different K blocks");
  int BN, splits;
  tc_gemm_shape(ctx, M, N, K, max_splits, B.ns, &BN, &splits, kb_cap);  // splits from K blocks of 64
  const int bk = A.bk;
  const int kblocks = (K + bk - 1) / bk;
  const int per = (kblocks + splits - 1) / splits;
  splits = (kblocks + per - 1) / per;
  long pi = prof_begin(ctx, prof_name);
  if (one && bk == kTcBK)
    launch_persist<128, 3, 3, 64, false, 1>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err);
  else if (A.ns == 3 && bk == 32)  // three-part operands in K blocks of 32: four stages
    launch<128, 4, 3, 32>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err);
  else if (bk != kTcBK)
    fail(EPSP_EINVAL, "K blocks of 32 are for three-part operands here (tc_gemm_launch_with takes two-part ones)");
  else if (A.ns == 3)  // the persistent kernel: each SM's tiles back to back, epilogues overlapped
    launch_persist<128, 2, 3, 64>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, 1, skip);
  else if (BN == 256)
    launch_persist<256, 2, 2, 64>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err);
  else
    launch_persist<128, 3, 2, 64>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err);
  prof_end(ctx, pi);
  return splits;
}

int tc_splits_for(Ctx* ctx, int M, int N, int K, int bn) {
  const int kblocks = (K + kTcBK - 1) / kTcBK;
  const int tiles = ((M + kTcBM - 1) / kTcBM) * ((N + bn - 1) / bn);
  int sp = std::min(std::max(1, (ctx->sm_count + tiles - 1) / tiles), std::max(1, std::min(16, kblocks)));
  const int per = (kblocks + sp - 1) / sp;
  return std::max(1, (kblocks + per - 1) / per);
}

int tc_gemm_launch_with(Ctx* ctx, const TcOperand& A, const TcOperand& B, int bn, int splits, int M, int N, int K,
                        float* out, long ld_out, long split_stride, int* d_err, const char* prof_name, bool persist,
                        bool pair, int gm) {
  if (bn != 128 && bn != 256) fail(EPSP_EINVAL, "tile width must be 128 or 256");
  if (pair && bn != 256) fail(EPSP_EINVAL, "the CTA-pair kernels take tile width 256");
  if (A.tf32 || B.tf32) {
    if (!(A.tf32 && B.tf32 && A.ns == 1 && B.ns == 1 && A.bk == 32 && B.bk == 32))
      fail(EPSP_EINVAL, "TF32 operands are one-part maps with K boxes of 32 on both sides");
    const int kblocks = (K + 31) / 32;
    if (splits <= 0) splits = tc_splits_for(ctx, M, N, K, bn);
    splits = std::max(1, std::min(splits, kblocks));
    const int per = (kblocks + splits - 1) / splits;
    splits = (kblocks + per - 1) / per;
    long pi = prof_begin(ctx, prof_name);
    if (pair && persist)
      launch_pair_persist<256, 6, 1, 32, true>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err,
                                               gm);
    else if (pair)
      launch_pair<256, 6, 1, 32, true>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
    else if (persist && bn == 256)
      launch_persist<256, 4, 1, 32, true>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
    else if (persist)
      launch_persist<128, 6, 1, 32, true>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
    else if (bn == 256)
      launch<256, 4, 1, 32, true>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
    else
      launch<128, 6, 1, 32, true>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
    prof_end(ctx, pi);
    return splits;
  }
  if (A.ns != 2 || B.ns != 2) fail(EPSP_EINVAL, "explicit tile shapes are for two-part operands");
  const int bk = A.bk;
  if (bk == 32 && bn != 256) fail(EPSP_EINVAL, "K blocks of 32 come with tile width 256");
  const int kblocks = (K + bk - 1) / bk;
  if (splits <= 0) splits = tc_splits_for(ctx, M, N, K, bn);
  splits = std::max(1, std::min(splits, kblocks));
  const int per = (kblocks + splits - 1) / splits;
  splits = (kblocks + per - 1) / per;
  if (persist && !(bk == 32 && bn == 256)) fail(EPSP_EINVAL, "the persistent kernel takes tile width 256 with K blocks of 32");
  if (pair && bk != 32) fail(EPSP_EINVAL, "the BF16x3 CTA-pair kernel takes K blocks of 32");
  long pi = prof_begin(ctx, prof_name);
  if (pair && persist)
    launch_pair_persist<256, 6, 2, 32, false>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err,
                                              gm);
  else if (pair)
    launch_pair<256, 6, 2, 32, false>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
  else if (persist)
    launch_persist<256, 4, 2, 32>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
  else if (bk == 32)
    launch<256, 4, 2, 32>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
  else if (bn == 256)
    launch<256, 2, 2>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
  else
    launch<128, 3, 2>(ctx, A, B, M, N, kblocks, per, splits, out, ld_out, split_stride, d_err, gm);
  prof_end(ctx, pi);
  return splits;
}

// Tuned shapes are kept for the process, per device and product shape, so later plans of the same
// sizes reuse the measurement.
namespace {
std::mutex g_tune_mu;
std::map<std::array<long, 5>, std::vector<TcTune>> g_tune_cache;
}  // namespace

TcTune tc_gemm_autotune(Ctx* ctx, const TcOperand& A, const TcOperand& B128, const TcOperand& B256, int M, int N, int K,
                        float* out, long ld_out, long split_stride, int max_splits, int* d_err, int reps,
                        std::vector<TcTune>* all, const TcOperand* A32, const TcOperand* B256_32, int gm) {
  const std::array<long, 5> key{ctx->device, M, N, K,
                                max_splits + (A32 && B256_32 ? 1000 : 0) + (A.tf32 ? 2000 : 0) + 10000l * gm};
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
      TcTune best = it->second.front();
      for (const auto& c : it->second)
        if (c.ms < best.ms) best = c;
      if (all) *all = it->second;
      return best;
    }
  }
  std::vector<TcTune> cand;
  for (int bn : {256, 128}) {
    const int tiles = ((M + kTcBM - 1) / kTcBM) * ((N + bn - 1) / bn);
    const int h = std::max(1, (ctx->sm_count + tiles - 1) / tiles);
    // the heuristic count and twice it, within max_splits (so that every shape has candidates)
    const int cap = std::max(1, max_splits);
    std::vector<int> counts{std::min(h, cap)};
    if (std::min(2 * h, cap) != counts[0]) counts.push_back(std::min(2 * h, cap));
    for (int sp : counts) {
      if (A.tf32) {  // TF32: either tile width, either kernel
        cand.push_back(TcTune{bn, sp, 32, 0.f});
        cand.push_back(TcTune{bn, sp, 32, 0.f, true});
        if (bn == 256) cand.push_back(TcTune{bn, sp, 32, 0.f, false, true});  // CTA pairs
        if (bn == 256) cand.push_back(TcTune{bn, sp, 32, 0.f, true, true});   // persistent CTA pairs
        for (int g : {gm, 4 * gm}) {  // the same kernels in grouped tile order, two group sizes
          if (gm <= 1) break;
          cand.push_back(TcTune{bn, sp, 32, 0.f, false, false, g});
          cand.push_back(TcTune{bn, sp, 32, 0.f, true, false, g});
          if (bn == 256) cand.push_back(TcTune{bn, sp, 32, 0.f, false, true, g});
          if (bn == 256) cand.push_back(TcTune{bn, sp, 32, 0.f, true, true, g});
        }
        continue;
      }
      cand.push_back(TcTune{bn, sp, kTcBK, 0.f});
      if (bn == 256 && A32 && B256_32) {
        cand.push_back(TcTune{bn, sp, 32, 0.f});
        cand.push_back(TcTune{bn, sp, 32, 0.f, true});
        cand.push_back(TcTune{bn, sp, 32, 0.f, false, true});  // CTA pairs
        cand.push_back(TcTune{bn, sp, 32, 0.f, true, true});   // persistent CTA pairs
        for (int g : {gm, 4 * gm}) {
          if (gm <= 1) break;
          cand.push_back(TcTune{bn, sp, 32, 0.f, false, false, g});
          cand.push_back(TcTune{bn, sp, 32, 0.f, true, false, g});
          cand.push_back(TcTune{bn, sp, 32, 0.f, false, true, g});
          cand.push_back(TcTune{bn, sp, 32, 0.f, true, true, g});
        }
      }
    }
  }
  cudaEvent_t e0, e1;
  EPSP_CUDA(cudaEventCreate(&e0));
  EPSP_CUDA(cudaEventCreate(&e1));
  TcTune best{};
  best.ms = 3.4e38f;
  // A32 / B256_32: the BF16 operands with K boxes of 32 (TF32 operands have one K box, 32)
  auto opA = [&](const TcTune& c) -> const TcOperand& { return c.bk == 32 && !A.tf32 ? *A32 : A; };
  auto opB = [&](const TcTune& c) -> const TcOperand& {
    return c.bk == 32 && !A.tf32 ? *B256_32 : (c.bn == 256 ? B256 : B128);
  };
  auto timed = [&](const TcTune& c) {
    float ms = 0.f;
    EPSP_CUDA(cudaEventRecord(e0, ctx->stream));
    tc_gemm_launch_with(ctx, opA(c), opB(c), c.bn, c.splits, M, N, K, out, ld_out, split_stride, d_err, "autotune",
                        c.persist, c.pair, c.gm);
    EPSP_CUDA(cudaEventRecord(e1, ctx->stream));
    EPSP_CUDA(cudaEventSynchronize(e1));
    EPSP_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    return ms;
  };
  // one untimed launch of each kernel the candidates use (tile width, K box, persistent, pairs;
  // split count and tile order are arguments), so that no timed launch pays a kernel's first-launch
  // costs (module loading); for a shape whose launch takes 20 ms or more those costs are noise, and
  // only the first kernel is launched ahead
  {
    std::set<std::array<int, 4>> seen;
    for (const auto& c : cand)
      if (seen.insert({c.bn, c.bk, int(c.persist), int(c.pair)}).second && timed(c) >= 20.f) break;
  }
  // every candidate once, then the kRetime fastest (under 20 ms) the best of `reps` more launches
  // timed one by one: candidates a few per cent apart are ranked by their undisturbed time rather
  // than by one launch, and the rest, well behind, cost one launch each
  constexpr size_t kRetime = 6;
  for (auto& c : cand) c.ms = timed(c);
  std::vector<size_t> rank(cand.size());
  for (size_t k = 0; k < rank.size(); ++k) rank[k] = k;
  std::stable_sort(rank.begin(), rank.end(), [&](size_t a, size_t b) { return cand[a].ms < cand[b].ms; });
  for (size_t k = 0; k < std::min(kRetime, rank.size()); ++k) {
    TcTune& c = cand[rank[k]];
    if (c.ms >= 20.f) break;
    for (int r = 0; r < reps; ++r) c.ms = std::min(c.ms, timed(c));
  }
  for (const auto& c : cand)
    if (c.ms < best.ms) best = c;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (all) *all = cand;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune_cache[key] = cand;
  }
  return best;
}

}  // namespace epsp
