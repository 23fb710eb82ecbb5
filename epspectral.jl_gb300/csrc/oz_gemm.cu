// oz_gemm.cu -- the FP64 GEMM of oz_gemm.cuh: splitting into digits, the tcgen05 kernel over digit
// planes, the sum of the orders.
#include "oz_gemm.cuh"
#include "tc_gemm.cuh"

#include <algorithm>

namespace epsp {

// ---- splitting ----

// x as 62-bit fixed point under 2^e, biased so that its bytes are the digits + 128.
__device__ __forceinline__ unsigned long long oz_fixed(double x, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int E = int((b >> 52) & 0x7ff);
  unsigned long long m = b & 0xfffffffffffffull;
  if (E) m |= 1ull << 52;
  const int sh = max(E, 1) - 1075 + 62 - e;  // x = m 2^(max(E, 1) - 1075)
  unsigned long long v;
  if (sh >= 0)
    v = m << sh;
  else if (sh > -55)
    v = (m + (1ull << (-sh - 1))) >> -sh;  // to nearest
  else
    v = 0;
  if (b >> 63) v = 0ull - v;
  return v + 0x8080808080808080ull;
}

// The exponent e of a row (|x| < 2^e) from the high word of its largest magnitude.
__device__ __forceinline__ int oz_exp(uint32_t mx) { return int(max(mx >> 20, 1u)) - 1022; }
__device__ __forceinline__ bool oz_finite(uint32_t mx) { return mx < 0x7ff00000u; }

// Two digits (bytes of two neighbouring values) as packed BF16: 2^23 + byte - (2^23 + 128) is exact.
__device__ __forceinline__ uint32_t oz_pack(uint32_t b0, uint32_t b1) {
  const float f0 = __uint_as_float(0x4B000000u | b0) - 8388736.f, f1 = __uint_as_float(0x4B000000u | b1) - 8388736.f;
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

// Writes the digits of eight neighbouring values (u: their fixed points) of row r at column k.
__device__ __forceinline__ void oz_store(const unsigned long long (&u)[8], long rows, long r, long Kp, long k,
                                         __nv_bfloat16* __restrict__ q) {
#pragma unroll
  for (int s = 0; s < kOzDigits; ++s) {
    uint32_t by[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) by[j] = uint32_t(u[j] >> (8 * (7 - s))) & 0xffu;
    uint4 o;
    o.x = oz_pack(by[0], by[1]);
    o.y = oz_pack(by[2], by[3]);
    o.z = oz_pack(by[4], by[5]);
    o.w = oz_pack(by[6], by[7]);
    *reinterpret_cast<uint4*>(q + (s * rows + r) * Kp + k) = o;
  }
}

__device__ __forceinline__ uint32_t oz_hi(double x) { return uint32_t(__double2hiint(x)) & 0x7fffffffu; }

// Rows contiguous in k: a block per row, its largest magnitude first, then the digits (the row's second
// read comes from L1/L2).
__global__ void __launch_bounds__(256) oz_split_k_kernel(const double* __restrict__ S, long ld, long rows, long K, long Kp,
                                                         __nv_bfloat16* __restrict__ q, uint32_t* __restrict__ mx) {
  pdl_wait();
  __shared__ uint32_t sm[8];
  const long r = blockIdx.x;
  const double* row = S + ld * r;
  uint32_t h = 0;
  for (long k = threadIdx.x; k < K; k += 256) h = max(h, oz_hi(row[k]));
  h = __reduce_max_sync(0xffffffffu, h);
  if (threadIdx.x % 32 == 0) sm[threadIdx.x / 32] = h;
  __syncthreads();
  h = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) h = max(h, sm[w]);
  if (threadIdx.x == 0) mx[r] = h;
  const bool fin = oz_finite(h);
  const int e = oz_exp(h);
  for (long k = 8 * long(threadIdx.x); k < Kp; k += 8 * 256) {
    unsigned long long u[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) u[j] = oz_fixed(fin && k + j < K ? row[k + j] : 0.0, e);
    oz_store(u, rows, r, Kp, k, q);
  }
}

// Rows contiguous in r: the largest magnitudes (mx zeroed before; an atomic maximum per block of 64 rows
// and kper k), then the digits through a 64 x 64 transpose.
__global__ void __launch_bounds__(256) oz_max_m_kernel(const double* __restrict__ S, long ld, long rows, long K, long kper,
                                                       uint32_t* __restrict__ mx) {
  pdl_wait();
  __shared__ uint32_t sm[4][64];
  const int tx = threadIdx.x % 64, ty = threadIdx.x / 64;
  const long r = long(blockIdx.x) * 64 + tx, k0 = long(blockIdx.y) * kper;
  uint32_t h = 0;
  if (r < rows)
#pragma unroll 4
    for (long k = k0 + ty; k < min(K, k0 + kper); k += 4) h = max(h, oz_hi(S[r + ld * k]));
  sm[ty][tx] = h;
  __syncthreads();
  if (ty == 0 && r < rows) atomicMax(mx + r, max(max(sm[0][tx], sm[1][tx]), max(sm[2][tx], sm[3][tx])));
}
__global__ void __launch_bounds__(256) oz_split_m_kernel(const double* __restrict__ S, long ld, long rows, long K, long Kp,
                                                         const uint32_t* __restrict__ mx, __nv_bfloat16* __restrict__ q) {
  pdl_wait();
  __shared__ unsigned long long tile[64][65];  // [k][r]
  const long r0 = long(blockIdx.x) * 64, k0 = (long(blockIdx.z) * gridDim.y + blockIdx.y) * 64;
  if (k0 >= Kp) return;
  {
    const int tx = threadIdx.x % 64, ty = threadIdx.x / 64;
    const long r = r0 + tx;
    const uint32_t h = r < rows ? mx[r] : 0u;
    const bool on = r < rows && oz_finite(h);
    const int e = oz_exp(h);
#pragma unroll 4
    for (int j = ty; j < 64; j += 4) {
      const long k = k0 + j;
      tile[j][tx] = oz_fixed(on && k < K ? S[r + ld * k] : 0.0, e);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 512; t += 256) {  // 8 lanes write one row's 64 values
    const int rl = t / 8, kg = t % 8;
    if (r0 + rl >= rows || k0 + 8 * kg >= Kp) continue;
    unsigned long long u[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) u[j] = tile[8 * kg + j][rl];
    oz_store(u, rows, r0 + rl, Kp, k0 + 8 * kg, q);
  }
}

// ---- the digit products ----

// The items of the persistent kernel: for each tile (M tile fastest) and K segment, order d's
// pairs(d) x nkc chunks of 256 terms in runs of `run` chunks, high orders (the most chunks) first.
struct OzShape {
  int M, N, kblocks;      // rows and columns of this launch, K blocks of 64 in all
  int rowsA, m0;          // rows of A's planes, the first of this launch
  int nM, nN, nseg, nkc;  // tiles, K segments, chunks of 256 terms per segment
  int run;
  int per_seg;            // items of one tile and segment
};

__host__ __device__ __forceinline__ int oz_pairs(int d) { return d < kOzDigits ? d + 1 : 2 * kOzDigits - 1 - d; }

template <int BN>
struct OzSmem {
  static constexpr int kStages = BN == 256 ? 4 : BN == 192 ? 5 : BN == 128 ? 6 : 8;
  static constexpr int kA = kTcBM * 128, kB = BN * 128;
  static constexpr int kStage = kA + kB;
  static constexpr int kBars = 2 * kStages + 5;
  static constexpr int kBytes = kStages * kStage + 8 * kBars + 16 + 1024;
  static constexpr int kTmem = BN == 64 ? 128 : BN == 128 ? 256 : 512;  // two accumulators
};

// Persistent, 320 threads: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 the sums. A chunk's four K
// blocks of 64 run into one of two TMEM accumulators; its exact integer sums are read while the next
// chunk runs and added into registers (adding 1.5 2^23 puts the integer into the mantissa, so a sum
// costs one FP32 and one integer addition); after an item's last chunk the registers go to
// sums[(seg, d)][n][m] by integer atomics (exact in any order), or by a store where the order is one item.
// Bound: shared memory (at BN = 256, 12 KB of operand reads and 12 KB of fills per 128 x 256 x 16 product, of 128 B a
// cycle: 0.72 of the tensor rate) and the issuing thread. The tile's width takes the fewest shared-memory cycles for
// N, its padding included (oz_tile_n: half of a 128-wide tile is padding at N = 65, most of a 64-wide one below 32), and
// `run` the shortest estimated time over the SMs (gemm_panel; a small product has fewer items than SMs).
// HOOK: the test hook's kernel, whose producer leaves out K block stall_kb and whose waits give up after hook_limit tries
// (with both as arguments of the one kernel it took 3 % longer: 7680 x 180 x 2880 541 -> 556 us).
template <int BN, bool HOOK>
__global__ void __launch_bounds__(320, 1)
    oz_mma_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const OzShape sh,
                  int* __restrict__ sums, int* __restrict__ err, int stall_kb, unsigned hook_limit) {
  using L = OzSmem<BN>;
  constexpr int STAGES = L::kStages;
  const unsigned wait_limit = HOOK ? hook_limit : kWaitLimit;
  constexpr int kCols = BN / 2;  // columns of one epilogue warp
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * L::kStage);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::kBars);
  __shared__ int s_abort;
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * STAGES, accf0 = full0 + 16 * STAGES, acce0 = accf0 + 16,
                 done_bar = accf0 + 32;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int ntile = sh.nM * sh.nN;
  const int nitems = ntile * sh.nseg * sh.per_seg;
  auto aborted = [&] { return *(volatile int*)&s_abort != 0; };
  // item -> tile, segment, order d, chunks [c0, c1) of it, and whether the order is this item alone
  struct Item {
    int mt, nt, seg, d, c0, c1;
    bool alone;
  };
  auto item_of = [&](int it) {
    Item o;
    const int tile = it % ntile;
    int rest = it / ntile;
    o.mt = tile % sh.nM;
    o.nt = tile / sh.nM;
    o.seg = rest % sh.nseg;
    rest /= sh.nseg;
    // orders from the one with the most pairs down: 7, 6, 8, 5, 4, 3, 2, 1, 0
    int d = 0, n = 0, tot = 0;
#pragma unroll
    for (int k = 0; k < kOzOrders; ++k) {
      d = k == 0 ? 7 : k == 1 ? 6 : k == 2 ? 8 : kOzOrders - 1 - k;
      tot = oz_pairs(d) * sh.nkc;
      n = (tot + sh.run - 1) / sh.run;
      if (rest < n) break;
      rest -= n;
    }
    o.d = d;
    o.c0 = rest * sh.run;
    o.c1 = min(tot, o.c0 + sh.run);
    o.alone = n == 1;
    return o;
  };
  // the chunks of an item in order: digits (s, d - s) and K blocks [b0, b1)
  struct Chunk {
    int s, k, b0, b1;
  };
  auto chunk_at = [&](const Item& o, Chunk& c) {
    c.b0 = (o.seg * sh.nkc + c.k) * (kOzChunk / 64);
    c.b1 = min(sh.kblocks, c.b0 + kOzChunk / 64);
  };
  auto chunk_first = [&](const Item& o) {
    Chunk c;
    c.s = max(0, o.d - (kOzDigits - 1)) + o.c0 / sh.nkc;
    c.k = o.c0 % sh.nkc;
    chunk_at(o, c);
    return c;
  };
  auto chunk_next = [&](const Item& o, Chunk& c) {
    if (++c.k == sh.nkc) {
      c.k = 0;
      ++c.s;
    }
    chunk_at(o, c);
  };

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < 2 * STAGES; ++s) mbar_init(smem_u32(bars + s), 1);
    mbar_init(accf0, 1);
    mbar_init(accf0 + 8, 1);
    mbar_init(acce0, 8);
    mbar_init(acce0 + 8, 8);
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(L::kTmem));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();  // (barriers and tensor memory are set up beside the kernel ahead)

  if (warp == 0 && lane == 0) {
    int g = 0;
    bool stop = false;
    for (int it = int(blockIdx.x); it < nitems && !stop; it += int(gridDim.x)) {
      const Item o = item_of(it);
      Chunk ch = chunk_first(o);
      for (int c = o.c0; c < o.c1 && !stop; ++c, chunk_next(o, ch)) {
        for (int kb = ch.b0; kb < ch.b1; ++kb) {
          const int st = g % STAGES;
          if (g >= STAGES && !mbar_wait(empty0 + 8 * st, ((g / STAGES) & 1) ^ 1, wait_limit)) {
            atomicExch(&s_abort, 1);
            stop = true;
            break;
          }
          if (aborted()) {
            stop = true;
            break;
          }
          if (HOOK && kb == stall_kb) {  // the issuer's wait for this block runs out
            ++g;
            continue;
          }
          const uint32_t dst = smem_u32(smem + st * L::kStage), fb = full0 + 8 * st;
          mbar_expect_tx(fb, L::kStage);
          // a tile past its plane's last row reads the next plane (or zeros): rows that are not stored
          tma_load_2d(dst, &mapA, kb * 64, ch.s * sh.rowsA + sh.m0 + o.mt * kTcBM, fb);
          tma_load_2d(dst + L::kA, &mapB, kb * 64, (o.d - ch.s) * sh.N + o.nt * BN, fb);
          ++g;
        }
      }
    }
    // wait (bounded) for the last copies, so that none is in flight when the block leaves, whichever warp gave up and when
    for (int k = max(0, g - STAGES); k < g; ++k) mbar_wait(full0 + 8 * (k % STAGES), (k / STAGES) & 1, wait_limit);
  } else if (warp == 1 && lane == 0) {
    constexpr uint32_t idesc = idesc_f32acc<false>(BN);
    const uint64_t desc0 = sw128_desc(smem_u32(smem));
    int st = 0, t = 0;
    uint32_t ph = 0;  // the ring's stage and the parity of its turn
    bool stop = false;
    for (int it = int(blockIdx.x); it < nitems && !stop; it += int(gridDim.x)) {
      const Item o = item_of(it);
      Chunk ch = chunk_first(o);
      for (int c = o.c0; c < o.c1 && !stop; ++c, ++t, chunk_next(o, ch)) {
        const int b = t & 1;
        const uint32_t acc = tmem + uint32_t(b * BN);
        if (t >= 2 && !mbar_wait_issuer(acce0 + 8 * b, ((t >> 1) & 1) ^ 1, &s_abort)) {
          atomicExch(&s_abort, 1);
          stop = true;
          break;
        }
        tc_fence_after();
        for (int kb = ch.b0; kb < ch.b1; ++kb) {
          if (!mbar_wait_issuer(full0 + 8 * st, ph, &s_abort)) {
            atomicExch(&s_abort, 1);
            stop = true;
            break;
          }
          tc_fence_after();
          // (an operand's descriptor holds its address / 16 in the low bits)
          const uint64_t da = desc0 + uint64_t(st * (L::kStage / 16)), db = da + L::kA / 16;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) umma<false>(acc, da + 2 * ks, db + 2 * ks, idesc, kb > ch.b0 || ks > 0);
          umma_commit(empty0 + 8 * st);
          if (++st == STAGES) {
            st = 0;
            ph ^= 1;
          }
        }
        umma_commit(accf0 + 8 * b);
      }
    }
    umma_commit(done_bar);
  } else if (warp >= 2) {
    const int q = warp % 4, half = (warp - 2) / 4;  // TMEM lane quarter, columns half kCols..
    int t = 0;
    bool stop = false;
    for (int it = int(blockIdx.x); it < nitems && !stop; it += int(gridDim.x)) {
      const Item o = item_of(it);
      uint32_t acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0u - uint32_t(o.c1 - o.c0) * 0x4B400000u;
      Chunk ch = chunk_first(o);
      for (int c = o.c0; c < o.c1; ++c, ++t, chunk_next(o, ch)) {
        const int b = t & 1;
        const bool got = mbar_wait(accf0 + 8 * b, (t >> 1) & 1, wait_limit);
        if (!got) atomicExch(&s_abort, 1);
        if (!__all_sync(0xffffffffu, got && !aborted())) {  // (the warp as one: the tensor memory loads are collective)
          stop = true;
          break;
        }
        tc_fence_after();
        const bool some = ch.b0 < ch.b1;  // a chunk past the last segment's end: no product, the sum is 0
#pragma unroll
        for (int j0 = 0; j0 < kCols; j0 += 32) {
          float v[32];
          tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(b * BN + half * kCols + j0), v);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[j0 + j] += __float_as_uint((some ? v[j] : 0.f) + 12582912.f);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acce0 + 8 * b);
      }
      if (stop) break;
      const int row = o.mt * kTcBM + q * 32 + lane;
      if (row < sh.M) {
        int* dst = sums + (long(o.seg * kOzOrders + o.d) * sh.N + o.nt * BN + half * kCols) * sh.M + row;
        const int nc = min(kCols, sh.N - o.nt * BN - half * kCols);
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
          if (j < nc) {
            if (o.alone)
              *dst = int(acc[j]);
            else
              atomicAdd(dst, int(acc[j]));
          }
          dst += sh.M;
        }
      }
    }
  }
  __syncwarp();
  // every MMA issued has completed before TMEM is freed (bounded)
  if (!mbar_wait(done_bar, 0)) atomicExch(&s_abort, 1);
  tc_fence_after();
  __syncthreads();
  if (aborted() && threadIdx.x == 0) atomicExch(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::kTmem));
}

// ---- the sum of the orders ----

// C = 2^(e_A + e_B - 76) Σ_d 2^(8 (8 - d)) sums[d] + beta C, the sum exact in 128 bits and rounded once.
__global__ void __launch_bounds__(256) oz_sum_kernel(const int* __restrict__ sums, int nseg, int M, int N, int K,
                                                     const uint32_t* __restrict__ mxA, const uint32_t* __restrict__ mxB,
                                                     const double* __restrict__ A, long lda, const double* __restrict__ B,
                                                     long ldb, double beta, double* __restrict__ C, long ldc) {
  pdl_wait();
  const long idx = long(blockIdx.x) * 256 + threadIdx.x;
  if (idx >= long(M) * N) return;
  const int m = int(idx % M), n = int(idx / M);
  const uint32_t ha = mxA[m], hb = mxB[n];
  double val;
  if (oz_finite(ha) && oz_finite(hb)) {
    __int128 tot = 0;
    for (int sg = 0; sg < nseg; ++sg) {
      const int* p = sums + (long(sg) * kOzOrders * N + n) * M + m;
      int v[kOzOrders];
#pragma unroll
      for (int d = 0; d < kOzOrders; ++d) v[d] = p[long(d) * N * M];
      __int128 t = 0;
#pragma unroll
      for (int d = 0; d < kOzOrders; ++d) t = t * 256 + v[d];
      tot += t;
    }
    const bool neg = tot < 0;
    const unsigned __int128 a = neg ? (unsigned __int128)(-tot) : (unsigned __int128)(tot);
    const unsigned long long hi = (unsigned long long)(a >> 64), lo = (unsigned long long)a;
    double x;
    int sc = 0;
    if (hi == 0) {
      x = __ull2double_rn(lo);
    } else {  // the top 64 bits with the rest as a sticky bit: one rounding
      const int z = __clzll((long long)hi);
      const unsigned long long top = z ? (hi << z) | (lo >> (64 - z)) : hi;
      const unsigned long long rest = z ? lo << z : lo;
      x = __ull2double_rn(top | (rest ? 1ull : 0ull));
      sc = 64 - z;
    }
    val = ldexp(neg ? -x : x, sc + oz_exp(ha) + oz_exp(hb) - 76);
  } else {  // an infinity or a NaN in the row or the column: as FP64 arithmetic has it
    val = 0;
    for (int k = 0; k < K; ++k) val = fma(A[m + lda * k], B[k + ldb * n], val);
  }
  double* c = C + m + ldc * n;
  *c = beta == 0 ? val : val + beta * *c;
}

// The same as FP64 sums, for a device without room for the smallest panel's work buffers.
__global__ void __launch_bounds__(256) oz_plain_kernel(long M, long N, long K, const double* __restrict__ A, long lda,
                                                       const double* __restrict__ B, long ldb, double beta,
                                                       double* __restrict__ C, long ldc) {
  pdl_wait();
  const long idx = long(blockIdx.x) * 256 + threadIdx.x, m = idx % M, n = idx / M;
  if (n >= N) return;
  double val = 0;
  for (long k = 0; k < K; ++k) val = fma(A[m + lda * k], B[k + ldb * n], val);
  double* c = C + m + ldc * n;
  *c = beta == 0 ? val : val + beta * *c;
}

// ---- host ----

int oz_tile_n(long N) {
  // shared-memory cycles of one 16-term step of all tiles: A's 128 rows and the tile's columns, padding included
  int best = 64;
  long cost = -1;
  for (int bn : {256, 192, 128, 64}) {
    const long c = ((N + bn - 1) / bn) * (4 + bn / 32) * 16;
    if (cost < 0 || c < cost) {
      cost = c;
      best = bn;
    }
  }
  return best;
}

constexpr long kMaxY = 65535;  // blocks of a grid's y dimension

void oz_split(Ctx* ctx, const double* S, long ld, long rows, long K, bool k_major, int box, OzPlanes& P) {
  cudaStream_t s = ctx->stream;
  const long Kp = (K + 63) / 64 * 64;
  if (rows * kOzDigits > (1l << 31) - 1) fail(EPSP_EINVAL, "sizes beyond the 32-bit tile grid");
  const bool grown = ensure(P.q, ctx, size_t(kOzDigits * rows * Kp));
  ensure(P.mx, ctx, size_t(rows));
  if (grown || P.rows != rows || P.K != K || P.box != box) {
    P.rows = rows;
    P.K = K;
    P.Kp = Kp;
    P.box = box;
    P.map = make_tmap_bf16(P.q.p, kOzDigits * rows, K, Kp, box, 64);  // k >= K reads zeros
  }
  if (k_major) {
    launch_after(s, oz_split_k_kernel, unsigned(rows), 256, 0, S, ld, rows, K, Kp, P.q.p, P.mx.p);
    EPSP_LAUNCHED(ctx);
    return;
  }
  EPSP_CUDA(cudaMemsetAsync(P.mx.p, 0, size_t(rows) * sizeof(uint32_t), s));
  // enough blocks of k for eight a multiprocessor, of 16 k at least (a block's fixed cost), 512 at most
  const long nb = div_up(size_t(rows), 64), kb = std::max<long>(1, 8l * ctx->sm_count / nb);
  const long kper = std::max<long>(std::min<long>(512, std::max<long>(16, (K + kb - 1) / kb)), (K + kMaxY - 1) / kMaxY);
  launch_after(s, oz_max_m_kernel, dim3(unsigned(nb), div_up(size_t(K), size_t(kper))), 256, 0, S, ld, rows, K, kper, P.mx.p);
  EPSP_LAUNCHED(ctx);
  launch_after(s, oz_split_m_kernel, dim3(div_up(size_t(rows), 64), unsigned(std::min(Kp / 64, kMaxY)), div_up(size_t(Kp / 64), size_t(kMaxY))), 256, 0, S, ld, rows, K, Kp, P.mx.p, P.q.p);
  EPSP_LAUNCHED(ctx);
}

template <int BN>
static void launch_mma(Ctx* ctx, const OzPlanes& A, const OzPlanes& B, const OzShape& sh, int* sums, int* err) {
  using L = OzSmem<BN>;
  const bool hook = ctx->stall_kb >= 0 || ctx->stall_wait_limit;
  auto* kern = hook ? oz_mma_kernel<BN, true> : oz_mma_kernel<BN, false>;
  EPSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
  const int items = sh.nM * sh.nN * sh.nseg * sh.per_seg;
  launch_after(ctx->stream, kern, std::min(items, ctx->sm_count), 320, L::kBytes, A.map, B.map, sh, sums, err, ctx->stall_kb,
               ctx->stall_wait_limit ? ctx->stall_wait_limit : kWaitLimit);
  EPSP_LAUNCHED(ctx);
}

// Rows [m0, m0 + M) of A's planes times B's planes.
static void gemm_panel(Ctx* ctx, OzWork& W, const OzPlanes& A, long m0, long M, const OzPlanes& B, const double* dA, long lda,
                       const double* dB, long ldb, double beta, double* C, long ldc) {
  cudaStream_t s = ctx->stream;
  OzShape sh{};
  sh.M = int(M);
  sh.N = int(B.rows);
  sh.rowsA = int(A.rows);
  sh.m0 = int(m0);
  sh.kblocks = int(A.Kp / 64);
  sh.nM = (sh.M + kTcBM - 1) / kTcBM;
  sh.nN = (sh.N + B.box - 1) / B.box;
  const int chunks = (sh.kblocks + 3) / 4;
  sh.nseg = (chunks + kOzSegChunks - 1) / kOzSegChunks;
  sh.nkc = (chunks + sh.nseg - 1) / sh.nseg;
  sh.nseg = (chunks + sh.nkc - 1) / sh.nkc;
  // Chunks per item: the shortest critical path of whole rounds over the SMs, a chunk being 16 products at shared
  // memory's rate and an item's end (registers to sums, pipeline drain) about four chunks; shared orders pay
  // atomics, so ties go to longer runs.
  bool shared = false;
  long best = -1;
  for (int run = 1; run <= 8 * sh.nkc; run += std::max(1, run / 16)) {
    long per_seg = 0;
    bool sh_ = false;
    for (int d = 0; d < kOzOrders; ++d) {
      const int n = (oz_pairs(d) * sh.nkc + run - 1) / run;
      per_seg += n;
      sh_ |= n > 1;
    }
    const long items = per_seg * sh.nseg * sh.nM * sh.nN;
    const long cost = (items + ctx->sm_count - 1) / ctx->sm_count * (std::min(run, 8 * sh.nkc) + 4);
    if (best < 0 || cost <= best) {
      best = cost;
      sh.run = run;
      sh.per_seg = int(std::min<long>(per_seg, 1l << 30));
      shared = sh_;
    }
  }
  if (long(sh.nM) * sh.nN * sh.nseg * sh.per_seg > (1l << 30)) fail(EPSP_EINVAL, "sizes beyond the 32-bit tile grid");
  const size_t n = size_t(sh.nseg) * kOzOrders * size_t(sh.M) * size_t(sh.N);
  if (shared) EPSP_CUDA(cudaMemsetAsync(W.sums.p, 0, n * sizeof(int), s));
  switch (B.box) {
    case 256: launch_mma<256>(ctx, A, B, sh, W.sums.p, W.err.p); break;
    case 192: launch_mma<192>(ctx, A, B, sh, W.sums.p, W.err.p); break;
    case 128: launch_mma<128>(ctx, A, B, sh, W.sums.p, W.err.p); break;
    default: launch_mma<64>(ctx, A, B, sh, W.sums.p, W.err.p); break;
  }
  launch_after(s, oz_sum_kernel, div_up(size_t(sh.M) * size_t(sh.N), 256), 256, 0, W.sums.p, sh.nseg, sh.M, sh.N, int(A.K),
                                                                        A.mx.p + m0, B.mx.p, dA, lda, dB, ldb, beta, C, ldc);
  EPSP_LAUNCHED(ctx);
}

bool OzKept::give_back() {
  if (!on || busy) return false;
  p.release();
  on = false;
  return true;
}

void OzKept::keep(Ctx* ctx, const double* S, long ld, long rows, long K, bool k_major, int box) {
  entry.enter(ctx->spares, this);
  const size_t values = size_t(kOzDigits) * size_t(rows) * size_t((K + 63) / 64 * 64);
  if (!(p.q.p && p.q.n >= values) && 2 * values > (size_t(64) << 20)) {  // (small ones without asking)
    size_t room = 0, all = 0;
    EPSP_CUDA(cudaMemGetInfo(&room, &all));
    if (2 * values > room / 4) {
      give_back();
      return;
    }
  }
  busy = true;
  try {
    oz_split(ctx, S, ld, rows, K, k_major, box, p);
    on = true;
  } catch (const Error& e) {
    on = false;
    p.release();
    if (e.code != EPSP_ENOMEM) {
      busy = false;
      throw;
    }
  }
  busy = false;
}

bool OzWork::give_back() {
  if (busy || !(a.q.p || b.q.p || sums.p)) return false;
  a.release();
  b.release();
  sums.release();
  return true;
}

static void reserve(Ctx* ctx, OzPlanes& P, long rows, long Kp) {
  bool grown = ensure(P.q, ctx, size_t(kOzDigits * rows * Kp));
  grown |= ensure(P.mx, ctx, size_t(rows));
  if (grown) P.rows = 0;  // the map's address is no longer the buffer's
}

void oz_gemm(Ctx* ctx, OzWork& W, long M, long N, long K, const double* A, long lda, const OzKept* kA, const double* B,
             long ldb, const OzKept* kB, double beta, double* C, long ldc) {
  if (M <= 0 || N <= 0) return;
  W.entry.enter(ctx->spares, &W);
  struct InUse {
    OzWork& w;
    ~InUse() { w.busy = false; }
  } use{W};
  W.busy = true;
  if (ensure(W.err, ctx, 1)) W.err.zero(ctx->stream);
  const long Kp = (K + 63) / 64 * 64, nseg = Kp / (kOzSegChunks * kOzChunk) + 1;
  long room = long(ctx->product_bytes ? ctx->product_bytes : size_t(4) << 30);  // of each buffer
  long pm = 0, pn = 0;
  const OzPlanes *pA = nullptr, *pB = nullptr;
  // the panels: every buffer is there before the first is used, since a product may add to C
  for (bool ready = false; !ready;) {
    if (room < (1l << 20)) {
      launch_after(ctx->stream, oz_plain_kernel, div_up(size_t(M) * size_t(N), 256), 256, 0, M, N, K, A, lda, B, ldb, beta, C, ldc);
      EPSP_LAUNCHED(ctx);
      return;
    }
    auto most = [&](long all, long tile, long bytes) { return std::min(all, std::max(tile, room / bytes / tile * tile)); };
    pA = kA ? kA->planes() : nullptr;
    pB = kB ? kB->planes() : nullptr;
    pn = pB ? N : most(N, 64, 2 * kOzDigits * Kp);
    pm = most(M, kOzBoxM, 4 * kOzOrders * nseg * pn);
    if (!pA) pm = std::min(pm, most(M, kOzBoxM, 2 * kOzDigits * Kp));
    try {
      if (!pA) reserve(ctx, W.a, pm, Kp);
      if (!pB) reserve(ctx, W.b, pn, Kp);
      ensure(W.sums, ctx, size_t(nseg * kOzOrders) * size_t(pm) * size_t(pn));
      // (what an allocation took may have been these operands' planes)
      ready = pA == (kA ? kA->planes() : nullptr) && pB == (kB ? kB->planes() : nullptr);
    } catch (const Error& e) {
      if (e.code != EPSP_ENOMEM) throw;
      W.a.release();
      W.b.release();
      W.sums.release();
      room /= 4;
    }
  }
  for (long m0 = 0; m0 < M; m0 += pm) {
    const long m = std::min(pm, M - m0);
    if (!pA) oz_split(ctx, A + m0, lda, m, K, false, kOzBoxM, W.a);
    for (long n0 = 0; n0 < N; n0 += pn) {
      const long n = std::min(pn, N - n0);
      if (!pB && (m0 == 0 || pn < N)) oz_split(ctx, B + ldb * n0, ldb, n, K, true, oz_tile_n(n), W.b);
      gemm_panel(ctx, W, pA ? *pA : W.a, pA ? m0 : 0, m, pB ? *pB : W.b, A + m0, lda, B + ldb * n0, ldb, beta,
                 C + m0 + ldc * n0, ldc);
    }
  }
}

void oz_check(Ctx* ctx, OzWork& W) {
  if (!W.err.p) return;
  int e = 0;
  W.err.download(&e, 1, ctx->stream);
  EPSP_CUDA(cudaStreamSynchronize(ctx->stream));
  if (e) {
    W.err.zero(ctx->stream);
    fail(EPSP_EDEVICE_TIMEOUT, "a tensor-core GEMM wait ran out (bounded device wait)");
  }
}

}  // namespace epsp
