// oz_gemm.cuh -- FP64 GEMMs on the BF16 tensor cores, for the FP64 paths (the Kramers-Kronig map, the
// recast Fan-Migdal contraction and the ladder's shift sums in FP64).
//
//   C[M, N] = op(A)[M, K] B[K, N] + beta C, column-major, FP64 in and out.
//
// GB300 has 1.25 TFLOP/s of FP64 and 1950 of BF16 (measured), so the product is formed from exact integer
// products (the error-free splitting of Ozaki, Ogita, Oishi and Rump, 2012, on integers): each row
// of A and each column of B is scaled by a power of two of its own (its largest magnitude < 2^e) and
// rounded to 62-bit fixed point, written as eight balanced base-256 digits q_0..q_7 (|q| <= 128, exact
// in BF16). The digit products of one order d = s + t share the weight 2^(e_A + e_B - 12 - 8 d) and are
// summed exactly: 256 terms of at most 2^14 stay within 2^22, below the 24 bits of an FP32 accumulator,
// and are then added as 32-bit integers. The nine orders d = 0..8 are kept (43 of the 64 digit
// products; order 9 starts at 2^-68 of the two largest magnitudes), summed as one 128-bit integer and
// rounded to FP64 once. So the result is reproducible bit for bit in any order of summation, and
//   |error| <= 2^-53 |C_mn| + K 2^-60 max_k |A_mk| max_k |B_kn|,
// the rounding of the inputs (2^-63 each) and the dropped orders. An operand's value that lies 2^-9 or more below the
// largest of its row (A) or column (B) thus keeps fewer bits than FP64's 53, and one 2^-63 below none: an element of C far
// below the products of those maxima is as accurate as the second term says. In the library's products, whose elements
// spread over six decades, each element was closer to the exact sum than FP64 sums are (1e-16 against 3e-15 at worst, 15
// modes x 30 states, widths of 1 and 10 meV). Rows or columns that hold an infinity or a NaN are summed in FP64
// directly, as IEEE arithmetic gives them.
//
// A 64 x 64-tile FP64 SIMT kernel stood here before (1.2 TFLOP/s at large sizes, one block per tile).
// Kernel time on one GB300, split of the changing operand and sum of the orders included:
//   Kramers-Kronig map  401 x 33 x 401                              491 -> 21 us
//   Fan-Migdal product  501 x 105 x 1575 and its 501 x 105 x 501    2492 -> 67 us
//   ladder contraction  7680 x 180 x 2880 and its 313 x 1440 x 313  9270 -> 600 us
// Relative error of Σ and σ after whole runs against 64-bit references: unchanged (3e-14, 3e-16).
#pragma once

#include "common.cuh"

#include <cuda.h>
#include <cuda_bf16.h>

namespace epsp {

constexpr int kOzDigits = 8;    // digits of an operand
constexpr int kOzOrders = 9;    // orders of digit products kept
constexpr int kOzBoxM = 128;    // rows of A's tiles
constexpr int kOzChunk = 256;   // terms of one exact FP32 accumulation
constexpr int kOzSegChunks = 63;  // chunks of one exact 32-bit sum: 8 pairs x 63 x 256 x 2^14 < 2^31

// One operand as digit planes: row r, digit s at row s rows + r of a [8 rows][Kp] BF16 matrix, k
// contiguous; mx[r] the high word of the row's largest |x| (its exponent; >= 0x7ff00000: not finite).
struct OzPlanes {
  DBuf<__nv_bfloat16> q;
  DBuf<uint32_t> mx;
  long rows = 0, K = 0, Kp = 0;
  int box = 0;  // rows of the tensor map's box
  CUtensorMap map;
  void release() {
    q.release();
    mx.release();
    rows = K = Kp = 0;
  }
};

// The planes of an operand that does not change, split once and kept beside it (16 bytes a value, twice the operand)
// while there is room: not where they would take more than a quarter of the free memory (asked from 64 MiB on), and
// given back to an allocation that finds none. The products split the operand themselves where they are not kept (the same results).
class OzKept final : Spare {
  OzPlanes p;
  bool on = false, busy = false;
  SpareEntry entry;
  bool give_back() override;

 public:
  void keep(Ctx* ctx, const double* S, long ld, long rows, long K, bool k_major, int box);
  const OzPlanes* planes() const { return on ? &p : nullptr; }
};

// Work buffers of a plan's products: the planes of the operands that are split for one product, the integer sums, and
// the flag a bounded wait sets. Given back, but for the flag, to an allocation that finds no room.
struct OzWork final : Spare {
  OzPlanes a, b;
  DBuf<int> sums;
  DBuf<int> err;
  bool busy = false;
  SpareEntry entry;
  bool give_back() override;
};

// The column tile for N columns: 64, 128, 192 or 256.
int oz_tile_n(long N);

// Splits `rows` rows of K values into planes for boxes of `box` rows: value (r, k) at S[ld r + k]
// (k_major) or S[r + ld k]. P's buffers are kept and grown as needed.
void oz_split(Ctx* ctx, const double* S, long ld, long rows, long K, bool k_major, int box, OzPlanes& P);

// C [M, N] = A B + beta C with A[m + lda k], B[k + ldb n]. An operand that does not change may be kept by the caller
// (kA with boxes of kOzBoxM rows, kB of oz_tile_n(N)); the others are split here, into W's buffers. Runs over
// panels of rows and, where B is split here, of columns, so that the planes and the sums hold 4 GiB each at most (of one
// tile at least), less where the device has no room, and by FP64 sums where it has none at all. Panels do
// not change an element: each is its own exact sum.
void oz_gemm(Ctx* ctx, OzWork& W, long M, long N, long K, const double* A, long lda, const OzKept* kA, const double* B,
             long ldb, const OzKept* kB, double beta, double* C, long ldc);

// Fails with EPSP_EDEVICE_TIMEOUT if a bounded wait of a product ran out (synchronises, clears the flag).
void oz_check(Ctx* ctx, OzWork& W);

}  // namespace epsp
