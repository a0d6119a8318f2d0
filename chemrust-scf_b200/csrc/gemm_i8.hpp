// FP64 complex GEMMs on the INT8 tensor cores (host interface).
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace chfsi {

// Rows of a complex FP64 matrix cut into eight signed 8-bit digits per part
// (re, im, re +- im), in the tile order the kernel copies: per part, row tile
// (`tile` rows) and 32-wide K slab one block of eight digit planes.  One
// exponent per row and chunk of `spc` slabs.
struct I8Operand {
    int8_t* data = nullptr;
    int8_t* mag = nullptr;  // magnitudes of the elements (or none)
    int* exps = nullptr;
    int rows = 0, tile = 0, tiles = 0;
    int K = 0, nslab = 0, spc = 0;
    bool ready() const { return data != nullptr; }
    int chunks() const { return (nslab + spc - 1) / spc; }
};

constexpr int kI8RowTile = 128;  // operand on the accumulator's lanes
constexpr int kI8ColTile = 64;   // operand on its columns
constexpr int kI8MaxK = 8192;    // longest exact INT32 accumulation used

// bytes of an operand's digits and exponents
size_t i8_operand_bytes(int rows, int tile, int K, int spc, bool mag = false);
// lays `op` out in buf; returns the bytes used
size_t i8_operand_place(I8Operand& op, void* buf, int rows, int tile, int K, int spc, bool mag = false);
// Digits of x: element (r, k) = x[r * ld + k], or x[k * ld + r] (transposed);
// third part re + sign * im.
void i8_slice(const double2* x, long long ld, bool transposed, int sign, const I8Operand& op,
              cudaStream_t st);

// K slabs per chunk of a projection M x N x K (the choice a cached operand is
// laid out with)
int i8_cn_chunk_slabs(int M, int N, int K);

// scratch that lets the products run in one group (callers may hand in less);
// check: with `unresolved`
size_t i8_cn_scratch_bytes(int M, int N, int K, bool cached_a, bool check = false);
size_t i8_tn_scratch_bytes(int M, int N, int K, bool cached_x, bool check = false);

// Whether the INT8 path is the faster one at these sizes.
bool i8_cn_pays(int M, int N, int K, bool herm, bool cached_a);
bool i8_tn_pays(int M, int N, int K, bool cached_x);

// out[m][n] = sum_k conj(A[m][k]) B[n][k] (herm: B = A or H A, upper tiles
// computed and mirrored).  pre: digits of A (kI8RowTile rows, sign -1) or
// null.  Returns false, with nothing launched, when the scratch cannot hold
// one group.  err: device word set when a bounded wait ran out.  unresolved (null,
// or a zeroed device word; not with pre or herm): set when some element's terms
// are so small against its rows' largest parts that the error may exceed the
// FP64 bound K 2^-53 sum |a||b|; the result then is not to be used.
bool gemm_cn_i8(const double2* A, int lda, const I8Operand* pre, const double2* B, int ldb, int M,
                int N, int K, bool herm, void* scratch, size_t bytes, double2* out, int* err,
                cudaStream_t st, int* unresolved = nullptr);

// O[m][n] = alpha sum_k W[k][m] X[k][n] + beta O[m][n]; pre: digits of the
// rows of X^T (kI8RowTile rows, sign +1) or null.  unresolved as above (not with
// pre); where it is set and beta is not zero, O is as it was.
bool gemm_tn_i8(const double2* W, int ldw, const double2* X, int ldx, const I8Operand* pre,
                double2* O, int ldo, int M, int N, int K, double alpha, double beta, void* scratch,
                size_t bytes, int* err, cudaStream_t st, int* unresolved = nullptr);

// Test hook: the launch that is `launches` from now (0: the next; negative:
// none) copies no operands, so that its waits run out.
void i8_inject_no_loads(long long launches);

}  // namespace chfsi
