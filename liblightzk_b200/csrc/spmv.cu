// spmv.cu -- R1CS evaluation: A*z, B*z, C*z over Fr for CSR matrices.
//
// Replaces batch_sparse_matrix_vector_multiplication (reference
// include/operator/poly.cuh:5-30): one launch covers all three matrices
// (blockIdx.y selects the matrix), each thread owns whole rows and
// accumulates z[col] * val in Montgomery form.  Row i covers
// [row_ptr[i], row_ptr[i+1]) and the last row ends at nnz -- the reference's
// descriptor (xpu-spmat.cuh:20-25, `row` row starts plus `cnt`); a standard
// CSR with rows+1 offsets works unchanged.  Indices may be 32- or 64-bit
// (the reference uses size_t).  Entries equal to one (Montgomery R mod r)
// skip the product: z * 1 = z exactly.
#include "r1cs.cuh"

namespace lzk {

struct SpmvArgs {
    CsrDev m[3];
    Fr* out[3];
};

// One thread a row; bound by the gathers of z beside the products, so what
// counts is warps in flight: four blocks an SM (64 registers).  The three
// descriptors stay in the parameter space and are indexed there: choosing
// between three parameters by blockIdx.y copied them to the stack, and every
// entry's loads then went through local memory.  A z, B z, C z of a circuit
// of 2^20 rows: 184 us before, 174 without the copies, 161 with the products
// on the FP64 pipe as well; a matrix product's rows of up to 100 entries
// 120 -> 109.  Slower: the next entry's operands loaded ahead (177), three
// blocks an SM (171), and, both tried before the copies were found, an entry
// a thread with the sums through shared memory (244) and one reduction for
// all products of a row (205).
//
// Rows of more than kLongRow entries wait for the end of the block's loop.  One
// of them in a thread is a chain of gathers and products while the rest of the
// device runs out of work, so each goes to a whole warp, 32 entries at a time;
// only where so many are long that this takes more steps does a thread keep
// one.  One row among 65536 of one entry: of 100 entries 19 us (in a thread 97
// with 32-bit products, 109 on the FP64 pipe), of 20000 0.64 ms (15.8, 18.6).
constexpr uint32_t kSpmvThreads = 256, kLongRow = 64, kLongRows = 256;

__global__ void __launch_bounds__(kSpmvThreads, 4) k_spmv3(const __grid_constant__ SpmvArgs args, const Fr* __restrict__ z)
{
    __shared__ uint64_t rows[kLongRows];
    __shared__ uint32_t count, longest;
    const CsrDev& M = args.m[blockIdx.y];
    Fr* out = args.out[blockIdx.y];
    if (!out) return;
    if (threadIdx.x == 0) count = longest = 0;
    __syncthreads();
    for (uint64_t i = gtid(); i < M.rows; i += gstride()) {
        uint64_t s, e;
        row_range(M, i, s, e);
        if (e > s + kLongRow) {
            const uint32_t at = atomicAdd(&count, 1u);
            if (at < kLongRows) {
                rows[at] = i;
                atomicMax(&longest, (uint32_t)min(e - s, (uint64_t)1 << 30));
                continue;
            }
        }
        st_elem(out + i, row_part<true>(M, s, e, 1, z));
    }
    __syncthreads();
    const uint32_t n = min(count, kLongRows), warps = kSpmvThreads / 32, lane = threadIdx.x & 31;
    if (!n) return;
    uint64_t s, e;
    if ((uint64_t)((n + warps - 1) / warps) * (longest / 32 + 3) > longest) {
        if (threadIdx.x < n) {
            const uint64_t i = rows[threadIdx.x];
            row_range(M, i, s, e);
            st_elem(out + i, row_part<true>(M, s, e, 1, z));
        }
        return;
    }
    for (uint32_t r = threadIdx.x / 32; r < n; r += warps) {
        row_range(M, rows[r], s, e);
        Fr acc = row_part<false>(M, s + lane, e, 32, z);
        for (int o = 16; o > 0; o >>= 1) {
            Fr y;
            _Pragma("unroll") for (int i = 0; i < 8; i++) y.v[i] = __shfl_xor_sync(0xffffffffu, acc.v[i], o);
            acc = add(acc, y);
        }
        if (lane == 0) st_elem(out + rows[r], acc);
    }
}

}  // namespace lzk

using namespace lzk;

extern "C" {

int lzk_spmv3(const lzk_csr* A, const lzk_csr* B, const lzk_csr* C, const lzk_fr_t* z, lzk_fr_t* Az, lzk_fr_t* Bz,
              lzk_fr_t* Cz, void* stream)
{
    if (!z && ((A && A->nnz) || (B && B->nnz) || (C && C->nnz))) return LZK_EINVAL;
    if ((A && !Az) || (B && !Bz) || (C && !Cz)) return LZK_EINVAL;
    CsrDev a, b, c;
    LZK_TRY(csr_to_dev(A, a));
    LZK_TRY(csr_to_dev(B, b));
    LZK_TRY(csr_to_dev(C, c));
    uint64_t rows = a.rows > b.rows ? a.rows : b.rows;
    rows = rows > c.rows ? rows : c.rows;
    if (rows == 0) return LZK_OK;
    const SpmvArgs args{{a, b, c},
                        {A ? reinterpret_cast<Fr*>(Az) : nullptr, B ? reinterpret_cast<Fr*>(Bz) : nullptr,
                         C ? reinterpret_cast<Fr*>(Cz) : nullptr}};
    k_spmv3<<<dim3(grid_for(rows, kSpmvThreads, sm_count() * 8), 3), kSpmvThreads, 0, as_stream(stream)>>>(
        args, reinterpret_cast<const Fr*>(z)); note_launch();
    return launch_status();
}

int lzk_spmv(const lzk_csr* M, const lzk_fr_t* z, lzk_fr_t* out, void* stream)
{
    if (!M) return LZK_EINVAL;
    return lzk_spmv3(M, nullptr, nullptr, z, out, nullptr, nullptr, stream);
}

}  // extern "C"
