// HBM-bound kernels of the quantized GEMM path: row / column reductions, the B re-layout done in
// prepare(), the S32 offset contribution, the stand-alone output stage, NHWC im2col and the weights
// reshape.  All of them move each byte once with 128-bit accesses where the addresses allow it.
#include "kernels.cuh"

#include <climits>

namespace cugl
{
namespace
{
constexpr int kThreads = 256;

__device__ __forceinline__ int32_t sum4(uint32_t w, bool is_signed, int32_t acc)
{
    return is_signed ? __dp4a(static_cast<int32_t>(w), 0x01010101, acc)
                     : static_cast<int32_t>(__dp4a(w, 0x01010101u, static_cast<uint32_t>(acc)));
}

__device__ __forceinline__ int32_t warp_sum(int32_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;
}

// A warp's share of the byte sum of n 16-byte vectors: four independent loads in flight per lane.
__device__ __forceinline__ int32_t sum_vectors(const uint4 *v, int n, int lane, bool is_signed, int32_t acc)
{
    int i = lane;
    for (; i + 96 < n; i += 128)
    {
        const uint4 q0 = __ldg(v + i), q1 = __ldg(v + i + 32), q2 = __ldg(v + i + 64), q3 = __ldg(v + i + 96);
        int32_t     a0 = sum4(q0.x, is_signed, 0), a1 = sum4(q1.x, is_signed, 0);
        int32_t     a2 = sum4(q2.x, is_signed, 0), a3 = sum4(q3.x, is_signed, 0);
        a0 = sum4(q0.y, is_signed, a0), a1 = sum4(q1.y, is_signed, a1);
        a2 = sum4(q2.y, is_signed, a2), a3 = sum4(q3.y, is_signed, a3);
        a0 = sum4(q0.z, is_signed, a0), a1 = sum4(q1.z, is_signed, a1);
        a2 = sum4(q2.z, is_signed, a2), a3 = sum4(q3.z, is_signed, a3);
        a0 = sum4(q0.w, is_signed, a0), a1 = sum4(q1.w, is_signed, a1);
        a2 = sum4(q2.w, is_signed, a2), a3 = sum4(q3.w, is_signed, a3);
        acc += (a0 + a1) + (a2 + a3);
    }
    for (; i < n; i += 32)
    {
        const uint4 q = __ldg(v + i);
        acc           = sum4(q.x, is_signed, acc);
        acc           = sum4(q.y, is_signed, acc);
        acc           = sum4(q.z, is_signed, acc);
        acc           = sum4(q.w, is_signed, acc);
    }
    return acc;
}

// ---- rowsum_A[m] = scalar * sum_k A[m,k] -------------------------------------------------------
// One warp per row: unaligned head bytes, a body of 16-byte vectors, tail bytes; shuffle reduction.
// CpuGemmLowpMatrixAReductionKernel::run_internal (CpuGemmLowpMatrixReductionKernel.cpp:133-204).
__global__ void __launch_bounds__(kThreads) reduce_rows_kernel(const uint8_t *__restrict__ a, bool is_signed, int M,
                                                               int K, int64_t lda, int32_t scalar,
                                                               int32_t *__restrict__ out)
{
    dependent_prologue(); // (launched by launch_prepare_operands)
    const int lane          = threadIdx.x & 31;
    const int warps_per_blk = kThreads / 32;
    for (int m = blockIdx.x * warps_per_blk + (threadIdx.x >> 5); m < M; m += gridDim.x * warps_per_blk)
    {
        const uint8_t *row  = a + static_cast<int64_t>(m) * lda;
        const int      head = min(K, static_cast<int>((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15));
        int32_t        acc  = 0;
        if (lane < head)
        {
            acc += load_q8(row, lane, is_signed);
        }
        const int nvec = (K - head) >> 4;
        acc            = sum_vectors(reinterpret_cast<const uint4 *>(row + head), nvec, lane, is_signed, acc);
        const int tail0 = head + (nvec << 4);
        if (tail0 + lane < K)
        {
            acc += load_q8(row, tail0 + lane, is_signed);
        }
        acc = warp_sum(acc);
        if (lane == 0)
        {
            out[m] = acc * scalar;
        }
    }
}

// ---- colsum_B[n] += sum over a K-slab of B[k,n] --------------------------------------------------
// A thread owns 16 consecutive columns and reads them with one 128-bit load per row, so a warp reads 512
// contiguous bytes of a row.  The bytes are summed as packed 16-bit pairs (signed bytes are biased by 128 first,
// the bias leaves again at the end): two adds per four columns and row.  A slab is at most 256 rows, which a
// 16-bit lane holds without overflow (256 * 255 < 2^16).  grid.y splits K; integer atomics combine the slabs
// (exact, order-independent).  out must be zero on entry; the scalar is applied by scale_vector_kernel.
// Needs B and ldb 16-byte aligned; reduce_cols_generic_kernel covers the rest and the ragged last columns.
// CpuGemmLowpMatrixBReductionKernel::run_internal (CpuGemmLowpMatrixReductionKernel.cpp:273-446).
constexpr int kColSlabRows = 256;
__global__ void __launch_bounds__(kThreads) reduce_cols_kernel(const uint8_t *__restrict__ b, bool is_signed, int K,
                                                               int n_vec, int64_t ldb, int k_per_block,
                                                               int32_t *__restrict__ out)
{
    const int unit = blockIdx.x * kThreads + threadIdx.x; // 16 columns
    if (unit >= n_vec)
    {
        return;
    }
    const int      k0   = blockIdx.y * k_per_block;
    const int      k1   = min(K, k0 + k_per_block);
    const uint32_t flip = is_signed ? 0x80808080u : 0u;
    uint32_t       even[4] = {0, 0, 0, 0}, odd[4] = {0, 0, 0, 0}; // columns 4w, 4w+2 | 4w+1, 4w+3 as 16-bit pairs
    const uint8_t *p = b + static_cast<int64_t>(k0) * ldb + 16 * static_cast<int64_t>(unit);
#pragma unroll 4
    for (int k = k0; k < k1; ++k, p += ldb)
    {
        const uint4    q    = __ldg(reinterpret_cast<const uint4 *>(p));
        const uint32_t w[4] = {q.x ^ flip, q.y ^ flip, q.z ^ flip, q.w ^ flip};
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            even[j] += w[j] & 0x00ff00ffu;
            odd[j] += (w[j] >> 8) & 0x00ff00ffu;
        }
    }
    const int32_t bias = is_signed ? 128 * (k1 - k0) : 0;
    int32_t      *o    = out + 16 * unit;
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        atomicAdd(o + 4 * j + 0, static_cast<int32_t>(even[j] & 0xffffu) - bias);
        atomicAdd(o + 4 * j + 1, static_cast<int32_t>(odd[j] & 0xffffu) - bias);
        atomicAdd(o + 4 * j + 2, static_cast<int32_t>(even[j] >> 16) - bias);
        atomicAdd(o + 4 * j + 3, static_cast<int32_t>(odd[j] >> 16) - bias);
    }
}

// any alignment: one thread per column of [n_first, N)
__global__ void __launch_bounds__(kThreads) reduce_cols_generic_kernel(const uint8_t *__restrict__ b, bool is_signed,
                                                                       int K, int n_first, int N, int64_t ldb,
                                                                       int k_per_block, int32_t *__restrict__ out)
{
    const int n = n_first + blockIdx.x * kThreads + threadIdx.x;
    if (n >= N)
    {
        return;
    }
    const int k0 = blockIdx.y * k_per_block;
    const int k1 = min(K, k0 + k_per_block);
    int32_t   s  = 0;
    for (int k = k0; k < k1; ++k)
    {
        s += load_q8(b + static_cast<int64_t>(k) * ldb, n, is_signed);
    }
    atomicAdd(out + n, s);
}

__global__ void scale_vector_kernel(int32_t *v, int n, int32_t scalar)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
    {
        v[i] *= scalar;
    }
}

// ---- operand preparation ---------------------------------------------------------------------------------
// One launch does everything the tensor-core kernel needs from its operands beforehand, for all products of a batch:
// blocks [0, b_blocks) turn B [K][N] (N contiguous) into Bt [N][ldbt] (K contiguous) with its column sums, the blocks
// behind them walk over the rows of A and produce row sums and, where the TMA engine cannot address A (base or pitch
// not a multiple of 16 bytes), a copy with 16-byte rows.  The work is bound by launches when the operands are small
// (16 products of 384 x 384 x 128 with a B that changes took 64 launches one after the other, 229 us; with this launch
// and a batched product 10.5 us.  923 x 429 x 873 with unaligned rows: copy + reduction + product 24.6 us, now 14) and
// by HBM when they are large.
struct PrepParams
{
    OperandPrep op;
    int         b_strips, b_splits, b_blocks, k_per_split; // strips of 64 columns, K splits of k_per_split rows
    int         row_lanes; // lanes that share a row of A (kThreads: a block each)
    bool        a_vec; // A rows 16-byte aligned
};

// Four consecutive bytes starting at p, of which `valid` (>= 1) exist; the rest read as zero.
__device__ __forceinline__ uint32_t load_bytes4(const uint8_t *p, int valid)
{
    uint32_t v = p[0];
    if (valid > 1) v |= static_cast<uint32_t>(p[1]) << 8;
    if (valid > 2) v |= static_cast<uint32_t>(p[2]) << 16;
    if (valid > 3) v |= static_cast<uint32_t>(p[3]) << 24;
    return v;
}

// B: a block owns 64 columns and a range of K and walks down it 128 rows at a time.  A thread reads 4 x 4 bytes (four
// rows of one 32-bit column word), transposes them with eight byte permutes and leaves four K-contiguous words in
// shared memory; the tile goes out as 128 contiguous bytes per column.  The column sums come from the transposed words
// (__dp4a); with one split per strip they are plain stores, else integer atomics on zeroed sums (exact in any order).
template <bool kWords>
__device__ __forceinline__ void prepare_b_strip(const PrepParams &p, int block, uint32_t (*tile)[33])
{
    const OperandPrep &o     = p.op;
    const int          split = block % p.b_splits, sz = block / p.b_splits;
    const int          strip = sz % p.b_strips, z = sz / p.b_strips;
    const int          n0 = strip * 64, k_begin = split * p.k_per_split, k_end = min(o.K, k_begin + p.k_per_split);
    const uint8_t     *b  = o.b + z * o.b_batch_stride;
    const uint8_t     *b_end = b + static_cast<int64_t>(o.K - 1) * o.ldb + o.N;
    uint8_t           *bt = o.bt + static_cast<int64_t>(z) * o.N * o.ldbt;
    const int          w = threadIdx.x & 15, g = threadIdx.x >> 4; // column word, group of four rows (of 16)
    const int          n = n0 + 4 * w;
    const int          piece = threadIdx.x & 7, col = threadIdx.x >> 3; // output: eight threads write 128 bytes of a column
    int32_t            sum[2] = {0, 0}; // columns col, col + 32 of the strip: this thread's share
    for (int k0 = k_begin; k0 < k_end; k0 += 128)
    {
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            const int kg = g + 16 * h, k = k0 + 4 * kg;
            uint32_t  r[4] = {0, 0, 0, 0};
            if (n < o.N)
            {
                const uint8_t *src = b + static_cast<int64_t>(k) * o.ldb + n;
                if (kWords && n + 4 <= o.N)
                {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (k + i < k_end) r[i] = __ldg(reinterpret_cast<const uint32_t *>(src + i * o.ldb));
                }
                else if (kWords)
                {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (k + i < k_end) r[i] = load_bytes4(src + i * o.ldb, o.N - n);
                }
                else
                {
                    // any alignment: two aligned words and a shift wherever both lie inside B (columns beyond N, whose bytes
                    // belong to the next row, are neither stored nor summed), single bytes at its very ends
                    uint32_t lo[4], hi[4];
                    bool     inside[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                    {
                        const uint8_t *q = src + i * o.ldb;
                        q -= reinterpret_cast<uintptr_t>(q) & 3;
                        inside[i] = k + i < k_end && q >= b && q + 8 <= b_end;
                        lo[i] = inside[i] ? __ldg(reinterpret_cast<const uint32_t *>(q)) : 0u;
                        hi[i] = inside[i] ? __ldg(reinterpret_cast<const uint32_t *>(q) + 1) : 0u;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                    {
                        r[i] = __funnelshift_r(lo[i], hi[i], 8 * static_cast<int>(reinterpret_cast<uintptr_t>(src + i * o.ldb) & 3));
                        if (!inside[i] && k + i < k_end) r[i] = load_bytes4(src + i * o.ldb, o.N - n);
                    }
                }
            }
            const uint32_t a0 = __byte_perm(r[0], r[1], 0x5140), a1 = __byte_perm(r[2], r[3], 0x5140);
            const uint32_t b0 = __byte_perm(r[0], r[1], 0x7362), b1 = __byte_perm(r[2], r[3], 0x7362);
            // column c of the strip, K word kg: row c of `tile`, 33 words apart
            tile[4 * w + 0][kg] = __byte_perm(a0, a1, 0x5410);
            tile[4 * w + 1][kg] = __byte_perm(a0, a1, 0x7632);
            tile[4 * w + 2][kg] = __byte_perm(b0, b1, 0x5410);
            tile[4 * w + 3][kg] = __byte_perm(b0, b1, 0x7632);
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            const int       c  = col + 32 * h;
            const uint32_t *tw = &tile[c][4 * piece];
            const uint4     v  = make_uint4(tw[0], tw[1], tw[2], tw[3]);
            sum[h] = sum4(v.x, o.b_signed, sum[h]);
            sum[h] = sum4(v.y, o.b_signed, sum[h]);
            sum[h] = sum4(v.z, o.b_signed, sum[h]);
            sum[h] = sum4(v.w, o.b_signed, sum[h]);
            // ldbt is a multiple of 128: what the tile holds beyond K is the zero padding of the row
            if (n0 + c < o.N)
            {
                *reinterpret_cast<uint4 *>(bt + static_cast<int64_t>(n0 + c) * o.ldbt + k0 + 16 * piece) = v;
            }
        }
        __syncthreads();
    }
    if (o.colsum != nullptr)
    {
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            int32_t s = sum[h];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            const int c = n0 + col + 32 * h;
            if (piece == 0 && c < o.N)
            {
                int32_t *out = o.colsum + static_cast<int64_t>(z) * o.N + c;
                if (p.b_splits == 1) *out = s;
                else atomicAdd(out, s);
            }
        }
    }
}

// A: 16 bytes per lane and step, as many lanes to a row as it has such pieces (a power of two, at most the warp; the
// pixels of a convolution input are rows of a few pieces).  A row that is not 16-byte aligned is read as five aligned
// words and shifted into place (the words of neighbouring lanes overlap and hit L1); the two ends of such a row, whose
// aligned words reach outside it, are read byte by byte.
__device__ __forceinline__ uint4 load_row16(const uint8_t *row, int k, int K, bool vec)
{
    const uint8_t *p = row + k;
    const int      o = static_cast<int>(reinterpret_cast<uintptr_t>(p) & 3);
    if (k + 16 <= K && vec)
    {
        return __ldg(reinterpret_cast<const uint4 *>(p));
    }
    if (k + 16 <= K && o == 0)
    {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(p);
        return make_uint4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
    }
    if (k >= 4 && k + 20 <= K) // the aligned words of [k - o, k - o + 20) lie inside the row
    {
        const uint32_t *w  = reinterpret_cast<const uint32_t *>(p - o);
        const uint32_t  w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3), w4 = __ldg(w + 4);
        return make_uint4(__funnelshift_r(w0, w1, 8 * o), __funnelshift_r(w1, w2, 8 * o), __funnelshift_r(w2, w3, 8 * o),
                          __funnelshift_r(w3, w4, 8 * o));
    }
    uint32_t v[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        if (k + 4 * j < K) v[j] = load_bytes4(p + 4 * j, K - k - 4 * j);
    }
    return make_uint4(v[0], v[1], v[2], v[3]);
}

// Few long rows: a block per row, so that no warp walks a whole row alone (16 rows of 5429 bytes: eleven steps of 512).
__device__ __forceinline__ void prepare_a_row_blocks(const PrepParams &p, int block, int32_t *partial)
{
    const OperandPrep &o   = p.op;
    const int64_t      m   = block;
    const int64_t      z   = o.batch_a > 1 ? m / o.rows : 0;
    const uint8_t     *row = o.a + z * o.a_batch_stride + (m - z * o.rows) * o.lda;
    uint8_t           *out = o.copy != nullptr ? o.copy + m * o.kp : nullptr;
    int32_t            acc = 0;
    for (int k = 16 * static_cast<int>(threadIdx.x); k < o.K; k += 16 * kThreads)
    {
        const uint4 v = load_row16(row, k, o.K, p.a_vec);
        if (out != nullptr) *reinterpret_cast<uint4 *>(out + k) = v;
        acc = sum4(v.x, o.a_signed, acc);
        acc = sum4(v.y, o.a_signed, acc);
        acc = sum4(v.z, o.a_signed, acc);
        acc = sum4(v.w, o.a_signed, acc);
    }
    if (o.rowsum != nullptr)
    {
        acc = warp_sum(acc);
        if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0)
        {
            for (int w = 1; w < kThreads / 32; ++w) acc += partial[w];
            o.rowsum[m] = acc;
        }
    }
}

__device__ __forceinline__ void prepare_a_rows(const PrepParams &p, int block, int n_blocks)
{
    const OperandPrep &o    = p.op;
    const int          lane = threadIdx.x & 31;
    const int          sub  = lane & (p.row_lanes - 1), per_warp = 32 / p.row_lanes;
    const int          k_all = o.copy != nullptr ? static_cast<int>(o.kp) : o.K; // what a row's sum covers
    const int64_t      rows = static_cast<int64_t>(o.rows) * o.batch_a;
    for (int64_t m0 = (static_cast<int64_t>(block) * (kThreads / 32) + (threadIdx.x >> 5)) * per_warp; m0 < rows;
         m0 += static_cast<int64_t>(n_blocks) * (kThreads / 32) * per_warp)
    {
        const int64_t m   = m0 + lane / p.row_lanes; // (lanes of a row beyond the last one only take part in the sum)
        int32_t       acc = 0;
        if (m < rows)
        {
            const int64_t  z   = o.batch_a > 1 ? m / o.rows : 0;
            const uint8_t *row = o.a + z * o.a_batch_stride + (m - z * o.rows) * o.lda;
            uint8_t       *out = o.copy != nullptr ? o.copy + m * o.kp : nullptr;
            int            k   = 16 * sub;
            if (p.a_vec && out == nullptr && p.row_lanes == 32) // long aligned rows, sums only
            {
                acc = sum_vectors(reinterpret_cast<const uint4 *>(row), o.K >> 4, lane, o.a_signed, 0);
                k   = (o.K >> 4) * 16 + 16 * sub; // the piece beyond the last whole one
            }
#pragma unroll 4
            for (; k < k_all; k += 16 * p.row_lanes)
            {
                uint4 v = load_row16(row, k, o.K, p.a_vec);
                if (o.fill != 0 && k + 16 > o.K) // bytes K .. kp - 1
                {
                    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                    {
                        if (k + j >= o.K) w[j >> 2] |= static_cast<uint32_t>(o.fill) << (8 * (j & 3));
                    }
                    v = make_uint4(w[0], w[1], w[2], w[3]);
                }
                if (out != nullptr) *reinterpret_cast<uint4 *>(out + k) = v;
                acc = sum4(v.x, o.a_signed, acc);
                acc = sum4(v.y, o.a_signed, acc);
                acc = sum4(v.z, o.a_signed, acc);
                acc = sum4(v.w, o.a_signed, acc);
            }
        }
        if (o.rowsum != nullptr)
        {
            for (int x = p.row_lanes >> 1; x > 0; x >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, x);
            if (sub == 0 && m < rows) o.rowsum[m] = acc;
        }
    }
}

// kWords: B's rows are 4-byte aligned (an instantiation of its own: the shifted loads cost the aligned ones registers and with them
// blocks per SM, 4096 x 4096 10.3 -> 12.4 us)
template <bool kWords>
__global__ void __launch_bounds__(kThreads) prepare_operands_kernel(const __grid_constant__ PrepParams p)
{
    __shared__ uint32_t tile[64][33];
    dependent_prologue(); // the tensor-core kernel behind this launch sets itself up meanwhile
    const int block = static_cast<int>(blockIdx.x);
    if (block < p.b_blocks)
    {
        prepare_b_strip<kWords>(p, block, tile);
    }
    else if (p.row_lanes == kThreads)
    {
        prepare_a_row_blocks(p, block - p.b_blocks, reinterpret_cast<int32_t *>(tile));
    }
    else
    {
        prepare_a_rows(p, block - p.b_blocks, static_cast<int>(gridDim.x) - p.b_blocks);
    }
}

// ---- weights reshape: [OFM][K] -> [K][OFM] -------------------------------------------------------
// CpuWeightsReshapeKernel::run_op (CpuWeightsReshapeKernel.cpp:121-183) for NHWC weights.
__global__ void __launch_bounds__(kThreads) transpose_bytes_kernel(const uint8_t *__restrict__ src, int rows,
                                                                   int cols, uint8_t *__restrict__ dst)
{
    __shared__ uint8_t tile[64][64 + 4];
    const int          r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
    const int          tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
    src += static_cast<int64_t>(blockIdx.z) * rows * cols; // blockIdx.z: which matrix of the batch
    dst += static_cast<int64_t>(blockIdx.z) * rows * cols;
    for (int r = ty; r < 64; r += 4)
    {
        tile[r][tx] = (r0 + r < rows && c0 + tx < cols) ? src[static_cast<int64_t>(r0 + r) * cols + c0 + tx] : 0;
    }
    __syncthreads();
    for (int c = ty; c < 64; c += 4)
    {
        if (c0 + c < cols && r0 + tx < rows)
        {
            dst[static_cast<int64_t>(c0 + c) * rows + r0 + tx] = tile[tx][c];
        }
    }
}

// ---- S32 offset contribution (output stage NONE) --------------------------------------------------
// CpuGemmLowpOffsetContributionKernel (CpuGemmLowpOffsetContributionKernel.cpp:116-229).
__global__ void __launch_bounds__(kThreads) offset_contribution_kernel(int32_t *__restrict__ mm, int M, int N,
                                                                       int64_t ld_elems,
                                                                       const int32_t *__restrict__ colsum,
                                                                       const int32_t *__restrict__ rowsum,
                                                                       int32_t a_off, int32_t b_off, int32_t k_term,
                                                                       bool vec_ok)
{
    // blockIdx.y strides over rows, x over groups of four columns: no division anywhere
    const int groups = (N + 3) >> 2;
    for (int m = blockIdx.y; m < M; m += gridDim.y)
    {
        int32_t      *row   = mm + m * ld_elems;
        const int32_t rterm = k_term + (rowsum != nullptr ? b_off * __ldg(rowsum + m) : 0);
        for (int g = blockIdx.x * kThreads + threadIdx.x; g < groups; g += gridDim.x * kThreads)
        {
            const int n0 = g * 4;
            if (vec_ok && n0 + 4 <= N)
            {
                int4 v = *reinterpret_cast<int4 *>(row + n0);
                if (colsum != nullptr)
                {
                    const int4 c = __ldg(reinterpret_cast<const int4 *>(colsum + n0));
                    v.x += a_off * c.x, v.y += a_off * c.y, v.z += a_off * c.z, v.w += a_off * c.w;
                }
                v.x += rterm, v.y += rterm, v.z += rterm, v.w += rterm;
                *reinterpret_cast<int4 *>(row + n0) = v;
            }
            else
            {
                for (int n = n0; n < min(n0 + 4, N); ++n)
                {
                    row[n] += rterm + (colsum != nullptr ? a_off * colsum[n] : 0);
                }
            }
        }
    }
}

// ---- stand-alone output stage ---------------------------------------------------------------------
// CpuGemmLowpQuantizeDownInt32To{Uint8,Int8}ScaleByFixedPointKernel::run_internal
// (…ToUint8ScaleByFixedPointKernel.cpp:78-186).  A thread owns four consecutive columns -- their bias, multipliers and
// shifts stay in registers -- and walks down the rows (blockIdx.y strides over them): one 128-bit load and one 32-bit
// (8-bit output) or 64-bit (16-bit output) store per row, a warp covering 512 contiguous input bytes; no division.
template <bool kOut16>
__global__ void __launch_bounds__(kThreads) output_stage_kernel(const int32_t *__restrict__ in, int64_t ld_in_elems,
                                                                const int32_t *__restrict__ bias,
                                                                uint8_t *__restrict__ out, int64_t ld_out, int M,
                                                                int N, const int32_t *__restrict__ mults,
                                                                const int32_t *__restrict__ shifts, int32_t mult,
                                                                int32_t shift, int32_t offset, int32_t lo, int32_t hi,
                                                                bool vec_ok, bool integer_stage)
{
    dependent_prologue(); // behind the product that writes its input
    const int n0 = (blockIdx.x * kThreads + threadIdx.x) * 4;
    if (n0 >= N)
    {
        return;
    }
    const bool full = n0 + 4 <= N;
    int32_t    cb[4], cm[4], cl[4], cr[4]; // bias, multiplier, left and right shift of this thread's columns
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        const int     n  = min(n0 + j, N - 1);
        const int32_t sh = shifts != nullptr ? shifts[n] : shift;
        cb[j]            = bias != nullptr ? bias[n] : 0;
        cm[j]            = mults != nullptr ? mults[n] : mult;
        cl[j]            = max(-sh, 0);
        cr[j]            = integer_stage ? sh : max(sh, 0);
    }
    for (int m = blockIdx.y; m < M; m += gridDim.y)
    {
        const int32_t *src = in + m * ld_in_elems + n0;
        uint8_t       *dst = out + m * ld_out + n0 * (kOut16 ? 2 : 1);
        int32_t        v[4];
        if (full && vec_ok)
        {
            const int4 q = __ldcs(reinterpret_cast<const int4 *>(src)); // read once: streaming
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        }
        else
        {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = (n0 + j < N) ? src[j] : 0;
        }
        uint32_t packed = 0, packed_hi = 0; // 8-bit: four bytes in packed; 16-bit: two halfwords in each
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const int32_t x = static_cast<int32_t>(static_cast<uint32_t>(v[j]) + static_cast<uint32_t>(cb[j]));
            const int32_t r = integer_stage
                                  ? finalize_int(static_cast<int32_t>(static_cast<uint32_t>(x) + static_cast<uint32_t>(offset)),
                                                 cm[j], cr[j], lo, hi)
                                  : finalize(x, cm[j], cl[j], cr[j], offset, lo, hi);
            if (kOut16)
            {
                (j < 2 ? packed : packed_hi) |= (static_cast<uint32_t>(r) & 0xffffu) << (16 * (j & 1));
            }
            else
            {
                packed |= (static_cast<uint32_t>(r) & 0xffu) << (8 * j);
            }
        }
        if (kOut16)
        {
            if (full && vec_ok)
            {
                *reinterpret_cast<uint2 *>(dst) = make_uint2(packed, packed_hi);
            }
            else
            {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n0 + j < N)
                        reinterpret_cast<uint16_t *>(dst)[j] = static_cast<uint16_t>((j < 2 ? packed : packed_hi) >> (16 * (j & 1)));
            }
        }
        else if (full && vec_ok)
        {
            *reinterpret_cast<uint32_t *>(dst) = packed;
        }
        else
        {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n0 + j < N) dst[j] = static_cast<uint8_t>(packed >> (8 * j));
        }
    }
}

// ---- NHWC im2col ------------------------------------------------------------------------------------
// dst row m = (b, yo, xo) holds kh*kw taps of C bytes in (ky, kx, c) order; an out-of-image tap is
// filled with the input zero point (directconv2d/impl.h:333-334).  VEC = bytes moved per thread and step.
// A block takes `rows_per_iter` consecutive output rows per step and spreads their VEC-byte units over its
// threads (consecutive threads write consecutive units: whole 128-byte lines); every index split is a 32-bit
// multiply-high division by a launch constant.
struct Im2colDivs
{
    FastDiv units, c, kw, wo, ho;
};

// weights of a convolution whose channels are padded (once per weight tensor): [rows][taps][C] -> [rows][taps][Cp]
__global__ void __launch_bounds__(kThreads) spread_channels_kernel(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst,
                                                                   int rows, int taps, int C, int Cp, int64_t ldd)
{
    const int64_t total = static_cast<int64_t>(rows) * taps * Cp;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * kThreads)
    {
        const int64_t t = i / Cp; // (row, tap)
        const int     c = static_cast<int>(i - t * Cp);
        const int64_t r = t / taps;
        dst[r * ldd + (t - r * taps) * Cp + c] = c < C ? src[t * C + c] : 0;
    }
}

// ---- sums over the windows of a convolution ----------------------------------------------------
// From the channel sums of the input pixels to the patch sum of every output pixel; eight lanes share a window, four loads in
// flight each.  Bound by launch and load latency (1 x 14 x 14, 11 x 11 with 16 channels: 16.2 us for all three launches, 32.8 with the sums inside the product).
__global__ void __launch_bounds__(kThreads) window_sums_kernel(const int32_t *__restrict__ pixel_sums, int32_t *__restrict__ out, int M,
                                                               const __grid_constant__ ConvOperands cv, FastDiv div_wo, FastDiv div_ho, FastDiv div_kw)
{
    dependent_prologue();
    const int sub = threadIdx.x & 7, taps = cv.kw * cv.kh;
    for (int64_t m0 = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x - (threadIdx.x & 31)) >> 3; m0 < M;
         m0 += static_cast<int64_t>(gridDim.x) * (kThreads / 8)) // the warp's four pixels
    {
        const int m  = min(static_cast<int>(m0) + static_cast<int>((threadIdx.x & 31) >> 3), M - 1);
        const int q  = fast_div(m, div_wo), xo = m - q * cv.Wo;
        const int bi = fast_div(q, div_ho), yo = q - bi * cv.Ho;
        const int y0 = yo * cv.sy - cv.pad_t, x0 = xo * cv.sx - cv.pad_l;
        const int32_t *image = pixel_sums + static_cast<int64_t>(bi) * cv.H * cv.W;
        int32_t        sum   = 0;
#pragma unroll 4
        for (int t = sub; t < taps; t += 8)
        {
            const int ky = fast_div(t, div_kw), kx = t - ky * cv.kw;
            const int y = y0 + ky * cv.dil_y, x = x0 + kx * cv.dil_x;
            const bool in = static_cast<unsigned>(y) < static_cast<unsigned>(cv.H) && static_cast<unsigned>(x) < static_cast<unsigned>(cv.W);
            sum += in ? __ldg(image + static_cast<int64_t>(y) * cv.W + x) : cv.pad_sum;
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (sub == 0) out[m] = sum; // (lanes beyond the last pixel repeat it: the same value twice)
    }
}

template <int VEC>
__global__ void __launch_bounds__(kThreads) im2col_nhwc_kernel(const uint8_t *__restrict__ src,
                                                               uint8_t *__restrict__ dst, int C, int W, int H,
                                                               int M, int kw, int kh, int sx, int sy, int pad_l,
                                                               int pad_t, int dil_x, int dil_y, int Wo, int Ho,
                                                               uint32_t pad_word, int64_t row_stride,
                                                               int rows_per_iter, const Im2colDivs dv)
{
    const int K             = kh * kw * C;
    const int units_per_row = static_cast<int>(row_stride / VEC);
    const int per_iter      = rows_per_iter * units_per_row;
    for (int64_t m0 = static_cast<int64_t>(blockIdx.x) * rows_per_iter; m0 < M;
         m0 += static_cast<int64_t>(gridDim.x) * rows_per_iter)
    {
        for (int i = threadIdx.x; i < per_iter; i += kThreads)
        {
            const int r = fast_div(i, dv.units);
            const int m = static_cast<int>(m0) + r;
            if (m >= M)
            {
                break;
            }
            const int off = (i - r * units_per_row) * VEC; // byte offset inside the row
            uint8_t  *d   = dst + static_cast<int64_t>(m) * row_stride + off;
            if (off >= K)
            {
                // zero the K padding that makes the row a multiple of 16 bytes
                if (VEC == 16) *reinterpret_cast<uint4 *>(d) = make_uint4(0, 0, 0, 0);
                else *d = 0;
                continue;
            }
            const int tap = fast_div(off, dv.c), c = off - tap * C;
            const int ky = fast_div(tap, dv.kw), kx = tap - ky * kw;
            const int q  = fast_div(m, dv.wo), xo = m - q * Wo;
            const int b  = fast_div(q, dv.ho), yo = q - b * Ho;
            const int yi = yo * sy - pad_t + ky * dil_y;
            const int xi = xo * sx - pad_l + kx * dil_x;
            const bool     inside = yi >= 0 && yi < H && xi >= 0 && xi < W;
            const uint8_t *sp     = src + ((static_cast<int64_t>(b) * H + yi) * W + xi) * C + c;
            if (VEC == 16)
            {
                uint4 v = make_uint4(pad_word, pad_word, pad_word, pad_word);
                if (inside) v = __ldg(reinterpret_cast<const uint4 *>(sp));
                *reinterpret_cast<uint4 *>(d) = v;
            }
            else
            {
                *d = inside ? *sp : static_cast<uint8_t>(pad_word);
            }
        }
    }
}

// ---- 2x2 space-to-depth lowering of stride-2 convolutions with at most four input channels -------------
// A 7x7 / stride 2 convolution over 3 channels has a 147-byte patch row, useless to a 16-byte gather.  Folding
// every 2x2 pixel block into 16 channels ((dy, dx, c) with c padded to 4) turns it into a 4x4 / stride 1
// convolution over 16 channels whose folded weights are zero wherever the original kernel has no tap:
// the sums are the same integers.  fold_input_kernel: dst[b][Y][X][(dy*2+dx)*4 + c] = src[b][2Y+dy][2X+dx][c];
// pixels beyond an odd edge and the padding channels hold the zero point (their weights are zero).
// One thread per folded pixel (16 output bytes).  kFast: three channels, an even image width and a 2-byte aligned
// tensor -- the two pixels of a row of the block are six contiguous bytes on a 2-byte boundary and come in as three
// 16-bit loads -- and fewer than 2^31 folded pixels, so that the index arithmetic is 32-bit.
template <bool kFast>
__global__ void __launch_bounds__(kThreads) fold_input_kernel(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst,
                                                              int B, int H, int W, int C, int H2, int W2, uint32_t zp)
{
    dependent_prologue();
    const int64_t total = static_cast<int64_t>(B) * H2 * W2;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * kThreads)
    {
        int     X, Y;
        int64_t b;
        if (kFast)
        {
            uint32_t q = static_cast<uint32_t>(i);
            X          = static_cast<int>(q % static_cast<uint32_t>(W2));
            q /= static_cast<uint32_t>(W2);
            Y = static_cast<int>(q % static_cast<uint32_t>(H2));
            b = q / static_cast<uint32_t>(H2);
        }
        else
        {
            X = static_cast<int>(i % W2);
            Y = static_cast<int>((i / W2) % H2);
            b = i / (static_cast<int64_t>(W2) * H2);
        }
        uint32_t w[4];
        if (kFast)
        {
            // W is even: the block's two columns both lie inside the image
#pragma unroll
            for (int dy = 0; dy < 2; ++dy)
            {
                const int y = 2 * Y + dy;
                uint32_t  p0 = zp * 0x01010101u, p1 = p0;
                if (y < H)
                {
                    const uint16_t *p = reinterpret_cast<const uint16_t *>(src + ((b * H + y) * W + 2 * X) * 3);
                    const uint32_t  h0 = __ldg(p), h1 = __ldg(p + 1), h2 = __ldg(p + 2); // c0 c1 | c2 c0' | c1' c2'
                    p0 = h0 | ((h1 & 0xffu) << 16) | (zp << 24);
                    p1 = (h1 >> 8) | (h2 << 8) | (zp << 24);
                }
                w[2 * dy]     = p0;
                w[2 * dy + 1] = p1;
            }
        }
        else
        {
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
                const int y = 2 * Y + (q >> 1), x = 2 * X + (q & 1);
                uint32_t  v = zp * 0x01010101u;
                if (y < H && x < W)
                {
                    const uint8_t *p = src + ((b * H + y) * W + x) * C;
                    v                = 0;
                    for (int c = 0; c < 4; ++c)
                    {
                        v |= (c < C ? static_cast<uint32_t>(p[c]) : zp) << (8 * c);
                    }
                }
                w[q] = v;
            }
        }
        reinterpret_cast<uint4 *>(dst)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// fold_weights_kernel: bt[n][((ty*kw2 + tx)*4 + dy*2 + dx)*4 + c] = w[n][2ty+dy-oy][2tx+dx-ox][c], zero where the
// original kernel has no such tap or channel.  (oy, ox) = parity of the top / left padding.
__global__ void __launch_bounds__(kThreads) fold_weights_kernel(const uint8_t *__restrict__ w, uint8_t *__restrict__ bt,
                                                                int64_t ldbt, int OFM, int kh, int kw, int C, int kh2,
                                                                int kw2, int oy, int ox)
{
    const int K2    = kh2 * kw2 * 16;
    const int total = OFM * K2;
    for (int i = blockIdx.x * kThreads + threadIdx.x; i < total; i += gridDim.x * kThreads)
    {
        const int n = i / K2, k = i % K2;
        const int c = k & 3, dx = (k >> 2) & 1, dy = (k >> 3) & 1, t = k >> 4;
        const int tx = t % kw2, ty = t / kw2;
        const int ky = 2 * ty + dy - oy, kx = 2 * tx + dx - ox;
        uint8_t   v  = 0;
        if (ky >= 0 && ky < kh && kx >= 0 && kx < kw && c < C)
        {
            v = w[((static_cast<int64_t>(n) * kh + ky) * kw + kx) * C + c];
        }
        bt[n * ldbt + k] = v;
    }
}

int grid_for(int64_t work_items, int sm_count, int per_thread = 1)
{
    const int64_t blocks = (work_items + static_cast<int64_t>(kThreads) * per_thread - 1) /
                           (static_cast<int64_t>(kThreads) * per_thread);
    const int64_t cap    = static_cast<int64_t>(sm_count) * 8; // whole multiples of the SM count
    return static_cast<int>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}
} // namespace

cugl_status launch_reduce_rows(cugl_context *ctx, const void *d_a, bool is_signed, int M, int K, int64_t lda,
                               int32_t scalar, int32_t *d_out)
{
    if (M <= 0) return CUGL_SUCCESS;
    const int rows_per_block = kThreads / 32;
    const int blocks         = grid_for(static_cast<int64_t>(M) * 32, ctx->sm_count);
    (void)rows_per_block;
    reduce_rows_kernel<<<blocks, kThreads, 0, ctx->stream>>>(static_cast<const uint8_t *>(d_a), is_signed, M, K, lda,
                                                             scalar, d_out);
    return check_cuda(ctx, cudaGetLastError(), "reduce_rows_kernel");
}

cugl_status launch_reduce_cols(cugl_context *ctx, const void *d_b, bool is_signed, int K, int N, int64_t ldb,
                               int32_t scalar, int32_t *d_out)
{
    if (N <= 0) return CUGL_SUCCESS;
    CUGL_CUDA_TRY(ctx, cudaMemsetAsync(d_out, 0, sizeof(int32_t) * N, ctx->stream));
    if (K > 0)
    {
        const bool aligned = ((reinterpret_cast<uintptr_t>(d_b) | static_cast<uint64_t>(ldb)) & 15) == 0;
        const int  n_vec   = aligned ? N / 16 : 0; // 16-column units read with 128-bit loads
        // enough K slabs to fill the machine a few times over, at least 32 rows each, at most kColSlabRows
        auto slab_rows = [&](int gx) {
            int slabs = (ctx->sm_count * 4 + gx - 1) / gx;
            slabs     = max(1, min(slabs, (K + 31) / 32));
            return min(kColSlabRows, (K + slabs - 1) / slabs);
        };
        if (n_vec > 0)
        {
            const int gx          = (n_vec + kThreads - 1) / kThreads;
            const int k_per_block = slab_rows(gx);
            reduce_cols_kernel<<<dim3(gx, (K + k_per_block - 1) / k_per_block), kThreads, 0, ctx->stream>>>(
                static_cast<const uint8_t *>(d_b), is_signed, K, n_vec, ldb, k_per_block, d_out);
            CUGL_TRY(check_cuda(ctx, cudaGetLastError(), "reduce_cols_kernel"));
        }
        if (16 * n_vec < N)
        {
            const int gx          = (N - 16 * n_vec + kThreads - 1) / kThreads;
            const int k_per_block = slab_rows(gx);
            reduce_cols_generic_kernel<<<dim3(gx, (K + k_per_block - 1) / k_per_block), kThreads, 0, ctx->stream>>>(
                static_cast<const uint8_t *>(d_b), is_signed, K, 16 * n_vec, N, ldb, k_per_block, d_out);
            CUGL_TRY(check_cuda(ctx, cudaGetLastError(), "reduce_cols_generic_kernel"));
        }
    }
    if (scalar != 1)
    {
        scale_vector_kernel<<<(N + 255) / 256, 256, 0, ctx->stream>>>(d_out, N, scalar);
        CUGL_TRY(check_cuda(ctx, cudaGetLastError(), "scale_vector_kernel"));
    }
    return CUGL_SUCCESS;
}

cugl_status launch_prepare_operands(cugl_context *ctx, const OperandPrep &op)
{
    PrepParams p{};
    p.op = op;
    bool b_words = true; // B rows 4-byte aligned
    if (op.b != nullptr && op.N > 0 && op.K > 0)
    {
        // One strip of 64 columns per block, all of K, when K is short or the strips alone give every SM six blocks: the column
        // sums then need neither zeroed memory nor atomics.  Else K is split until about six blocks per SM exist: a block
        // waits for one tile's loads at a time (4096 x 14336: a block per strip 67 us, six blocks per SM 41; 4096 x 4096: two
        // blocks per SM 12.6, six 10.5).
        p.b_strips = (op.N + 63) / 64;
        const int64_t strips = static_cast<int64_t>(p.b_strips) * op.batch_b;
        const int64_t k_tiles = (op.K + 127) / 128;
        int64_t splits = strips >= 6 * ctx->sm_count ? 1 : (6 * ctx->sm_count + strips - 1) / strips;
        splits         = splits < k_tiles ? splits : k_tiles;
        if (k_tiles <= 4) splits = 1; // a strip of a few tiles is finished sooner than a memset and its launch
        const int64_t tiles_per_split = (k_tiles + splits - 1) / splits;
        p.k_per_split = static_cast<int>(tiles_per_split * 128);
        p.b_splits    = static_cast<int>((k_tiles + tiles_per_split - 1) / tiles_per_split);
        const int64_t blocks = strips * p.b_splits;
        if (blocks > INT32_MAX / 2) return fail(ctx, CUGL_UNSUPPORTED_CONFIG, "B operand: too many column strips");
        p.b_blocks = static_cast<int>(blocks);
        b_words    = ((reinterpret_cast<uintptr_t>(op.b) | static_cast<uint64_t>(op.ldb) |
                       static_cast<uint64_t>(op.batch_b > 1 ? op.b_batch_stride : 0)) & 3) == 0;
        if (p.b_splits > 1 && op.colsum != nullptr)
        {
            CUGL_CUDA_TRY(ctx, cudaMemsetAsync(op.colsum, 0, sizeof(int32_t) * static_cast<size_t>(op.N) * op.batch_b, ctx->stream));
        }
    }
    int a_blocks = 0;
    if (op.a != nullptr && op.rows > 0)
    {
        p.a_vec = ((reinterpret_cast<uintptr_t>(op.a) | static_cast<uint64_t>(op.lda) |
                    static_cast<uint64_t>(op.batch_a > 1 ? op.a_batch_stride : 0)) & 15) == 0;
        p.row_lanes = 1;
        while (p.row_lanes < 32 && p.row_lanes * 16 < op.K) p.row_lanes *= 2;
        a_blocks = grid_for(static_cast<int64_t>(op.rows) * op.batch_a * p.row_lanes, ctx->sm_count);
        // rows of more than one step per warp, and at most two blocks per SM if every row gets its own
        const int64_t all_rows = static_cast<int64_t>(op.rows) * op.batch_a;
        if (op.K > 512 && op.fill == 0 && all_rows <= 2 * ctx->sm_count)
        {
            p.row_lanes = kThreads;
            a_blocks    = static_cast<int>(all_rows);
        }
        else if (p.b_blocks == 0 && op.copy == nullptr && op.batch_a <= 1 && op.K > 512)
        {
            // Nothing but the sums of many long rows: the kernel that does only that holds more warps per SM (32768 x 1024:
            // together with its product 15.4 us against 19.2, 10000 x 2064 13.7 / 16.1).
            CUGL_CUDA_TRY(ctx, launch_dependent(ctx, reduce_rows_kernel, a_blocks, kThreads, 0, a_blocks, op.a, op.a_signed, op.rows, op.K, op.lda,
                                                1, op.rowsum));
            return check_cuda(ctx, cudaGetLastError(), "reduce_rows_kernel");
        }
    }
    if (p.b_blocks + a_blocks == 0) return CUGL_SUCCESS;
    CUGL_CUDA_TRY(ctx, launch_dependent(ctx, p.b_blocks == 0 || b_words ? prepare_operands_kernel<true> : prepare_operands_kernel<false>, p.b_blocks + a_blocks,
                                        kThreads, 0, p.b_blocks + a_blocks, p));
    return check_cuda(ctx, cudaGetLastError(), "prepare_operands_kernel");
}

cugl_status launch_transpose_colsum(cugl_context *ctx, const void *d_b, bool is_signed, int K, int N, int64_t ldb,
                                    void *d_bt, int64_t ldbt, int32_t *d_colsum, int batch, int64_t b_batch_stride)
{
    OperandPrep op{};
    op.b = static_cast<const uint8_t *>(d_b), op.ldb = ldb, op.b_batch_stride = b_batch_stride;
    op.bt = static_cast<uint8_t *>(d_bt), op.ldbt = ldbt, op.colsum = d_colsum, op.b_signed = is_signed;
    op.N = N, op.K = K, op.batch_b = batch;
    return launch_prepare_operands(ctx, op);
}

cugl_status launch_transpose_bytes(cugl_context *ctx, const void *d_src, int rows, int cols, void *d_dst, int batch)
{
    if (rows <= 0 || cols <= 0 || batch <= 0) return CUGL_SUCCESS;
    dim3 grid((cols + 63) / 64, (rows + 63) / 64, batch);
    transpose_bytes_kernel<<<grid, kThreads, 0, ctx->stream>>>(static_cast<const uint8_t *>(d_src), rows, cols,
                                                               static_cast<uint8_t *>(d_dst));
    return check_cuda(ctx, cudaGetLastError(), "transpose_bytes_kernel");
}

cugl_status launch_offset_contribution(cugl_context *ctx, int32_t *d_mm, int M, int N, int K, int64_t ld_bytes,
                                       const int32_t *d_colsum, const int32_t *d_rowsum, int32_t a_off,
                                       int32_t b_off)
{
    if (M <= 0 || N <= 0) return CUGL_SUCCESS;
    const int32_t k_term = (a_off != 0 && b_off != 0)
                               ? static_cast<int32_t>(static_cast<uint32_t>(a_off) * static_cast<uint32_t>(b_off) *
                                                      static_cast<uint32_t>(K))
                               : 0;
    const int  groups = (N + 3) / 4;
    const int  gx     = max(1, min((groups + kThreads - 1) / kThreads, 8));
    const int  gy     = max(1, min(M, ctx->sm_count * 16 / gx));
    const bool vec_ok = ((reinterpret_cast<uintptr_t>(d_mm) | static_cast<uint64_t>(ld_bytes) |
                          reinterpret_cast<uintptr_t>(d_colsum)) & 15) == 0;
    offset_contribution_kernel<<<dim3(gx, gy), kThreads, 0, ctx->stream>>>(d_mm, M, N, ld_bytes / 4,
                                                                           a_off != 0 ? d_colsum : nullptr,
                                                                           b_off != 0 ? d_rowsum : nullptr, a_off, b_off,
                                                                           k_term, vec_ok);
    return check_cuda(ctx, cudaGetLastError(), "offset_contribution_kernel");
}

cugl_status launch_output_stage(cugl_context *ctx, const int32_t *d_in, int64_t ld_in_bytes, const int32_t *d_bias,
                                void *d_out, int64_t ld_out_bytes, int M, int N, const int32_t *d_mults,
                                const int32_t *d_shifts, int32_t mult, int32_t shift, int32_t offset, int32_t lo,
                                int32_t hi, bool integer_stage, bool out16)
{
    if (M <= 0 || N <= 0) return CUGL_SUCCESS;
    const bool vec_ok = ((reinterpret_cast<uintptr_t>(d_in) | static_cast<uint64_t>(ld_in_bytes)) & 15) == 0 &&
                        ((reinterpret_cast<uintptr_t>(d_out) | static_cast<uint64_t>(ld_out_bytes)) & (out16 ? 7 : 3)) == 0;
    const int  gx = ((N + 3) / 4 + kThreads - 1) / kThreads;
    const int  gy = max(1, min(M, (ctx->sm_count * 16 + gx - 1) / gx));
    const dim3 blocks(gx, gy);
    if (out16)
    {
        CUGL_CUDA_TRY(ctx, launch_dependent(ctx, output_stage_kernel<true>, blocks, kThreads, 0, gx * gy,
            d_in, ld_in_bytes / 4, d_bias, static_cast<uint8_t *>(d_out), ld_out_bytes, M, N, d_mults, d_shifts, mult,
            shift, offset, lo, hi, vec_ok, integer_stage));
    }
    else
    {
        CUGL_CUDA_TRY(ctx, launch_dependent(ctx, output_stage_kernel<false>, blocks, kThreads, 0, gx * gy,
            d_in, ld_in_bytes / 4, d_bias, static_cast<uint8_t *>(d_out), ld_out_bytes, M, N, d_mults, d_shifts, mult,
            shift, offset, lo, hi, vec_ok, integer_stage));
    }
    return check_cuda(ctx, cudaGetLastError(), "output_stage_kernel");
}

cugl_status launch_spread_channels(cugl_context *ctx, const void *d_src, void *d_dst, int rows, int taps, int C, int Cp, int64_t ldd)
{
    const int blocks = grid_for(static_cast<int64_t>(rows) * taps * Cp, ctx->sm_count);
    spread_channels_kernel<<<blocks, kThreads, 0, ctx->stream>>>(static_cast<const uint8_t *>(d_src), static_cast<uint8_t *>(d_dst), rows,
                                                                 taps, C, Cp, ldd);
    return check_cuda(ctx, cudaGetLastError(), "spread_channels_kernel");
}

cugl_status launch_window_sums(cugl_context *ctx, const int32_t *d_pixel_sums, const ConvOperands &cv, int M, int32_t *d_out)
{
    if (M <= 0) return CUGL_SUCCESS;
    const int blocks = grid_for(static_cast<int64_t>(M) * 8, ctx->sm_count);
    CUGL_CUDA_TRY(ctx, launch_blocks(ctx, window_sums_kernel, blocks, d_pixel_sums, d_out, M, cv, make_fastdiv(cv.Wo), make_fastdiv(cv.Ho),
                                     make_fastdiv(cv.kw)));
    return check_cuda(ctx, cudaGetLastError(), "window_sums_kernel");
}

cugl_status launch_im2col_nhwc(cugl_context *ctx, const void *d_src, void *d_dst, int C, int W, int H, int B, int kw,
                               int kh, int sx, int sy, int pad_l, int pad_t, int dil_x, int dil_y, int Wo, int Ho,
                               int pad_value, int64_t row_stride)
{
    const int64_t M64 = static_cast<int64_t>(B) * Ho * Wo;
    if (M64 <= 0) return CUGL_SUCCESS;
    if (M64 >= (1ll << 31) || row_stride >= (1ll << 24))
    {
        return fail(ctx, CUGL_UNSUPPORTED_CONFIG, "im2col: more than 2^31 output rows or rows of 16 MB and more");
    }
    const int      M        = static_cast<int>(M64);
    const uint32_t pb       = static_cast<uint32_t>(pad_value) & 0xffu;
    const uint32_t pad_word = pb * 0x01010101u;
    const bool     vec16    = (C % 16 == 0) && (row_stride % 16 == 0) &&
                       ((reinterpret_cast<uintptr_t>(d_src) | reinterpret_cast<uintptr_t>(d_dst)) & 15) == 0;
    const int vec   = vec16 ? 16 : 1;
    const int units = static_cast<int>(row_stride / vec);
    // about four units per thread and step, whole rows
    const int rows_per_iter = max(1, min(M, (4 * kThreads + units - 1) / units));
    Im2colDivs dv;
    dv.units = make_fastdiv(units);
    dv.c     = make_fastdiv(C);
    dv.kw    = make_fastdiv(kw);
    dv.wo    = make_fastdiv(Wo);
    dv.ho    = make_fastdiv(Ho);
    const int blocks = grid_for((static_cast<int64_t>(M) + rows_per_iter - 1) / rows_per_iter * kThreads, ctx->sm_count);
    if (vec16)
    {
        im2col_nhwc_kernel<16><<<blocks, kThreads, 0, ctx->stream>>>(
            static_cast<const uint8_t *>(d_src), static_cast<uint8_t *>(d_dst), C, W, H, M, kw, kh, sx, sy, pad_l,
            pad_t, dil_x, dil_y, Wo, Ho, pad_word, row_stride, rows_per_iter, dv);
    }
    else
    {
        im2col_nhwc_kernel<1><<<blocks, kThreads, 0, ctx->stream>>>(
            static_cast<const uint8_t *>(d_src), static_cast<uint8_t *>(d_dst), C, W, H, M, kw, kh, sx, sy, pad_l,
            pad_t, dil_x, dil_y, Wo, Ho, pad_word, row_stride, rows_per_iter, dv);
    }
    return check_cuda(ctx, cudaGetLastError(), "im2col_nhwc_kernel");
}
cugl_status launch_fold_input(cugl_context *ctx, const void *d_src, void *d_dst, int B, int H, int W, int C, int H2,
                              int W2, int zero_point)
{
    const int blocks = grid_for(static_cast<int64_t>(B) * H2 * W2, ctx->sm_count);
    const bool fast = C == 3 && (W & 1) == 0 && (reinterpret_cast<uintptr_t>(d_src) & 1) == 0 &&
                      static_cast<int64_t>(B) * H2 * W2 <= 0x7fffffff;
    if (fast)
    {
        CUGL_CUDA_TRY(ctx, launch_blocks(ctx, fold_input_kernel<true>, blocks, static_cast<const uint8_t *>(d_src),
                                            static_cast<uint8_t *>(d_dst), B, H, W, C, H2, W2, static_cast<uint32_t>(zero_point) & 0xffu));
    }
    else
    {
        CUGL_CUDA_TRY(ctx, launch_blocks(ctx, fold_input_kernel<false>, blocks, static_cast<const uint8_t *>(d_src),
                                            static_cast<uint8_t *>(d_dst), B, H, W, C, H2, W2, static_cast<uint32_t>(zero_point) & 0xffu));
    }
    return check_cuda(ctx, cudaGetLastError(), "fold_input_kernel");
}

cugl_status launch_fold_weights(cugl_context *ctx, const void *d_w, void *d_bt, int64_t ldbt, int OFM, int kh, int kw,
                                int C, int kh2, int kw2, int oy, int ox)
{
    const int blocks = grid_for(static_cast<int64_t>(OFM) * kh2 * kw2 * 16, ctx->sm_count);
    fold_weights_kernel<<<blocks, kThreads, 0, ctx->stream>>>(static_cast<const uint8_t *>(d_w),
                                                              static_cast<uint8_t *>(d_bt), ldbt, OFM, kh, kw, C, kh2,
                                                              kw2, oy, ox);
    return check_cuda(ctx, cudaGetLastError(), "fold_weights_kernel");
}
} // namespace cugl
