// Y[M,N] (+)= X[M,K] * W[N,K]^T (+ bias[N]) for any sizes and types.
//
// Float operands and a float result, the product of the true 32-bit path, run on the tensor cores with every operand in
// three bf16 parts (gemm_split_kernel): no reduced precision, the error is below that of one fmaf a product.  Everything
// else, the operand types the tensor-core kernels do not take, runs on the CUDA cores (gemm_generic_kernel).  The
// reference's products are `y[r] = sum_c W[r,c]*x[c]` with float accumulation over widened weights
// (src/cuda_bridge.cu:963-1018, src/math.zig:121-176); it runs one such GEMV per token (src/cuda_bridge.cu:1439-1444),
// these kernels tile tokens instead.
//
// Both cut the K range into at most eight segments of equal length and add the segments' sums, so that rounding errors
// grow with the length of a segment and not of K.
#include "common.cuh"
#include "tc_common.cuh"

#include <mutex>

namespace zlm {

// The K range is cut into 1, 2, 4 or 8 segments of about 256 elements or more.
constexpr int MAX_SEGMENTS = 8;
__host__ __device__ inline int segment_count(int K) { return K <= 256 ? 1 : K <= 512 ? 2 : K <= 1024 ? 4 : 8; }
__host__ __device__ inline int segment_length(int K) {
    const int n = segment_count(K);
    return ((K + n - 1) / n + 63) / 64 * 64;
}

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TX, typename TW, typename TY, typename TB, bool ACC>
__global__ void __launch_bounds__(256)
gemm_generic_kernel(const TX* __restrict__ X, const TW* __restrict__ W, const TB* __restrict__ bias,
                    TY* __restrict__ Y, int M, int N, int K, long ldx, long ldw, long ldy) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    // loader coordinates: 64 rows x 16 k, four consecutive k per thread
    const int lr = tid >> 2, lk = (tid & 3) * 4;

    float acc[TM][TN], total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    const int seg = segment_length(K);                       // a multiple of BK
    int k_next = seg;                                        // where the running segment ends
    for (int k0 = 0; k0 < K; k0 += BK) {
        if (k0 == k_next) {                                  // a segment is complete
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    total[i][j] = k0 == seg ? acc[i][j] : total[i][j] + acc[i][j];
                    acc[i][j] = 0.f;
                }
            k_next += seg;
        }
        {
            const int gm = m0 + lr;
            const TX* src = X + (long)gm * ldx + k0 + lk;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int gk = k0 + lk + i;
                As[lk + i][lr] = (gm < M && gk < K) ? to_float(src[i]) : 0.f;
            }
            const int gn = n0 + lr;
            const TW* wsrc = W + (long)gn * ldw + k0 + lk;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int gk = k0 + lk + i;
                Bs[lk + i][lr] = (gn < N && gk < K) ? to_float(wsrc[i]) : 0.f;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Bs[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn >= N) continue;
            float v = K > seg ? total[i][j] + acc[i][j] : acc[i][j];
            if (bias) v += to_float(bias[gn]);
            TY* dst = Y + (long)gm * ldy + gn;
            if (ACC) *dst = from_float<TY>(to_float(*dst) + v);
            else *dst = from_float<TY>(v);
        }
    }
}

// ------------------------------------------------- float operands: tensor cores, every operand in three bf16 parts
// A float is the sum of three bf16 numbers, a = a0 + a1 2^-8 + a2 2^-16, each the rounded rest of what came before it
// (the factors keep the parts in the range of a itself, so that no part of a normal number is lost among the smallest
// bf16 numbers); the idea is published (Henry, Tang, Heinecke: Leveraging the bfloat16 artificial intelligence datatype for
// higher-precision computations, 2019).  Of the nine products of parts the six largest are taken, on the tensor cores with
// 32-bit sums: what is left out is at most 2^-24 of a product, a rounding of one fmaf (a = b = 1 + 2^-8 - 2^-17), and
// mostly a tenth of that.  They go to three sums in tensor memory,
// g0 = a0 b0, g1 = a0 b1 + a1 b0, g2 = a0 b2 + a1 b1 + a2 b0.  The tensor core cuts what does not fit a 32-bit sum
// instead of rounding it, so g0 holds SPLIT_PERIOD k at a time and threads add it up in registers, rounded; g1 and g2
// are added 2^8 and 2^16 times smaller at the end of a segment, where the cuts do not count.
//
// The order of an output's additions is fixed by K alone (the segments above, the periods, one order of the products
// in a period): a value does not depend on M, on where the row sits in the batch or on the tile it falls in.
//
// A result that is not finite is summed again with fmaf (sum_again): a part of an infinity, or of a number that bf16 rounds
// up to one, makes NaN where float has an answer.
//
// Error against 64 bits, relative, of sums of normal numbers: 1.0e-7 over K = 4096 and 1.3e-7 over K = 14336 (one fmaf a
// product in at most eight segments: 5.7e-7, 7.6e-7).  With 32, 128 or 1024 k a period 1.2e-7, 1.4e-7, 9.9e-7: shorter
// periods round oftener, longer ones cut oftener (a bias of -4.9e-8 with 64).
//
// Measured in a captured run of launches against FFMA tiles and streaming kernels: 600 tokens x 28672 x 4096 3351 -> 943 to
// 989 us, 600 x 4096 x 14336 1809 -> 412, 64 x 28672 x 4096 387 -> 147, 32 x 28672 x 4096 224 -> 99, 8 x 28672 x 4096 99 -> 79
// (6.0 TB/s).  Fewer than 8 tokens on few weight rows or a short K lose: 1 x 2048 x 8192 15 -> 22, 1 x 5120 x 5120 22 -> 29,
// 1 x 5120 x 13824 56 -> 63 to 72, 1 x 4096 x 4096 15.0 -> 16.9, 1 x 1024 x 256 2.7 -> 4.6, and one of at most 65 to 128 tokens
// with K = 64 7.1 -> 8.9; all of float32 decoding gains or stays (1 sequence at the 1B and 8B shapes 605 -> 579, 1,201 ->
// 1,209 us, four layers) but for one or two sequences at the 13B shape (1,255 -> 1,325).  A launch's start and end take some 7 us
// there and a block's stage, one block an SM, some 450 ns: its waits and hand-overs, not its bytes.  Without effect on that or
// slower, each with the same bits: a second sum for g0, three buffers of weights, a second issuing warp, a0's products in one
// instruction of 48 columns, tokens split ahead of their buffer by two groups of warps.  With 128 tokens splitting and adding
// up share the issue slots (without the splitting 858 us of 943, without the small products 836, without both 706).  Two
// blocks as one (cta_group::2, 256 x 128) took 1370 us: its hand-overs between the SMs are longer than what it saves in loads.
constexpr int SPLIT_K = 32;                 // k of a stage: 128 bytes of float, two tensor-core instructions' worth
constexpr int SPLIT_ROWS = 128;             // weight rows of a tile: the instruction's M, a lane of tensor memory each
constexpr int SPLIT_PERIOD = 64;            // k whose products meet in the tensor core before a rounded addition

struct SegArgs {
    const float* X;
    const float* W;
    const void* bias;        // float or bf16 (bias_dtype), or null
    float* Y;
    const __nv_bfloat16* planes;   // the tokens' parts as split_rows_kernel leaves them, or null: the kernel makes them itself
    int bias_dtype, accumulate;
    int M, N, K;
    long ldx, ldw, ldy;
    int seg, segs;           // length and number of the segments
    int parts;               // blocks of a cluster; each owns segs / parts neighbouring segments
    int bound;               // W is older than every kernel that may still run: it is read before the kernel before has ended
};

__device__ int split_error;                 // first bounded wait that ran out (tc::ERR_*)

// TOK tokens a tile.  Up to 32 tokens the work is streaming the weights: two blocks an SM.  Tiles of 128 tokens take the
// tokens' parts from memory, where split_rows_kernel has put them.
template <int TOK> struct SplitCfg {
    static constexpr bool PRE = TOK == 128;
    static constexpr int GROUPS = TOK == 32 ? 1 : 2;                         // of four warps that split weights, a stage each in turn
    static constexpr int EPI = TOK > 32 ? 8 : 4;                             // warps that add up the results
    static constexpr int X0 = 4 * GROUPS, EPI0 = X0 + (PRE ? 0 : 4), MMA = EPI0 + EPI;   // first warps of the roles
    static constexpr int LOAD = MMA + 1, WARPS = LOAD + (PRE ? 2 : 1), THREADS = 32 * WARPS;
    static constexpr int BLOCKS = TOK > 32 ? 1 : 2;
    static constexpr int RAW_W = SPLIT_ROWS * SPLIT_K * 4, RAW_X = PRE ? 0 : TOK * SPLIT_K * 4;   // a stage as it lies in memory
    static constexpr int STAGES_W = TOK == 128 ? 4 : TOK == 32 ? 5 : TOK == 64 ? 10 : 6, STAGES_X = 4;
    static constexpr int PLANE = TOK * SPLIT_K * 2, PLANES = 3 * PLANE;      // the tokens' parts, bf16
    static constexpr int BUFS = PRE ? 4 : 2;                                 // stages of them
    static constexpr int DEPTH = TOK == 128 ? 0 : TOK == 32 ? 2 : 3;         // sums of tensor memory that wait for their other half
    static constexpr int KEPT = TOK == 128 ? TOK * SPLIT_ROWS * 4 : 0;       // ... and the one of shared memory
    static constexpr int MAX_OWN = TOK == 128 ? 2 : 1 << DEPTH;              // segments a block may own
    static constexpr int A0 = (3 + DEPTH) * TOK;                             // first tensor-memory column of the weights' parts
    static constexpr int COLS = A0 + 96 > 256 ? 512 : 256;
    static constexpr int RINGS = STAGES_W * RAW_W + STAGES_X * RAW_X;
    static constexpr int SMEM = 1024 + RINGS + BUFS * PLANES + KEPT + 384;
    static_assert(A0 + 96 <= 512 && TOK * SPLIT_ROWS * 4 <= RINGS && BLOCKS * (SMEM + 1024) <= 233472, "room");
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, int src_bytes) {
    // copies src_bytes (0..16) and fills the rest of the 16 bytes with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float4 ld_shared_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared_u32x2(uint32_t addr, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void st_shared_u32x4(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Two floats into their three parts, packed as the operands take them (the first in the lower half).
__device__ __forceinline__ void split_pair(float lo, float hi, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    asm("{\n\t.reg .b32 l, h;\n\t.reg .b64 v, t, m, s;\n\t"
        "mov.b32 l, 0fBF800000;\n\tmov.b64 m, {l, l};\n\t"                   // -1
        "mov.b32 l, 0f43800000;\n\tmov.b64 s, {l, l};\n\t"                   // 256
        "mov.b64 v, {%3, %4};\n\t"
        "cvt.rn.bf16x2.f32 %0, %4, %3;\n\t"
        "shl.b32 l, %0, 16;\n\tand.b32 h, %0, 0xffff0000;\n\tmov.b64 t, {l, h};\n\t"
        "fma.rn.f32x2 v, t, m, v;\n\tmul.rn.f32x2 v, v, s;\n\t"
        "mov.b64 {l, h}, v;\n\tcvt.rn.bf16x2.f32 %1, h, l;\n\t"
        "shl.b32 l, %1, 16;\n\tand.b32 h, %1, 0xffff0000;\n\tmov.b64 t, {l, h};\n\t"
        "fma.rn.f32x2 v, t, m, v;\n\tmul.rn.f32x2 v, v, s;\n\t"
        "mov.b64 {l, h}, v;\n\tcvt.rn.bf16x2.f32 %2, h, l;\n\t}"
        : "=&r"(p0), "=&r"(p1), "=&r"(p2) : "f"(lo), "f"(hi));
}

// Descriptor of a K-major bf16 tile of 32 elements a row in the 64-byte swizzle: groups of 8 rows 512 bytes apart, 16-byte
// piece c of row r at piece c ^ ((r >> 1) & 3).  Layout type 4; the other fields as in smem_desc_sw128.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

// 8 registers to 8 consecutive columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ float bias_at(const SegArgs& a, int gn) {
    return a.bias_dtype == ZLM_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.bias)[gn])
                                    : reinterpret_cast<const float*>(a.bias)[gn];
}

// Four neighbouring outputs of a token, as far as they exist: the bias, then the sum that is there (accumulate).
__device__ __forceinline__ void store4(const SegArgs& a, bool vec, int gm, int gn, float (&o)[4]) {
    if (a.bias != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (gn + i < a.N)
                o[i] += bias_at(a, gn + i);
    }
    float* dst = a.Y + (long)gm * a.ldy + gn;
    if (vec && gn + 4 <= a.N) {
        float4 y = make_float4(o[0], o[1], o[2], o[3]);
        if (a.accumulate) {
            const float4 was = *reinterpret_cast<const float4*>(dst);
            y = make_float4(was.x + o[0], was.y + o[1], was.z + o[2], was.w + o[3]);
        }
        *reinterpret_cast<float4*>(dst) = y;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (gn + i < a.N) dst[i] = a.accumulate ? dst[i] + o[i] : o[i];
    }
}
__device__ __forceinline__ bool rows_on_16_bytes(const SegArgs& a) { return (a.ldy & 3) == 0 && ((uintptr_t)a.Y & 15) == 0; }

// Every block of the cluster holds the sum of its segments of the tile at `part`: [TOK][SPLIT_ROWS] floats.  The blocks
// share the tile's pieces of four neighbouring outputs and add each piece's sums pairwise.  All threads call this; the
// sums must be written and visible in the cluster, and no block may leave before all are done.
template <int TOK, int THREADS>
__device__ __forceinline__ void add_parts(const SegArgs& a, uint32_t part, int rank, int m0, int n0) {
    constexpr int Q = SPLIT_ROWS / 4;
    uint32_t remote[MAX_SEGMENTS];
#pragma unroll
    for (int r = 0; r < MAX_SEGMENTS; ++r) remote[r] = r < a.parts ? tc::map_to_rank(part, (uint32_t)r) : 0u;
    const int per = TOK * Q / a.parts;
    const bool vec = rows_on_16_bytes(a);
    for (int e = rank * per + (int)threadIdx.x; e < (rank + 1) * per; e += THREADS) {
        const int t = e / Q, c = (e - t * Q) * 4;
        const int gm = m0 + t, gn = n0 + c;
        if (gm >= a.M || gn >= a.N) continue;
        float4 p[MAX_SEGMENTS];
#pragma unroll
        for (int r = 0; r < MAX_SEGMENTS; ++r)
            if (r < a.parts) p[r] = ld_cluster_f32x4(remote[r] + 4u * (t * SPLIT_ROWS + c));
#pragma unroll
        for (int d = 1; d < MAX_SEGMENTS; d *= 2)
#pragma unroll
            for (int r = 0; r < MAX_SEGMENTS; r += 2 * d)
                if (r + d < a.parts) {
                    p[r].x += p[r + d].x; p[r].y += p[r + d].y; p[r].z += p[r + d].z; p[r].w += p[r + d].w;
                }
        float o[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
        store4(a, vec, gm, gn, o);
    }
}

// One warp's rows of a stage, the first `rows` of R rows from `src` on, k0..k0+31 of a row in 128 bytes of shared memory,
// 16-byte piece c of row r at piece c ^ (r & 7).  Rows from `rows` on and k from k_end on are zeros and not read (`src`
// is a row that exists): rows that repeated the last one asked a single token's lines 16 times over in
// every block (1 x 28672 x 4096 93 -> 82 us).
template <int R, bool WIDE>
__device__ __forceinline__ void copy_rows(uint32_t dst, const float* src, long ld, int rows, int k0, int k_end, int lane) {
    if constexpr (WIDE) {
        const int c = lane & 7, k = k0 + 4 * c;
        const bool have = k < k_end;                        // K is a multiple of 4: a piece is whole or absent
        const float* from = src + (have ? k : 0);
#pragma unroll
        for (int i = 0; i < (R + 3) / 4; ++i) {
            const int r = 4 * i + (lane >> 3);
            cp_async_16(dst + r * 128 + ((c ^ (r & 7)) << 4), r < rows ? from + (long)r * ld : from, have && r < rows ? 16 : 0);
        }
    } else {
        const bool have = k0 + lane < k_end;
        const float* from = src + (have ? k0 + lane : 0);
#pragma unroll 4
        for (int r = 0; r < R; ++r)
            cp_async_4(dst + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4, r < rows ? from + (long)r * ld : from,
                       have && r < rows ? 4 : 0);
    }
}

// The tokens' parts for tiles of 128 tokens: blocks [tile][stage][part][128 tokens][32 k], swizzled as the tensor core
// reads them, zeros beyond M and K.  A thread takes eight k of a token.
template <bool WIDE>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* X, long ldx, int M, int K, int stages, __nv_bfloat16* planes) {
    pdl_launch_dependents();
    pdl_wait();
    const int c = threadIdx.x & 3, st = (int)blockIdx.x % stages, m = (int)blockIdx.x / stages * 64 + (threadIdx.x >> 2);
    const int k = st * SPLIT_K + 8 * c, row = m & 127;
    float v[8];
    if (WIDE) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 f = m < M && k + 4 * h < K ? *reinterpret_cast<const float4*>(X + (long)m * ldx + k + 4 * h) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[4 * h] = f.x; v[4 * h + 1] = f.y; v[4 * h + 2] = f.z; v[4 * h + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = m < M && k + i < K ? X[(long)m * ldx + k + i] : 0.f;
    }
    uint32_t p[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) split_pair(v[2 * i], v[2 * i + 1], p[0][i], p[1][i], p[2][i]);
    uint4* to = reinterpret_cast<uint4*>(planes) + ((long)(m >> 7) * stages + st) * (3 * 128 * 4) + row * 4 + (c ^ ((row >> 1) & 3));
#pragma unroll
    for (int i = 0; i < 3; ++i) to[i * 128 * 4] = make_uint4(p[i][0], p[i][1], p[i][2], p[i][3]);
}

// A copy of contiguous memory into shared memory (16-byte boundaries and size), counted on `bar` in bytes.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// A warp's results of a segment (`sums`: this lane's weight row, `tokens` of them), those that are not finite summed again over
// n k of the tokens' rows `x` and this lane's row `w` (null: there is none), by the whole warp: the first eight k a row a lane,
// which is all where the token's numbers are NaN; then row after row, the lanes on neighbouring k.  A sum that is NaN stays
// so, and is left there.  No wait of the kernel runs out meanwhile: a poll takes 4 us, the limit is 17 s.
// 64 x 2048 x 8192, of which are not finite: one row of weights 90 us, one number of every token 2,440, all tokens' numbers
// 140 (finite 58; a thread by itself with 32 sums one after another took tens of milliseconds for the first).
// A function of its own, called with everything in memory: inlined it cost the way past it registers and 2 percent.
__device__ __noinline__ void sum_again(float* sums, int tokens, const float* x, long ldx, const float* w, int n, int lane) {
#pragma unroll 1
    for (int t = 0; t < tokens; ++t, x += ldx) {
        unsigned who = __ballot_sync(0xffffffffu, w != nullptr && !(fabsf(sums[t]) <= 3.402823466e38f));
        if (who == 0) continue;
        float v = 0.f;
        const bool mine = (who >> lane) & 1u;
        if (mine)
            for (int k = 0; k < min(n, 8); ++k) v = fmaf(x[k], w[k], v);
        for (who &= __ballot_sync(0xffffffffu, v == v); who != 0; who &= who - 1) {
            const int l = __ffs(who) - 1;
            const float* row = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, (unsigned long long)w, l));
            float sum = 0.f;
            for (int k = lane; k - lane < n && !__any_sync(0xffffffffu, sum != sum); k += 256) {
                float p[8], q[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const bool have = k + 32 * i < n;
                    p[i] = have ? x[k + 32 * i] : 0.f;
                    q[i] = have ? row[k + 32 * i] : 0.f;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) sum = fmaf(p[i], q[i], sum);
            }
            sum = warp_sum(sum);
            if (lane == l) v = sum;
        }
        if (mine) sums[t] = v;
    }
}

// Roles of the warps.  One thread asks for the weights (TMA, 128 rows x 32 k a stage); with rows off 16-byte boundaries
// the warps that split them copy them themselves.  Weights (in groups of four warps that take the stages in turn): 32
// weight rows a warp, a row a thread from shared memory into its parts in tensor memory (operand A).  Tokens: the
// same into three planes of shared memory (operand B), or one thread that copies planes made before.  One warp issues the
// tensor-core instructions, four or eight add up the results.
template <int TOK, bool WIDE>
__global__ void __launch_bounds__(SplitCfg<TOK>::THREADS, SplitCfg<TOK>::BLOCKS)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, SegArgs a) {
    using C = SplitCfg<TOK>;
    extern __shared__ uint8_t split_smem[];
    const uint32_t raw = tc::smem_u32(split_smem), base = (raw + 1023u) & ~1023u;
    const uint32_t ring_x = base + C::STAGES_W * C::RAW_W, planes = base + C::RINGS, kept = planes + C::BUFS * C::PLANES, bars = kept + C::KEPT;
    // barriers: weights' parts ready [2] and read [2] (tokens that are split here share them: one wait and one commit a stage
    // less, 6144 x 4096 at 8 tokens 25.4 -> 24.2 us, at 64 44.8 -> 41.5), planes ready [BUFS] and read [BUFS], the sums of a
    // period and of a segment ready and read, no instruction in flight, weights in memory ready [STAGES_W] and read [STAGES_W]; then the
    // tensor memory's address and the abort flag
    const uint32_t w_full = bars, w_empty = bars + 16;
    const uint32_t x_full = C::PRE ? bars + 32 : w_full, x_empty = C::PRE ? bars + 64 : w_empty;   // one pair for both
    const uint32_t sums_full = bars + 96, sums_free = bars + 104, seg_full = bars + 112, seg_free = bars + 120, drained = bars + 128;
    const uint32_t raw_full = bars + 136, raw_empty = raw_full + 8 * C::STAGES_W;
    uint32_t* holder = reinterpret_cast<uint32_t*>(split_smem + (bars - raw) + 136 + 16 * C::STAGES_W);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(holder + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int tiles_m = (a.M + TOK - 1) / TOK;
    // the tiles of one stripe of weight rows are neighbours: its weights are read from memory once
    const int tile_m = (int)blockIdx.x % tiles_m, m0 = tile_m * TOK, n0 = ((int)blockIdx.x / tiles_m) * SPLIT_ROWS;
    const int rank = (int)blockIdx.z, own = a.segs / a.parts;
    const int k_lo = min(a.K, rank * own * a.seg), k_hi = min(a.K, k_lo + own * a.seg);
    const int n_stages = (k_hi - k_lo + SPLIT_K - 1) / SPLIT_K, seg_stages = a.seg / SPLIT_K;
    constexpr int PERIOD = SPLIT_PERIOD / SPLIT_K;
    int* err = &split_error;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(w_full + 8 * s, C::PRE ? 4 : 8);
            tc::mbar_init(w_empty + 8 * s, 1);
        }
        for (int s = 0; C::PRE && s < C::BUFS; ++s) {
            tc::mbar_init(x_full + 8 * s, 1);
            tc::mbar_init(x_empty + 8 * s, 1);
        }
        for (int s = 0; s < C::STAGES_W; ++s) {
            tc::mbar_init(raw_full + 8 * s, 1);
            tc::mbar_init(raw_empty + 8 * s, 4);
        }
        tc::mbar_init(sums_full, 1);
        tc::mbar_init(sums_free, C::EPI);
        tc::mbar_init(seg_full, 1);
        tc::mbar_init(seg_free, C::EPI);
        tc::mbar_init(drained, 1);
        *abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == C::MMA) {
        tc::tmem_alloc(tc::smem_u32(holder), C::COLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem = *holder;
    pdl_launch_dependents();

    if (warp < C::X0) {
        // ------------------------------------------------------------ weights into their parts
        constexpr int G = C::GROUPS, OWN = C::STAGES_W / G;                  // slots of the ring a group fills itself
        const int w = warp & 3, group = warp >> 2;
        const int rows = a.N - (n0 + 32 * w);
        const float* src = a.W + (long)min(n0 + 32 * w, a.N - 1) * a.ldw;
        const uint32_t mine = base + 32 * w * 128;
        int ahead = group;
        auto fetch = [&]() {
            const int slot = group * OWN + ahead / G % OWN;
            if (ahead < n_stages) copy_rows<32, false>(mine + slot * C::RAW_W, src, a.ldw, rows, k_lo + ahead * SPLIT_K, k_hi, lane);
            cp_async_commit();
            ahead += G;
        };
        if constexpr (!WIDE) {
            if (!a.bound) pdl_wait();
#pragma unroll 1
            for (int s = 0; s < OWN - 1; ++s) fetch();
        }
        for (int st = group; st < n_stages; st += G) {
            const int slot = WIDE ? st % C::STAGES_W : group * OWN + st / G % OWN;
            if constexpr (WIDE) {
                if (!tc::warp_wait(raw_full + 8 * slot, (st / C::STAGES_W) & 1, abort_flag, err, tc::ERR_WAIT_FULL)) break;
            } else {
                cp_async_wait<OWN - 2>();                                    // this lane's copies of the stage have landed
                __syncwarp();                                                // ... and the warp's; the stage before has been read
                fetch();
            }
            const uint32_t from = mine + slot * C::RAW_W + lane * 128;
            const int buf = st & 1;
            const uint32_t to = tmem + ((uint32_t)(w * 32) << 16) + C::A0 + 48 * buf;
            // as much as the registers hold is ready before the tensor core has read the buffer
            constexpr int H = TOK == 128 ? 2 : 1;                            // 16 k each: 8 columns of each part
            bool alive = true;
#pragma unroll
            for (int h0 = 0; h0 < 2; h0 += H) {
                uint32_t p[H][3][8];
#pragma unroll
                for (int h = 0; h < H; ++h) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 v = ld_shared_f32x4(from + (((4 * (h0 + h) + c) ^ (lane & 7)) << 4));
                        split_pair(v.x, v.y, p[h][0][2 * c], p[h][1][2 * c], p[h][2][2 * c]);
                        split_pair(v.z, v.w, p[h][0][2 * c + 1], p[h][1][2 * c + 1], p[h][2][2 * c + 1]);
                    }
                }
                if (WIDE && h0 + H == 2) {                                   // the weights have been read
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(raw_empty + 8 * slot);
                }
                if (h0 == 0) {
                    alive = tc::warp_wait(w_empty + 8 * buf, ((st >> 1) & 1) ^ 1u, abort_flag, err, tc::ERR_WAIT_EMPTY);
                    if (!alive) break;
                    tc::tc_fence_after_sync();
                }
#pragma unroll
                for (int h = 0; h < H; ++h)
#pragma unroll
                    for (int i = 0; i < 3; ++i) tmem_st8(to + 16 * i + 8 * (h0 + h), p[h][i]);
            }
            if (!alive) break;
            tc::tmem_st_wait();
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(w_full + 8 * buf);
        }
        cp_async_wait<0>();                                                  // gives up with no copy in flight
    } else if (warp == C::LOAD) {
        // ------------------------------------------------------------ weights as they lie in memory
        // bound weights do not depend on the kernel before: the first are asked for before it has ended
        if (WIDE && lane == 0) {
            if (!a.bound) pdl_wait();
            int st = 0;
            for (; st < n_stages; ++st) {
                const int slot = st % C::STAGES_W;
                if (!tc::mbar_wait(raw_empty + 8 * slot, ((st / C::STAGES_W) & 1) ^ 1u, abort_flag, err, tc::ERR_WAIT_EMPTY)) break;
                tc::mbar_expect_tx(raw_full + 8 * slot, C::RAW_W);
                tc::tma_load_2d(base + slot * C::RAW_W, &map_w, raw_full + 8 * slot, k_lo + st * SPLIT_K, n0);
            }
            if (st < n_stages)                                               // gives up with no copy in flight
                for (int s = st > C::STAGES_W ? st - C::STAGES_W : 0; s < st; ++s)
                    for (uint32_t i = 0; i < tc::WAIT_POLLS && !tc::mbar_try_wait(raw_full + 8 * (s % C::STAGES_W), (s / C::STAGES_W) & 1); ++i) {}
        }
    } else if (C::PRE && warp == C::LOAD + 1) {
        // ------------------------------------------------------------ tokens' planes
        if (lane == 0) {
            const uint8_t* src = reinterpret_cast<const uint8_t*>(a.planes) + ((long)tile_m * ((a.K + SPLIT_K - 1) / SPLIT_K) + k_lo / SPLIT_K) * C::PLANES;
            pdl_wait();
            int st = 0;
            for (; st < n_stages; ++st) {
                const int buf = st % C::BUFS;
                if (!tc::mbar_wait(x_empty + 8 * buf, ((st / C::BUFS) & 1) ^ 1u, abort_flag, err, tc::ERR_WAIT_EMPTY)) break;
                tc::mbar_expect_tx(x_full + 8 * buf, C::PLANES);
                bulk_load(planes + buf * C::PLANES, src + (long)st * C::PLANES, C::PLANES, x_full + 8 * buf);
            }
            if (st < n_stages)                                               // gives up with no copy in flight
                for (int s = st > C::BUFS ? st - C::BUFS : 0; s < st; ++s)
                    for (uint32_t i = 0; i < tc::WAIT_POLLS && !tc::mbar_try_wait(x_full + 8 * (s % C::BUFS), (s / C::BUFS) & 1); ++i) {}
        }
    } else if (!C::PRE && warp < C::EPI0) {
        // ------------------------------------------------------------ tokens into their parts
        constexpr int XR = TOK / 4;                                          // a warp's token rows
        const int w = warp & 3;
        const int rows = a.M - (m0 + XR * w);
        const float* src = a.X + (long)min(m0 + XR * w, a.M - 1) * a.ldx;
        const uint32_t ring = ring_x + XR * w * 128;
        auto fetch = [&](int st) {
            if (st < n_stages) copy_rows<XR, WIDE>(ring + (st % C::STAGES_X) * C::RAW_X, src, a.ldx, rows, k_lo + st * SPLIT_K, k_hi, lane);
            cp_async_commit();
        };
        pdl_wait();
#pragma unroll 1
        for (int s = 0; s < C::STAGES_X - 1; ++s) fetch(s);
        for (int st = 0; st < n_stages; ++st) {
            cp_async_wait<C::STAGES_X - 2>();
            __syncwarp();
            fetch(st + C::STAGES_X - 1);
            const int buf = st & 1;
            if (!tc::warp_wait(x_empty + 8 * buf, ((st >> 1) & 1) ^ 1u, abort_flag, err, tc::ERR_WAIT_EMPTY)) break;
            constexpr int CPT = TOK / 16;                                    // pieces of four k a thread takes
            const int r = lane % XR, c0 = (lane / XR) * CPT, row = XR * w + r;
            const uint32_t from = ring + (st % C::STAGES_X) * C::RAW_X + r * 128;
            const uint32_t to = planes + buf * C::PLANES + row * 64;
            const int turn = (row >> 1) & 3;
            if constexpr (CPT == 1) {
                const float4 v = ld_shared_f32x4(from + ((c0 ^ (r & 7)) << 4));
                uint32_t p[3][2];
                split_pair(v.x, v.y, p[0][0], p[1][0], p[2][0]);
                split_pair(v.z, v.w, p[0][1], p[1][1], p[2][1]);
#pragma unroll
                for (int i = 0; i < 3; ++i) st_shared_u32x2(to + i * C::PLANE + (((c0 >> 1) ^ turn) << 4) + (c0 & 1) * 8, p[i][0], p[i][1]);
            } else {
#pragma unroll
                for (int c = 0; c < CPT; c += 2) {
                    uint32_t p[3][4];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float4 v = ld_shared_f32x4(from + (((c0 + c + j) ^ (r & 7)) << 4));
                        split_pair(v.x, v.y, p[0][2 * j], p[1][2 * j], p[2][2 * j]);
                        split_pair(v.z, v.w, p[0][2 * j + 1], p[1][2 * j + 1], p[2][2 * j + 1]);
                    }
#pragma unroll
                    for (int i = 0; i < 3; ++i)
                        st_shared_u32x4(to + i * C::PLANE + ((((c0 + c) >> 1) ^ turn) << 4), p[i][0], p[i][1], p[i][2], p[i][3]);
                }
            }
            tc::fence_proxy_async();                                         // the tensor core reads what threads wrote
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(x_full + 8 * buf);
        }
        cp_async_wait<0>();
    } else if (warp == C::MMA) {
        // ------------------------------------------------------------ tensor-core instructions
        constexpr uint32_t one = tc::idesc_bf16(128, TOK), two = tc::idesc_bf16(128, 2 * TOK);
        int in_seg = 0, period = 0, segment = 0, st = 0;
        // a segment is an even number of stages and starts a period: a stage's buffer and its place in the period go together
        static_assert(PERIOD == 2 && C::BUFS % 2 == 0, "two stages a period, two buffers of weights");
        // (two stages at a time spill at 16 and 32 tokens: 1 x 2048 x 8192 23.7 us, 22.4 without; at 128 they save 3 percent)
#pragma unroll (TOK <= 32 ? 1 : 2)
        for (; st < n_stages; ++st) {
            const int buf = st & 1, xb = C::PRE ? st % C::BUFS : buf;
            const bool starts = buf == 0, seg_ends = in_seg + 1 == seg_stages || st + 1 == n_stages, ends = buf == 1 || seg_ends;
            if (C::PRE && !tc::warp_wait(x_full + 8 * xb, (st / C::BUFS) & 1, abort_flag, err, tc::ERR_WAIT_FULL)) break;
            if (!tc::warp_wait(w_full + 8 * buf, (st >> 1) & 1, abort_flag, err, tc::ERR_WAIT_FULL)) break;
            if (starts && period > 0 && !tc::warp_wait(sums_free, (period - 1) & 1, abort_flag, err, tc::ERR_WAIT_ACCUM)) break;
            tc::tc_fence_after_sync();
            const uint32_t A = tmem + C::A0 + 48 * buf;
            const uint64_t B0 = smem_desc_sw64(planes + xb * C::PLANES), B1 = smem_desc_sw64(planes + xb * C::PLANES + C::PLANE);
            auto large = [&]() {
#pragma unroll
                for (int h = 0; h < 2; ++h) tc::umma_bf16_ts(tmem, A + 8 * h, B0 + 2 * h, one, !(starts && h == 0));
                if (ends) tc::umma_commit(sums_full);                        // g0 is read while g1 and g2 are summed
            };
            auto small = [&]() {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    tc::umma_bf16_ts(tmem + TOK, A + 8 * h, B1 + 2 * h, two, !(in_seg == 0 && h == 0));
                    tc::umma_bf16_ts(tmem + TOK, A + 16 + 8 * h, B0 + 2 * h, two, 1);
                    tc::umma_bf16_ts(tmem + 2 * TOK, A + 32 + 8 * h, B0 + 2 * h, one, 1);
                }
                tc::umma_commit(w_empty + 8 * buf);
                if (C::PRE) tc::umma_commit(x_empty + 8 * xb);
                if (seg_ends) tc::umma_commit(seg_full);
            };
            if (in_seg == 0 && segment > 0) {
                if (tc::elect_one()) large();
                __syncwarp();
                if (!tc::warp_wait(seg_free, (segment - 1) & 1, abort_flag, err, tc::ERR_WAIT_ACCUM)) break;
                tc::tc_fence_after_sync();
                if (tc::elect_one()) small();
            } else if (tc::elect_one()) {
                large();
                small();
            }
            __syncwarp();
            if (ends) ++period;
            if (seg_ends) { in_seg = 0; ++segment; } else ++in_seg;
        }
        if (st < n_stages) {                                                 // gives up with no instruction in flight
            if (tc::elect_one()) tc::umma_commit(drained);
            __syncwarp();
            tc::warp_wait(drained, 0, abort_flag, err, tc::ERR_WAIT_DRAIN);
        }
    } else {
        // ------------------------------------------------------------ results
        constexpr int COLS = TOK * 4 / C::EPI, CH = COLS / 16;               // a warp's tokens
        const int q = warp & 3, t0 = ((warp - C::EPI0) >> 2) * COLS;
        const int gn = n0 + q * 32 + lane;
        const uint32_t mine = tmem + ((uint32_t)(q * 32) << 16) + t0;
        float* part = reinterpret_cast<float*>(split_smem + (base - raw)) + t0 * SPLIT_ROWS + q * 32 + lane;
        float* kept_at = reinterpret_cast<float*>(split_smem + (kept - raw)) + t0 * SPLIT_ROWS + q * 32 + lane;
        pdl_wait();                                                          // Y may be read by the kernel before
        int period = 0;
        for (int s = 0; s < own; ++s) {
            float acc[COLS];
#pragma unroll
            for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
            const int stages = min(seg_stages, n_stages - s * seg_stages);   // none: beyond K, zeros
            if (stages > 0) {
                bool alive = true;
                for (int p = 0; p < (stages + PERIOD - 1) / PERIOD; ++p, ++period) {
                    if (!tc::warp_wait(sums_full, period & 1, abort_flag, err, tc::ERR_WAIT_ACCUM)) { alive = false; break; }
                    tc::tc_fence_after_sync();
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        uint32_t v[16];
                        tc::tmem_ld16(mine + 16 * c, v);
                        tc::tmem_ld_wait();
                        if (c == CH - 1) {
                            tc::tc_fence_before_sync();
                            __syncwarp();
                            if (lane == 0) tc::mbar_arrive(sums_free);
                        }
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[16 * c + i] += __uint_as_float(v[i]);
                    }
                }
                if (!alive || !tc::warp_wait(seg_full, s & 1, abort_flag, err, tc::ERR_WAIT_ACCUM)) break;
                tc::tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    uint32_t v[16], u[16];
                    tc::tmem_ld16(mine + TOK + 16 * c, v);
                    tc::tmem_ld16(mine + 2 * TOK + 16 * c, u);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        acc[16 * c + i] += fmaf(__uint_as_float(u[i]), 0x1p-16f, __uint_as_float(v[i]) * 0x1p-8f);
                }
                tc::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(seg_free);
                bool again = false;                                          // results that are not finite
#pragma unroll
                for (int i = 0; i < COLS; ++i) again |= !(fabsf(acc[i]) <= 3.402823466e38f);
                if (__builtin_expect(__any_sync(0xffffffffu, again && gn < a.N), 0)) {
                    float all[COLS];
#pragma unroll
                    for (int i = 0; i < COLS; ++i) all[i] = acc[i];
                    const int k0 = k_lo + s * a.seg;
                    sum_again(all, min(COLS, a.M - m0 - t0), a.X + (long)(m0 + t0) * a.ldx + k0, a.ldx,
                              gn < a.N ? a.W + (long)gn * a.ldw + k0 : nullptr, min(a.seg, k_hi - k0), lane);
#pragma unroll
                    for (int i = 0; i < COLS; ++i) acc[i] = all[i];
                }
            }
            // neighbouring segments are added pairwise, then the pairs, then the fours: the sums that wait for their
            // other half lie in tensor memory, a level each (128 tokens: in shared memory, one level)
            if constexpr (C::DEPTH > 0) {
                int level = 0;
#pragma unroll 1
                for (; (s >> level) & 1; ++level) {
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        uint32_t v[16];
                        tc::tmem_ld16(mine + (3 + level) * TOK + 16 * c, v);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[16 * c + i] = __uint_as_float(v[i]) + acc[16 * c + i];
                    }
                }
                if (s + 1 < own) {
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        uint32_t v[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(acc[16 * c + i]);
                        tc::tmem_st16(mine + (3 + level) * TOK + 16 * c, v);
                    }
                    tc::tmem_st_wait();
                    continue;
                }
            } else if (own > 1) {
                if (s == 0) {
#pragma unroll
                    for (int i = 0; i < COLS; ++i) kept_at[i * SPLIT_ROWS] = acc[i];
                    continue;
                }
#pragma unroll
                for (int i = 0; i < COLS; ++i) acc[i] = kept_at[i * SPLIT_ROWS] + acc[i];
            }
            if (a.parts > 1) {                                               // all stages have been read: their memory takes the sums
#pragma unroll
                for (int i = 0; i < COLS; ++i) part[i * SPLIT_ROWS] = acc[i];
            } else if (gn < a.N) {
                const float bias = a.bias != nullptr ? bias_at(a, gn) : 0.f;
#pragma unroll
                for (int i = 0; i < COLS; ++i) {
                    const int gm = m0 + t0 + i;
                    if (gm < a.M) {
                        float* dst = a.Y + (long)gm * a.ldy + gn;
                        float v = acc[i];
                        if (a.bias != nullptr) v += bias;
                        *dst = a.accumulate ? *dst + v : v;
                    }
                }
            }
        }
    }
    if (a.parts > 1) {
        pdl_wait();
        tc::cluster_sync_arrive_wait();
        add_parts<TOK, C::THREADS>(a, base, rank, m0, n0);
        tc::cluster_sync_arrive_wait();                                      // the others may still read this block's sums
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == C::MMA) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc(tmem, C::COLS);
    }
}

// The weights in boxes of 32 k x 128 rows with the 128-byte swizzle; what lies beyond K or N is read as zeros.
static int weight_map(CUtensorMap* m, const SegArgs& a) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<Encode>(p);
    });
    if (!fn) return ZLM_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)a.K, (cuuint64_t)a.N}, strides[1] = {(cuuint64_t)a.ldw * 4};
    const cuuint32_t box[2] = {SPLIT_K, SPLIT_ROWS}, steps[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(a.W), dims, strides, box, steps,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : ZLM_ERR_UNSUPPORTED;
}

template <int TOK, bool WIDE> static int launch_split(const CUtensorMap& map_w, const SegArgs& a, long tiles, cudaStream_t stream) {
    using C = SplitCfg<TOK>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<TOK, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(gemm_split_kernel<TOK, WIDE>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles, 1, a.parts);
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // may start while its predecessor drains
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = a.parts;
    cfg.attrs = attr;
    cfg.numAttrs = a.parts > 1 ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_split_kernel<TOK, WIDE>, map_w, a);
    return e == cudaSuccess ? launch_status() : (int)e;
}

// Blocks a cluster: as few as fill the device, the segments' sums then meeting in fewer places.
template <int TOK> static int launch_tokens(SegArgs a, bool wide, cudaStream_t stream) {
    using C = SplitCfg<TOK>;
    const long tiles = (long)((a.N + SPLIT_ROWS - 1) / SPLIT_ROWS) * ((a.M + TOK - 1) / TOK);
    if (tiles > 0x7fffffffL) return ZLM_ERR_UNSUPPORTED;
    const long room = (long)tc::sm_count() * C::BLOCKS;
    a.parts = a.segs > C::MAX_OWN ? a.segs / C::MAX_OWN : 1;
    while (a.parts < a.segs && tiles * a.parts * 2 <= room) a.parts *= 2;
    CUtensorMap map_w = {};
    return wide && weight_map(&map_w, a) == 0 ? launch_split<TOK, true>(map_w, a, tiles, stream)
                                              : launch_split<TOK, false>(map_w, a, tiles, stream);
}

// Tokens whose parts one call of the tile kernel finds in memory; the scratch they take.
constexpr long SPLIT_CHUNK_BYTES = 128l << 20;
static long split_row_bytes(int K) { return (long)((K + SPLIT_K - 1) / SPLIT_K) * SPLIT_K * 6; }
static int split_chunk(int M, int K) {
    const long tiles = SPLIT_CHUNK_BYTES / (128 * split_row_bytes(K)), need = (M + 127) / 128;
    return (int)(need < tiles ? need : tiles > 1 ? tiles : 1) * 128;
}

static int launch_float(const void* X, const void* W, const void* bias, int bias_dtype, void* Y, int accumulate, int M, int N,
                        int K, long ldx, long ldw, long ldy, int bound, void* scratch, long scratch_bytes, cudaStream_t stream) {
    if (bias != nullptr && bias_dtype != ZLM_F32 && bias_dtype != ZLM_BF16) return ZLM_ERR_UNSUPPORTED;
    SegArgs a;
    a.X = (const float*)X; a.W = (const float*)W; a.bias = bias; a.Y = (float*)Y;
    a.planes = nullptr;
    a.bound = bound;
    a.bias_dtype = bias_dtype; a.accumulate = accumulate;
    a.M = M; a.N = N; a.K = K; a.ldx = ldx; a.ldw = ldw; a.ldy = ldy;
    a.segs = segment_count(K);
    a.seg = segment_length(K);
    // rows that start on 16-byte boundaries are copied by TMA and 16 bytes at a time, others 4 bytes at a time
    const bool wide = !((K & 3) || (ldx & 3) || (ldw & 3) || ((uintptr_t)X & 15) || ((uintptr_t)W & 15));
    if (M <= 16) return launch_tokens<16>(a, wide, stream);
    if (M <= 32) return launch_tokens<32>(a, wide, stream);
    const int chunk = split_chunk(M, K);
    if (M <= 64 || scratch == nullptr || ((uintptr_t)scratch & 15) || scratch_bytes < chunk * split_row_bytes(K))
        return launch_tokens<64>(a, wide, stream);
    const int stages = (K + SPLIT_K - 1) / SPLIT_K;
    a.planes = (const __nv_bfloat16*)scratch;
    for (int m = 0; m < M; m += chunk) {
        a.M = M - m < chunk ? M - m : chunk;
        a.X = (const float*)X + (long)m * ldx;
        a.Y = (float*)Y + (long)m * ldy;
        const dim3 grid((unsigned)((a.M + 127) / 128 * 2 * stages));
        cudaError_t e = wide ? launch_pdl(split_rows_kernel<true>, grid, dim3(256), 0, stream, a.X, ldx, a.M, K, stages, (__nv_bfloat16*)scratch)
                             : launch_pdl(split_rows_kernel<false>, grid, dim3(256), 0, stream, a.X, ldx, a.M, K, stages, (__nv_bfloat16*)scratch);
        if (e != cudaSuccess) return (int)e;
        const int rc = launch_tokens<128>(a, wide, stream);
        if (rc != 0) return rc;
    }
    return 0;
}

template <typename TX, typename TW, typename TY, typename TB>
static int launch(const void* X, const void* W, const void* bias, void* Y, int accumulate, int M, int N, int K,
                  long ldx, long ldw, long ldy, cudaStream_t stream) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (accumulate)
        gemm_generic_kernel<TX, TW, TY, TB, true><<<grid, 256, 0, stream>>>(
            (const TX*)X, (const TW*)W, (const TB*)bias, (TY*)Y, M, N, K, ldx, ldw, ldy);
    else
        gemm_generic_kernel<TX, TW, TY, TB, false><<<grid, 256, 0, stream>>>(
            (const TX*)X, (const TW*)W, (const TB*)bias, (TY*)Y, M, N, K, ldx, ldw, ldy);
    return launch_status();
}

template <typename TX, typename TW, typename TY>
static int pick_bias(int bias_dtype, const void* X, const void* W, const void* bias, void* Y, int accumulate, int M,
                     int N, int K, long ldx, long ldw, long ldy, cudaStream_t stream) {
    if (bias == nullptr || bias_dtype == ZLM_F32)
        return launch<TX, TW, TY, float>(X, W, bias, Y, accumulate, M, N, K, ldx, ldw, ldy, stream);
    if (bias_dtype == ZLM_BF16)
        return launch<TX, TW, TY, __nv_bfloat16>(X, W, bias, Y, accumulate, M, N, K, ldx, ldw, ldy, stream);
    return ZLM_ERR_UNSUPPORTED;
}

template <typename TX, typename TW>
static int pick_y(int y_dtype, int bias_dtype, const void* X, const void* W, const void* bias, void* Y,
                  int accumulate, int M, int N, int K, long ldx, long ldw, long ldy, cudaStream_t stream) {
    if (y_dtype == ZLM_F32)
        return pick_bias<TX, TW, float>(bias_dtype, X, W, bias, Y, accumulate, M, N, K, ldx, ldw, ldy, stream);
    if (y_dtype == ZLM_BF16)
        return pick_bias<TX, TW, __nv_bfloat16>(bias_dtype, X, W, bias, Y, accumulate, M, N, K, ldx, ldw, ldy,
                                                 stream);
    return ZLM_ERR_UNSUPPORTED;
}

}  // namespace zlm

using namespace zlm;

// accumulate != 0: Y += X*W^T (+bias); the running sum is read and written in Y's type.
ZLM_EXPORT int zlm_gemm_generic(const void* X, int x_dtype, const void* W, int w_dtype, const void* bias,
                                int bias_dtype, void* Y, int y_dtype, int accumulate, int M, int N, int K,
                                long ldx, long ldw, long ldy, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || ldx < K || ldw < K || ldy < N) return ZLM_ERR_BAD_ARG;
    if (x_dtype == ZLM_F32 && w_dtype == ZLM_F32 && y_dtype == ZLM_F32)
        return launch_float(X, W, bias, bias_dtype, Y, accumulate, M, N, K, ldx, ldw, ldy, 0, nullptr, 0, stream);
    if (x_dtype == ZLM_F32 && w_dtype == ZLM_F32)
        return y_dtype == ZLM_BF16 ? pick_bias<float, float, __nv_bfloat16>(bias_dtype, X, W, bias, Y, accumulate, M, N, K, ldx,
                                                                            ldw, ldy, stream)
                                   : ZLM_ERR_UNSUPPORTED;
    if (x_dtype == ZLM_F32 && w_dtype == ZLM_BF16)
        return pick_y<float, __nv_bfloat16>(y_dtype, bias_dtype, X, W, bias, Y, accumulate, M, N, K, ldx, ldw, ldy,
                                            stream);
    if (x_dtype == ZLM_BF16 && w_dtype == ZLM_F32)
        return pick_y<__nv_bfloat16, float>(y_dtype, bias_dtype, X, W, bias, Y, accumulate, M, N, K, ldx, ldw, ldy,
                                            stream);
    if (x_dtype == ZLM_BF16 && w_dtype == ZLM_BF16)
        return pick_y<__nv_bfloat16, __nv_bfloat16>(y_dtype, bias_dtype, X, W, bias, Y, accumulate, M, N, K, ldx,
                                                    ldw, ldy, stream);
    return ZLM_ERR_UNSUPPORTED;
}

// The same product of float operands, which is faster with scratch memory from 65 tokens on (16-byte aligned; its
// contents are of no use afterwards).  zlm_gemm_float_scratch: the bytes it takes.  bound != 0: W holds what it is to hold
// before any kernel that may still run when this one starts (a model's weights); its first rows are then read while the
// kernels before finish.  Otherwise W may come from the kernel just before.
ZLM_EXPORT long zlm_gemm_float_scratch(int M, int K) { return M <= 64 || K <= 0 ? 0 : split_chunk(M, K) * split_row_bytes(K); }

ZLM_EXPORT int zlm_gemm_float(const void* X, const void* W, const void* bias, int bias_dtype, void* Y, int accumulate, int M,
                              int N, int K, long ldx, long ldw, long ldy, int bound, void* scratch, long scratch_bytes,
                              cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || ldx < K || ldw < K || ldy < N) return ZLM_ERR_BAD_ARG;
    return launch_float(X, W, bias, bias_dtype, Y, accumulate, M, N, K, ldx, ldw, ldy, bound, scratch, scratch_bytes, stream);
}

// Reads and clears the error word the float kernels report bounded-wait failures through (synchronises the device).
ZLM_EXPORT int zlm_gemm_generic_status(int* out) {
    cudaError_t e = cudaMemcpyFromSymbol(out, split_error, sizeof(int));
    if (e == cudaSuccess && *out != 0) {
        const int none = 0;
        e = cudaMemcpyToSymbol(split_error, &none, sizeof(int));
    }
    return (int)e;
}
