// Y[M,N] (+)= X[M,K] * W[N,K]^T (+ bias[N]) on the CUDA cores, any sizes.
//
// This is the matrix product of the true 32-bit path (plain FFMA, no reduced
// precision tensor-core mode) and the catch-all for operand types the tensor-core
// kernels do not take.  The reference's products are `y[r] = sum_c W[r,c]*x[c]`
// with float accumulation over widened weights (src/cuda_bridge.cu:963-1018,
// src/math.zig:121-176); it runs one such GEMV per token
// (src/cuda_bridge.cu:1439-1444), this kernel tiles tokens instead.
//
// The order of an output's additions is fixed by K alone: the K range is cut into at most eight segments
// (segment_length below), one thread adds a segment's products in ascending k with fmaf, and the segments' sums are
// added in ascending order.  So a value does not depend on M, on where the row sits in the batch, on the kernel or
// on the tile it falls in.  The segments exist so that a product of few tiles can give every segment to a block of
// its own (the blocks of a cluster exchange their sums through shared memory); they also halve the rounding error
// (5.7e-7 relative over K = 4096 instead of 1.15e-6 of one long sum, 7.6e-7 instead of 2.1e-6 over K = 14336).
//
// Three kernels keep that rule.  gemm_generic_kernel tiles 64 tokens x 64 weight rows, one block for all segments,
// and takes every operand type.  Float operands whose rows start on 16-byte boundaries take gemm_rows_kernel with
// at most 64 tokens (it streams the weights through a ring of asynchronous copies) and gemm_tiles_kernel with more,
// unless that has one segment and few tiles (launch_float).
#include "common.cuh"
#include "tc_common.cuh"

namespace zlm {

// The length of a segment of the K range: about 1,024 elements, more where that would make more than eight segments.
constexpr int MAX_SEGMENTS = 8;
__host__ __device__ inline int segment_length(int K) {
    int n = (K + 1023) / 1024;
    n = n > MAX_SEGMENTS ? MAX_SEGMENTS : n;
    return ((K + n - 1) / n + 127) / 128 * 128;
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

// ------------------------------------------------- float operands, a cluster of blocks over the segments
struct SegArgs {
    const float* X;
    const float* W;
    const void* bias;        // float or bf16 (bias_dtype), or null
    float* Y;
    int bias_dtype, accumulate;
    int M, N, K;
    long ldx, ldw, ldy;
    int seg, segs;           // length and number of the segments; block z of a cluster of `segs` owns segment z
};

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// Four neighbouring outputs of a token, as far as they exist: the bias, then the sum that is there (accumulate).
__device__ __forceinline__ void store4(const SegArgs& a, bool vec, int gm, int gn, float (&o)[4]) {
    if (a.bias != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (gn + i < a.N)
                o[i] += a.bias_dtype == ZLM_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.bias)[gn + i])
                                                 : reinterpret_cast<const float*>(a.bias)[gn + i];
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

// Every block of the cluster holds its segment's sums of the tile at `part`: [TOK][PP] floats, ROWS of them used.
// The blocks share the tile's pieces of four neighbouring outputs and add each piece's segments in order.  All
// threads call this; the sums must be written and visible in the cluster, and no block may leave before all are done.
template <int TOK, int ROWS, int PP, int THREADS>
__device__ __forceinline__ void add_segments(const SegArgs& a, uint32_t part, int rank, int m0, int n0) {
    constexpr int Q = ROWS / 4;
    uint32_t remote[MAX_SEGMENTS];
#pragma unroll
    for (int r = 0; r < MAX_SEGMENTS; ++r) remote[r] = r < a.segs ? tc::map_to_rank(part, (uint32_t)r) : 0u;
    const int per = (TOK * Q + a.segs - 1) / a.segs;
    const bool vec = rows_on_16_bytes(a);
    for (int e = rank * per + (int)threadIdx.x; e < min(TOK * Q, (rank + 1) * per); e += THREADS) {
        const int t = e / Q, c = (e - t * Q) * 4;
        const int gm = m0 + t, gn = n0 + c;
        if (gm >= a.M || gn >= a.N) continue;
        float4 p[MAX_SEGMENTS];
#pragma unroll
        for (int r = 0; r < MAX_SEGMENTS; ++r)
            if (r < a.segs) p[r] = ld_cluster_f32x4(remote[r] + 4u * (t * PP + c));
        float o[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
        for (int r = 1; r < MAX_SEGMENTS; ++r)
            if (r < a.segs) { o[0] += p[r].x; o[1] += p[r].y; o[2] += p[r].z; o[3] += p[r].w; }
        store4(a, vec, gm, gn, o);
    }
}

// More than 64 tokens: tiles of 64 WM tokens x 64 WN weight rows, a warp 64 x 64 and a thread 8 x 16 of it (two
// groups of four tokens, four groups of four rows).  Shared memory returns 128 bytes a clock to the registers,
// broadcast or not: an 8 x 8 thread tile reads 64 bytes for 64 multiply-adds a k, as many clocks as the multiply-adds
// take; 8 x 16 reads 96 for 128, three quarters of them.  What keeps it at 34 to 44 of 74 TFLOP/s is not measured: with
// eight warps an SM (237 registers a thread) the issue of loads and multiply-adds in turn, the two barriers and the
// staging stores of a step of 8 k are candidates.  K comes in steps of 8 through two buffers: the next step's 16-byte
// global loads are in flight while this step is summed.  A tile whose K is one segment is stored from registers.  At
// 600 tokens (8 x 8 tiles of 128 x 128 without segments before): 600 x 4096 x 14336 2.99 -> 1.69 ms, 600 x 4096 x 4096
// 0.82 -> 0.59 (34 TFLOP/s), 600 x 28672 x 4096 3.31 -> 3.17 ms (44).
template <int WM, int WN> struct TileCfg {
    static constexpr int LM = 64 * WM, LN = 64 * WN, LK = 8;
    static constexpr int THREADS = 32 * WM * WN;
    static constexpr int AP = LM + 4, BP = LN + 4;           // floats of a staged k: tokens, weight rows
    static constexpr int PP = LN + 4;                        // floats of a token's sums in the exchange
    static constexpr int STAGES_BYTES = 2 * LK * (AP + BP) * 4, PART_BYTES = LM * PP * 4;
    static constexpr int SMEM = PART_BYTES > STAGES_BYTES ? PART_BYTES : STAGES_BYTES;
};

// ONE: K is one segment (a form of its own, so that neither form's registers weigh on the other).
template <int WM, int WN, bool ONE>
__global__ void __launch_bounds__(32 * WM * WN, 8 / (WM * WN))
gemm_tiles_kernel(SegArgs a) {
    using C = TileCfg<WM, WN>;
    constexpr int LM = C::LM, LN = C::LN, LK = C::LK;
    extern __shared__ __align__(16) float seg_smem[];
    float* As = seg_smem;                                    // [2][LK][AP]
    float* Bs = seg_smem + 2 * LK * C::AP;                   // [2][LK][BP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp / WN, wn = warp % WN;
    const int tm = lane >> 2, tn = lane & 3;
    const int tiles_m = (a.M + LM - 1) / LM, tiles = tiles_m * ((a.N + LN - 1) / LN);
    const int rank = (int)blockIdx.z;
    const int k_lo = rank * a.seg, k_hi = min(a.K, k_lo + a.seg);
    // loader: pieces of four k (K is a multiple of 4: a piece is whole or absent); rows beyond M or N repeat the
    // last one and are not stored
    constexpr int RS = C::THREADS / 2, XN = LM / RS, WNP = LN / RS;
    const int lr = tid >> 1, lk = (tid & 1) * 4;
    // With one segment the grid is what fits the device at once and a block goes on from tile to tile: the last tiles are
    // then spread over the SMs.  (A block a tile: those on one SM end together, and the next tiles fill it in pairs while
    // other SMs idle; 128 x 50257 x 768, 1.3 waves, took as long as two.)
    for (int tile = (int)blockIdx.x;;) {
        // the tiles of one stripe of weight rows are neighbours: its weights are read from memory once
        const int m0 = (tile % tiles_m) * LM, n0 = (tile / tiles_m) * LN;
        const float* xsrc[XN];
        const float* wsrc[WNP];
#pragma unroll
        for (int h = 0; h < XN; ++h) xsrc[h] = a.X + (long)min(m0 + lr + RS * h, a.M - 1) * a.ldx + lk;
#pragma unroll
        for (int h = 0; h < WNP; ++h) wsrc[h] = a.W + (long)min(n0 + lr + RS * h, a.N - 1) * a.ldw + lk;
        float4 xa[XN], wb[WNP];
        auto fetch = [&](int k0) {
            const bool have = k0 + lk < k_hi;
#pragma unroll
            for (int h = 0; h < XN; ++h)
                xa[h] = have ? *reinterpret_cast<const float4*>(xsrc[h] + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int h = 0; h < WNP; ++h)
                wb[h] = have ? *reinterpret_cast<const float4*>(wsrc[h] + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        auto stage = [&](int buf) {
            float* A = As + buf * LK * C::AP + lk * C::AP + lr;
            float* B = Bs + buf * LK * C::BP + lk * C::BP + lr;
#pragma unroll
            for (int h = 0; h < XN; ++h) {
                A[RS * h] = xa[h].x; A[C::AP + RS * h] = xa[h].y;
                A[2 * C::AP + RS * h] = xa[h].z; A[3 * C::AP + RS * h] = xa[h].w;
            }
#pragma unroll
            for (int h = 0; h < WNP; ++h) {
                B[RS * h] = wb[h].x; B[C::BP + RS * h] = wb[h].y;
                B[2 * C::BP + RS * h] = wb[h].z; B[3 * C::BP + RS * h] = wb[h].w;
            }
        };
        float acc[8][16];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[i][j] = 0.f;

        fetch(k_lo);
        stage(0);
        __syncthreads();
        int buf = 0;
        for (int k0 = k_lo; k0 < k_hi; k0 += LK) {
            const bool more = k0 + LK < k_hi;
            if (more) fetch(k0 + LK);
            const float* A = As + buf * LK * C::AP + wm * 64 + 4 * tm;
            const float* B = Bs + buf * LK * C::BP + wn * 64 + 4 * tn;
#pragma unroll
            for (int k = 0; k < LK; ++k) {
                float x[8], w[16];
#pragma unroll
                for (int i = 0; i < 2; ++i) *reinterpret_cast<float4*>(x + 4 * i) = *reinterpret_cast<const float4*>(A + k * C::AP + 32 * i);
#pragma unroll
                for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(w + 4 * j) = *reinterpret_cast<const float4*>(B + k * C::BP + 16 * j);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[i][j] = fmaf(x[i], w[j], acc[i][j]);
            }
            if (more) {
                stage(buf ^ 1);                                  // the other buffer was last read one step ago
                __syncthreads();
                buf ^= 1;
            }
        }
        if constexpr (ONE) {
            const bool vec = rows_on_16_bytes(a);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int gm = m0 + wm * 64 + 4 * tm + 32 * (i >> 2) + (i & 3);
                if (gm >= a.M) continue;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float o[4] = {acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]};
                    if (const int gn = n0 + wn * 64 + 4 * tn + 16 * j; gn < a.N) store4(a, vec, gm, gn, o);
                }
            }
            tile += (int)gridDim.x;
            if (tile >= tiles) return;
            __syncthreads();                                     // the stages have been read: the next tile may fill them
        } else {
            __syncthreads();                                         // the stages have been read: their memory takes the sums
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float* row = seg_smem + (wm * 64 + 4 * tm + 32 * (i >> 2) + (i & 3)) * C::PP + wn * 64 + 4 * tn;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<float4*>(row + 16 * j) = make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
            }
            tc::cluster_sync();
            add_segments<LM, LN, C::PP, C::THREADS>(a, tc::smem_u32(seg_smem), rank, m0, n0);
            tc::cluster_sync();                                      // the others may still read this block's sums
            return;
        }
    }
}

// At most 64 tokens: a block owns ROWS weight rows and all tokens (padded to TOK) of a segment, a thread RT rows x
// TT tokens; a block that has all of K stores from registers, else the blocks of a cluster add their segments.  The
// segment comes in chunks of BK floats through a ring of STAGES stages: all threads issue 16-byte asynchronous copies,
// and sum the oldest stage while the younger ones are in flight.  A staged row is padded by four floats, so that
// neighbouring rows' 16-byte reads fall in different banks.  What bounds it, beside the weights' bytes, is what shared
// memory returns to the registers (128 bytes a clock): 4 (1 / RT + 1 / TT) bytes a multiply-add, so a thread takes
// several rows and tokens where there are tokens enough.  Against one thread's sum over all of K with 1 x 2 or 1 x 8
// outputs a thread: 8 x 4096 x 14336 102 -> 57 us (4.1 TB/s), 8 x 28672 x 4096 146 -> 98 us, 32 x 28672 x 4096
// 471 -> 222 us, 64 x 4096 x 14336 1263 -> 218 us.
template <int TOK, int ROWS, int TT, int RT, int BKC, int STAGES> struct RowsCfg {
    static constexpr int TL = TOK / TT, RL = ROWS / RT, THREADS = TL * RL;
    static constexpr int PITCH = BKC + 4, STAGE = (ROWS + TOK) * PITCH;      // floats
    static constexpr int SMEM = (STAGES * STAGE > TOK * ROWS ? STAGES * STAGE : TOK * ROWS) * 4;
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, int src_bytes) {
    // copies src_bytes (0..16) and fills the rest of the 16 bytes with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int TOK, int ROWS, int TT, int RT, int BKC, int STAGES, bool ONE>
__global__ void __launch_bounds__(RowsCfg<TOK, ROWS, TT, RT, BKC, STAGES>::THREADS)
gemm_rows_kernel(SegArgs a) {
    using C = RowsCfg<TOK, ROWS, TT, RT, BKC, STAGES>;
    constexpr int T = C::THREADS, PPR = BKC / 4, RS = T / PPR;               // pieces a row, rows a pass of the threads
    static_assert(T % PPR == 0 && ROWS % RS == 0, "every pass copies whole rows");
    extern __shared__ __align__(16) float seg_smem[];
    const uint32_t base = tc::smem_u32(seg_smem);
    const int tid = threadIdx.x;
    const int n0 = (int)blockIdx.x * ROWS;
    const int rank = (int)blockIdx.z;
    const int k_lo = rank * a.seg, k_hi = min(a.K, k_lo + a.seg);
    const int n_chunks = (k_hi - k_lo + BKC - 1) / BKC;
    const int pr = tid / PPR, pc = (tid % PPR) * 4;
    auto issue = [&](int chunk) {
        const int k = k_lo + chunk * BKC + pc;
        // pieces beyond the segment are zeros (K is a multiple of 4: a piece is whole or absent); rows beyond N or M
        // repeat the last one and are not stored
        const bool have = k < k_hi;
        const int at = have ? k : 0, bytes = have ? 16 : 0;
        const uint32_t dst = base + ((chunk % STAGES) * C::STAGE + pr * C::PITCH + pc) * 4;
#pragma unroll
        for (int r = 0; r < ROWS; r += RS)
            cp_async_16(dst + r * C::PITCH * 4, a.W + (long)min(n0 + r + pr, a.N - 1) * a.ldw + at, bytes);
#pragma unroll
        for (int r = 0; r < TOK; r += RS)
            if (TOK % RS == 0 || r + pr < TOK)
                cp_async_16(dst + (ROWS + r) * C::PITCH * 4, a.X + (long)min(r + pr, a.M - 1) * a.ldx + at, bytes);
    };
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) {
        if (c < n_chunks) issue(c);
        cp_async_commit();
    }
    const int tl = tid % C::TL, rl = tid / C::TL;            // tokens tl + TL j, rows rl + RL i
    float acc[RT][TT];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < TT; ++j) acc[i][j] = 0.f;
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
        cp_async_wait<STAGES - 2>();                         // this thread's copies of the oldest stage have landed
        __syncthreads();                                     // ... and everyone's; the stage summed last is free
        if (chunk + STAGES - 1 < n_chunks) issue(chunk + STAGES - 1);
        cp_async_commit();
        const float* ws = seg_smem + (chunk % STAGES) * C::STAGE + rl * C::PITCH;
        const float* xs = seg_smem + (chunk % STAGES) * C::STAGE + (ROWS + tl) * C::PITCH;
        // with one or two outputs a thread the loads of eight steps are in flight together (2 to 8 percent)
#pragma unroll (RT * TT <= 2 ? 8 : 4)
        for (int k = 0; k < BKC; k += 4) {
            float4 w[RT], x[TT];
#pragma unroll
            for (int i = 0; i < RT; ++i) w[i] = *reinterpret_cast<const float4*>(ws + i * C::RL * C::PITCH + k);
#pragma unroll
            for (int j = 0; j < TT; ++j) x[j] = *reinterpret_cast<const float4*>(xs + j * C::TL * C::PITCH + k);
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < TT; ++j) {
                    acc[i][j] = fmaf(x[j].x, w[i].x, acc[i][j]);
                    acc[i][j] = fmaf(x[j].y, w[i].y, acc[i][j]);
                    acc[i][j] = fmaf(x[j].z, w[i].z, acc[i][j]);
                    acc[i][j] = fmaf(x[j].w, w[i].w, acc[i][j]);
                }
        }
    }
    cp_async_wait<0>();
    // (The form for one segment keeps the other way in: without it the compiler has fewer loads in flight in the loop above,
    // 32 to 48 registers instead of 64, and 3 x 2560 x 1024 takes 11.0 us instead of 8.2.)
    if (ONE && a.segs == 1) {
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < TT; ++j) {
                const int gm = tl + C::TL * j, gn = n0 + rl + C::RL * i;
                if (gm >= a.M || gn >= a.N) continue;
                float v = acc[i][j];
                if (a.bias != nullptr)
                    v += a.bias_dtype == ZLM_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.bias)[gn])
                                                  : reinterpret_cast<const float*>(a.bias)[gn];
                float* dst = a.Y + (long)gm * a.ldy + gn;
                *dst = a.accumulate ? *dst + v : v;
            }
    } else {
        __syncthreads();                                     // the stages have been read: their memory takes the sums
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < TT; ++j) seg_smem[(tl + C::TL * j) * ROWS + rl + C::RL * i] = acc[i][j];
        tc::cluster_sync();
        add_segments<TOK, ROWS, ROWS, T>(a, base, rank, 0, n0);
        tc::cluster_sync();                                      // the others may still read this block's sums
    }
}

// Launches a cluster of `segs` blocks for each of `blocks` tiles.
static int launch_segments(void (*kernel)(SegArgs), const SegArgs& a, int blocks, int threads, int smem, bool* configured,
                           cudaStream_t stream) {
    if (!*configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        *configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, 1, a.segs);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = a.segs;
    cfg.attrs = attr;
    cfg.numAttrs = a.segs > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
    return e == cudaSuccess ? launch_status() : (int)e;
}

template <int WM, int WN> static int launch_tiles(const SegArgs& a, cudaStream_t stream) {
    using C = TileCfg<WM, WN>;
    static bool configured[2] = {false, false};
    const int tiles = ((a.M + C::LM - 1) / C::LM) * ((a.N + C::LN - 1) / C::LN);
    const int room = tc::sm_count() * (8 / (WM * WN));       // blocks the registers admit at once
    if (a.segs == 1)
        return launch_segments(gemm_tiles_kernel<WM, WN, true>, a, tiles > room ? room : tiles, C::THREADS, C::STAGES_BYTES,
                               &configured[0], stream);
    return launch_segments(gemm_tiles_kernel<WM, WN, false>, a, tiles, C::THREADS, C::SMEM, &configured[1], stream);
}

template <int TOK, int ROWS, int TT, int RT, int BKC, int STAGES> static int launch_rows(const SegArgs& a, cudaStream_t stream) {
    using C = RowsCfg<TOK, ROWS, TT, RT, BKC, STAGES>;
    static bool configured[2] = {false, false};
    if (a.segs == 1)
        return launch_segments(gemm_rows_kernel<TOK, ROWS, TT, RT, BKC, STAGES, true>, a, (a.N + ROWS - 1) / ROWS, C::THREADS,
                               C::SMEM, &configured[0], stream);
    return launch_segments(gemm_rows_kernel<TOK, ROWS, TT, RT, BKC, STAGES, false>, a, (a.N + ROWS - 1) / ROWS, C::THREADS,
                           C::SMEM, &configured[1], stream);
}

// Float operands whose rows start on 16-byte boundaries; ZLM_ERR_UNSUPPORTED: gemm_generic_kernel takes the call.
static int launch_float(const void* X, const void* W, const void* bias, int bias_dtype, void* Y, int accumulate, int M, int N,
                        int K, long ldx, long ldw, long ldy, cudaStream_t stream) {
    if ((K & 3) || (ldx & 3) || (ldw & 3) || ((uintptr_t)X & 15) || ((uintptr_t)W & 15)) return ZLM_ERR_UNSUPPORTED;
    if (bias != nullptr && bias_dtype != ZLM_F32 && bias_dtype != ZLM_BF16) return ZLM_ERR_UNSUPPORTED;
    SegArgs a;
    a.X = (const float*)X; a.W = (const float*)W; a.bias = bias; a.Y = (float*)Y;
    a.bias_dtype = bias_dtype; a.accumulate = accumulate;
    a.M = M; a.N = N; a.K = K; a.ldx = ldx; a.ldw = ldw; a.ldy = ldy;
    a.seg = segment_length(K);
    a.segs = (K + a.seg - 1) / a.seg;
    // At most 32 tokens: 64 weight rows a block where that gives at least every other SM a block.  Fewer blocks leave SMs
    // idle: 32 rows then, or 16 where those are few, too (M = 8: 1024 x 1024 16.7 -> 8.1 us; M = 12, 4096 x 1024: 19.0 with
    // 64 rows, 14.0 with 32; 8192 x 1024: 19.5 with 64, 31.6 with 16).  At most four tokens and a few more blocks of 64
    // than the three an SM that run at once: 128 rows make it one wave (16384 x 2048: M = 1 33.4 -> 27.3, M = 2
    // 35.4 -> 27.5, M = 4 31.3 -> 28.3; 24000 x 1024, one wave either way, 21.6 with 64 rows, 24.1 with 128).
    const int sms = tc::sm_count();
    const long blocks = (N + 63) / 64 * (long)a.segs;
    if (M <= 32 && 2 * blocks <= sms) {
        if (4 * blocks > sms) {
            if (M <= 2) return launch_rows<2, 32, 1, 1, 64, 4>(a, stream);
            if (M <= 4) return launch_rows<4, 32, 1, 1, 64, 4>(a, stream);
            if (M <= 8) return launch_rows<8, 32, 1, 2, 64, 4>(a, stream);
            if (M <= 16) return launch_rows<16, 32, 2, 2, 64, 4>(a, stream);
            return launch_rows<32, 32, 2, 4, 64, 4>(a, stream);
        }
        if (M <= 2) return launch_rows<2, 16, 1, 1, 64, 4>(a, stream);
        if (M <= 4) return launch_rows<4, 16, 1, 1, 128, 4>(a, stream);
        if (M <= 8) return launch_rows<8, 16, 1, 1, 128, 4>(a, stream);
        if (M <= 16) return launch_rows<16, 16, 1, 2, 128, 4>(a, stream);
        return launch_rows<32, 16, 2, 2, 128, 4>(a, stream);
    }
    if (M <= 4 && blocks > 3L * sms && blocks <= 4L * sms) {
        if (M <= 1) return launch_rows<1, 128, 1, 1, 32, 4>(a, stream);
        if (M <= 2) return launch_rows<2, 128, 1, 2, 32, 4>(a, stream);
        return launch_rows<4, 128, 2, 4, 32, 4>(a, stream);
    }
    const bool most_sms = 8 * blocks > 7L * sms;
    if (M <= 1 && most_sms) return launch_rows<1, 64, 1, 1, 64, 4>(a, stream);
    if (M <= 2) return launch_rows<2, 64, 1, 1, 64, 4>(a, stream);
    if (M <= 4) return launch_rows<4, 64, 2, 1, 64, 4>(a, stream);
    if (M <= 8 && !most_sms) return launch_rows<8, 64, 4, 1, 64, 4>(a, stream);
    if (M <= 8) return launch_rows<8, 64, 4, 2, 32, 4>(a, stream);
    if (M <= 16) return launch_rows<16, 64, 2, 4, 32, 4>(a, stream);
    if (M <= 32) return launch_rows<32, 64, 4, 4, 32, 4>(a, stream);
    if (M <= 64) return launch_rows<64, 64, 4, 8, 32, 3>(a, stream);
    // One segment and few tiles: the catch-all's blocks of 256 threads, four outputs a thread wide and high, finish a lone
    // tile sooner (96 x 1024 x 1024 120 -> 84 us, 200 x 4096 x 1024 129 -> 118; two waves of it are the line: 300 x 4096 x
    // 1024 133 against 154).
    if (a.segs == 1 && (long)((M + BM - 1) / BM) * ((N + BN - 1) / BN) <= 2L * sms) return ZLM_ERR_UNSUPPORTED;
    // Tiles of 128 x 128 where their tokens are nearly all real, tiles of 64 x 128 (half the registers' worth of work, so
    // four blocks an SM) where that many fewer tokens are padding (1024 k: 130 x 28672 408 -> 333 us, 300 x 16384
    // 415 -> 336, 200 x 28672, 256 tokens either way, 414 against 418).
    const long whole = (M + 127) / 128 * 128L, half = (M + 63) / 64 * 64L;
    if (half * 105 < whole * 100) return launch_tiles<1, 2>(a, stream);
    return launch_tiles<2, 2>(a, stream);
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
    if (x_dtype == ZLM_F32 && w_dtype == ZLM_F32 && y_dtype == ZLM_F32) {
        const int rc = launch_float(X, W, bias, bias_dtype, Y, accumulate, M, N, K, ldx, ldw, ldy, stream);
        if (rc != ZLM_ERR_UNSUPPORTED) return rc;
    }
    if (x_dtype == ZLM_F32 && w_dtype == ZLM_F32)
        return pick_y<float, float>(y_dtype, bias_dtype, X, W, bias, Y, accumulate, M, N, K, ldx, ldw, ldy, stream);
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
