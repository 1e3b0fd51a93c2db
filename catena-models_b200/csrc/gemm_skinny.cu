// Y[M,N] = X[M,K] * W[N,K]^T for a handful of rows (decode steps): the weights are streamed
// once from HBM and are the 16-row operand of mma.sync.m16n8k16, the M <= 8*NT activation
// rows are its 8-wide operand ("swap A and B"), accumulation is float.
//
// A block owns 16 consecutive rows of W (gated modes: 16 gate rows and the matching 16 up rows) and one of gridDim.y slices of
// K; its 4 warps take the slice's steps of 64 values in turns and their partial sums are added through shared memory in warp
// order.  The gridDim.y blocks of a row tile form a thread-block cluster: block 0 of the cluster reads
// the others' sums from their shared memory (distributed shared memory) and adds them in rank
// order.  Every order is fixed, so the result does not depend on what else runs.  The two mma steps of 32 values
// use a lane's 8 values in an order that is the same for the W and the X fragment, so the sum over k is complete and each
// product is formed once (the instruction's own k order is irrelevant to a dot product).
//
// What bounds it: bytes on their way from HBM.  Loads into registers (this kernel's former form: 64 registers a thread, 32 warps an
// SM) kept 64 to 128 KB an SM in flight while a kernel ran and nothing between kernels: a chain of a layer's products took
// 41 us for 134 MB, its parts 3.5 to 4.8 TB/s.  Now each warp streams its weights through a ring of its own in shared memory
// (cp.async), which costs no registers, so that the next kernel's blocks become resident while this one's still run, and they fill
// their rings (weights are constants) before they wait for this kernel's results.  A chain of plain streaming kernels of that form
// reads 5.4 TB/s with the small kernels between, one with register loads 4.8.  Measured on B200, decode steps at 500 tokens
// of context: 1.7B-class, 1 row 1,044 -> 869 us, 8 rows 1,095 -> 955; 350M-class, 4 rows 465 -> 385; 2.6B-class, 3 rows 1,544 -> 1,230.
// The same kernel without the early launch: 1,032 and 1,093 us at 1 and 8 rows.  More stages are worse (four of a gated block:
// 1,066 and 1,194): their shared memory keeps the next kernel out.
//
// MODE_SWIGLU: W is the row-packed [Wgate; Wup] (2F rows); a block computes 16 gate rows and the matching 16 up rows and
// stores a = T(silu(T(g)) * T(u)) -- the reference's rounding points (lfm3_wmma.hex:10790-10815).
#include "common.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define SK_WARPS 4
#define SK_MODE_PLAIN 0
#define SK_MODE_SWIGLU 1
#define SK_MODE_GEGLU 3                      // as SWIGLU with the tanh form of gelu on the gate
#define SK_MODE_CLAMPED 4                    // both halves clamped at a limit L: min(g, L) sigmoid(1.702 min(g, L)) (clamp(u, -L, L) + 1)
#define SK_GATED(M) ((M) == SK_MODE_SWIGLU || (M) == SK_MODE_GEGLU || (M) == SK_MODE_CLAMPED)
#define SK_MODE_GELU 5                       // no gate: the tanh form of gelu on every output
#define SK_MODE_PARTS 2          // float partial sums per k-slice, no exchange between the blocks of a row tile

__device__ __forceinline__ void mma_bf16_16816(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 sk_lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// A warp's ring of weights in shared memory: a stage is 64 values of k of SETS x 16 weight rows (2 KB a set, 128 bytes a
// row).  Rows alternate between the two halves of the banks (the 16-byte pieces of an odd row are stored with their index
// xor 4), so that the fragment reads, four pieces of two rows per quarter of a warp, meet no conflict.
#define SK_SET_BYTES 2048
__device__ __forceinline__ uint32_t sk_piece(int row, int piece) { return (uint32_t)(row * 128 + ((piece ^ ((row & 1) << 2)) << 4)); }

// One warp's share of the product: of the k-blocks b0 .. b1 (of 32 values), which the block's WARPS warps take in turns of 64
// values (side by side they read 128 x WARPS consecutive bytes of a row),
// SETS x 16 weight rows against all M activation rows.  w0[s] points at the first of the set's 16 rows, of which rows[s] exist.  The ring is filled before the wait for the
// kernel before this one: weights are constants.
template <int NT, int SETS, int STAGES, int WARPS>
__device__ __forceinline__ void skinny_stream(float (&acc)[SETS][NT][4], const bf16* __restrict__ X, const bf16* const (&w0)[SETS],
                                              const int (&rows)[SETS], int b0, int b1, int M, int K, long long ldx,
                                              long long ldw, uint32_t ring, int warp, int lane) {
    constexpr int STEP = 64 * WARPS;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int s = 0; s < SETS; ++s)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[s][n][j] = 0.f;
    const int k_begin = b0 * 32 + warp * 64, k_end = min(K, b1 * 32);
    const int n_stages = k_end > k_begin ? (k_end - k_begin + STEP - 1) / STEP : 0;
    const int c_row = lane >> 3, c_piece = lane & 7;                   // this lane copies piece c_piece of rows c_row, + 4, + 8, + 12
    const uint32_t d0 = ring + sk_piece(c_row, c_piece);               // (rows 4 apart have the same parity)
    const bf16* src0[SETS];
#pragma unroll
    for (int s = 0; s < SETS; ++s) src0[s] = w0[s] + (long long)c_row * ldw + k_begin + c_piece * 8;
    auto load_w = [&](int i, int slot) {
        const bool kv = k_begin + i * STEP + c_piece * 8 < k_end;
#pragma unroll
        for (int s = 0; s < SETS; ++s)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool ok = kv && c_row + 4 * q < rows[s];
                const bf16* src = ok ? src0[s] + 4 * q * ldw + i * STEP : X;
                const int n = ok ? 16 : 0;                             // 0 source bytes: the destination is zero-filled
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d0 + (uint32_t)((slot * SETS + s) * SK_SET_BYTES + q * 512)),
                             "l"(src), "r"(n)
                             : "memory");
            }
    };
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const bf16* xp[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) xp[n] = X + (long long)(n * 8 + g < M ? n * 8 + g : 0) * ldx + k_begin + t * 8;
    auto load_x = [&](int i, uint4 (&x)[2][NT]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = k_begin + i * STEP + h * 32 + t * 8;
#pragma unroll
            for (int n = 0; n < NT; ++n)
                x[h][n] = (k < k_end && n * 8 + g < M) ? __ldg(reinterpret_cast<const uint4*>(xp[n] + i * STEP + h * 32)) : zero;
        }
    };
#pragma unroll
    for (int i = 0; i < STAGES; ++i) {
        if (i < n_stages) load_w(i, i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    pdl_wait();
    uint4 xv[2][NT], xn[2][NT];
    load_x(0, xv);
    const uint32_t f0 = ring + sk_piece(g, t), f1 = ring + sk_piece(g, t + 4);      // rows g; rows g + 8 lie 1 KB further
    int slot = 0;
    for (int i = 0; i < n_stages; ++i) {
        if (i + 1 < n_stages) load_x(i + 1, xn);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        __syncwarp();
        uint4 wa[SETS][2], wb[SETS][2];
#pragma unroll
        for (int s = 0; s < SETS; ++s) {
            const uint32_t off = (uint32_t)((slot * SETS + s) * SK_SET_BYTES);
            wa[s][0] = sk_lds128(f0 + off);
            wb[s][0] = sk_lds128(f0 + off + 1024);
            wa[s][1] = sk_lds128(f1 + off);
            wb[s][1] = sk_lds128(f1 + off + 1024);
        }
        __syncwarp();                                                  // every lane has its fragments: the slot may be filled again
        if (i + STAGES < n_stages) load_w(i + STAGES, slot);
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int s = 0; s < SETS; ++s)
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    mma_bf16_16816(acc[s][n], wa[s][h].x, wb[s][h].x, wa[s][h].y, wb[s][h].y, xv[h][n].x, xv[h][n].y);
                    mma_bf16_16816(acc[s][n], wa[s][h].z, wb[s][h].z, wa[s][h].w, wb[s][h].w, xv[h][n].z, xv[h][n].w);
                }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < NT; ++n) xv[h][n] = xn[h][n];
        slot = slot + 1 == STAGES ? 0 : slot + 1;
    }
}

// Where output (row of the tile, activation row m) lies among a warp's accumulators: [n][lane][j].
__device__ __forceinline__ int sk_slot(int row, int m) {
    return (m >> 3) * 128 + (((row & 7) << 2) | ((m & 7) >> 1)) * 4 + (((row >> 3) << 1) | (m & 1));
}

template <int NT, typename TY, int MODE, int STAGES>
__global__ void __launch_bounds__(SK_WARPS * 32)
gemm_skinny_kernel(TY* __restrict__ Y, const bf16* __restrict__ X, const bf16* __restrict__ W, int M, int N,
                   int K, long long ldx, long long ldw, long long ldy, long long part_stride, float gate_limit) {
    constexpr int SETS = SK_GATED(MODE) ? 2 : 1;                       // gated: 16 gate rows and the matching 16 up rows
    extern __shared__ __align__(128) uint8_t sk_smem[];
    __shared__ float red[SK_WARPS][SETS][NT * 128];
    __shared__ float csum[SETS][NT * 128];
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = blockIdx.x * 16;
    const int nblk = (K + 31) >> 5;
    const int ksplit = gridDim.y;
    const int per_cta = (nblk + ksplit - 1) / ksplit;
    const int c0 = min(nblk, (int)blockIdx.y * per_cta), c1 = min(nblk, c0 + per_cta);
    const bf16* w0[SETS];
    int rows[SETS];
#pragma unroll
    for (int s = 0; s < SETS; ++s) {
        w0[s] = W + (long long)(s * N + r0) * ldw;                     // N = F in the gated modes
        rows[s] = N - r0;
    }
    float acc[SETS][NT][4];
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(sk_smem) + warp * (STAGES * SETS * SK_SET_BYTES);
    skinny_stream<NT, SETS, STAGES, SK_WARPS>(acc, X, w0, rows, c0, c1, M, K, ldx, ldw, ring, warp, lane);
#pragma unroll
    for (int s = 0; s < SETS; ++s)
#pragma unroll
        for (int n = 0; n < NT; ++n)
            *reinterpret_cast<float4*>(&red[warp][s][n * 128 + lane * 4]) = make_float4(acc[s][n][0], acc[s][n][1], acc[s][n][2], acc[s][n][3]);
    __syncthreads();
    if (MODE == SK_MODE_PARTS) {
        // every k-slice leaves its sums where whoever consumes the product adds them in slice order
        for (int o = threadIdx.x; o < NT * 128; o += SK_WARPS * 32) {
            const int row = o & 15, m = o >> 4, e = sk_slot(row, m);
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < SK_WARPS; ++w) v += red[w][0][e];
            if (r0 + row < N && m < M) Y[(long long)blockIdx.y * part_stride + (long long)m * ldy + r0 + row] = from_f32<TY>(v);
        }
        return;
    }
    cg::cluster_group cluster = cg::this_cluster();
    if (ksplit > 1) {
        for (int e = threadIdx.x; e < NT * 128; e += SK_WARPS * 32)
#pragma unroll
            for (int s = 0; s < SETS; ++s) {
                float v = 0.f;
#pragma unroll
                for (int w = 0; w < SK_WARPS; ++w) v += red[w][s][e];
                csum[s][e] = v;
            }
        cluster.sync();
    }
    if (blockIdx.y == 0) {
        for (int o = threadIdx.x; o < NT * 128; o += SK_WARPS * 32) {
            const int row = o & 15, m = o >> 4, e = sk_slot(row, m);
            float tot[SETS];
#pragma unroll
            for (int s = 0; s < SETS; ++s) {
                if (ksplit > 1) {
                    tot[s] = csum[s][e];
                    for (int r = 1; r < ksplit; ++r) tot[s] += cluster.map_shared_rank(&csum[s][0], r)[e];
                } else {
                    tot[s] = 0.f;
#pragma unroll
                    for (int w = 0; w < SK_WARPS; ++w) tot[s] += red[w][s][e];
                }
            }
            if (r0 + row >= N || m >= M) continue;
            TY* dst = Y + (long long)m * ldy + r0 + row;
            if (SK_GATED(MODE)) {
                const float gr = rounded<TY>(tot[0]), ur = rounded<TY>(tot[SETS - 1]);
                float th = 0.f;      // the hardware's tanh, as in the tensor-core products' epilogue: the same digits from every product
                if (MODE == SK_MODE_GEGLU) asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(0.7978845608028654f * (gr + 0.044715f * gr * gr * gr)));
                if (MODE == SK_MODE_CLAMPED) {
                    *dst = from_f32<TY>(gated_act(gr, ur, CM_ACT_CLAMPED_SWISH, gate_limit));
                    continue;
                }
                const float ag = MODE == SK_MODE_GEGLU ? 0.5f * gr * (1.f + th) : gr * sigmoid_f32(gr);
                *dst = from_f32<TY>(ag * ur);
            } else {
                *dst = from_f32<TY>(MODE == SK_MODE_GELU ? gelu_tanh_fast(tot[0]) : tot[0]);
            }
        }
    }
    // The others' shared memory must outlive the reads.  Nothing is handed over here, so the arrival needs no
    // release (which would wait for this block's stores to Y): each thread arrives after its own reads.
    if (ksplit > 1) {
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    }
}

template <int NT, typename TY, int MODE, int STAGES>
static int launch_skinny_stages(TY* Y, const bf16* X, const bf16* W, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                                long long part_stride, int ksplit, int cluster, float gate_limit, cudaStream_t st) {
    constexpr size_t smem = SK_WARPS * STAGES * (SK_GATED(MODE) ? 2 : 1) * SK_SET_BYTES;
    auto kernel = gemm_skinny_kernel<NT, TY, MODE, STAGES>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            cm_set_error("gemm_skinny: %zu bytes of shared memory refused", smem);
            return CM_ERR_LAUNCH;
        }
        configured = true;
    }
    cm_launch_cluster(kernel, dim3((N + 15) / 16, ksplit), SK_WARPS * 32, smem, st, cluster, true, Y, X, W, M, N, K, ldx, ldw, ldy,
                      part_stride, gate_limit);
    CM_CHECK_LAUNCH();
    return CM_OK;
}

template <int NT, typename TY, int MODE>
static int launch_skinny(void* Y, const void* X, const void* W, int M, int N, int K, long long ldx, long long ldw,
                         long long ldy, cudaStream_t st, float gate_limit = 0.f) {
    const int tiles = (N + 15) / 16;
    // Few row tiles with long rows leave most SMs idle: split K over a cluster of 4 blocks then.
    // (Measured on B200: 2048 x 8192 goes from 15.3 to 10.2 us; with K = 2048 the cluster's
    // barriers cost more than the extra blocks gain.)
    const int ksplit = (tiles <= 160 && K >= 4096) ? 4 : 1;
    if constexpr (SK_GATED(MODE)) {
        // Three stages while four such blocks an SM (48 KB each) hold the whole grid at once, else two (five blocks of 32 KB,
        // as many as the registers allow): a second wave of a few blocks streams alone.  Whole decode steps, us, three /
        // two stages: 8 rows over 16,384 x 2,048 (512 blocks) 958 / 955, 4 over 9,216 x 1,024 (288) 384 / 397, 3 over
        // 21,504 x 2,048 (672) 1,340 / 1,230.
        static int sm_count = 0;
        if (!sm_count) {
            int dev = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
            if (sm_count <= 0) sm_count = 1;
        }
        if (tiles * ksplit > 4 * sm_count)
            return launch_skinny_stages<NT, TY, MODE, 2>((TY*)Y, (const bf16*)X, (const bf16*)W, M, N, K, ldx, ldw, ldy, 0, ksplit,
                                                         ksplit, gate_limit, st);
        return launch_skinny_stages<NT, TY, MODE, 3>((TY*)Y, (const bf16*)X, (const bf16*)W, M, N, K, ldx, ldw, ldy, 0, ksplit, ksplit,
                                                     gate_limit, st);
    } else {
        return launch_skinny_stages<NT, TY, MODE, 4>((TY*)Y, (const bf16*)X, (const bf16*)W, M, N, K, ldx, ldw, ldy, 0, ksplit, ksplit,
                                                     gate_limit, st);
    }
}

// Stages as the slice needs them, six at most: shared memory that a block does not use would keep the next kernel's blocks out.
template <int NT>
static int launch_skinny_parts(float* P, const void* X, const void* W, int M, int N, int K, long long ldx, long long ldw,
                               long long ldp, long long part_stride, int ksplit, cudaStream_t st) {
    const int need = ((((K + 31) / 32 + ksplit - 1) / ksplit + 1) / 2 + SK_WARPS - 1) / SK_WARPS;
    const bf16 *x = (const bf16*)X, *w = (const bf16*)W;
    if (need <= 2) return launch_skinny_stages<NT, float, SK_MODE_PARTS, 2>(P, x, w, M, N, K, ldx, ldw, ldp, part_stride, ksplit, 1, 0.f, st);
    if (need <= 4) return launch_skinny_stages<NT, float, SK_MODE_PARTS, 4>(P, x, w, M, N, K, ldx, ldw, ldp, part_stride, ksplit, 1, 0.f, st);
    return launch_skinny_stages<NT, float, SK_MODE_PARTS, 6>(P, x, w, M, N, K, ldx, ldw, ldp, part_stride, ksplit, 1, 0.f, st);
}

template <typename TY, int MODE>
static int dispatch_skinny(void* Y, const void* X, const void* W, int M, int N, int K, long long ldx, long long ldw,
                           long long ldy, cudaStream_t st, float gate_limit = 0.f) {
    if (M <= 8) return launch_skinny<1, TY, MODE>(Y, X, W, M, N, K, ldx, ldw, ldy, st, gate_limit);
    if (M <= 16) return launch_skinny<2, TY, MODE>(Y, X, W, M, N, K, ldx, ldw, ldy, st, gate_limit);
    if (M <= 32) return launch_skinny<4, TY, MODE>(Y, X, W, M, N, K, ldx, ldw, ldy, st, gate_limit);
    static_assert(CM_SKINNY_MAX_ROWS == 64, "cm_limits.h: CM_SKINNY_MAX_ROWS");
    if (M <= CM_SKINNY_MAX_ROWS) return launch_skinny<8, TY, MODE>(Y, X, W, M, N, K, ldx, ldw, ldy, st, gate_limit);
    CM_REFUSE("gemm_skinny: %d rows (at most %d)", M, CM_SKINNY_MAX_ROWS);
}

// P[s][m][n] = sum over the s-th of `ksplit` slices of K of X[m,k] W[n,k], float: the product with its
// inner dimension cut over independent blocks.  The slices are part_stride elements apart; the
// consumer (cm_add_norm with m_parts) adds them in slice order.  At most 16 rows.
extern "C" int cm_gemm_skinny_parts(float* P, const void* X, const void* W, int M, int N, int K, long long ldx,
                                    long long ldw, long long ldp, long long part_stride, int ksplit, cudaStream_t st) {
    if (M <= 0 || N <= 0) return CM_OK;
    if (M > 16) CM_REFUSE("gemm_skinny_parts: %d rows (at most 16)", M);
    if (ksplit < 1 || ksplit > 8) CM_REFUSE("gemm_skinny_parts: %d slices (1 to 8)", ksplit);
    if (K <= 0 || K % 8 || ldx % 8 || ldw % 8)
        CM_REFUSE("gemm_skinny_parts: inner size %d and row strides %lld, %lld must be multiples of 8", K, ldx, ldw);
    if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15)
        CM_REFUSE("gemm_skinny_parts: operands must be 16-byte aligned");
    if (M <= 8) return launch_skinny_parts<1>(P, X, W, M, N, K, ldx, ldw, ldp, part_stride, ksplit, st);
    return launch_skinny_parts<2>(P, X, W, M, N, K, ldx, ldw, ldp, part_stride, ksplit, st);
}

// in_proj and the gated short convolution of a decode step in one kernel (one token per sequence).
// W is the in_proj matrix [B: H rows | C: H rows | X: H rows] x K.  A block owns 16 channels; its warps split K
// and form the B, C and X rows of these channels side by side; the sums are rounded to bfloat16 as the unfused
// product's output is, and then
//     bx = B * X;  z = sum_j taps[c][j] * s[j]  with s = (state[0 .. KT-2], bx);  y = T(z * C);
//     state <- s[1 .. KT-1]
// runs once per (sequence, channel), in the same order as shortconv_kernel does it.
#define SKC_WARPS 8
#define SKC_STAGES 2

template <int NT, int STAGES>
__global__ void __launch_bounds__(SKC_WARPS * 32)
gemm_skinny_conv_kernel(bf16* __restrict__ Y, const bf16* __restrict__ X, const bf16* __restrict__ W,
                        const float* __restrict__ taps, float* __restrict__ state, const int* __restrict__ seq_slot,
                        int M, int H, int K, int KT, long long ldx, long long ldw, long long ldy) {
    extern __shared__ __align__(128) uint8_t sk_smem[];
    __shared__ float red[SKC_WARPS][3][NT * 128];
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = blockIdx.x * 16;
    const int nblk = (K + 31) >> 5;
    const bf16* w0[3];
    int rows[3];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        w0[s] = W + ((long long)s * H + r0) * ldw;
        rows[s] = H - r0;
    }
    float acc[3][NT][4];
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(sk_smem) + warp * (STAGES * 3 * SK_SET_BYTES);
    skinny_stream<NT, 3, STAGES, SKC_WARPS>(acc, X, w0, rows, 0, nblk, M, K, ldx, ldw, ring, warp, lane);
#pragma unroll
    for (int s = 0; s < 3; ++s)
#pragma unroll
        for (int n = 0; n < NT; ++n)
            *reinterpret_cast<float4*>(&red[warp][s][n * 128 + lane * 4]) = make_float4(acc[s][n][0], acc[s][n][1], acc[s][n][2], acc[s][n][3]);
    // one output per thread (NT * 128 of them, at most as many as the block has threads): its state and taps are on
    // their way while the block meets (up to 4 taps; more are read at the end)
    static_assert(NT * 128 <= SKC_WARPS * 32, "a thread per output");
    const int row = threadIdx.x & 15, m = threadIdx.x >> 4, c = r0 + row;
    const bool owner = threadIdx.x < NT * 128 && c < H && m < M;
    const bool early = KT <= 4;
    float* st = nullptr;
    const float* wc = taps + (long long)c * KT;
    float s_pre[3] = {0.f, 0.f, 0.f}, w_pre[4] = {0.f, 0.f, 0.f, 0.f};
    if (owner) {
        st = state + (long long)seq_slot[m] * (KT - 1) * H + c;
        if (early) {
#pragma unroll
            for (int q = 0; q < 3; ++q)
                if (q < KT - 1) s_pre[q] = st[(long long)q * H];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < KT) w_pre[q] = wc[q];
        }
    }
    __syncthreads();
    if (!owner) return;
    const int e = sk_slot(row, m);
    float sum[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < SKC_WARPS; ++w) v += red[w][q][e];
        sum[q] = rounded<bf16>(v);
    }
    const float bx = sum[0] * sum[2];
    float z = 0.f;
    if (early) {
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (q < KT - 1) {
                z += w_pre[q] * s_pre[q];
                if (q > 0) st[(long long)(q - 1) * H] = s_pre[q];        // shift: entry q becomes entry q - 1
            }
#pragma unroll
        for (int q = 1; q < 4; ++q)
            if (q == KT - 1) z += w_pre[q] * bx;
    } else {
        for (int q = 0; q < KT - 1; ++q) {
            const float sv = st[(long long)q * H];
            z += wc[q] * sv;
            if (q > 0) st[(long long)(q - 1) * H] = sv;
        }
        z += wc[KT - 1] * bx;
    }
    st[(long long)(KT - 2) * H] = bx;
    Y[(long long)m * ldy + c] = from_f32<bf16>(z * sum[1]);
}

template <int NT>
static int launch_skinny_conv(void* Y, const void* X, const void* W, const float* taps, float* state, const int* seq_slot, int M,
                              int H, int K, int KT, long long ldx, long long ldw, long long ldy, cudaStream_t st) {
    constexpr size_t smem = SKC_WARPS * SKC_STAGES * 3 * SK_SET_BYTES;
    auto kernel = gemm_skinny_conv_kernel<NT, SKC_STAGES>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            cm_set_error("gemm_skinny_shortconv: %zu bytes of shared memory refused", smem);
            return CM_ERR_LAUNCH;
        }
        configured = true;
    }
    cm_launch_cluster(kernel, dim3((H + 15) / 16), SKC_WARPS * 32, smem, st, 1, true, (bf16*)Y, (const bf16*)X,
                      (const bf16*)W, taps, state, seq_slot, M, H, K, KT, ldx, ldw, ldy);
    CM_CHECK_LAUNCH();
    return CM_OK;
}

// y[M, H] = the short convolution's output for M sequences that bring one token each; x [M, K],
// w [3H, K] bfloat16, taps [H][KT] float, state [slots][KT-1][H] float, seq_slot [M].
extern "C" int cm_gemm_skinny_shortconv(void* Y, const void* X, const void* W, const float* taps, float* state,
                                        const int* seq_slot, int M, int H, int K, int KT, long long ldx,
                                        long long ldw, long long ldy, cudaStream_t st) {
    if (M <= 0 || H <= 0) return CM_OK;
    if (M > 16) CM_REFUSE("gemm_skinny_shortconv: %d rows (at most 16)", M);
    if (KT < 2 || KT > CM_MAX_CONV_TAPS) CM_REFUSE("gemm_skinny_shortconv: %d taps (2..%d)", KT, CM_MAX_CONV_TAPS);
    if (K <= 0 || K % 8 || ldx % 8 || ldw % 8)
        CM_REFUSE("gemm_skinny_shortconv: inner size %d and row strides %lld, %lld must be multiples of 8", K, ldx, ldw);
    if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15)
        CM_REFUSE("gemm_skinny_shortconv: operands must be 16-byte aligned");
    if (M <= 8) return launch_skinny_conv<1>(Y, X, W, taps, state, seq_slot, M, H, K, KT, ldx, ldw, ldy, st);
    return launch_skinny_conv<2>(Y, X, W, taps, state, seq_slot, M, H, K, KT, ldx, ldw, ldy, st);
}

// X and W bfloat16; Y bfloat16 (dty = DT_BF16) or float (DT_F32).  swiglu: W has 2N rows
// ([gate; up]) and Y is [M, N].  K, ldx and ldw must be multiples of 8 (16-byte loads).
extern "C" int cm_gemm_skinny(int dty, void* Y, const void* X, const void* W, int M, int N, int K, long long ldx,
                              long long ldw, long long ldy, int swiglu, float gate_limit, cudaStream_t st) {
    if (M <= 0 || N <= 0) return CM_OK;
    if (K <= 0 || K % 8 || ldx % 8 || ldw % 8)
        CM_REFUSE("gemm_skinny: inner size %d and row strides %lld, %lld must be multiples of 8", K, ldx, ldw);
    if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15)
        CM_REFUSE("gemm_skinny: operands must be 16-byte aligned");
    if (swiglu == 4) {                       // no gate: W has N rows
        if (dty != DT_BF16) return CM_ERR_DTYPE;
        return dispatch_skinny<bf16, SK_MODE_GELU>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    }
    if (swiglu) {
        if (dty != DT_BF16) return CM_ERR_DTYPE;
        if (swiglu == 2) return dispatch_skinny<bf16, SK_MODE_GEGLU>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
        if (swiglu == 3) {
            if (!(gate_limit > 0.f)) CM_REFUSE("gemm_skinny: the clamped gate needs a positive limit");
            return dispatch_skinny<bf16, SK_MODE_CLAMPED>(Y, X, W, M, N, K, ldx, ldw, ldy, st, gate_limit);
        }
        return dispatch_skinny<bf16, SK_MODE_SWIGLU>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    }
    if (dty == DT_BF16) return dispatch_skinny<bf16, SK_MODE_PLAIN>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (dty == DT_F32) return dispatch_skinny<float, SK_MODE_PLAIN>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    return CM_ERR_DTYPE;
}
