// Y[M,N] = X[M,K] * W[N,K]^T on the CUDA cores, float accumulation with plain FMAs.
//
// This is the matrix product of the true 32-bit path (no tensor-core mode of reduced
// precision is involved) and the any-size fallback of the bfloat16 path.  Every output
// element is formed in one order whatever kernel forms it: K is cut into slices of GS_SLICE, a
// slice's sum runs over its k in increasing order, and the slices' sums are added in slice order.  A
// row's result therefore does not depend on M, on the tile it falls in, or on its batch-mates, and
// the shorter running sums round less than one sum over all of K would.
//
// Three kernels:
//  - gemm_simt_rows_kernel, up to 16 rows at a time (decode steps, short prompts): bound by the stream of
//    weights, whose slices are spread over warps and blocks;
//  - gemm_simt_tile_kernel, more rows: bound by the FMA pipe, 8 x 8 outputs a thread in packed pairs;
//  - gemm_simt_kernel, any types and alignment.
#include "common.cuh"

#define GS_BM 64
#define GS_BN 64
#define GS_BK 16
#define GS_SLICE 128                   // k of one slice: a multiple of every kernel's k-step

template <typename TX, typename TW, typename TY>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(TY* __restrict__ Y, const TX* __restrict__ X, const TW* __restrict__ W, int M,
                 int N, int K, long long ldx, long long ldw, long long ldy) {
    pdl_wait();
    __shared__ float xs[GS_BK][GS_BM + 1];
    __shared__ float ws[GS_BK][GS_BN + 1];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 x 16 threads, 4 x 4 outputs each
    const int m0 = blockIdx.y * GS_BM, n0 = blockIdx.x * GS_BN;
    float acc[4][4], total[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = total[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += GS_BK) {
        // 64 rows x 16 k per operand = 1024 elements, 4 per thread
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 256;
            const int r = e >> 4, k = e & 15;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + k;
            xs[k][r] = (gm < M && gk < K) ? to_f32(X[(long long)gm * ldx + gk]) : 0.f;
            ws[k][r] = (gn < N && gk < K) ? to_f32(W[(long long)gn * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GS_BK; ++k) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if ((k0 + GS_BK) % GS_SLICE == 0 || k0 + GS_BK >= K) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    total[i][j] += acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
        __syncthreads();
    }
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn < N) Y[(long long)gm * ldy + gn] = from_f32<TY>(total[i][j]);
        }
    }
}

// ---- float, 16-byte aligned operands, up to MR rows of X at a time --------------------------------------
// A warp takes R rows of W (lanes) x Q slices of K (R * Q = 32): a lane forms the MR sums of its row over its
// slice.  The block's warps take the slices of a round side by side and the block adds the round's sums in slice order.
// W and X come through a ring of the warp's own in shared memory (cp.async, chunks of 32 k = 128 bytes of a row); the
// pitch of 36 floats spreads the lanes' 16-byte reads over all banks.  The first stages' weights are requested before
// the wait for the kernel before this one.  Bound by the stream of weights up to about eight rows: 4 x 65,536 x 1,024 55 us
// (4.9 TB/s; before 446), 4 x 3,072 x 1,024 5.6 us (before 118).
#define GSR_STAGES 4
#define GSR_CHUNK 32
#define GSR_PITCH 36

__device__ __forceinline__ void gs_cp16(uint32_t dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;                 // 0 source bytes: the 16 destination bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

template <int MR, int R>
__global__ void __launch_bounds__(256)
gemm_simt_rows_kernel(float* __restrict__ Y, const float* __restrict__ X, const float* __restrict__ W, int M, int N, int K,
                      long long ldx, long long ldw, long long ldy) {
    constexpr int Q = 32 / R;
    constexpr int W_FLOATS = 32 * GSR_PITCH, X_FLOATS = MR * Q * GSR_PITCH;
    constexpr int STAGE = W_FLOATS + X_FLOATS;
    constexpr int CHUNKS = GS_SLICE / GSR_CHUNK;
    extern __shared__ __align__(16) float gsr_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int row = lane % R, q = lane / R;
    const int n0 = blockIdx.x * R, m0 = blockIdx.y * MR;
    float* ring = gsr_smem + warp * GSR_STAGES * STAGE;
    float* red = gsr_smem + warps * GSR_STAGES * STAGE;                // [warps * Q][MR][R]
    const int slices = (K + GS_SLICE - 1) / GS_SLICE;
    const int per_round = warps * Q;
    const int rounds = (slices + per_round - 1) / per_round;
    const int stages = rounds * CHUNKS;

    const int piece = (lane & 7) * 4;                                  // floats of the chunk that this lane copies
    const uint32_t ring_addr = (uint32_t)__cvta_generic_to_shared(ring);
    auto chunk_k = [&](int stage, int qq) { return ((stage / CHUNKS) * per_round + warp * Q + qq) * GS_SLICE + (stage % CHUNKS) * GSR_CHUNK; };
    auto load_w = [&](int stage) {
        const uint32_t dst = ring_addr + (stage % GSR_STAGES) * STAGE * 4;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = i * 4 + (lane >> 3), r = c % R;              // the chunk of lane c
            const int k = chunk_k(stage, c / R) + piece;
            const bool ok = n0 + r < N && k < K;
            gs_cp16(dst + (c * GSR_PITCH + piece) * 4, ok ? W + (long long)(n0 + r) * ldw + k : W, ok);
        }
    };
    auto load_x = [&](int stage) {
        const uint32_t dst = ring_addr + ((stage % GSR_STAGES) * STAGE + W_FLOATS) * 4;
#pragma unroll
        for (int i = 0; i < (MR * Q + 3) / 4; ++i) {
            const int c = i * 4 + (lane >> 3), m = c / Q;              // chunk c: row m of X, slice c % Q
            const int k = chunk_k(stage, c % Q) + piece;
            const bool ok = m < MR && m0 + m < M && k < K;
            if (MR * Q % 4 == 0 || c < MR * Q) gs_cp16(dst + (c * GSR_PITCH + piece) * 4, ok ? X + (long long)(m0 + m) * ldx + k : X, ok);
        }
    };
#pragma unroll
    for (int s = 0; s < GSR_STAGES - 1; ++s)
        if (s < stages) load_w(s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < GSR_STAGES - 1; ++s) {
        if (s < stages) load_x(s);
        asm volatile("cp.async.commit_group;" ::: "memory");           // the first group holds every weight requested above
    }
    float acc[MR];
    constexpr int OUTS = (MR * R + 31) / 32;                           // outputs of a block per thread, at most (one warp)
    float total[OUTS];
#pragma unroll
    for (int i = 0; i < OUTS; ++i) total[i] = 0.f;
    for (int rd = 0; rd < rounds; ++rd) {
#pragma unroll
        for (int m = 0; m < MR; ++m) acc[m] = 0.f;
#pragma unroll 1
        for (int c = 0; c < CHUNKS; ++c) {
            const int st = rd * CHUNKS + c;
            if (st + GSR_STAGES - 1 < stages) {
                load_w(st + GSR_STAGES - 1);
                load_x(st + GSR_STAGES - 1);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group %0;" ::"n"(GSR_STAGES - 1) : "memory");
            __syncwarp();
            const float* base = ring + (st % GSR_STAGES) * STAGE;
            const float* wp = base + lane * GSR_PITCH;
            const float* xp = base + W_FLOATS + q * GSR_PITCH;
#pragma unroll
            for (int k = 0; k < GSR_CHUNK; k += 4) {
                const float4 w = *reinterpret_cast<const float4*>(wp + k);
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    const float4 x = *reinterpret_cast<const float4*>(xp + m * Q * GSR_PITCH + k);
                    acc[m] = fmaf(x.x, w.x, acc[m]);
                    acc[m] = fmaf(x.y, w.y, acc[m]);
                    acc[m] = fmaf(x.z, w.z, acc[m]);
                    acc[m] = fmaf(x.w, w.w, acc[m]);
                }
            }
            __syncwarp();                                              // the stage may be filled again
        }
        const int s = warp * Q + q;
#pragma unroll
        for (int m = 0; m < MR; ++m) red[(s * MR + m) * R + row] = acc[m];
        __syncthreads();
        const int here = min(per_round, slices - rd * per_round);
#pragma unroll
        for (int i = 0; i < OUTS; ++i) {
            const int o = threadIdx.x + i * blockDim.x;
            if (o < MR * R)
                for (int j = 0; j < here; ++j) total[i] += red[j * (MR * R) + o];
        }
        __syncthreads();
    }
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < OUTS; ++i) {
        const int o = threadIdx.x + i * blockDim.x;
        const int m = m0 + o / R, n = n0 + o % R;
        if (o < MR * R && m < M && n < N) Y[(long long)m * ldy + n] = total[i];
    }
}

// ---- float, 16-byte aligned operands, many rows -----------------------------------------------------------
// BM x 128 outputs a block, 2 BM threads of 8 x 8 each: rows ty * 4 (+ BM / 2), columns tx * 4 (+ 64).  Operands are
// kept k-major in shared memory (two buffers of 16 k); columns are
// multiplied in packed pairs (fma.rn.f32x2: each half is an IEEE fused multiply-add, as the scalar one; with scalar ones
// 1,000 x 9,216 x 1,024 took 515 us in place of 410).  The sums over whole slices are kept in shared memory, which leaves
// registers for two blocks per SM (128 rows with them in registers, one block: 473 us).  Bound by the FMA pipe where tiles fill
// the device: 46 of the 75 TFLOP/s at 1,000 x 9,216 x 1,024.  With one block of 64 rows an SM it was the loads, a k-step (0.5 us
// of arithmetic) ahead: a ring of four k-steps took 1,000 x 1,024 x 4,608 from 455 to 286 us.
#define GST_BN 128
#define GST_BK 16

__device__ __forceinline__ uint64_t gs_dup(float a) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ void gs_fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ void gs_add2(uint64_t& d, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }

template <int BM>
__global__ void __launch_bounds__(2 * BM, 2)
gemm_simt_tile_kernel(float* __restrict__ Y, const float* __restrict__ X, const float* __restrict__ W, int M, int N, int K,
                      long long ldx, long long ldw, long long ldy) {
    constexpr int THREADS = 2 * BM;
    constexpr int LW = 512 / THREADS;                                  // 16-byte pieces of W per thread and k-step (of X: 2)
    constexpr int ROWS = THREADS / 4;                                  // rows that one piece of every thread covers
    // RAW > 0: the operands come through a ring of RAW k-steps in shared memory, as they lie in memory (cp.async), and a thread
    // moves the pieces that it copied itself into the k-major buffers when their step is next: a lone block's loads then have
    // RAW k-steps to arrive instead of one.  RAW 0: through registers, one step ahead (two blocks an SM cover for each other).
    constexpr int RAW = BM == 64 ? 4 : 0;
    constexpr int PIECES = 2 + LW;                                     // 16-byte pieces of a k-step per thread
    extern __shared__ __align__(16) float gst_smem[];
    uint64_t* total = reinterpret_cast<uint64_t*>(gst_smem);           // [32][THREADS]: a thread's sums over whole slices
    float (*xs)[GST_BK][BM + 4] = reinterpret_cast<float (*)[GST_BK][BM + 4]>(gst_smem + 64 * THREADS);
    float (*ws)[GST_BK][GST_BN + 4] = reinterpret_cast<float (*)[GST_BK][GST_BN + 4]>(gst_smem + 64 * THREADS + 2 * GST_BK * (BM + 4));
    float4* raw = reinterpret_cast<float4*>(gst_smem + 64 * THREADS + 2 * GST_BK * (BM + 4 + GST_BN + 4));      // [RAW][PIECES][THREADS]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * GST_BN;
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    float4 xa[2], wa[LW];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto copy_w = [&](int step) {
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int r = n0 + lr + ROWS * i, k = step * GST_BK + lk;
            const bool ok = r < N && k < K;
            gs_cp16((uint32_t)__cvta_generic_to_shared(raw + ((step % (RAW ? RAW : 1)) * PIECES + 2 + i) * THREADS + tid),
                    ok ? W + (long long)r * ldw + k : W, ok);
        }
    };
    auto copy_x = [&](int step) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = m0 + lr + ROWS * i, k = step * GST_BK + lk;
            const bool ok = r < M && k < K;
            gs_cp16((uint32_t)__cvta_generic_to_shared(raw + ((step % (RAW ? RAW : 1)) * PIECES + i) * THREADS + tid),
                    ok ? X + (long long)r * ldx + k : X, ok);
        }
    };
    auto take = [&](int step) {                                        // this thread's pieces of a step that has arrived
#pragma unroll
        for (int i = 0; i < 2; ++i) xa[i] = raw[((step % (RAW ? RAW : 1)) * PIECES + i) * THREADS + tid];
#pragma unroll
        for (int i = 0; i < LW; ++i) wa[i] = raw[((step % (RAW ? RAW : 1)) * PIECES + 2 + i) * THREADS + tid];
    };
    auto fetch_w = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int r = n0 + lr + ROWS * i;
            wa[i] = (r < N && k0 + lk < K) ? __ldg(reinterpret_cast<const float4*>(W + (long long)r * ldw + k0 + lk)) : zero;
        }
    };
    auto fetch_x = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = m0 + lr + ROWS * i;
            xa[i] = (r < M && k0 + lk < K) ? *reinterpret_cast<const float4*>(X + (long long)r * ldx + k0 + lk) : zero;
        }
    };
    auto put = [&](int b) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float v[4] = {xa[i].x, xa[i].y, xa[i].z, xa[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) xs[b][lk + j][lr + ROWS * i] = v[j];
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const float v[4] = {wa[i].x, wa[i].y, wa[i].z, wa[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) ws[b][lk + j][lr + ROWS * i] = v[j];
        }
    };
    const int steps = (K + GST_BK - 1) / GST_BK;
    if (RAW) {
#pragma unroll
        for (int i = 0; i < RAW; ++i)
            if (i < steps) copy_w(i);
        pdl_wait();
#pragma unroll
        for (int i = 0; i < RAW; ++i) {
            if (i < steps) copy_x(i);
            asm volatile("cp.async.commit_group;" ::: "memory");       // the first group holds every weight requested above
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(RAW > 0 ? RAW - 1 : 0) : "memory");
        take(0);
    } else {
        fetch_w(0);
        pdl_wait();
        fetch_x(0);
    }
    put(0);
    __syncthreads();
    int b = 0;
    for (int k0 = 0; k0 < K; k0 += GST_BK, b ^= 1) {
        const bool more = k0 + GST_BK < K;
        if (RAW) {
            const int next = k0 / GST_BK + RAW;                        // into the place of the step in the buffers now
            if (next < steps) {
                copy_w(next);
                copy_x(next);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else if (more) {
            fetch_w(k0 + GST_BK);
            fetch_x(k0 + GST_BK);
        }
#pragma unroll
        for (int k = 0; k < GST_BK; ++k) {
            uint64_t w2[4];
            const ulonglong2 wl = *reinterpret_cast<const ulonglong2*>(&ws[b][k][tx * 4]);
            const ulonglong2 wh = *reinterpret_cast<const ulonglong2*>(&ws[b][k][64 + tx * 4]);
            w2[0] = wl.x; w2[1] = wl.y; w2[2] = wh.x; w2[3] = wh.y;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 x = *reinterpret_cast<const float4*>(&xs[b][k][(BM / 2) * h + ty * 4]);
                const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t x2 = gs_dup(xv[i]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) gs_fma2(acc[4 * h + i][j], x2, w2[j]);
                }
            }
        }
        if ((k0 + GST_BK) % GS_SLICE == 0 || !more) {
            // a slice ends: its sums join the slices before it (kept in shared memory, a column of it per thread); the
            // last slice's total stays in the registers
            const bool first = k0 < GS_SLICE;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint64_t* t = total + (i * 4 + j) * THREADS + tid;
                    if (!first) gs_add2(acc[i][j], *t);
                    if (more) {
                        *t = acc[i][j];
                        acc[i][j] = 0;
                    }
                }
        }
        if (more) {
            if (RAW) {
                asm volatile("cp.async.wait_group %0;" ::"n"(RAW > 0 ? RAW - 1 : 0) : "memory");
                take(k0 / GST_BK + 1);
            }
            put(b ^ 1);
        }
        __syncthreads();
    }
    pdl_trigger();
    const bool vec = (ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + (BM / 2) * (i / 4) + ty * 4 + (i & 3);
        if (m >= M) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = n0 + 64 * h + tx * 4;
            float v[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][2 * h]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[i][2 * h + 1]));
            float* dst = Y + (long long)m * ldy + n;
            if (vec && n + 3 < N) {
                *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n + j < N) dst[j] = v[j];
            }
        }
    }
}

template <int MR, int R>
static int launch_simt_rows(float* Y, const float* X, const float* W, int M, int N, int K, long long ldx, long long ldw,
                            long long ldy, cudaStream_t st) {
    constexpr int Q = 32 / R;
    constexpr int STAGE = (32 + MR * Q) * GSR_PITCH;
    constexpr int PER_WARP = (GSR_STAGES * STAGE + Q * MR * R) * 4;    // 28 to 39 KB: the ring and the round's sums
    constexpr int MAX_WARPS = 232448 / PER_WARP < 8 ? 232448 / PER_WARP : 8;
    const int slices = (K + GS_SLICE - 1) / GS_SLICE;
    const int rounds = (slices + MAX_WARPS * Q - 1) / (MAX_WARPS * Q);
    const int warps = (slices + rounds * Q - 1) / (rounds * Q);
    const size_t most = (size_t)MAX_WARPS * PER_WARP;
    const size_t smem = (size_t)warps * PER_WARP;
    auto kernel = gemm_simt_rows_kernel<MR, R>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) {
            cudaGetLastError();
            cm_set_error("gemm_simt: %zu bytes of shared memory refused", most);
            return CM_ERR_LAUNCH;
        }
        configured = true;
    }
    cm_launch(kernel, dim3((N + R - 1) / R, (M + MR - 1) / MR), warps * 32, smem, st, Y, X, W, M, N, K, ldx, ldw, ldy);
    CM_CHECK_LAUNCH();
    return CM_OK;
}

template <int BM>
static int launch_simt_tile(float* Y, const float* X, const float* W, int M, int N, int K, long long ldx, long long ldw,
                            long long ldy, cudaStream_t st) {
    constexpr size_t smem = (64 * 2 * BM + 2 * GST_BK * (BM + 4 + GST_BN + 4) + (BM == 64 ? 4 * GST_BK * (BM + GST_BN) : 0)) * 4;
    auto kernel = gemm_simt_tile_kernel<BM>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            cm_set_error("gemm_simt: %zu bytes of shared memory refused", smem);
            return CM_ERR_LAUNCH;
        }
        configured = true;
    }
    cm_launch(kernel, dim3((N + GST_BN - 1) / GST_BN, (M + BM - 1) / BM), 2 * BM, smem, st, Y, X, W, M, N, K, ldx, ldw, ldy);
    CM_CHECK_LAUNCH();
    return CM_OK;
}
// Which kernel (all give the same bits).  Measured on B200, us (the kernel before: 64 x 64 tiles, 4 x 4 outputs a thread,
// one k-step's loads at a time):
//  - up to 4 rows: eight rows of W a warp where there are few of them, so that enough warps stream (4 x 1,024 x 4,608: 7.9,
//    with 16 rows a warp 9.3, before 527), else 16 (4 x 9,216 x 1,024: 13.1 / 11.4, before 119);
//  - up to 8 rows: one pass of eight (8 x 9,216 x 1,024 14.0), or two of four for a narrow W (8 x 1,024 x 1,024 3.3 / 3.9);
//  - more: whichever of the passes of eight rows and the two tiles is estimated faster.  A pass costs its arithmetic at
//    15.5 TFLOP/s (128 x 1,024 x 4,608: 87 us, before 510).  Two tiles of either height fit an SM: a round of them costs 0.110 us
//    (64 rows) or 0.205 us (128) per k, and a last round with at most one tile an SM 0.062 or 0.123: 500 x 3,072 x 1,024 115 us
//    with 64 rows (before 178), 1,000 x 1,024 x 4,608 286 (before 546), 1,000 x 9,216 x 1,024 410 with 128 rows (before 897),
//    1,000 x 16,384 x 2,048 1,427 (before 3,260).
static int launch_simt_float(float* Y, const float* X, const float* W, int M, int N, int K, long long ldx, long long ldw,
                             long long ldy, cudaStream_t st) {
    if (M <= 4 && N < 2048) return launch_simt_rows<4, 8>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (M <= 4 || (M <= 8 && N <= 2048)) return launch_simt_rows<4, 16>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (M <= 16) return launch_simt_rows<8, 16>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    static int sm_count = 0;
    if (!sm_count) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (sm_count <= 0) sm_count = 1;
    }
    const long long cols = (N + GST_BN - 1) / GST_BN, round = 2LL * sm_count;
    auto tiles_us = [&](long long tiles, double full, double half) {
        const long long left = tiles % round;
        return K * (tiles / round * full + (left == 0 ? 0.0 : left <= sm_count ? half : full));
    };
    const double rows = 2.0 * ((M + 7) / 8 * 8) * N * K / 15.5e6;
    const double tile64 = tiles_us(cols * ((M + 63) / 64), 0.110, 0.062), tile128 = tiles_us(cols * ((M + 127) / 128), 0.205, 0.123);
    // (a grid has at most 65,535 rows of blocks, which ends the passes of eight at half a million rows)
    if (rows <= tile64 && rows <= tile128 && M <= 8 * 65535) return launch_simt_rows<8, 16>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (tile64 <= tile128 && M <= 64 * 65535) return launch_simt_tile<64>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    return launch_simt_tile<128>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
}

template <typename TX, typename TW, typename TY>
static int launch_simt(void* Y, const void* X, const void* W, int M, int N, int K, long long ldx,
                       long long ldw, long long ldy, cudaStream_t st) {
    dim3 grid((N + GS_BN - 1) / GS_BN, (M + GS_BM - 1) / GS_BM);
    cm_launch(gemm_simt_kernel<TX, TW, TY>, grid, 256, 0, st, (TY*)Y, (const TX*)X, (const TW*)W, M, N, K,
                                                       ldx, ldw, ldy);
    CM_CHECK_LAUNCH();
    return CM_OK;
}

// dtx / dtw / dty: DT_F32 or DT_BF16 of X, W and Y.  Supported: all-float; bf16 X and W with
// bf16 or float Y; bf16 X with float W (a matrix that the file stores in 32 bits) and bf16 or
// float Y.
extern "C" int cm_gemm_simt(int dtx, int dtw, int dty, void* Y, const void* X, const void* W, int M,
                            int N, int K, long long ldx, long long ldw, long long ldy,
                            cudaStream_t st) {
    if (M <= 0 || N <= 0) return CM_OK;
    if (K <= 0) CM_REFUSE("gemm: inner size %d", K);
    if (dtx == DT_F32 && dtw == DT_F32 && dty == DT_F32 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 &&
        ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15) == 0)
        return launch_simt_float((float*)Y, (const float*)X, (const float*)W, M, N, K, ldx, ldw, ldy, st);
    if (dtx == DT_F32 && dtw == DT_F32 && dty == DT_F32)
        return launch_simt<float, float, float>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (dtx == DT_BF16 && dtw == DT_BF16 && dty == DT_BF16)
        return launch_simt<bf16, bf16, bf16>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (dtx == DT_BF16 && dtw == DT_BF16 && dty == DT_F32)
        return launch_simt<bf16, bf16, float>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (dtx == DT_BF16 && dtw == DT_F32 && dty == DT_BF16)
        return launch_simt<bf16, float, bf16>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    if (dtx == DT_BF16 && dtw == DT_F32 && dty == DT_F32)
        return launch_simt<bf16, float, float>(Y, X, W, M, N, K, ldx, ldw, ldy, st);
    return CM_ERR_DTYPE;
}
