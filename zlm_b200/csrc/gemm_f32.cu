// True 32-bit matrix product Y[T,N] = X[T,K] . W[N,K]^T on the FFMA pipe: no
// tensor cores, no reduced-precision mode.  Every output element is one chain of
// FMAs over k = 0..K-1 in ascending order, so a token's result is bit-identical
// whatever the batch around it and however the step was cut.
// out_i = sum_j W[i,j] x_j with fp32 accumulation, row-major [out][in] weights
// (src/kernels/linear/matvec/kernels/float.zig:69-80).
#include "common.cuh"

#define F32_BM 64
#define F32_BN 64
#define F32_BK 32
#define F32_LD (F32_BK + 4)      // rows 16 bytes apart modulo the banks
#define F32_STAGES 3
#define F32_THREADS 128

// A block: 64 tokens x 64 outputs; a thread 8 tokens x 4 outputs.  Both operands stand in shared memory as they are in memory,
// 32 columns a row, two stages on their way (asynchronous copies, zeros beyond the edges) while one is multiplied; a thread
// reads four columns of a row at a time: 12 reads of 16 bytes for 128 FMAs.
// Bound by those reads (a warp's takes the shared-memory pipe 4 cycles, four warps' FMAs one) and, with few blocks an SM, by
// the latency of a step.  509 x 2,048 by 3,072 x 2,048 and by 2,048 x 2,048: 241 and 192 us with 4 x 4 outputs a thread,
// scalar loads and one stage, 174 and 126 us so.  Tried: operands transposed through registers one step ahead, packed FMAs
// (253 and 182 us: a step of 16 columns waits 1,400 of its 1,900 cycles for memory); 8 x 8 outputs on 64 threads, which halves
// the reads an FMA (213 and 208: one warp or two a scheduler do not cover their own latencies).
// mode 0: Y = acc (fp32); mode 1: Y += acc (fp32 residual stream).  Rows of 16-byte pieces: the next kernel takes the others.
template <int MODE>
__global__ void __launch_bounds__(F32_THREADS)
gemm_f32_kernel(float* __restrict__ Y, const float* __restrict__ X, const float* __restrict__ W,
                int T, int N, int K, int ldy) {
    extern __shared__ __align__(16) float f32_smem[];       // [F32_STAGES][F32_BM + F32_BN][F32_LD]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * F32_BM, n0 = blockIdx.x * F32_BN;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const int steps = (K + F32_BK - 1) / F32_BK;
    auto stage = [&](int step) {
        if (step < steps) {
            float* base = f32_smem + (size_t)(step % F32_STAGES) * (F32_BM + F32_BN) * F32_LD;
#pragma unroll
            for (int x = tid; x < (F32_BM + F32_BN) * (F32_BK / 4); x += F32_THREADS) {
                const int row = x / (F32_BK / 4), k = step * F32_BK + (x % (F32_BK / 4)) * 4;
                const bool w = row >= F32_BM;
                const int g = w ? n0 + row - F32_BM : m0 + row;
                const float* src = (w ? W : X) + (size_t)g * K + k;
                const bool in = g < (w ? N : T) && k < K && ZLM_CHK(src, 16);
                const unsigned dst = (unsigned)__cvta_generic_to_shared(base + row * F32_LD + (x % (F32_BK / 4)) * 4);
                const int bytes = in ? 16 : 0;                 // (the rest of the copy is zeros)
                if (!in) src = X;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
#pragma unroll
    for (int x = 0; x < F32_STAGES - 1; ++x) stage(x);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(F32_STAGES - 2) : "memory");
        __syncthreads();
        stage(step + F32_STAGES - 1);             // (into the stage that every thread has read before this barrier)
        const float* xs = f32_smem + (size_t)(step % F32_STAGES) * (F32_BM + F32_BN) * F32_LD + ty * F32_LD;
        const float* ws = f32_smem + (size_t)(step % F32_STAGES) * (F32_BM + F32_BN) * F32_LD + (F32_BM + tx) * F32_LD;
#pragma unroll
        for (int kk = 0; kk < F32_BK; kk += 4) {
            float4 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = *(const float4*)(ws + 16 * j * F32_LD + kk);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 x = *(const float4*)(xs + 8 * i * F32_LD + kk);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    acc[i][j] = fmaf(x.w, w[j].w, fmaf(x.z, w[j].z, fmaf(x.y, w[j].y, fmaf(x.x, w[j].x, acc[i][j]))));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gm = m0 + ty + 8 * i;
        if (gm >= T) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx + 16 * j;
            if (gn >= N || !ZLM_CHK(Y + (size_t)gm * ldy + gn, 4)) continue;
            float* y = Y + (size_t)gm * ldy + gn;
            if (MODE == 0) *y = acc[i][j];
            else *y = *y + acc[i][j];
        }
    }
}

// The same for rows whose columns come one at a time (K no multiple of four, or an operand off its 16 bytes): 4 x 4 outputs a
// thread, operands through registers and transposed, one stage.  Copies of 4 bytes are as many as the columns, and issuing
// them costs more than they hide: 1 and 2,048 tokens of 2,049 columns by 2,048 outputs take 98 and 536 us here, 110 and 622
// with the stages above.  The sums' order is the same, and so are the bits.
#define F32P_BK 16
template <int MODE>
__global__ void __launch_bounds__(256)
gemm_f32_plain_kernel(float* __restrict__ Y, const float* __restrict__ X, const float* __restrict__ W, int T, int N, int K, int ldy) {
    __shared__ float xs[F32P_BK][F32_BM + 4], ws[F32P_BK][F32_BN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, m0 = blockIdx.y * F32_BM, n0 = blockIdx.x * F32_BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += F32P_BK) {
        const int k = k0 + tx;                       // a thread loads column k of rows ty, ty + 16, ...
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int r = ty + 16 * p;
            const float *x = X + (size_t)(m0 + r) * K + k, *w = W + (size_t)(n0 + r) * K + k;
            xs[tx][r] = (m0 + r < T && k < K && ZLM_CHK(x, 4)) ? *x : 0.f;
            ws[tx][r] = (n0 + r < N && k < K && ZLM_CHK(w, 4)) ? *w : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < F32P_BK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { a[i] = xs[kk][ty * 4 + i]; b[i] = ws[kk][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gm = m0 + ty * 4 + i, gn = n0 + tx * 4 + j;
            float* y = Y + (size_t)gm * ldy + gn;
            if (gm < T && gn < N && ZLM_CHK(y, 4)) *y = MODE == 0 ? acc[i][j] : *y + acc[i][j];
        }
}

template <int MODE>
static int launch_f32(dim3 grid, cudaStream_t st, bool vec, float* Y, const float* X, const float* W, int T, int N, int K, int ldy) {
    if (!vec) {
        zlm_count_launch();
        gemm_f32_plain_kernel<MODE><<<grid, 256, 0, st>>>(Y, X, W, T, N, K, ldy);
        return zlm_check_launch("gemm_f32");
    }
    const size_t smem = (size_t)F32_STAGES * (F32_BM + F32_BN) * F32_LD * sizeof(float);
    static bool attr_set_dev[64] = {};
    bool& attr_set = attr_set_dev[zlm_device_index()];
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            zlm_set_error("gemm_f32: cannot reserve shared memory: %s", cudaGetErrorString(e));
            return ZLM_ERR_CUDA;
        }
        attr_set = true;
    }
    zlm_count_launch();
    gemm_f32_kernel<MODE><<<grid, F32_THREADS, smem, st>>>(Y, X, W, T, N, K, ldy);
    return zlm_check_launch("gemm_f32");
}

extern "C" int zlm_gemm_f32(float* Y, const float* X, const float* W, int T, int N, int K, int ldy,
                            int accumulate, cudaStream_t st) {
    if (T == 0 || N == 0) return ZLM_OK;
    ZLM_REQUIRE(T > 0 && N > 0 && K > 0 && ldy >= N, "gemm_f32: bad sizes T=%d N=%d K=%d ldy=%d", T, N, K, ldy);
    dim3 grid((N + F32_BN - 1) / F32_BN, (T + F32_BM - 1) / F32_BM);
    ZLM_REQUIRE(grid.y <= 65535, "gemm_f32: more than %d tokens in one step", 65535 * F32_BM);
    const bool vec = K % 4 == 0 && (uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0;
    return accumulate ? launch_f32<1>(grid, st, vec, Y, X, W, T, N, K, ldy) : launch_f32<0>(grid, st, vec, Y, X, W, T, N, K, ldy);
}

ZLM_TRANSLATION_UNIT(gemm_f32)
