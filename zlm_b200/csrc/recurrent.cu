// Recurrent mixers whose state is carried from token to token in fp32:
//
//   * a real-gated linear recurrent unit (one number of state per channel) behind a short causal convolution:
//       u = conv(x + b_x) + b_c                      x, y: two projections of the mixer's input
//       r = sigmoid(A_r[b] u_b + c_r),  i = sigmoid(A_i[b] u_b + c_i)      block-diagonal: u in `blocks` equal parts
//       log a = -c * r * softplus(lam),  S_t = a S_(t-1) + sqrt(1 - a^2) * i * u,   out = S_t * gelu_tanh(y + b_y)
//   * linear attention with a decay per key channel and token (gated linear attention) or per head:
//       S_t = diag(alpha_t) S_(t-1) + k_t v_t^T,  o_t = S_t^T q_t            S [dim][v_dim] per head
//     and the kernel that makes alpha from a low-rank projection: alpha = sigmoid(W2 lo + b)^(1/tau).
//
// Everything after the projections (convolution sums, gates, decays and their logarithms, softplus, exponentials,
// the state, the read-out) is fp32 in both element types.  A sequence's state is [slots][...] fp32 and is read at
// a step's start and written at its end; nothing is special about a sequence's first token: its state is zero.
#include "common.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define RC_MAX_TAPS 8

__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float gelu_tanh_f(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

// ---------------------------------------------------------------------------- convolution of the x branch
// u[t][c] = sum_j w[c][j] * (x_(t-taps+1+j)[c] + bx[c]) + cb[c]; x of the step's earlier tokens from `proj`, of earlier
// steps from the state's rows 1 .. taps-1 (row taps-1 the newest; they hold x + bx), zeros before the start.  u16, if
// given, receives u in the element type as well (the operand of the gates' product on the tensor cores).
template <typename TA>
__global__ void __launch_bounds__(256)
rglru_conv_kernel(float* __restrict__ u, TA* __restrict__ u16, const TA* __restrict__ proj, int proj_stride, int x_off,
                  const TA* __restrict__ bx, const TA* __restrict__ conv_w, const TA* __restrict__ cb,
                  const float* __restrict__ state, const int* __restrict__ token_pos, const int* __restrict__ token_slot,
                  const int* __restrict__ token_seq, const int* __restrict__ seq_start, const int* __restrict__ cu_seqlens,
                  int W, int taps) {
    pdl_trigger();
    const int t = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
    pdl_wait();
    if (c >= W) return;
    if (!ZLM_CHK(token_pos + t, 4) || !ZLM_CHK(token_slot + t, 4) || !ZLM_CHK(token_seq + t, 4)) return;
    const int pos = token_pos[t], slot = token_slot[t], r = token_seq[t];
    if (!ZLM_CHK(seq_start + r, 4) || !ZLM_CHK(cu_seqlens + r, 4)) return;
    const int i = pos - seq_start[r], row0 = cu_seqlens[r];
    const float b = bx ? to_f32(bx[c]) : 0.f;
    float a = cb ? to_f32(cb[c]) : 0.f;
    for (int j = 0; j < taps; ++j) {
        const int s = i - (taps - 1) + j;
        if (pos - (taps - 1) + j < 0) continue;
        float x;
        if (s >= 0) {
            const TA* p = proj + (size_t)(row0 + s) * proj_stride + x_off + c;
            if (!ZLM_CHK(p, sizeof(TA))) continue;
            x = to_f32(*p) + b;
        } else {
            const float* p = state + ((size_t)slot * taps + (taps + s)) * W + c;
            if (!ZLM_CHK(p, 4)) continue;
            x = *p;
        }
        a = fmaf(to_f32(conv_w[(size_t)c * taps + j]), x, a);
    }
    if (ZLM_CHK(u + (size_t)t * W + c, 4)) u[(size_t)t * W + c] = a;
    if (u16 && ZLM_CHK(u16 + (size_t)t * W + c, sizeof(TA))) u16[(size_t)t * W + c] = from_f32<TA>(a);
}

// ---------------------------------------------------------------------------- block-diagonal gate logits
// z [T][blocks][2][bs] fp32: z[t][b][g][o] = sum_i A_g[b][o][i] u[t][b*bs + i], g = 0 (recurrence gate), 1 (input gate);
// the gates' biases are added where z is read.  (The same layout as the product u_b [T, bs] x [A_r[b] ; A_i[b]]^T
// leaves, block by block, when the tensor cores compute it.)
// A block: 16 tokens x 64 outputs of one diagonal block, both gates; u and the weights in tiles of 32 inputs in shared
// memory; fp32 multiply-adds in a fixed order.
#define RG_TT 16
#define RG_OT 64
#define RG_KT 32
template <typename TA>
__global__ void __launch_bounds__(RG_OT * 4)
rglru_gates_kernel(float* __restrict__ z, const float* __restrict__ u, const TA* __restrict__ Ar,
                   const TA* __restrict__ Ai, int T, int W, int bs) {
    __shared__ float su[RG_TT][RG_KT + 1];
    __shared__ float sw[2][RG_OT][RG_KT + 1];
    pdl_trigger();
    const int t0 = blockIdx.x * RG_TT, b = blockIdx.z, o0 = blockIdx.y * RG_OT;
    const int tid = threadIdx.x, ol = tid % RG_OT, tq = tid / RG_OT;          // the thread's output, and its quarter of the tokens
    pdl_wait();
    float acc[2][RG_TT / 4];
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int j = 0; j < RG_TT / 4; ++j) acc[g][j] = 0.f;
    for (int k0 = 0; k0 < bs; k0 += RG_KT) {
        for (int x = tid; x < RG_TT * RG_KT; x += RG_OT * 4) {
            const int tt = x / RG_KT, kk = x % RG_KT;
            const float* p = u + (size_t)(t0 + tt) * W + b * bs + k0 + kk;
            su[tt][kk] = (t0 + tt < T && k0 + kk < bs && ZLM_CHK(p, 4)) ? *p : 0.f;
        }
        for (int x = tid; x < 2 * RG_OT * RG_KT; x += RG_OT * 4) {
            const int g = x / (RG_OT * RG_KT), oo = (x / RG_KT) % RG_OT, kk = x % RG_KT;
            const TA* p = (g ? Ai : Ar) + ((size_t)b * bs + o0 + oo) * bs + k0 + kk;
            sw[g][oo][kk] = (o0 + oo < bs && k0 + kk < bs && ZLM_CHK(p, sizeof(TA))) ? to_f32(*p) : 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < RG_KT; ++kk) {
            const float wr = sw[0][ol][kk], wi = sw[1][ol][kk];
#pragma unroll
            for (int j = 0; j < RG_TT / 4; ++j) {
                const float x = su[tq * (RG_TT / 4) + j][kk];
                acc[0][j] = fmaf(wr, x, acc[0][j]);
                acc[1][j] = fmaf(wi, x, acc[1][j]);
            }
        }
        __syncthreads();
    }
    if (o0 + ol >= bs) return;
#pragma unroll
    for (int j = 0; j < RG_TT / 4; ++j) {
        const int t = t0 + tq * (RG_TT / 4) + j;
        if (t >= T) continue;
        float* zp = z + ((size_t)t * 2 * W) + (size_t)b * 2 * bs + o0 + ol;
        if (ZLM_CHK(zp, 4)) zp[0] = acc[0][j];
        if (ZLM_CHK(zp + bs, 4)) zp[bs] = acc[1][j];
    }
}

// The same for steps of up to 16 tokens: a warp per output channel reads its two rows of the gates' matrices once
// (lanes over the inputs), every token's sums in registers; the lanes' parts meet in a butterfly.
#define RG_FEW 16
// eight neighbouring elements as floats (16 bytes of bf16, 32 of fp32; the caller has checked the alignment)
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f) {
    const uint4 u = *(const uint4*)p;
    f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
    f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
    f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
}
__device__ __forceinline__ void load8(const float* p, float* f) {
    const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// VEC 8: a lane reads eight neighbouring inputs at a time (block sizes that are multiples of 8); VEC 1: one
template <typename TA, int VEC>
__global__ void __launch_bounds__(256)
rglru_gates_few_kernel(float* __restrict__ z, const float* __restrict__ u, const TA* __restrict__ Ar,
                       const TA* __restrict__ Ai, int T, int W, int bs) {
    pdl_trigger();
    const int lane = threadIdx.x & 31, c = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (c >= W) return;
    const int b = c / bs, o = c - b * bs;
    float acc[2][RG_FEW];
#pragma unroll
    for (int t = 0; t < RG_FEW; ++t) acc[0][t] = acc[1][t] = 0.f;
    pdl_wait();
    for (int i = lane * VEC; i < bs; i += 32 * VEC) {
        const TA* pr = Ar + (size_t)c * bs + i;
        const TA* pi = Ai + (size_t)c * bs + i;
        if (!ZLM_CHK(pr, VEC * sizeof(TA)) || !ZLM_CHK(pi, VEC * sizeof(TA))) continue;
        float wr[VEC], wi[VEC];
        if (VEC == 8) { load8(pr, wr); load8(pi, wi); } else { wr[0] = to_f32(*pr); wi[0] = to_f32(*pi); }
#pragma unroll
        for (int t = 0; t < RG_FEW; ++t) {
            if (t >= T) break;
            const float* up = u + (size_t)t * W + b * bs + i;
            if (!ZLM_CHK(up, VEC * 4)) continue;
            float x[VEC];
            if (VEC == 8) load8(up, x); else x[0] = *up;
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                acc[0][t] = fmaf(wr[e], x[e], acc[0][t]);
                acc[1][t] = fmaf(wi[e], x[e], acc[1][t]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < RG_FEW; ++t) {
        if (t >= T) break;
        const float sr = warp_sum(acc[0][t]), si = warp_sum(acc[1][t]);
        float* zp = z + ((size_t)t * 2 * W) + (size_t)b * 2 * bs + o;
        if (lane == 0 && ZLM_CHK(zp, 4)) zp[0] = sr;
        if (lane == 0 && ZLM_CHK(zp + bs, 4)) zp[bs] = si;
    }
}

// a token's decay and input: a = exp(-c r softplus(lam)), b = sqrt(1 - a^2) i u, from the gates' logits
__device__ __forceinline__ void rglru_ab(float zr, float zi, float u, float sl, float& a, float& b) {
    const float log_a = -sigmoid_f(zr) * sl;
    a = expf(log_a);
    b = sqrtf(fmaxf(-expm1f(2.0f * log_a), 0.f)) * sigmoid_f(zi) * u;           // sqrt(1 - a^2) without the cancellation
}

// the convolution's newest inputs after a step of n tokens: row m holds the input (taps - m) tokens back from the next
template <typename TA>
__device__ __forceinline__ void rglru_keep_inputs(float* sp, const TA* proj, int proj_stride, int x_off, int c, int row0, int n,
                                                  int W, int taps, float xb) {
    float keep[RC_MAX_TAPS];
    for (int m = 1; m < taps; ++m) {
        const int s = n - taps + m;
        if (s >= 0) {
            const TA* p = proj + (size_t)(row0 + s) * proj_stride + x_off + c;
            keep[m] = ZLM_CHK(p, sizeof(TA)) ? to_f32(*p) + xb : 0.f;
        } else {
            keep[m] = sp[(size_t)(taps + s) * W];
        }
    }
    for (int m = 1; m < taps; ++m) sp[(size_t)m * W] = keep[m];
}

// ---------------------------------------------------------------------------- the recurrence and the y branch
// Short steps: a thread owns one channel of one sequence and walks the step's tokens (eight tokens' loads in flight),
// then leaves the state: row 0 the recurrence's S, rows 1 .. taps-1 the newest x + bx.
#define RS_AHEAD 8
#define PIECE_AHEAD 16          // the pieces' walks: a piece is two such rounds
template <typename TA>
__global__ void __launch_bounds__(128)
rglru_scan_kernel(TA* __restrict__ out, int out_stride, const float* __restrict__ u, const float* __restrict__ z,
                  const TA* __restrict__ proj, int proj_stride, int x_off, int y_off, const TA* __restrict__ bx,
                  const TA* __restrict__ by, const TA* __restrict__ cr, const TA* __restrict__ ci, const TA* __restrict__ lam,
                  float c_decay, float* __restrict__ state, const int* __restrict__ seq_slot,
                  const int* __restrict__ cu_seqlens, int W, int bs, int taps, float out_scale) {
    pdl_trigger();
    const int r = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
    pdl_wait();
    if (c >= W || !ZLM_CHK(seq_slot + r, 4) || !ZLM_CHK(cu_seqlens + r, 8)) return;
    const int slot = seq_slot[r], row0 = cu_seqlens[r], n = cu_seqlens[r + 1] - row0;
    float* sp = state + (size_t)slot * taps * W + c;
    if (!ZLM_CHK(sp, 4)) return;
    float S = *sp;
    const float sl = softplus_f(to_f32(lam[c])) * c_decay;
    const float yb = by ? to_f32(by[c]) : 0.f, rb = cr ? to_f32(cr[c]) : 0.f, ib = ci ? to_f32(ci[c]) : 0.f;
    const size_t zc = (size_t)(c / bs) * 2 * bs + (c % bs);
    for (int s0 = 0; s0 < n; s0 += RS_AHEAD) {
        float vu[RS_AHEAD], vr[RS_AHEAD], vi[RS_AHEAD], vy[RS_AHEAD];
#pragma unroll
        for (int j = 0; j < RS_AHEAD; ++j) {
            const size_t row = (size_t)(row0 + s0 + j);
            const bool ok = s0 + j < n && ZLM_CHK(u + row * W + c, 4) && ZLM_CHK(z + row * 2 * W + zc, 4) &&
                            ZLM_CHK(z + row * 2 * W + zc + bs, 4) && ZLM_CHK(proj + row * proj_stride + y_off + c, sizeof(TA));
            vu[j] = ok ? u[row * W + c] : 0.f;
            vr[j] = ok ? z[row * 2 * W + zc] : 0.f;
            vi[j] = ok ? z[row * 2 * W + zc + bs] : 0.f;
            vy[j] = ok ? to_f32(proj[row * proj_stride + y_off + c]) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < RS_AHEAD; ++j) {
            if (s0 + j >= n) break;
            float a, b;
            rglru_ab(vr[j] + rb, vi[j] + ib, vu[j], sl, a, b);
            S = fmaf(a, S, b);
            TA* dst = out + (size_t)(row0 + s0 + j) * out_stride + c;
            if (ZLM_CHK(dst, sizeof(TA))) *dst = from_f32<TA>(S * gelu_tanh_f(vy[j] + yb) * out_scale);
        }
    }
    *sp = S;
    rglru_keep_inputs<TA>(sp, proj, proj_stride, x_off, c, row0, n, W, taps, bx ? to_f32(bx[c]) : 0.f);
}

// Long steps run in pieces of L tokens side by side.  First pass: a thread owns one channel of one piece, turns the
// gates' logits of its tokens into (a, b) in place (a where the recurrence gate's logit stood, b where the input
// gate's stood) and leaves what the piece does to a state: S_out = PA * S_in + PB.
__global__ void __launch_bounds__(128)
rglru_piece_ab_kernel(float* __restrict__ z, const float* __restrict__ u, const void* __restrict__ cr, const void* __restrict__ ci,
                      const void* __restrict__ lam, int dtype, float c_decay, float* __restrict__ PA, float* __restrict__ PB,
                      const int* __restrict__ cu_seqlens, int W, int bs, int maxp, int L) {
    pdl_trigger();
    const int r = blockIdx.x / maxp, p = blockIdx.x % maxp, c = blockIdx.y * blockDim.x + threadIdx.x;
    pdl_wait();
    if (c >= W || !ZLM_CHK(cu_seqlens + r, 8)) return;
    const int row0 = cu_seqlens[r], n = cu_seqlens[r + 1] - row0;
    const int lo = p * L, hi = min(n, lo + L);
    if (lo >= hi) return;
    const VecW vr{cr, dtype}, vi{ci, dtype}, vl{lam, dtype};
    const float sl = softplus_f(vl[c]) * c_decay;
    const float rb = cr ? vr[c] : 0.f, ib = ci ? vi[c] : 0.f;
    const size_t zc = (size_t)(c / bs) * 2 * bs + (c % bs);
    float A = 1.f, B = 0.f;
    for (int s0 = lo; s0 < hi; s0 += PIECE_AHEAD) {
        float fu[PIECE_AHEAD], fr[PIECE_AHEAD], fi[PIECE_AHEAD];
#pragma unroll
        for (int j = 0; j < PIECE_AHEAD; ++j) {
            const size_t row = (size_t)(row0 + s0 + j);
            const bool ok = s0 + j < hi && ZLM_CHK(u + row * W + c, 4) && ZLM_CHK(z + row * 2 * W + zc, 4) && ZLM_CHK(z + row * 2 * W + zc + bs, 4);
            fu[j] = ok ? u[row * W + c] : 0.f;
            fr[j] = ok ? z[row * 2 * W + zc] : 0.f;
            fi[j] = ok ? z[row * 2 * W + zc + bs] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < PIECE_AHEAD; ++j) {
            if (s0 + j >= hi) break;
            float a, b;
            rglru_ab(fr[j] + rb, fi[j] + ib, fu[j], sl, a, b);
            const size_t row = (size_t)(row0 + s0 + j);
            z[row * 2 * W + zc] = a;
            z[row * 2 * W + zc + bs] = b;
            A *= a;
            B = fmaf(a, B, b);
        }
    }
    const size_t at = ((size_t)r * maxp + p) * W + c;
    if (ZLM_CHK(PA + at, 4)) PA[at] = A;
    if (ZLM_CHK(PB + at, 4)) PB[at] = B;
}

// The pieces' states in order: PA[piece] becomes the state the piece starts from; the sequence's state is left.
template <typename TA>
__global__ void __launch_bounds__(128)
rglru_chain_kernel(float* __restrict__ PA, const float* __restrict__ PB, float* __restrict__ state, const TA* __restrict__ proj,
                   int proj_stride, int x_off, const TA* __restrict__ bx, const int* __restrict__ seq_slot,
                   const int* __restrict__ cu_seqlens, int W, int taps, int maxp, int L) {
    pdl_trigger();
    const int r = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
    pdl_wait();
    if (c >= W || !ZLM_CHK(seq_slot + r, 4) || !ZLM_CHK(cu_seqlens + r, 8)) return;
    const int slot = seq_slot[r], row0 = cu_seqlens[r], n = cu_seqlens[r + 1] - row0;
    float* sp = state + (size_t)slot * taps * W + c;
    if (!ZLM_CHK(sp, 4)) return;
    float S = *sp;
    const int np = (n + L - 1) / L;
    for (int p0 = 0; p0 < np; p0 += RS_AHEAD) {
        float A[RS_AHEAD], B[RS_AHEAD];
#pragma unroll
        for (int j = 0; j < RS_AHEAD; ++j) {
            const size_t at = ((size_t)r * maxp + p0 + j) * W + c;
            const bool ok = p0 + j < np && ZLM_CHK(PA + at, 4) && ZLM_CHK(PB + at, 4);
            A[j] = ok ? PA[at] : 1.f;
            B[j] = ok ? PB[at] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < RS_AHEAD; ++j) {
            if (p0 + j >= np) break;
            const size_t at = ((size_t)r * maxp + p0 + j) * W + c;
            if (ZLM_CHK(PA + at, 4)) PA[at] = S;
            S = fmaf(A[j], S, B[j]);
        }
    }
    *sp = S;
    rglru_keep_inputs<TA>(sp, proj, proj_stride, x_off, c, row0, n, W, taps, bx ? to_f32(bx[c]) : 0.f);
}

// Second pass: every piece walks its tokens again from the state it starts from.
template <typename TA>
__global__ void __launch_bounds__(128)
rglru_piece_out_kernel(TA* __restrict__ out, int out_stride, const float* __restrict__ z, const float* __restrict__ S0,
                       const TA* __restrict__ proj, int proj_stride, int y_off, const TA* __restrict__ by,
                       const int* __restrict__ cu_seqlens, int W, int bs, int maxp, int L, float out_scale) {
    pdl_trigger();
    const int r = blockIdx.x / maxp, p = blockIdx.x % maxp, c = blockIdx.y * blockDim.x + threadIdx.x;
    pdl_wait();
    if (c >= W || !ZLM_CHK(cu_seqlens + r, 8)) return;
    const int row0 = cu_seqlens[r], n = cu_seqlens[r + 1] - row0;
    const int lo = p * L, hi = min(n, lo + L);
    if (lo >= hi) return;
    const size_t at = ((size_t)r * maxp + p) * W + c;
    float S = ZLM_CHK(S0 + at, 4) ? S0[at] : 0.f;
    const float yb = by ? to_f32(by[c]) : 0.f;
    const size_t zc = (size_t)(c / bs) * 2 * bs + (c % bs);
    for (int s0 = lo; s0 < hi; s0 += PIECE_AHEAD) {
        float fa[PIECE_AHEAD], fb[PIECE_AHEAD], fy[PIECE_AHEAD];
#pragma unroll
        for (int j = 0; j < PIECE_AHEAD; ++j) {
            const size_t row = (size_t)(row0 + s0 + j);
            const bool ok = s0 + j < hi && ZLM_CHK(z + row * 2 * W + zc, 4) && ZLM_CHK(z + row * 2 * W + zc + bs, 4) &&
                            ZLM_CHK(proj + row * proj_stride + y_off + c, sizeof(TA));
            fa[j] = ok ? z[row * 2 * W + zc] : 0.f;
            fb[j] = ok ? z[row * 2 * W + zc + bs] : 0.f;
            fy[j] = ok ? to_f32(proj[row * proj_stride + y_off + c]) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < PIECE_AHEAD; ++j) {
            if (s0 + j >= hi) break;
            S = fmaf(fa[j], S, fb[j]);
            TA* dst = out + (size_t)(row0 + s0 + j) * out_stride + c;
            if (ZLM_CHK(dst, sizeof(TA))) *dst = from_f32<TA>(S * gelu_tanh_f(fy[j] + yb) * out_scale);
        }
    }
}

#define RGLRU_PIECE 32
template <typename TA>
static void launch_rglru(void* out, int out_stride, float* u, void* u16, float* z, int gates_done, const void* proj,
                         int proj_stride, int x_off, int y_off, const void* bx, const void* by, const void* conv_w,
                         const void* cb, const void* Ar, const void* Ai, const void* cr, const void* ci, const void* lam,
                         float c_decay, float* state, const int* token_pos, const int* token_slot, const int* token_seq,
                         const int* seq_start, const int* cu_seqlens, const int* seq_slot, int T, int R, int W, int blocks,
                         int taps, float out_scale, int max_new, float* pieces, int phase, cudaStream_t st) {
    const int bs = W / blocks;
    if (phase == 0 || phase == 1)
        zlm_launch(rglru_conv_kernel<TA>, dim3(T, (W + 255) / 256), dim3(256), 0, st, u, (TA*)u16, (const TA*)proj, proj_stride,
                   x_off, (const TA*)bx, (const TA*)conv_w, (const TA*)cb, (const float*)state, token_pos, token_slot, token_seq,
                   seq_start, cu_seqlens, W, taps);
    if (phase == 1) return;
    if (!gates_done) {
        // (eight inputs a lane where every row of a block starts at a multiple of 16 bytes, and u's rows at 32)
        const bool vec = bs % 8 == 0 && (uintptr_t)Ar % 16 == 0 && (uintptr_t)Ai % 16 == 0 && (uintptr_t)u % 16 == 0;
        if (T <= RG_FEW && vec)
            zlm_launch(rglru_gates_few_kernel<TA, 8>, dim3((W + 7) / 8), dim3(256), 0, st, z, (const float*)u, (const TA*)Ar,
                       (const TA*)Ai, T, W, bs);
        else if (T <= RG_FEW)
            zlm_launch(rglru_gates_few_kernel<TA, 1>, dim3((W + 7) / 8), dim3(256), 0, st, z, (const float*)u, (const TA*)Ar,
                       (const TA*)Ai, T, W, bs);
        else
            zlm_launch(rglru_gates_kernel<TA>, dim3((T + RG_TT - 1) / RG_TT, (bs + RG_OT - 1) / RG_OT, blocks), dim3(RG_OT * 4), 0,
                       st, z, (const float*)u, (const TA*)Ar, (const TA*)Ai, T, W, bs);
    }
    if (pieces) {
        const int L = RGLRU_PIECE, maxp = (max_new + L - 1) / L;
        float* PA = pieces;
        float* PB = pieces + (size_t)R * maxp * W;
        const int dtype = sizeof(TA) == 4 ? ZLM_DTYPE_F32 : ZLM_DTYPE_BF16;
        zlm_launch(rglru_piece_ab_kernel, dim3(R * maxp, (W + 127) / 128), dim3(128), 0, st, z, (const float*)u, cr, ci, lam, dtype,
                   c_decay, PA, PB, cu_seqlens, W, bs, maxp, L);
        zlm_launch(rglru_chain_kernel<TA>, dim3(R, (W + 127) / 128), dim3(128), 0, st, PA, (const float*)PB, state, (const TA*)proj,
                   proj_stride, x_off, (const TA*)bx, seq_slot, cu_seqlens, W, taps, maxp, L);
        zlm_launch(rglru_piece_out_kernel<TA>, dim3(R * maxp, (W + 127) / 128), dim3(128), 0, st, (TA*)out, out_stride,
                   (const float*)z, (const float*)PA, (const TA*)proj, proj_stride, y_off, (const TA*)by, cu_seqlens, W, bs, maxp, L,
                   out_scale);
        return;
    }
    zlm_launch(rglru_scan_kernel<TA>, dim3(R, (W + 127) / 128), dim3(128), 0, st, (TA*)out, out_stride, (const float*)u,
               (const float*)z, (const TA*)proj, proj_stride, x_off, y_off, (const TA*)bx, (const TA*)by, (const TA*)cr,
               (const TA*)ci, (const TA*)lam, c_decay, state, seq_slot, cu_seqlens, W, bs, taps, out_scale);
}

// proj [T][proj_stride] holds the x branch from column x_off and the y branch from y_off (W columns each), without their
// biases bx, by [W]; conv_w [W][taps], cb [W]; Ar, Ai [blocks][W/blocks][W/blocks] (out, in), cr, ci [W]; lam [W]; all in
// the element type.  u: fp32 scratch [T][W]; u16: null, or scratch [T][W] in the element type that receives u as well;
// z: fp32 scratch [T][blocks][2][W/blocks].  state [slots][taps][W] fp32.  out [T][out_stride] receives
// S * gelu_tanh(y) * out_scale in the element type.
// phase 0: everything; 1: the convolution only (the caller then computes z = u16_b [A_r[b] ; A_i[b]]^T block by block
// with a product of its own); 2: what follows the gates' logits (gates_done 1: z holds them).
// pieces: null (a thread walks a sequence's tokens), or 2 * R * ceil(max_new / 32) * W floats: sequences run in pieces of
// 32 tokens side by side.
extern "C" int zlm_rglru(void* out, int out_stride, float* u, void* u16, float* z, const void* proj, int proj_stride, int x_off,
                         int y_off, const void* bx, const void* by, const void* conv_w, const void* cb, const void* Ar,
                         const void* Ai, const void* cr, const void* ci, const void* lam, float c_decay, float* state, int dtype,
                         const int* token_pos, const int* token_slot, const int* token_seq, const int* seq_start,
                         const int* cu_seqlens, const int* seq_slot, int T, int R, int W, int blocks, int taps, float out_scale,
                         int max_new, float* pieces, int phase, cudaStream_t st) {
    if (T == 0) return ZLM_OK;
    ZLM_REQUIRE(W > 0 && blocks > 0 && W % blocks == 0, "rglru: %d channels in %d blocks", W, blocks);
    ZLM_REQUIRE(taps >= 1 && taps <= RC_MAX_TAPS, "rglru: %d taps (at most %d)", taps, RC_MAX_TAPS);
    ZLM_REQUIRE(blocks <= 65535 && (W / blocks + RG_OT - 1) / RG_OT <= 65535 && (W + 127) / 128 <= 65535, "rglru: too many channels");
    ZLM_REQUIRE(phase >= 0 && phase <= 2 && (!pieces || max_new > 0), "rglru: phase %d, longest sequence %d", phase, max_new);
    const int gates_done = phase == 2 ? 1 : 0;
    if (dtype == ZLM_DTYPE_F32)
        launch_rglru<float>(out, out_stride, u, u16, z, gates_done, proj, proj_stride, x_off, y_off, bx, by, conv_w, cb, Ar, Ai, cr,
                            ci, lam, c_decay, state, token_pos, token_slot, token_seq, seq_start, cu_seqlens, seq_slot, T, R, W,
                            blocks, taps, out_scale, max_new, pieces, phase, st);
    else if (dtype == ZLM_DTYPE_BF16)
        launch_rglru<__nv_bfloat16>(out, out_stride, u, u16, z, gates_done, proj, proj_stride, x_off, y_off, bx, by, conv_w, cb, Ar,
                                    Ai, cr, ci, lam, c_decay, state, token_pos, token_slot, token_seq, seq_start, cu_seqlens,
                                    seq_slot, T, R, W, blocks, taps, out_scale, max_new, pieces, phase, st);
    else
        ZLM_REQUIRE(false, "rglru: unsupported dtype %d", dtype);
    return zlm_check_launch("rglru");
}

// ---------------------------------------------------------------------------- long bfloat16 prompts: three launches
// (1) the convolution, in bfloat16 and block by block: u16 [blocks][Tp][bs], Tp = T rounded up to 128, so that (2) all
// diagonal blocks' gate logits are one grouped product, z [blocks][Tp][2][bs] fp32; (3) the recurrence on thread-block
// clusters in one pass over z and the two branches, with u formed again from the x branch (the same sum: the same bits) instead
// of stored in fp32.  1,999 tokens of 2,048 channels in 8 blocks: convolution 37, eight products 45, three passes of the
// recurrence 88 us before (u, z and the pieces' decays written and read by each); 11, 25 and 53 us now, one by one in a layer, and
// 67 for the three where they follow each other as dependent launches (144 before).

// A thread: 8 neighbouring channels of RC_RUN tokens, each token's row of x read once for all its taps.
#define RC_RUN 8
template <int TAPS>
__global__ void __launch_bounds__(128)
rglru_conv_blocks_kernel(__nv_bfloat16* __restrict__ u16, int* __restrict__ table, const __nv_bfloat16* __restrict__ proj,
                         int proj_stride, int x_off, const __nv_bfloat16* __restrict__ bx, const __nv_bfloat16* __restrict__ conv_w,
                         const __nv_bfloat16* __restrict__ cb, const float* __restrict__ state, const int* __restrict__ token_pos,
                         const int* __restrict__ token_slot, const int* __restrict__ token_seq, const int* __restrict__ seq_start,
                         int T, int Tp, int W, int bs, int blocks) {
    pdl_trigger();
    const int c = (blockIdx.y * 128 + threadIdx.x) * 8, t0 = blockIdx.x * RC_RUN;
    float w[8][TAPS], b[8], bias[8];
    if (c < W) {
        // (eight channels' taps and biases stand next to each other: eight numbers a read where they start at 16 bytes)
        if (((uintptr_t)conv_w | (uintptr_t)bx | (uintptr_t)cb) % 16 == 0) {
            auto read8 = [](const __nv_bfloat16* p, float* f) {
                const uint4 u = p && ZLM_CHK(p, 16) ? *(const uint4*)p : make_uint4(0, 0, 0, 0);
                const unsigned x[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(i & 1 ? x[i / 2] & 0xffff0000u : x[i / 2] << 16);
            };
            read8(bx ? bx + c : nullptr, b);
            read8(cb ? cb + c : nullptr, bias);
#pragma unroll
            for (int x = 0; x < TAPS; ++x) {
                float f[8];
                read8(conv_w + (size_t)c * TAPS + 8 * x, f);
#pragma unroll
                for (int i = 0; i < 8; ++i) w[(8 * x + i) / TAPS][(8 * x + i) % TAPS] = f[i];
            }
        } else {
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                b[v] = bx && ZLM_CHK(bx + c + v, 2) ? to_f32(bx[c + v]) : 0.f;
                bias[v] = cb && ZLM_CHK(cb + c + v, 2) ? to_f32(cb[c + v]) : 0.f;
#pragma unroll
                for (int j = 0; j < TAPS; ++j)
                    w[v][j] = ZLM_CHK(conv_w + (size_t)(c + v) * TAPS + j, 2) ? to_f32(conv_w[(size_t)(c + v) * TAPS + j]) : 0.f;
            }
        }
    }
    pdl_wait();
    const int per = (T + 255) / 256, tiles = blocks * per;       // (for the product: tiles of up to 256 rows of one diagonal block)
    if (blockIdx.x == 0)
        for (int x = blockIdx.y * 128 + threadIdx.x; x < tiles; x += gridDim.y * 128)
            if (ZLM_CHK(table + x, 4) && ZLM_CHK(table + tiles + x, 4) && ZLM_CHK(table + 2 * tiles + x, 4)) {
                table[x] = x / per;
                table[tiles + x] = x / per * Tp + x % per * 256;
                table[2 * tiles + x] = min(256, T - x % per * 256);
            }
    if (c >= W) return;
    uint4 x[RC_RUN + TAPS - 1];
#pragma unroll
    for (int j = 0; j < RC_RUN + TAPS - 1; ++j) {
        const int t = t0 - (TAPS - 1) + j;
        const __nv_bfloat16* p = proj + (size_t)t * proj_stride + x_off + c;
        x[j] = (t >= 0 && t < T && ZLM_CHK(p, 16)) ? *(const uint4*)p : make_uint4(0, 0, 0, 0);
    }
    __nv_bfloat16* dst = u16 + ((size_t)(c / bs) * Tp + t0) * bs + c % bs;
#pragma unroll
    for (int k = 0; k < RC_RUN; ++k) {
        const int t = t0 + k;
        if (t >= T || !ZLM_CHK(token_pos + t, 4) || !ZLM_CHK(token_seq + t, 4) || !ZLM_CHK(token_slot + t, 4)) break;
        const int pos = token_pos[t], i = pos - seq_start[token_seq[t]];
        float a[8];
#pragma unroll
        for (int v = 0; v < 8; ++v) a[v] = bias[v];
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const int s = i - (TAPS - 1) + j;         // the tap's token among the sequence's tokens of this step
            if (pos - (TAPS - 1) + j < 0) continue;   // before the sequence's start
            float f[8];
            if (s >= 0) {
                const uint4 q = x[k + j];
                f[0] = __uint_as_float(q.x << 16); f[1] = __uint_as_float(q.x & 0xffff0000u);
                f[2] = __uint_as_float(q.y << 16); f[3] = __uint_as_float(q.y & 0xffff0000u);
                f[4] = __uint_as_float(q.z << 16); f[5] = __uint_as_float(q.z & 0xffff0000u);
                f[6] = __uint_as_float(q.w << 16); f[7] = __uint_as_float(q.w & 0xffff0000u);
#pragma unroll
                for (int v = 0; v < 8; ++v) f[v] += b[v];
            } else {
                const float* p = state + ((size_t)token_slot[t] * TAPS + (TAPS + s)) * W + c;
                const bool ok = ZLM_CHK(p, 32);
#pragma unroll
                for (int v = 0; v < 8; ++v) f[v] = ok ? p[v] : 0.f;
            }
#pragma unroll
            for (int v = 0; v < 8; ++v) a[v] = fmaf(w[v][j], f[v], a[v]);
        }
        unsigned h[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(a[2 * v], a[2 * v + 1]);
            h[v] = *(const unsigned*)&p;
        }
        if (ZLM_CHK(dst + (size_t)k * bs, 16)) *(uint4*)(dst + (size_t)k * bs) = make_uint4(h[0], h[1], h[2], h[3]);
    }
}

// The recurrence's functions without branches, so that the numbers of a thread's tokens are worked out side by side (the
// library's division, square root, expm1f and tanhf each branch for arguments that do not occur here: 62 us of the kernel
// below with them, 55 us without).  Each is an approximation and one step of Newton's rule x - f(x) / f'(x) (Abramowitz and Stegun,
// Handbook of Mathematical Functions, 3.9.5), or the exponential's series (4.2.1): a few units in the last place of fp32 over
// the whole range, which a test compares with 64-bit values (zlm_rglru_functions).  NaN stays NaN.
// 1 / (1 + e^-x).  With e = e^-|x| the denominator is in [1, 2], where neither it nor its reciprocal can overflow or vanish:
// 1/d from r by f(r) = 1/r - d.  Below zero e / (1 + e): what underflows is the result itself (a clamped argument instead would
// leave 1.8e-35 there, which gelu multiplies with numbers as large as the type has).
__device__ __forceinline__ float rl_sigmoid(float x) {
    const float e = expf(-fabsf(x)), d = 1.0f + e, r0 = __fdividef(1.0f, d), r = fmaf(r0, fmaf(-d, r0, 1.0f), r0);
    return x < 0.f ? e * r : r;
}
// 1 - e^y for y <= 0, a = e^(y/2): above -1, where the difference would cancel, the series of (e^y - 1) / y, Horner's form
__device__ __forceinline__ float rl_one_minus_exp(float y, float a) {
    float p = 1.0f / 479001600.0f;                   // sum of y^k / k!, k = 1 .. 12; y^13 / 13! is below 2^-32 on [-1, 0]
    constexpr float c[11] = {1.0f / 39916800.0f, 1.0f / 3628800.0f, 1.0f / 362880.0f, 1.0f / 40320.0f, 1.0f / 5040.0f, 1.0f / 720.0f,
                             1.0f / 120.0f, 1.0f / 24.0f, 1.0f / 6.0f, 0.5f, 1.0f};
#pragma unroll
    for (int k = 0; k < 11; ++k) p = fmaf(p, y, c[k]);
    return y < -1.0f ? fmaf(-a, a, 1.0f) : -y * p;
}
// sqrt x from s = x rsqrt x by f(s) = s^2 - x; where the difference would be of the order of the smallest fp32 numbers, s as it is
__device__ __forceinline__ float rl_sqrt(float x) {
    const float r = rsqrtf(x), s = x * r, q = fmaf(fmaf(-s, s, x), 0.5f * r, s);
    return x < 1e-30f ? (x == 0.f ? 0.f : s) : q;
}
__device__ __forceinline__ void rl_ab(float zr, float zi, float u, float sl, float& a, float& b) {
    const float log_a = -rl_sigmoid(zr) * sl;
    a = expf(log_a);
    b = rl_sqrt(rl_one_minus_exp(2.0f * log_a, a)) * rl_sigmoid(zi) * u;
}
// gelu_tanh as z sigmoid(2 t): 1 + tanh(t) = 2 sigmoid(2 t)
__device__ __forceinline__ float rl_gelu(float z) { return z * rl_sigmoid(1.5957691216057308f * (z + 0.044715f * z * z * z)); }

// The four of them on n numbers, for their test: which 0 sigmoid, 1 one_minus_exp (of y, with e^(y/2) formed here), 2 sqrt, 3 gelu.
__global__ void rglru_functions_kernel(float* __restrict__ out, const float* __restrict__ in, int n, int which) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !ZLM_CHK(in + i, 4) || !ZLM_CHK(out + i, 4)) return;
    const float x = in[i];
    out[i] = which == 0 ? rl_sigmoid(x) : which == 1 ? rl_one_minus_exp(x, expf(0.5f * x)) : which == 2 ? rl_sqrt(x) : rl_gelu(x);
}
extern "C" int zlm_rglru_functions(float* out, const float* in, int n, int which, cudaStream_t st) {
    ZLM_REQUIRE(n > 0 && which >= 0 && which < 4, "rglru_functions: %d numbers, function %d", n, which);
    zlm_count_launch();
    rglru_functions_kernel<<<(n + 255) / 256, 256, 0, st>>>(out, in, n, which);
    return zlm_check_launch("rglru_functions");
}

// A cluster of up to RL_CLUSTER blocks owns 64 channels of one sequence, a warp RL_P neighbouring tokens of two channels a lane, whose
// decays and inputs it keeps in registers.  What a warp's tokens do to a state, S_out = A S_in + B, is folded over the block in
// shared memory and over the cluster in distributed shared memory; then every warp knows the state it starts from and walks
// its tokens.  Longer sequences go round again; of a shorter one the warps without a token only meet the barriers, and the
// blocks without one leave at once (a barrier waits for the threads that are left).  Bound by its exponentials and divisions: about
// 150 instructions a number, half of the issue slots busy with 16 warps an SM (128 registers; 16 to 20 bytes of spills up to 4
// taps, up to 132 beyond).
#define RL_CLUSTER 8
#define RL_WARPS 8
#define RL_P 8
template <int TAPS>
__global__ void __launch_bounds__(RL_WARPS * 32, 2)
rglru_cluster_kernel(__nv_bfloat16* __restrict__ out, int out_stride, const float* __restrict__ z, const __nv_bfloat16* __restrict__ proj,
                     int proj_stride, int x_off, int y_off, const __nv_bfloat16* __restrict__ bx, const __nv_bfloat16* __restrict__ by,
                     const __nv_bfloat16* __restrict__ conv_w, const __nv_bfloat16* __restrict__ cb, const __nv_bfloat16* __restrict__ cr,
                     const __nv_bfloat16* __restrict__ ci, const __nv_bfloat16* __restrict__ lam, float c_decay,
                     float* __restrict__ state, const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                     const int* __restrict__ cu_seqlens, int Tp, int W, int bs, float out_scale) {
    // two sets, for rounds in turn: a block that is a round ahead does not overwrite what another still reads
    __shared__ float2 piece[2][RL_WARPS][64];
    __shared__ float2 total[2][64];
    __shared__ float begin[RL_WARPS][64];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), r = blockIdx.x / (int)cluster.num_blocks();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.y * 64 + lane * 2;
    pdl_trigger();
    // (the step's integer arrays are copied in ahead of its first kernel: they may be read before pdl_wait())
    int row0 = 0, n = 0, slot = 0, start = 0;
    if (ZLM_CHK(seq_slot + r, 4) && ZLM_CHK(cu_seqlens + r, 8) && ZLM_CHK(seq_start + r, 4)) {
        row0 = cu_seqlens[r];
        n = cu_seqlens[r + 1] - row0;
        slot = seq_slot[r];
        start = seq_start[r];
    }
    // the blocks of the cluster that the sequence has tokens for
    const int ranks = min((int)cluster.num_blocks(), max(1, (n + RL_WARPS * RL_P - 1) / (RL_WARPS * RL_P)));
    if (rank >= ranks) return;
    bool live = c < W;                               // (no thread leaves its block: the block's others wait for it)
    const bool own = live && ((rank * RL_WARPS + warp) * RL_P < n || warp == 0);      // (a warp without a token needs nothing of these)
    float w[2][TAPS], xb[2], ub[2], yb[2], rb[2], ib[2], sl[2], S0[2] = {0.f, 0.f};
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        xb[v] = (own && bx && ZLM_CHK(bx + c + v, 2)) ? to_f32(bx[c + v]) : 0.f;
        ub[v] = (own && cb && ZLM_CHK(cb + c + v, 2)) ? to_f32(cb[c + v]) : 0.f;
        yb[v] = (own && by && ZLM_CHK(by + c + v, 2)) ? to_f32(by[c + v]) : 0.f;
        rb[v] = (own && cr && ZLM_CHK(cr + c + v, 2)) ? to_f32(cr[c + v]) : 0.f;
        ib[v] = (own && ci && ZLM_CHK(ci + c + v, 2)) ? to_f32(ci[c + v]) : 0.f;
        sl[v] = own && ZLM_CHK(lam + c + v, 2) ? softplus_f(to_f32(lam[c + v])) * c_decay : 0.f;
#pragma unroll
        for (int j = 0; j < TAPS; ++j)
            w[v][j] = own && ZLM_CHK(conv_w + (size_t)(c + v) * TAPS + j, 2) ? to_f32(conv_w[(size_t)(c + v) * TAPS + j]) : 0.f;
    }
    pdl_wait();
    float* sp = state + (size_t)slot * TAPS * W + c;
    live = live && ZLM_CHK(sp, 8);
    if (live) { S0[0] = sp[0]; S0[1] = sp[1]; }
    const float* zp = z + ((size_t)(c / bs) * Tp + row0) * 2 * bs + c % bs;
    int par = 0;
    for (int base = 0; base < n; base += ranks * RL_WARPS * RL_P, par ^= 1) {
        const int lo = base + (rank * RL_WARPS + warp) * RL_P, cnt = live ? min(n - lo, RL_P) : 0;
        float2 zr[RL_P], zi[RL_P];
        unsigned xr[RL_P + TAPS - 1], yr[RL_P];
        float A[2] = {1.f, 1.f}, B[2] = {0.f, 0.f};
        if (lo < n) {
#pragma unroll
            for (int j = 0; j < RL_P; ++j) {
                const float* q = zp + (size_t)(lo + j) * 2 * bs;
                const bool ok = j < cnt && ZLM_CHK(q, 8) && ZLM_CHK(q + bs, 8);
                zr[j] = ok ? *(const float2*)q : make_float2(0.f, 0.f);
                zi[j] = ok ? *(const float2*)(q + bs) : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < RL_P + TAPS - 1; ++j) {
                const int i = lo - (TAPS - 1) + j;
                const __nv_bfloat16* q = proj + (size_t)(row0 + i) * proj_stride + x_off + c;
                xr[j] = (live && i >= 0 && i < n && ZLM_CHK(q, 4)) ? *(const unsigned*)q : 0u;
            }
#pragma unroll
            for (int j = 0; j < RL_P; ++j) {
                const __nv_bfloat16* q = proj + (size_t)(row0 + lo + j) * proj_stride + y_off + c;
                yr[j] = (j < cnt && ZLM_CHK(q, 4)) ? *(const unsigned*)q : 0u;
            }
            float u[RL_P][2];
            if (lo >= TAPS - 1) {                        // (every tap of every token is one of the step's)
                float x[2][RL_P + TAPS - 1];
#pragma unroll
                for (int j = 0; j < RL_P + TAPS - 1; ++j) {
                    x[0][j] = __uint_as_float(xr[j] << 16) + xb[0];
                    x[1][j] = __uint_as_float(xr[j] & 0xffff0000u) + xb[1];
                }
#pragma unroll
                for (int j = 0; j < RL_P; ++j)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        u[j][v] = ub[v];
#pragma unroll
                        for (int k = 0; k < TAPS; ++k) u[j][v] = fmaf(w[v][k], x[v][j + k], u[j][v]);
                    }
            } else {
#pragma unroll
                for (int j = 0; j < RL_P; ++j)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        u[j][v] = ub[v];
#pragma unroll
                        for (int k = 0; k < TAPS; ++k) {
                            const int i = lo + j - (TAPS - 1) + k;
                            if (start + i < 0) continue;
                            float x;
                            if (i >= 0) x = __uint_as_float(v ? xr[j + k] & 0xffff0000u : xr[j + k] << 16) + xb[v];
                            else x = (j < cnt && ZLM_CHK(sp + (size_t)(TAPS + i) * W + v, 4)) ? sp[(size_t)(TAPS + i) * W + v] : 0.f;
                            u[j][v] = fmaf(w[v][k], x, u[j][v]);
                        }
                    }
            }
#pragma unroll
            for (int j = 0; j < RL_P; ++j) {
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    float a, b;
                    rl_ab((v ? zr[j].y : zr[j].x) + rb[v], (v ? zi[j].y : zi[j].x) + ib[v], u[j][v], sl[v], a, b);
                    if (v) { zr[j].y = a; zi[j].y = b; } else { zr[j].x = a; zi[j].x = b; }
                    if (j < cnt) {
                        A[v] *= a;
                        B[v] = fmaf(a, B[v], b);
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) piece[par][warp][lane * 2 + v] = make_float2(A[v], B[v]);
        __syncthreads();
        if (warp == 0)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                float2 t = piece[par][0][lane * 2 + v];
                for (int x = 1; x < RL_WARPS; ++x) {
                    const float2 q = piece[par][x][lane * 2 + v];
                    t = make_float2(q.x * t.x, fmaf(q.x, t.y, q.y));
                }
                total[par][lane * 2 + v] = t;
            }
        if (ranks > 1) cluster.sync();               // (one block: the totals are this warp's own lanes')
        // the states that the block's warps start from, and the one the whole round ends with
        if (warp == 0)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                float2 t[RL_CLUSTER];
#pragma unroll
                for (int k = 0; k < RL_CLUSTER; ++k) t[k] = k < ranks ? cluster.map_shared_rank(&total[par][0], k)[lane * 2 + v] : make_float2(1.f, 0.f);
                float q = S0[v], s = q;
#pragma unroll
                for (int k = 0; k < RL_CLUSTER; ++k) {
                    q = fmaf(t[k].x, q, t[k].y);
                    if (k + 1 == rank) s = q;
                }
                S0[v] = q;
#pragma unroll
                for (int x = 0; x < RL_WARPS; ++x) {
                    begin[x][lane * 2 + v] = s;
                    const float2 p = piece[par][x][lane * 2 + v];
                    s = fmaf(p.x, s, p.y);
                }
            }
        __syncthreads();
        float S[2] = {begin[warp][lane * 2], begin[warp][lane * 2 + 1]};
#pragma unroll
        for (int j = 0; j < RL_P; ++j) {
            if (j >= cnt) break;
            S[0] = fmaf(zr[j].x, S[0], zi[j].x);
            S[1] = fmaf(zr[j].y, S[1], zi[j].y);
            const float y0 = S[0] * rl_gelu(__uint_as_float(yr[j] << 16) + yb[0]) * out_scale;
            const float y1 = S[1] * rl_gelu(__uint_as_float(yr[j] & 0xffff0000u) + yb[1]) * out_scale;
            __nv_bfloat16* o = out + (size_t)(row0 + lo + j) * out_stride + c;
            if (ZLM_CHK(o, 4)) *(__nv_bfloat162*)o = __floats2bfloat162_rn(y0, y1);
        }
    }
    // (every block has read the old state ahead of the first barrier, and its older inputs only this warp has read)
    if (live && rank == 0 && warp == 0)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            sp[v] = S0[v];
            rglru_keep_inputs<__nv_bfloat16>(sp + v, proj, proj_stride, x_off, c + v, row0, n, W, TAPS, xb[v]);
        }
    if (ranks > 1) cluster.sync();                   // no block leaves while another may still read its shared memory
}

// bfloat16, with everything as in zlm_rglru: the first of the three launches.  u16 [blocks][Tp][W/blocks], Tp = T rounded up to
// 128; table [3][blocks * ceil(T / 256)] for zlm_gemm_tc_experts.
extern "C" int zlm_rglru_conv_blocks(void* u16, int* table, const void* proj, int proj_stride, int x_off, const void* bx,
                                     const void* conv_w, const void* cb, const float* state, const int* token_pos,
                                     const int* token_slot, const int* token_seq, const int* seq_start, int T, int W, int blocks, int taps,
                                     cudaStream_t st) {
    if (T == 0) return ZLM_OK;
    ZLM_REQUIRE(W > 0 && blocks > 0 && W % blocks == 0 && (W / blocks) % 8 == 0, "rglru: %d channels in %d blocks", W, blocks);
    ZLM_REQUIRE(taps >= 1 && taps <= RC_MAX_TAPS, "rglru: %d taps (at most %d)", taps, RC_MAX_TAPS);
    ZLM_REQUIRE(proj_stride % 8 == 0 && x_off % 8 == 0 && (uintptr_t)proj % 16 == 0 && (uintptr_t)u16 % 16 == 0 && (W + 1023) / 1024 <= 65535,
                "rglru: rows of %d from column %d", proj_stride, x_off);
    const int Tp = (T + 127) / 128 * 128;
    const dim3 grid((T + RC_RUN - 1) / RC_RUN, (W + 1023) / 1024);
#define ZLM_RC(N)                                                                                                               \
    case N:                                                                                                                     \
        zlm_launch(rglru_conv_blocks_kernel<N>, grid, dim3(128), 0, st, (__nv_bfloat16*)u16, table, (const __nv_bfloat16*)proj, \
                   proj_stride, x_off, (const __nv_bfloat16*)bx, (const __nv_bfloat16*)conv_w, (const __nv_bfloat16*)cb, state, token_pos, \
                   token_slot, token_seq, seq_start, T, Tp, W, W / blocks, blocks);                                            \
        break;
    switch (taps) { ZLM_RC(1) ZLM_RC(2) ZLM_RC(3) ZLM_RC(4) ZLM_RC(5) ZLM_RC(6) ZLM_RC(7) ZLM_RC(8) }
#undef ZLM_RC
    return zlm_check_launch("rglru_conv_blocks");
}

// Blocks of a sequence's cluster, in a step of T tokens: the size of the least estimate.  In rounds of the longest sequence, which
// follow one another (4 us each), the GPU takes three for as many blocks with tokens as fit on it (two an SM) and one for as many
// that leave at once.  What the other sequences bring is taken as their mean.  Us of the three launches in clusters of 1 / 2 / 4 / 8,
// and of the passes over pieces, 2,048 channels: 1 sequence of 2,048 tokens 182 / 120 / 79 / 67 and 147; 64 of 128 239 / 278 / 308 /
// 372 and 394; 1 of 128 beside 63 single tokens 76 / 123 / 142 / 183 and 83 (665 in full clusters that neither left nor skipped); 1
// of 1,024 beside 20 of 40 148 / 123 / 109 / 113 and 151.
extern "C" int zlm_rglru_cluster_size(int R, int T, int max_new, int W) {
    constexpr int ROUND = RL_WARPS * RL_P;
    const int longest = (max_new + ROUND - 1) / ROUND, mean = R > 1 ? (T - max_new) / (R - 1) : 0, other = mean > ROUND ? (mean + ROUND - 1) / ROUND : 1;
    int best = 1;
    float least = 0.f;
    for (int c = 1; c <= RL_CLUSTER; c <<= 1) {
        const float with = (float)(longest < c ? longest : c) + (R - 1.f) * (float)(other < c ? other : c), leave = (float)R * c - with;
        const float est = (float)((longest + c - 1) / c) + (3.f * with + leave) * (float)((W + 63) / 64) / 296.f;
        if (c == 1 || est < least) { best = c; least = est; }
    }
    return best;
}

// The third: z [blocks][Tp][2][W/blocks] fp32 holds the gates' logits without their biases; `cluster` blocks a sequence.
extern "C" int zlm_rglru_cluster(void* out, int out_stride, const float* z, const void* proj, int proj_stride, int x_off, int y_off,
                                 const void* bx, const void* by, const void* conv_w, const void* cb, const void* cr, const void* ci,
                                 const void* lam, float c_decay, float* state, const int* seq_slot, const int* seq_start,
                                 const int* cu_seqlens, int T, int R, int W, int blocks, int taps, float out_scale, int cluster,
                                 cudaStream_t st) {
    if (T == 0) return ZLM_OK;
    ZLM_REQUIRE(W > 0 && blocks > 0 && W % blocks == 0 && (W / blocks) % 8 == 0, "rglru: %d channels in %d blocks", W, blocks);
    ZLM_REQUIRE(taps >= 1 && taps <= RC_MAX_TAPS, "rglru: %d taps (at most %d)", taps, RC_MAX_TAPS);
    ZLM_REQUIRE(cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8, "rglru: clusters of %d blocks", cluster);
    ZLM_REQUIRE(proj_stride % 2 == 0 && x_off % 2 == 0 && y_off % 2 == 0 && out_stride % 2 == 0 && (uintptr_t)proj % 4 == 0 &&
                    (uintptr_t)out % 4 == 0 && (uintptr_t)z % 8 == 0 && (W + 63) / 64 <= 65535 && R > 0 && R <= (1 << 27),
                "rglru: rows of %d and %d, %d sequences", proj_stride, out_stride, R);
    const int Tp = (T + 127) / 128 * 128;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(R * cluster, (W + 63) / 64);
    cfg.blockDim = dim3(RL_WARPS * 32);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = zlm_pdl_enabled() ? 2 : 1;
    zlm_count_launch();
#define ZLM_RL(N)                                                                                                               \
    case N:                                                                                                                     \
        cudaLaunchKernelEx(&cfg, rglru_cluster_kernel<N>, (__nv_bfloat16*)out, out_stride, z, (const __nv_bfloat16*)proj,       \
                           proj_stride, x_off, y_off, (const __nv_bfloat16*)bx, (const __nv_bfloat16*)by, (const __nv_bfloat16*)conv_w, \
                           (const __nv_bfloat16*)cb, (const __nv_bfloat16*)cr, (const __nv_bfloat16*)ci, (const __nv_bfloat16*)lam, \
                           c_decay, state, seq_slot, seq_start, cu_seqlens, Tp, W, W / blocks, out_scale);                      \
        break;
    switch (taps) { ZLM_RL(1) ZLM_RL(2) ZLM_RL(3) ZLM_RL(4) ZLM_RL(5) ZLM_RL(6) ZLM_RL(7) ZLM_RL(8) }
#undef ZLM_RL
    return zlm_check_launch("rglru_cluster");
}

// ---------------------------------------------------------------------------- decays from a low-rank projection
// alpha[t][c] = sigmoid(z)^(1/tau) = exp(-softplus(-z) / tau), z = sum_r W2[c][r] lo[t][r] + b[c]; lo: `rank` columns of
// proj from lo_off on.  fp32 throughout.
// TOK tokens a block: a thread reads its channel's row of W2 once for all of them
template <typename TA, int TOK>
__global__ void __launch_bounds__(256)
lowrank_decay_kernel(float* __restrict__ alpha, const TA* __restrict__ proj, int proj_stride, int lo_off, const TA* __restrict__ W2,
                     const TA* __restrict__ b, int T, int C, int rank, float inv_tau) {
    extern __shared__ float ld_lo[];            // [TOK][rank]
    pdl_trigger();
    const int t0 = blockIdx.x * TOK;
    pdl_wait();
    for (int x = threadIdx.x; x < TOK * rank; x += blockDim.x) {
        const int tt = x / rank, r = x - tt * rank;
        const TA* p = proj + (size_t)(t0 + tt) * proj_stride + lo_off + r;
        ld_lo[x] = (t0 + tt < T && ZLM_CHK(p, sizeof(TA))) ? to_f32(*p) : 0.f;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        float z[TOK];
        const float bias = b ? to_f32(b[c]) : 0.f;
#pragma unroll
        for (int tt = 0; tt < TOK; ++tt) z[tt] = bias;
        for (int r = 0; r < rank; ++r) {
            if (!ZLM_CHK(W2 + (size_t)c * rank + r, sizeof(TA))) continue;
            const float w = to_f32(W2[(size_t)c * rank + r]);
#pragma unroll
            for (int tt = 0; tt < TOK; ++tt) z[tt] = fmaf(w, ld_lo[tt * rank + r], z[tt]);
        }
#pragma unroll
        for (int tt = 0; tt < TOK; ++tt) {
            if (t0 + tt >= T) break;
            float* ap = alpha + (size_t)(t0 + tt) * C + c;
            if (ZLM_CHK(ap, 4)) *ap = expf(-softplus_f(-z[tt]) * inv_tau);
        }
    }
}

extern "C" int zlm_lowrank_decay(float* alpha, const void* proj, int proj_stride, int lo_off, const void* W2, const void* b,
                                 int dtype, int T, int C, int rank, float tau, cudaStream_t st) {
    if (T == 0) return ZLM_OK;
    ZLM_REQUIRE(C > 0 && rank > 0 && rank <= 512 && tau > 0.f, "lowrank_decay: %d channels of rank %d, tau %g", C, rank, (double)tau);
    // many tokens: sixteen a block; few: one, so that the blocks are many
#define ZLM_LD(TA, TOK)                                                                                                  \
    zlm_launch(lowrank_decay_kernel<TA, TOK>, dim3((T + TOK - 1) / TOK), dim3(256), (size_t)TOK * rank * sizeof(float), st, alpha, \
               (const TA*)proj, proj_stride, lo_off, (const TA*)W2, (const TA*)b, T, C, rank, 1.0f / tau)
    if (dtype == ZLM_DTYPE_F32) {
        if (T >= 256) ZLM_LD(float, 16); else ZLM_LD(float, 1);
    } else if (dtype == ZLM_DTYPE_BF16) {
        if (T >= 256) ZLM_LD(__nv_bfloat16, 16); else ZLM_LD(__nv_bfloat16, 1);
    } else {
        ZLM_REQUIRE(false, "lowrank_decay: unsupported dtype %d", dtype);
    }
#undef ZLM_LD
    return zlm_check_launch("lowrank_decay");
}

// ---------------------------------------------------------------------------- linear attention with decays per channel
// A block: one head of one sequence (or of one piece of a sequence) and 512 / DS value columns, DS = DR / DPT.  A thread owns
// DPT rows of four columns of the state in registers (rows from `dim` on stay zero), two rows a packed instruction, so that a
// number of q, k or the decays read from shared memory serves four columns; the DS lanes that share columns add their parts of
// an output by shuffles, dealing the columns out.  Tokens are staged LA_CH at a time as fp32: q (scaled), k, the decays, v.
//   MODE 0: a sequence's tokens in order, from and to the sequence's state.
//   MODE 1: a piece of L tokens from a zero state; leaves the piece's outputs, the state it ends with (part) and the
//           product of its decays per key channel (pdecay): S_out = diag(pdecay) S_in + part.  o [T][H*V] fp32.
// Bound by the packed FMAs and, with one column a thread, by shared-memory reads before: 2,048 tokens of 8 heads of 64 x 128 in
// pieces 37 us with a column a thread (62 with two threads a column), 32 us so.
#define LA_CH 16
#define LA_CPT 4
template <typename TA, int DR, int DPT, int MODE>
__global__ void __launch_bounds__(128, MODE == 0 || DR == 128 ? 4 : 5)
linear_attention_kernel(float* __restrict__ o, const TA* __restrict__ proj, int proj_stride, int q_off, int k_off, int v_off,
                        const float* __restrict__ alpha, const float* __restrict__ head_decay, float* __restrict__ state,
                        const int* __restrict__ seq_slot, const int* __restrict__ cu_seqlens, int H, int D, int V,
                        float q_scale, float* __restrict__ part, float* __restrict__ pdecay, int maxp, int L) {
    constexpr int DS = DR / DPT, COLS = 128 / DS * LA_CPT, SEG = DPT + 4, DP = DS * SEG;      // (segments in different banks)
    static_assert(DS == 4 || DS == 8, "the sums below deal four columns out to four lanes or eight");
    __shared__ __align__(16) float sq[LA_CH][DP], sk[LA_CH][DP], sa[LA_CH][DP];
    __shared__ __align__(16) float sv[LA_CH][COLS];
    pdl_trigger();
    const int unit = blockIdx.x / H, h = blockIdx.x % H, v0 = blockIdx.y * COLS, tid = threadIdx.x;
    const int r = MODE == 0 ? unit : unit / maxp, p = MODE == 0 ? 0 : unit % maxp;
    const int grp = tid / DS, lane_d = tid % DS, v = v0 + grp * LA_CPT;
    pdl_wait();
    if (!ZLM_CHK(seq_slot + r, 4) || !ZLM_CHK(cu_seqlens + r, 8)) return;
    const int slot = seq_slot[r], row0 = cu_seqlens[r], n = cu_seqlens[r + 1] - row0;
    const int lo = MODE == 0 ? 0 : p * L, hi = MODE == 0 ? n : min(n, lo + L);
    if (lo >= hi) return;
    float* sp = (MODE == 0 ? state + (((size_t)slot * H + h) * D) * V : part + ((((size_t)r * maxp + p) * H + h) * D) * V) + v;
    float2 S[DPT / 2][LA_CPT];
#pragma unroll
    for (int j = 0; j < DPT / 2; ++j)
#pragma unroll
        for (int c = 0; c < LA_CPT; ++c) {
            float t[2] = {0.f, 0.f};
            if (MODE == 0)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int d = lane_d * DPT + 2 * j + e;
                    if (d < D && v + c < V && ZLM_CHK(sp + (size_t)d * V + c, 4)) t[e] = sp[(size_t)d * V + c];
                }
            S[j][c] = make_float2(t[0], t[1]);
        }
    const float hd = head_decay ? head_decay[h] : 1.0f;
    float pd = 1.0f;                              // MODE 1: the product of the piece's decays of key channel `tid`
    for (int s0 = lo; s0 < hi; s0 += LA_CH) {
        const int m = min(LA_CH, hi - s0);
        __syncthreads();
#pragma unroll 4
        for (int x = tid; x < LA_CH * DR; x += 128) {
            const int j = x / DR, d = x % DR, at = (d / DPT) * SEG + d % DPT;
            float fq = 0.f, fk = 0.f, fa = 1.f;
            if (j < m && d < D) {
                const TA* row = proj + (size_t)(row0 + s0 + j) * proj_stride;
                if (ZLM_CHK(row + q_off + h * D + d, sizeof(TA))) fq = to_f32(row[q_off + h * D + d]) * q_scale;
                if (ZLM_CHK(row + k_off + h * D + d, sizeof(TA))) fk = to_f32(row[k_off + h * D + d]);
                if (alpha) {
                    const float* ap = alpha + ((size_t)(row0 + s0 + j) * H + h) * D + d;
                    if (ZLM_CHK(ap, 4)) fa = *ap;
                } else {
                    fa = hd;
                }
            }
            sq[j][at] = fq; sk[j][at] = fk; sa[j][at] = fa;
        }
#pragma unroll 8
        for (int x = tid; x < LA_CH * COLS; x += 128) {
            const int j = x / COLS, e = x % COLS;
            float fv = 0.f;
            if (j < m && v0 + e < V) {
                const TA* pv = proj + (size_t)(row0 + s0 + j) * proj_stride + v_off + h * V + v0 + e;
                if (ZLM_CHK(pv, sizeof(TA))) fv = to_f32(*pv);
            }
            sv[j][e] = fv;
        }
        __syncthreads();
        if (MODE == 1 && tid < DR)
            for (int j = 0; j < m; ++j) pd *= sa[j][(tid / DPT) * SEG + tid % DPT];
        for (int j = 0; j < m; ++j) {
            const float4 v4 = *(const float4*)&sv[j][grp * LA_CPT];
            const float2 vv[LA_CPT] = {make_float2(v4.x, v4.x), make_float2(v4.y, v4.y), make_float2(v4.z, v4.z), make_float2(v4.w, v4.w)};
            float2 acc2[LA_CPT];
#pragma unroll
            for (int c = 0; c < LA_CPT; ++c) acc2[c] = make_float2(0.f, 0.f);
#pragma unroll
            for (int d = 0; d < DPT; d += 4) {
                const int at = lane_d * SEG + d;
                const float4 a4 = *(const float4*)&sa[j][at], q4 = *(const float4*)&sq[j][at], k4 = *(const float4*)&sk[j][at];
                const float2 a2[2] = {make_float2(a4.x, a4.y), make_float2(a4.z, a4.w)}, q2[2] = {make_float2(q4.x, q4.y), make_float2(q4.z, q4.w)},
                             k2[2] = {make_float2(k4.x, k4.y), make_float2(k4.z, k4.w)};
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int c = 0; c < LA_CPT; ++c) {
                        S[d / 2 + e][c] = __ffma2_rn(a2[e], S[d / 2 + e][c], __fmul2_rn(k2[e], vv[c]));
                        acc2[c] = __ffma2_rn(S[d / 2 + e][c], q2[e], acc2[c]);
                    }
            }
            float acc[LA_CPT];
#pragma unroll
            for (int c = 0; c < LA_CPT; ++c) acc[c] = acc2[c].x + acc2[c].y;
            // half of the lanes go on with columns 0-1, half with 2-3, then one column each
            const bool up = (lane_d & (DS >> 1)) != 0, up2 = (lane_d & (DS >> 2)) != 0;
            const float r0 = __shfl_xor_sync(0xffffffffu, up ? acc[0] : acc[2], DS >> 1), r1 = __shfl_xor_sync(0xffffffffu, up ? acc[1] : acc[3], DS >> 1);
            const float b0 = (up ? acc[2] : acc[0]) + r0, b1 = (up ? acc[3] : acc[1]) + r1;
            float sum = (up2 ? b1 : b0) + __shfl_xor_sync(0xffffffffu, up2 ? b0 : b1, DS >> 2);
            if (DS == 8) sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            const int mine = (up ? 2 : 0) + (up2 ? 1 : 0);
            float* op = o + ((size_t)(row0 + s0 + j) * H + h) * V + v + mine;
            if ((DS == 4 || (lane_d & 1) == 0) && v + mine < V && ZLM_CHK(op, 4)) *op = sum;
        }
    }
#pragma unroll
    for (int j = 0; j < DPT / 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int d = lane_d * DPT + 2 * j + e;
            float* dst = sp + (size_t)d * V;
            if (d >= D) continue;
            const float t[LA_CPT] = {e ? S[j][0].y : S[j][0].x, e ? S[j][1].y : S[j][1].x, e ? S[j][2].y : S[j][2].x, e ? S[j][3].y : S[j][3].x};
            if (V % 4 == 0 && v < V && (uintptr_t)dst % 16 == 0 && ZLM_CHK(dst, 16)) {
                *(float4*)dst = make_float4(t[0], t[1], t[2], t[3]);
            } else {
#pragma unroll
                for (int c = 0; c < LA_CPT; ++c)
                    if (v + c < V && ZLM_CHK(dst + c, 4)) dst[c] = t[c];
            }
        }
    if (MODE == 1 && blockIdx.y == 0 && tid < D) {
        float* pp = pdecay + (((size_t)r * maxp + p) * H + h) * D + tid;
        if (ZLM_CHK(pp, 4)) *pp = pd;
    }
}

// The walk of steps that bring one token or two a sequence, where many heads and sequences fill the GPU (la_by_columns): a block is
// one head of one sequence and up to 128 value columns, a thread owns one column of the state, DR rows in registers, so that
// a warp reads and writes a row of the state 128 bytes at a time.  Bound by the state's way through memory then; the four columns
// by sixteen rows a thread above read and write it in pieces.  Every sum is in the order of the kernel above (segments of DPT
// rows, even and odd rows apart, the segments' sums as its shuffles pair them): a token's bits do not tell which of them ran.
template <typename TA, int DR, int DPT>
__global__ void __launch_bounds__(128)
linear_attention_columns_kernel(float* __restrict__ o, const TA* __restrict__ proj, int proj_stride, int q_off, int k_off, int v_off,
                                const float* __restrict__ alpha, const float* __restrict__ head_decay, float* __restrict__ state,
                                const int* __restrict__ seq_slot, const int* __restrict__ cu_seqlens, int H, int D, int V,
                                float q_scale) {
    constexpr int DS = DR / DPT;
    __shared__ __align__(16) float sq[LA_CH][DR], sk[LA_CH][DR], sa[LA_CH][DR];
    __shared__ float sv[LA_CH][128];
    pdl_trigger();
    const int r = blockIdx.x / H, h = blockIdx.x % H, v0 = blockIdx.y * 128, tid = threadIdx.x, v = v0 + tid;
    pdl_wait();
    if (!ZLM_CHK(seq_slot + r, 4) || !ZLM_CHK(cu_seqlens + r, 8)) return;
    const int slot = seq_slot[r], row0 = cu_seqlens[r], n = cu_seqlens[r + 1] - row0;
    if (n <= 0) return;
    float* sp = state + (((size_t)slot * H + h) * D) * V + v;
    float S[DR];
#pragma unroll
    for (int d = 0; d < DR; ++d) S[d] = (d < D && v < V && ZLM_CHK(sp + (size_t)d * V, 4)) ? sp[(size_t)d * V] : 0.f;
    const float hd = head_decay ? head_decay[h] : 1.0f;
    for (int s0 = 0; s0 < n; s0 += LA_CH) {
        const int m = min(LA_CH, n - s0);
        __syncthreads();
        for (int x = tid; x < LA_CH * DR; x += 128) {
            const int j = x / DR, d = x % DR;
            float fq = 0.f, fk = 0.f, fa = 1.f;
            if (j < m && d < D) {
                const TA* row = proj + (size_t)(row0 + s0 + j) * proj_stride;
                if (ZLM_CHK(row + q_off + h * D + d, sizeof(TA))) fq = to_f32(row[q_off + h * D + d]) * q_scale;
                if (ZLM_CHK(row + k_off + h * D + d, sizeof(TA))) fk = to_f32(row[k_off + h * D + d]);
                if (alpha) {
                    const float* ap = alpha + ((size_t)(row0 + s0 + j) * H + h) * D + d;
                    if (ZLM_CHK(ap, 4)) fa = *ap;
                } else {
                    fa = hd;
                }
            }
            sq[j][d] = fq; sk[j][d] = fk; sa[j][d] = fa;
        }
        for (int x = tid; x < LA_CH * 128; x += 128) {
            const int j = x / 128, e = x % 128;
            float fv = 0.f;
            if (j < m && v0 + e < V) {
                const TA* pv = proj + (size_t)(row0 + s0 + j) * proj_stride + v_off + h * V + v0 + e;
                if (ZLM_CHK(pv, sizeof(TA))) fv = to_f32(*pv);
            }
            sv[j][e] = fv;
        }
        __syncthreads();
        for (int j = 0; j < m; ++j) {
            const float vv = sv[j][tid];
            float sum[DS], odd[DS];
#pragma unroll
            for (int g = 0; g < DS; ++g) sum[g] = odd[g] = 0.f;
#pragma unroll
            for (int e = 0; e < DPT; e += 4)
#pragma unroll
                for (int g = 0; g < DS; ++g) {
                    const int d = g * DPT + e;
                    const float4 a4 = *(const float4*)&sa[j][d], q4 = *(const float4*)&sq[j][d], k4 = *(const float4*)&sk[j][d];
                    S[d] = fmaf(a4.x, S[d], __fmul_rn(k4.x, vv));         sum[g] = fmaf(S[d], q4.x, sum[g]);
                    S[d + 1] = fmaf(a4.y, S[d + 1], __fmul_rn(k4.y, vv)); odd[g] = fmaf(S[d + 1], q4.y, odd[g]);
                    S[d + 2] = fmaf(a4.z, S[d + 2], __fmul_rn(k4.z, vv)); sum[g] = fmaf(S[d + 2], q4.z, sum[g]);
                    S[d + 3] = fmaf(a4.w, S[d + 3], __fmul_rn(k4.w, vv)); odd[g] = fmaf(S[d + 3], q4.w, odd[g]);
                }
#pragma unroll
            for (int g = 0; g < DS; ++g) sum[g] += odd[g];
#pragma unroll
            for (int x = DS / 2; x; x >>= 1)
#pragma unroll
                for (int g = 0; g < x; ++g) sum[g] += sum[g + x];
            float* op = o + ((size_t)(row0 + s0 + j) * H + h) * V + v;
            if (v < V && ZLM_CHK(op, 4)) *op = sum[0];
        }
    }
    if (v < V) {                                     // (a branch of its own: as part of the next test it kept every row's address in registers)
#pragma unroll
        for (int d = 0; d < DR; ++d)
            if (d < D && ZLM_CHK(sp + (size_t)d * V, 4)) sp[(size_t)d * V] = S[d];
    }
}

// The pieces' states in order: part[piece] becomes the state the piece starts from, the sequence's state is left.
// (a thread owns VEC neighbouring numbers of one row of the state; eight pieces' loads in flight.)  grid (R * H, ceil(D * V / (128 VEC)))
#define CHAIN_AHEAD 8
template <int VEC>
__global__ void __launch_bounds__(128)
linear_attention_chain_kernel(float* __restrict__ part, const float* __restrict__ pdecay, float* __restrict__ state,
                              const int* __restrict__ seq_slot, const int* __restrict__ cu_seqlens, int H, int D, int V,
                              int maxp, int L) {
    struct alignas(4 * VEC) Num { float v[VEC]; };
    pdl_trigger();
    const int rh = blockIdx.x, r = rh / H, h = rh % H, e = (blockIdx.y * 128 + threadIdx.x) * VEC, d = e / V;
    pdl_wait();
    if (e >= D * V || !ZLM_CHK(seq_slot + r, 4) || !ZLM_CHK(cu_seqlens + r, 8)) return;
    const int slot = seq_slot[r], n = cu_seqlens[r + 1] - cu_seqlens[r];
    const int np = (n + L - 1) / L;
    Num* sp = (Num*)(state + ((size_t)slot * H + h) * D * V + e);
    if (!ZLM_CHK(sp, 4 * VEC)) return;
    Num S = *sp;
    const size_t pstride = (size_t)H * D * V, dstride = (size_t)H * D;
    float* pp = part + ((size_t)r * maxp * H + h) * D * V + e;
    const float* dp = pdecay + ((size_t)r * maxp * H + h) * D + d;
    for (int p0 = 0; p0 < np; p0 += CHAIN_AHEAD, pp += CHAIN_AHEAD * pstride, dp += CHAIN_AHEAD * dstride) {
        Num A[CHAIN_AHEAD];
        float g[CHAIN_AHEAD];
#pragma unroll
        for (int j = 0; j < CHAIN_AHEAD; ++j) {
            g[j] = 1.f;
            memset(&A[j], 0, sizeof(Num));
            if (p0 + j < np && ZLM_CHK(pp + j * pstride, 4 * VEC) && ZLM_CHK(dp + j * dstride, 4)) {
                A[j] = *(const Num*)(pp + j * pstride);
                g[j] = dp[j * dstride];
            }
        }
#pragma unroll
        for (int j = 0; j < CHAIN_AHEAD; ++j) {
            if (p0 + j >= np) break;
            if (ZLM_CHK(pp + j * pstride, 4 * VEC)) *(Num*)(pp + j * pstride) = S;
#pragma unroll
            for (int x = 0; x < VEC; ++x) S.v[x] = fmaf(g[j], S.v[x], A[j].v[x]);
        }
    }
    *sp = S;
}

// What the state ahead of a piece gives its tokens, as a product: o_t += S_in^T (diag(alpha_lo .. alpha_t) q_t), 32 tokens by 128
// columns a block, a warp eight tokens, a lane four columns of each.  With y (heads of up to 128 columns) the outputs go on to
// what follows them in the mixer: every head divided by its root mean square, times a weight, times the gate.
// 2,048 tokens of 8 heads of 64 x 128: walked token by token 27 us, and 18 us for norm and gate; 19 us so, about 5 more with both.
#define LA_PIECE 32
#define LA_LD (LA_PIECE + 4)
struct LaOut {
    void* y;                         // null: o
    int y_stride;
    const void* g;
    int g_stride;
    VecW w;                          // [V]
    float eps;
    int act;                         // 1: silu, 0: sigmoid
};
template <typename TA, int DR>
__global__ void __launch_bounds__(128, DR == 128 ? 2 : 4)
linear_attention_out_kernel(float* __restrict__ o, const TA* __restrict__ proj, int proj_stride, int q_off,
                            const float* __restrict__ alpha, const float* __restrict__ head_decay, const float* __restrict__ part,
                            const int* __restrict__ cu_seqlens, int H, int D, int V, float q_scale, int maxp, LaOut out) {
    struct alignas(4 * sizeof(TA)) Four { TA v[4]; };
    extern __shared__ __align__(16) float la_smem[];
    float* S = la_smem;                              // [DR][128]
    float* Q = S + DR * 128;                         // [DR][LA_LD]: the decayed queries, tokens innermost
    pdl_trigger();
    const int unit = blockIdx.x / H, h = blockIdx.x % H, v0 = blockIdx.y * 128, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = unit / maxp, p = unit % maxp;
    pdl_wait();
    if (!ZLM_CHK(cu_seqlens + r, 8)) return;
    const int row0 = cu_seqlens[r] + p * LA_PIECE, m = min(LA_PIECE, cu_seqlens[r + 1] - row0);
    if (m <= 0) return;
    const float* src = part + ((((size_t)r * maxp + p) * H + h) * D) * V + v0;
    const bool vec = V % 4 == 0 && (uintptr_t)part % 16 == 0;
    for (int x = tid; x < D * 32; x += 128) {
        const int d = x >> 5, c = (x & 31) * 4;
        const float* q = src + (size_t)d * V + c;
        float* dst = S + d * 128 + c;
        if (vec && v0 + c < V && ZLM_CHK(q, 16)) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(q));
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = (v0 + c + e < V && ZLM_CHK(q + e, 4)) ? q[e] : 0.f;
        }
    }
    asm volatile("cp.async.commit_group;\n" ::);
    if (tid < D) {
        const float hd = head_decay ? head_decay[h] : 1.0f;
        float pd = 1.0f;
#pragma unroll 16
        for (int j = 0; j < LA_PIECE; ++j) {
            const TA* q = proj + (size_t)(row0 + j) * proj_stride + q_off + h * D + tid;
            const float* a = alpha + ((size_t)(row0 + j) * H + h) * D + tid;
            const bool ok = j < m && ZLM_CHK(q, sizeof(TA)) && (!alpha || ZLM_CHK(a, 4));
            pd *= ok ? (alpha ? *a : hd) : 1.0f;
            Q[tid * LA_LD + j] = ok ? to_f32(*q) * q_scale * pd : 0.f;
        }
    }
    const int c = v0 + lane * 4;
    const bool vo = V % 4 == 0 && c < V && (uintptr_t)o % 16 == 0;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
    // sixteen coordinates at a time from zero, then added: the roundings of a short chain
    for (int d0 = 0; d0 < D; d0 += 16) {
        float t[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) t[i][e] = 0.f;
#pragma unroll 8
        for (int d = d0; d < min(D, d0 + 16); ++d) {
            const float4 qa = *(const float4*)(Q + d * LA_LD + warp * 8), qb = *(const float4*)(Q + d * LA_LD + warp * 8 + 4);
            const float4 s = *(const float4*)(S + d * 128 + lane * 4);
            const float q[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                t[i][0] = fmaf(q[i], s.x, t[i][0]);
                t[i][1] = fmaf(q[i], s.y, t[i][1]);
                t[i][2] = fmaf(q[i], s.z, t[i][2]);
                t[i][3] = fmaf(q[i], s.w, t[i][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] += t[i][e];
    }
    // the piece's own outputs and the gate's logits, all of them on their way before the first is used
    float own[8][4];
    Four z[8];
    const bool yv = out.y && V % 4 == 0 && c < V && (out.y_stride | out.g_stride) % 4 == 0 &&
                    ((uintptr_t)out.y | (uintptr_t)out.g) % sizeof(Four) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int j = warp * 8 + i;
        const float* op = o + ((size_t)(row0 + j) * H + h) * V + c;
        const TA* gp = (const TA*)out.g + (size_t)(row0 + j) * out.g_stride + (size_t)h * V + c;
        memset(&z[i], 0, sizeof(Four));
#pragma unroll
        for (int e = 0; e < 4; ++e) own[i][e] = 0.f;
        if (j >= m) continue;
        if (vo && ZLM_CHK(op, 16)) {
            const float4 f = *(const float4*)op;
            own[i][0] = f.x; own[i][1] = f.y; own[i][2] = f.z; own[i][3] = f.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (c + e < V && ZLM_CHK(op + e, 4)) own[i][e] = op[e];
        }
        if (!out.y) continue;
        if (yv && ZLM_CHK(gp, sizeof(Four))) {
            z[i] = *(const Four*)gp;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (c + e < V && ZLM_CHK(gp + e, sizeof(TA))) z[i].v[e] = gp[e];
        }
    }
    float wn[4] = {0.f, 0.f, 0.f, 0.f};
    if (out.y)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (c + e < V && out.w.ok(c + e, 1)) wn[e] = out.w[c + e];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int j = warp * 8 + i;
        if (j >= m) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] += own[i][e];
        if (!out.y) {
            float* op = o + ((size_t)(row0 + j) * H + h) * V + c;
            if (vo && ZLM_CHK(op, 16)) *(float4*)op = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + e < V && ZLM_CHK(op + e, 4)) op[e] = acc[i][e];
            continue;
        }
        float ss = 0.f;                              // (columns beyond V are zero)
#pragma unroll
        for (int e = 0; e < 4; ++e) ss = fmaf(acc[i][e], acc[i][e], ss);
        const float f = 1.0f / sqrtf(warp_sum(ss) / (float)V + out.eps);
        TA* yp = (TA*)out.y + (size_t)(row0 + j) * out.y_stride + (size_t)h * V + c;
        Four y;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float zz = to_f32(z[i].v[e]), sg = 1.0f / (1.0f + expf(-zz));
            y.v[e] = from_f32<TA>(acc[i][e] * f * wn[e] * (out.act == 1 ? zz * sg : sg));
        }
        if (yv && ZLM_CHK(yp, sizeof(Four))) {
            *(Four*)yp = y;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (c + e < V && ZLM_CHK(yp + e, sizeof(TA))) yp[e] = y.v[e];
        }
    }
}

template <typename TA, int DR>
static int launch_la_out(dim3 grid, cudaStream_t st, float* o, const void* proj, int proj_stride, int q_off, const float* alpha,
                         const float* head_decay, const float* part, const int* cu_seqlens, int H, int D, int V, float q_scale,
                         int maxp, const LaOut& out) {
    const size_t smem = (size_t)DR * (128 + LA_LD) * sizeof(float);
    auto kern = linear_attention_out_kernel<TA, DR>;
    static bool attr_set_dev[64] = {};
    bool& attr_set = attr_set_dev[zlm_device_index()];
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            zlm_set_error("linear_attention: cannot reserve shared memory: %s", cudaGetErrorString(e));
            return ZLM_ERR_CUDA;
        }
        attr_set = true;
    }
    zlm_launch(kern, grid, dim3(128), smem, st, o, (const TA*)proj, proj_stride, q_off, alpha, head_decay, part, cu_seqlens, H, D, V,
               q_scale, maxp, out);
    return ZLM_OK;
}

// R sequences in maxp pieces each (1: whole)
extern "C" int zlm_linear_attention_fits(int R, int H, int D, int V, int maxp) {
    return (long long)R * H * maxp <= 2147483647LL && (long long)R * H * D <= 2147483647LL && (V + 127) / 128 <= 65535;
}

// A step of R sequences of up to `longest` tokens: by columns, or four columns a thread?  By columns from so many blocks on, where no
// sequence brings more than three tokens: with more of them the arithmetic counts, with fewer blocks the depth of a thread's chain does.  Us by
// columns / with four a thread, 8 heads, one token a sequence: 64 x 128, 8 sequences 4.6 / 4.3, 16 5.5 / 5.7, 64 7.1 / 7.8; 128 x
// 128, 4 sequences 7.3 / 5.1, 16 8.8 / 11.0, 64 16 / 22; 32 x 128, 64 sequences 4 to 5, a fifth less with four, 96 a fifth more.
// Heads of up to 64 columns leave half of a block of columns idle (64 x 64, 80 sequences 9.7 / 9.1).
extern "C" int zlm_linear_attention_by_columns(int longest, int R, int H, int D, int V) {
    const long long blocks = (long long)R * H * ((V + 127) / 128);
    return longest <= 3 && blocks >= (D <= 32 ? 600 : D <= 64 ? 112 : 64) && (V > 64 || D <= 32 || D > 64);
}

// q, k [H*D], v [H*V]: columns of proj from q_off, k_off, v_off on (element type); alpha [T][H*D] fp32 decays per token
// and key channel, or null with head_decay [H] fp32 (one decay a head); state [slots][H][D][V] fp32; o [T][H*V] fp32.
// pieces: null, or R * ceil(max_new / 32) * H * D * (V + 1) floats: sequences run in pieces of 32 tokens side by side
// (a walk of every piece, a chain of their states, a product that adds what the state ahead of a piece gives).
// y (null: none; with pieces, V <= 128): [T][y_stride] in the element type receives every head of o divided by its root mean
// square, times w [V], times silu (act 1) or sigmoid (0) of g [T][g_stride]; o is then scratch.
extern "C" int zlm_linear_attention(float* o, const void* proj, int proj_stride, int q_off, int k_off, int v_off,
                                    const float* alpha, const float* head_decay, float* state, int dtype, const int* seq_slot,
                                    const int* cu_seqlens, int T, int R, int H, int D, int V, float q_scale, int max_new,
                                    float* pieces, void* y, int y_stride, const void* g, int g_stride, const void* w, int w_dtype,
                                    float eps, int act, cudaStream_t st) {
    if (T == 0) return ZLM_OK;
    ZLM_REQUIRE(H > 0 && D > 0 && V > 0 && D <= 128, "linear_attention: %d heads of %d key and %d value columns (keys up to 128)", H, D, V);
    ZLM_REQUIRE(alpha || head_decay, "linear_attention: neither decays per channel nor per head");
    ZLM_REQUIRE(!pieces || max_new > 0, "linear_attention: pieces without the longest sequence");
    ZLM_REQUIRE(!y || (pieces && V <= 128 && g && w), "linear_attention: heads of %d columns do not take their gate along", V);
    const int L = LA_PIECE, maxp = pieces ? (max_new + L - 1) / L : 1;
    ZLM_REQUIRE(zlm_linear_attention_fits(R, H, D, V, maxp), "linear_attention: too many sequences or columns");
    const dim3 pgrid(R * maxp * H, (V + 127) / 128);
    float* part = pieces;
    float* pdecay = pieces ? pieces + (size_t)R * maxp * H * D * V : nullptr;
    const LaOut out{y, y_stride, g, g_stride, VecW{w, w_dtype}, eps, act};
    int rc = ZLM_OK;
    // a grid's second dimension ends at 65,535.  Heads with more blocks of 64 columns, or more blocks of the chain, than that (four
    // million columns, or 33 million numbers of state) walk by columns whatever their tokens: one head fills the GPU.  (Carrying on
    // in the third dimension cost every walk 5 to 25 %: the column's range is no longer known to the compiler.)
    const bool wide = (D > 64 && (V + 63) / 64 > 65535) || (pieces && (D * V + (V % 4 ? 127 : 511)) / (V % 4 ? 128 : 512) > 65535);
    const bool columns = wide || (!pieces && zlm_linear_attention_by_columns(max_new > 0 ? max_new : T, R, H, D, V));
#define ZLM_LA(TA, DR, SP, MODE, G)                                                                                            \
    zlm_launch(linear_attention_kernel<TA, DR, SP, MODE>, dim3(G, (V + 512 * SP / DR - 1) / (512 * SP / DR)), dim3(128), 0, st, o, (const TA*)proj, proj_stride, q_off, k_off, v_off, \
               alpha, head_decay, state, seq_slot, cu_seqlens, H, D, V, q_scale, part, pdecay, maxp, L)
#define ZLM_LA_RUN(TA, DR, SP)                                                                                              \
    do {                                                                                                                   \
        if (columns) {                                                                                                      \
            zlm_launch(linear_attention_columns_kernel<TA, DR, SP>, dim3(R * H, (V + 127) / 128), dim3(128), 0, st, o, (const TA*)proj,  \
                       proj_stride, q_off, k_off, v_off, alpha, head_decay, state, seq_slot, cu_seqlens, H, D, V, q_scale); \
            break;                                                                                                          \
        }                                                                                                                   \
        if (!pieces) { ZLM_LA(TA, DR, SP, 0, R * H); break; }                                                               \
        ZLM_LA(TA, DR, SP, 1, R * maxp * H);                                                                                      \
        if (V % 4 == 0 && (uintptr_t)state % 16 == 0 && (uintptr_t)part % 16 == 0)                                         \
            zlm_launch(linear_attention_chain_kernel<4>, dim3(R * H, (D * V + 511) / 512), dim3(128), 0, st, part,         \
                       (const float*)pdecay, state, seq_slot, cu_seqlens, H, D, V, maxp, L);                               \
        else                                                                                                               \
            zlm_launch(linear_attention_chain_kernel<1>, dim3(R * H, (D * V + 127) / 128), dim3(128), 0, st, part,         \
                       (const float*)pdecay, state, seq_slot, cu_seqlens, H, D, V, maxp, L);                               \
        rc = launch_la_out<TA, DR>(pgrid, st, o, proj, proj_stride, q_off, alpha, head_decay, part, cu_seqlens, H, D, V,   \
                                   q_scale, maxp, out);                                                                    \
    } while (0)
#define ZLM_LA_D(TA)                                                                     \
    if (D <= 32) ZLM_LA_RUN(TA, 32, 8); else if (D <= 64) ZLM_LA_RUN(TA, 64, 16); else ZLM_LA_RUN(TA, 128, 16)
    if (dtype == ZLM_DTYPE_F32) {
        ZLM_LA_D(float);
    } else if (dtype == ZLM_DTYPE_BF16) {
        ZLM_LA_D(__nv_bfloat16);
    } else {
        ZLM_REQUIRE(false, "linear_attention: unsupported dtype %d", dtype);
    }
#undef ZLM_LA_D
#undef ZLM_LA_RUN
#undef ZLM_LA
    if (rc) return rc;
    return zlm_check_launch("linear_attention");
}

ZLM_TRANSLATION_UNIT(recurrent)
