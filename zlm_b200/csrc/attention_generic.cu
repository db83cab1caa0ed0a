// Attention of packed query tokens over the paged cache, any head size up to 512,
// fp32 or bf16 storage, fp32 arithmetic.  One block per (query head, token); the
// keys are walked in chunks of 32 that are aligned to absolute positions and
// dealt round-robin to the 4 warps, so the order of every sum depends only on
// the query's own position and window, never on the batch or on how the
// sequence was cut into steps.
// Formula: s_t = (q . k_t) * scale, softmax over t in [t_start, pos],
// o = sum p_t v_t with a running maximum and sum
// (src/kernels/transformer/attention.zig:86-164); kv head = q head / group
// (:104-105); window start: seq = pos + 1, t_start = seq - w if w and seq > w
// (src/runtime/executor.zig:93-98).
// Options: `chunk` (keys of the query's own chunk of that many positions, counted from position 0, only),
// `softcap` (s <- cap * tanh(s / cap) after the scale), `sinks` (one number per query head whose exponential
// joins the softmax's denominator without a value; without the array the flag `sink` stands for a 0), and
// `v_share` (that many neighbouring key heads read one value head: the page is [nkv key heads | nkv / v_share
// value heads] of [ZLM_PAGE][hd] each), `keep` (with a window: the sequence's first `keep` keys stay visible) and `bias`
// (bias_n numbers a head, added after the cap by distance, the last one for all greater distances; attn_common.cuh).
#include "common.cuh"
#include "attn_common.cuh"

#define ATT_WARPS 4
#define ATT_MAX_PER_LANE 16   // head_dim <= 512

template <typename TA>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attention_generic_kernel(TA* __restrict__ out, int out_stride, const TA* __restrict__ q,
                         int q_stride, const TA* __restrict__ pool,
                         const int* __restrict__ block_table, int table_stride,
                         const int* __restrict__ token_pos, const int* __restrict__ token_slot,
                         int nq, int nkv, int hd, float scale, int window, int sink, int chunk, float softcap,
                         const float* __restrict__ sinks, int v_share, int keep, const float* __restrict__ bias, int bias_n) {
    extern __shared__ float sm[];
    float* qs = sm;                         // [hd]
    float* accs = sm + hd;                  // [ATT_WARPS][hd]
    __shared__ float ms[ATT_WARPS], ls[ATT_WARPS];

    const int t = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kvh = h / (nq / nkv);
    if (!ZLM_CHK(token_pos + t, 4) || !ZLM_CHK(token_slot + t, 4)) return;
    const int pos = token_pos[t];
    const int slot = token_slot[t];
    const int seq = pos + 1;
    int t_start = (window != 0 && seq > window) ? seq - window : 0;
    if (chunk > 0) t_start = max(t_start, pos - pos % chunk);
    const int* pages = block_table + (size_t)slot * table_stride;
    const size_t page_stride = (size_t)(nkv + nkv / v_share) * ZLM_PAGE * hd;
    const size_t v_off = (size_t)(nkv - kvh + kvh / v_share) * ZLM_PAGE * hd;       // from this key head to its value head

    const TA* qp = q + (size_t)t * q_stride + (size_t)h * hd;
    if (!ZLM_CHK(qp, (size_t)hd * sizeof(TA)) ||
        !ZLM_CHK(out + (size_t)t * out_stride + (size_t)h * hd, (size_t)hd * sizeof(TA)))
        return;
    for (int e = threadIdx.x; e < hd; e += blockDim.x) qs[e] = to_f32(qp[e]);
    __syncthreads();

    float m = -INFINITY, l = 0.f;
    if (sink && warp == 0) {      // one more term in the sum, without a value: exp(sinks[h]), or exp(0)
        m = (sinks && ZLM_CHK(sinks + h, 4)) ? sinks[h] : 0.f;
        l = 1.f;
    }
    float acc[ATT_MAX_PER_LANE];
#pragma unroll
    for (int r = 0; r < ATT_MAX_PER_LANE; ++r) acc[r] = 0.f;

    const int c0 = t_start / 32, c1 = pos / 32;
    const int kept = keep > 0 ? min((keep - 1) / 32 + 1, c0) : 0;         // chunks of the first kept keys ahead of the window's
    const float* brow = attn_bias_row(AttnOpts{chunk, softcap, sinks, v_share, keep, bias, bias_n}, h);
    for (int c = warp; c <= c1; c += ATT_WARPS) {
        // chunk c holds keys [32c, 32c+32); chunk c belongs to warp c % ATT_WARPS
        if (c >= kept && c < c0) {                 // between the kept keys and the window: on to this warp's first chunk there
            c = c0 + ((warp - c0 % ATT_WARPS + ATT_WARPS) % ATT_WARPS);
            if (c > c1) break;
        }
        const int key = c * 32 + lane;
        const bool valid = attn_sees(key, pos, t_start, keep);
        if (!ZLM_CHK(pages + (c * 32) / ZLM_PAGE, 4)) continue;
        const int page = pages[(c * 32) / ZLM_PAGE];
        const TA* kbase = pool + (size_t)page * page_stride + (size_t)kvh * ZLM_PAGE * hd;
        // this head's 64 keys and 64 values of the page
        if (!ZLM_CHK(kbase, (size_t)ZLM_PAGE * hd * sizeof(TA)) || !ZLM_CHK(kbase + v_off, (size_t)ZLM_PAGE * hd * sizeof(TA)))
            continue;
        float s = -INFINITY;
        if (valid) {
            const TA* kr = kbase + (size_t)(key % ZLM_PAGE) * hd;
            float d = 0.f;
            for (int e = 0; e < hd; ++e) d = fmaf(qs[e], to_f32(kr[e]), d);
            s = __fmul_rn(d, scale);
            if (softcap > 0.f) s = softcap * tanhf(s / softcap);
            if (brow) s += attn_bias_at(brow, min(pos - key, bias_n - 1));
        }
        const float cm = warp_max(s);          // the chunk holds at least one valid key
        const float mn = fmaxf(m, cm);
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - mn);
        const float p = valid ? expf(s - mn) : 0.f;
        l = fmaf(l, alpha, warp_sum(p));
        m = mn;
#pragma unroll
        for (int r = 0; r < ATT_MAX_PER_LANE; ++r) acc[r] *= alpha;
        const TA* vbase = kbase + v_off;
        const int nvalid_hi = min(31, pos - c * 32);
        const int lo = keep > 0 ? 0 : max(0, t_start - c * 32);
        for (int jk = lo; jk <= nvalid_hi; ++jk) {
            const float pj = __shfl_sync(0xffffffffu, p, jk);
            if (keep > 0 && !attn_sees(c * 32 + jk, pos, t_start, keep)) continue;
            const TA* vr = vbase + (size_t)((c * 32 + jk) % ZLM_PAGE) * hd;
#pragma unroll
            for (int r = 0; r < ATT_MAX_PER_LANE; ++r) {
                const int e = lane + 32 * r;
                if (e < hd) acc[r] = fmaf(pj, to_f32(vr[e]), acc[r]);
            }
        }
    }
    if (lane == 0) { ms[warp] = m; ls[warp] = l; }
#pragma unroll
    for (int r = 0; r < ATT_MAX_PER_LANE; ++r) {
        const int e = lane + 32 * r;
        if (e < hd) accs[warp * hd + e] = acc[r];
    }
    __syncthreads();
    // merge the warps in the fixed order 0..3
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) M = fmaxf(M, ms[w]);
    float L = 0.f;
    float f[ATT_WARPS];
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) {
        f[w] = (ms[w] == -INFINITY) ? 0.f : expf(ms[w] - M);
        L = fmaf(ls[w], f[w], L);
    }
    const float invL = 1.0f / L;
    TA* op = out + (size_t)t * out_stride + (size_t)h * hd;
    for (int e = threadIdx.x; e < hd; e += blockDim.x) {
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) o = fmaf(accs[w * hd + e], f[w], o);
        op[e] = from_f32<TA>(__fmul_rn(o, invL));
    }
}

extern "C" int zlm_attention_generic(void* out, int out_stride, const void* q, int q_stride,
                                     int dtype, const void* pool, const int* block_table,
                                     int table_stride, const int* token_pos,
                                     const int* token_slot, int T, int nq, int nkv, int hd,
                                     float scale, int window, int sink, int chunk, float softcap,
                                     const float* sinks, int v_share, int keep, const float* bias, int bias_n, cudaStream_t st) {
    if (T == 0) return ZLM_OK;
    ZLM_REQUIRE_ATTN_OPTS("attention");
    ZLM_REQUIRE(hd > 0 && hd <= 32 * ATT_MAX_PER_LANE, "attention: head_dim=%d must be at most %d", hd,
                32 * ATT_MAX_PER_LANE);
    ZLM_REQUIRE(nq > 0 && nkv > 0 && nq % nkv == 0, "attention: %d query heads over %d kv heads", nq, nkv);
    ZLM_REQUIRE(window >= 0, "attention: window=%d", window);
    ZLM_REQUIRE(nq <= 65535, "attention: more than 65535 query heads");
    dim3 grid(T, nq);
    const size_t smem = (size_t)(1 + ATT_WARPS) * hd * sizeof(float);
    zlm_count_launch();
    if (dtype == ZLM_DTYPE_F32)
        attention_generic_kernel<float><<<grid, ATT_WARPS * 32, smem, st>>>(
            (float*)out, out_stride, (const float*)q, q_stride, (const float*)pool, block_table,
            table_stride, token_pos, token_slot, nq, nkv, hd, scale, window, sink, chunk, softcap, sinks, v_share, keep, bias, bias_n);
    else if (dtype == ZLM_DTYPE_BF16)
        attention_generic_kernel<__nv_bfloat16><<<grid, ATT_WARPS * 32, smem, st>>>(
            (__nv_bfloat16*)out, out_stride, (const __nv_bfloat16*)q, q_stride,
            (const __nv_bfloat16*)pool, block_table, table_stride, token_pos, token_slot, nq, nkv,
            hd, scale, window, sink, chunk, softcap, sinks, v_share, keep, bias, bias_n);
    else
        ZLM_REQUIRE(false, "attention: unsupported dtype %d", dtype);
    return zlm_check_launch("attention_generic");
}

// ---------------------------------------------------------------------------- many tokens of a sequence, 32-bit
// The same attention over tiles of 32 queries of one sequence and head: the keys and values of a chunk are read from
// memory once for 32 queries instead of once for each, and the dot products run as register tiles.  Bit for bit what the
// kernel above computes: a score is the same ascending chain of FMAs, chunk c belongs to the (c % 4)-th of four running
// softmaxes (here a group of 64 threads each, there a warp), the sum over a chunk's 32 weights is the same tree, and the
// four are merged in the same order; so a token's result still depends on nothing but its own sequence.  (Every product
// that is followed by a sum is written as fmaf or as a rounded product in both kernels: nothing is left to contraction.)
// Bound by shared-memory reads (4 x 4 scores a thread: 8 reads of 16 bytes for 64 FMAs) and the FFMA pipe.  509 queries
// behind 515 cached tokens, 16 heads of 128: 3,498 us a query a block (every query reads all its keys from L2, a row a
// lane), 132 us here (two blocks an SM leave heads of 96 and 128 with 150 to 160 bytes of spills).
#define AT_Q 32                  // queries of a block
#define AT_GROUPS ATT_WARPS      // running softmaxes, a group of threads each
#define AT_GT 64                 // threads of a group
template <bool B> struct AtBool { static constexpr bool value = B; };
__device__ __forceinline__ void at_group_sync(int group) { asm volatile("bar.sync %0, %1;\n" ::"r"(group + 1), "r"(AT_GT) : "memory"); }

template <int HD>
__global__ void __launch_bounds__(AT_GROUPS * AT_GT, 2)
attention_f32_tile_kernel(float* __restrict__ out, int out_stride, const float* __restrict__ q, int q_stride,
                          const float* __restrict__ pool, const int* __restrict__ block_table, int table_stride,
                          const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                          int nq, int nkv, float scale, int window, int sink, int chunk, const float* __restrict__ sinks) {
    constexpr int LD = HD + 4;             // rows 16 bytes apart modulo the banks: eight neighbouring rows meet no bank twice
    constexpr int PLD = AT_Q + 4;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                         // [AT_Q][LD]
    float* kv = qs + AT_Q * LD;                             // [AT_GROUPS][32][LD]: a chunk's keys, then its values
    float* ps = kv + AT_GROUPS * 32 * LD;                   // [AT_GROUPS][32 keys][PLD queries]
    __shared__ float al[AT_GROUPS][AT_Q], ms[AT_GROUPS][AT_Q], ls[AT_GROUPS][AT_Q];
    const int h = blockIdx.x, r = blockIdx.z, tid = threadIdx.x;
    const int t0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * AT_Q;          // the tiles with the most keys first
    if (!ZLM_CHK(cu_seqlens + r, 8) || !ZLM_CHK(seq_slot + r, 4) || !ZLM_CHK(seq_start + r, 4)) return;
    const int row0 = cu_seqlens[r] + t0, rows = min(AT_Q, cu_seqlens[r + 1] - row0);
    if (rows <= 0) return;
    const int pos0 = seq_start[r] + t0, last = pos0 + rows - 1;
    const int kvh = h / (nq / nkv);
    const int* pages = block_table + (size_t)seq_slot[r] * table_stride;
    const size_t page_stride = (size_t)2 * nkv * ZLM_PAGE * HD, v_off = (size_t)nkv * ZLM_PAGE * HD;
    for (int x = tid; x < AT_Q * (HD / 4); x += AT_GROUPS * AT_GT) {
        const int i = x / (HD / 4), e = (x % (HD / 4)) * 4;
        const float* p = q + (size_t)(row0 + i) * q_stride + (size_t)h * HD + e;
        *(float4*)(qs + i * LD + e) = (i < rows && ZLM_CHK(p, 16)) ? *(const float4*)p : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const int g = tid / AT_GT, gt = tid % AT_GT;
    float* kg = kv + g * 32 * LD;
    float* pg = ps + g * 32 * PLD;
    // scores: queries qi + 8 i and keys ki + 8 j of the chunk; values: queries 8 vq + i, columns 4 ve + 64 x ..
    const int qi = gt >> 3, ki = gt & 7, vq = gt >> 4, ve = gt & 15;
    constexpr int VX = (HD + 63) / 64;
    float m[4], l[4], acc[8][VX][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
        if (sink && g == 0) {
            m[i] = (sinks && ZLM_CHK(sinks + h, 4)) ? sinks[h] : 0.f;
            l[i] = 1.f;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int x = 0; x < VX; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][x][e] = 0.f;
    const int c_lo = attn_first_key(pos0, window, chunk) / 32, c_hi = last / 32;
    for (int c = c_lo + ((g - c_lo % AT_GROUPS + AT_GROUPS) % AT_GROUPS); c <= c_hi; c += AT_GROUPS) {
        if (!ZLM_CHK(pages + (c * 32) / ZLM_PAGE, 4)) break;
        const float* kbase = pool + (size_t)pages[(c * 32) / ZLM_PAGE] * page_stride + ((size_t)kvh * ZLM_PAGE + (c * 32) % ZLM_PAGE) * HD;
        auto stage = [&](const float* src) {
#pragma unroll
            for (int x = gt; x < 32 * (HD / 4); x += AT_GT) dec_cp_async16(kg + x / (HD / 4) * LD + (x % (HD / 4)) * 4, src + x * 4);
            dec_commit();
        };
        stage(kbase);
        dec_wait<0>();
        at_group_sync(g);
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int e = 0; e < HD; e += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *(const float4*)(qs + (qi + 8 * i) * LD + e);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *(const float4*)(kg + (ki + 8 * j) * LD + e);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
        }
        at_group_sync(g);                          // the keys are read: the values take their place
        stage(kbase + v_off);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + qi + 8 * i, lo = attn_first_key(pos, window, chunk);
            bool sees[4];
            float cm = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = c * 32 + ki + 8 * j;
                sees[j] = key <= pos && key >= lo;
                s[i][j] = sees[j] ? __fmul_rn(s[i][j], scale) : -INFINITY;
                cm = fmaxf(cm, s[i][j]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
            const float mn = fmaxf(m[i], cm);
            const float alpha = (m[i] == -INFINITY) ? 0.f : expf(m[i] - mn);
            float p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = sees[j] ? expf(s[i][j] - mn) : 0.f;
            // the tree of warp_sum over the chunk's 32 keys: keys 16 apart, then 8 (both in this thread), then 4, 2, 1
            float sum = (p[0] + p[2]) + (p[1] + p[3]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            // (a query that sees no key of the chunk keeps its sums to the bit: alpha is 1, or they are zero)
            l[i] = fmaf(l[i], alpha, sum);
            m[i] = mn;
#pragma unroll
            for (int j = 0; j < 4; ++j) pg[(ki + 8 * j) * PLD + qi + 8 * i] = p[j];
            if (ki == 0) al[g][qi + 8 * i] = alpha;
        }
        dec_wait<0>();
        at_group_sync(g);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float alpha = al[g][vq * 8 + i];
#pragma unroll
            for (int x = 0; x < VX; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][x][e] *= alpha;
        }
        const bool whole = c * 32 + 31 <= pos0 && c * 32 >= attn_first_key(last, window, chunk);
        // (a key that a query does not see takes no part, whatever its value is: not even as zero times it)
        unsigned see[8];
        if (!whole) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int pos = pos0 + vq * 8 + i, hi = pos - c * 32, lo = attn_first_key(pos, window, chunk) - c * 32;
                see[i] = hi < 0 || lo > 31 ? 0u : (hi >= 31 ? 0xffffffffu : (2u << hi) - 1u) & (lo <= 0 ? 0xffffffffu : ~((1u << lo) - 1u));
            }
        }
        auto values = [&](auto all) {
#pragma unroll 4
            for (int j = 0; j < 32; ++j) {
                const float4 pa = *(const float4*)(pg + j * PLD + vq * 8), pb = *(const float4*)(pg + j * PLD + vq * 8 + 4);
                const float p[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
#pragma unroll
                for (int x = 0; x < VX; ++x) {
                    if (HD % 64 != 0 && ve * 4 + 64 * x >= HD) continue;
                    const float4 v = *(const float4*)(kg + j * LD + ve * 4 + 64 * x);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (!decltype(all)::value && !(see[i] >> j & 1u)) continue;
                        acc[i][x][0] = fmaf(p[i], v.x, acc[i][x][0]);
                        acc[i][x][1] = fmaf(p[i], v.y, acc[i][x][1]);
                        acc[i][x][2] = fmaf(p[i], v.z, acc[i][x][2]);
                        acc[i][x][3] = fmaf(p[i], v.w, acc[i][x][3]);
                    }
                }
            }
        };
        if (whole) values(AtBool<true>()); else values(AtBool<false>());
        at_group_sync(g);
    }
    // merge the groups in the fixed order 0..3 (their sums through the chunks' buffers)
    if (ki == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { ms[g][qi + 8 * i] = m[i]; ls[g][qi + 8 * i] = l[i]; }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int x = 0; x < VX; ++x)
            if (HD % 64 == 0 || ve * 4 + 64 * x < HD)
                *(float4*)(kg + (vq * 8 + i) * LD + ve * 4 + 64 * x) = make_float4(acc[i][x][0], acc[i][x][1], acc[i][x][2], acc[i][x][3]);
    __syncthreads();
    for (int x = tid; x < rows * (HD / 4); x += AT_GROUPS * AT_GT) {
        const int i = x / (HD / 4), e = (x % (HD / 4)) * 4;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < AT_GROUPS; ++w) M = fmaxf(M, ms[w][i]);
        float L = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < AT_GROUPS; ++w) {
            const float f = (ms[w][i] == -INFINITY) ? 0.f : expf(ms[w][i] - M);
            L = fmaf(ls[w][i], f, L);
            const float4 a = *(const float4*)(kv + (w * 32 + i) * LD + e);
            o[0] = fmaf(a.x, f, o[0]);
            o[1] = fmaf(a.y, f, o[1]);
            o[2] = fmaf(a.z, f, o[2]);
            o[3] = fmaf(a.w, f, o[3]);
        }
        const float inv = 1.0f / L;
        float* op = out + (size_t)(row0 + i) * out_stride + (size_t)h * HD + e;
        if (ZLM_CHK(op, 16))
            *(float4*)op = make_float4(__fmul_rn(o[0], inv), __fmul_rn(o[1], inv), __fmul_rn(o[2], inv), __fmul_rn(o[3], inv));
    }
}

// head sizes that the tile kernel is built for, and rows it can read 16 bytes at a time; no cap, no bias, no kept first
// keys, every key head with its own value head (the kernel above takes those, and everything else)
extern "C" int zlm_attention_f32_tile_supported(int nq, int nkv, int hd, int q_stride, int out_stride, float softcap, int v_share,
                                                int keep, int has_bias, int R, int max_new) {
    // (a grid's second and third dimension end at 65,535: two million tokens of one sequence, and as many sequences)
    if (R > 65535 || (max_new - 1) / AT_Q >= 65535) return 0;
    return (hd == 64 || hd == 96 || hd == 128) && nq > 0 && nkv > 0 && nq % nkv == 0 && q_stride % 4 == 0 && out_stride % 4 == 0 &&
           softcap == 0.f && v_share == 1 && keep == 0 && !has_bias;
}

template <int HD>
static int launch_f32_tile(dim3 grid, cudaStream_t st, float* out, int out_stride, const float* q, int q_stride, const float* pool,
                           const int* block_table, int table_stride, const int* cu_seqlens, const int* seq_slot, const int* seq_start,
                           int nq, int nkv, float scale, int window, int sink, int chunk, const float* sinks) {
    const size_t smem = (size_t)(AT_Q * (HD + 4) + AT_GROUPS * 32 * (HD + 4) + AT_GROUPS * 32 * (AT_Q + 4)) * sizeof(float);
    static bool attr_set_dev[64] = {};
    bool& attr_set = attr_set_dev[zlm_device_index()];
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(attention_f32_tile_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            zlm_set_error("attention: cannot reserve shared memory: %s", cudaGetErrorString(e));
            return ZLM_ERR_CUDA;
        }
        attr_set = true;
    }
    zlm_count_launch();
    attention_f32_tile_kernel<HD><<<grid, AT_GROUPS * AT_GT, smem, st>>>(out, out_stride, q, q_stride, pool, block_table, table_stride,
                                                                        cu_seqlens, seq_slot, seq_start, nq, nkv, scale, window, sink,
                                                                        chunk, sinks);
    return zlm_check_launch("attention_f32_tile");
}

extern "C" int zlm_attention_f32_tile(float* out, int out_stride, const float* q, int q_stride, const float* pool,
                                      const int* block_table, int table_stride, const int* cu_seqlens, const int* seq_slot,
                                      const int* seq_start, int R, int max_new, int nq, int nkv, int hd, float scale, int window,
                                      int sink, int chunk, const float* sinks, cudaStream_t st) {
    if (R == 0 || max_new == 0) return ZLM_OK;
    ZLM_REQUIRE(zlm_attention_f32_tile_supported(nq, nkv, hd, q_stride, out_stride, 0.f, 1, 0, 0, R, max_new) && (uintptr_t)q % 16 == 0 &&
                    (uintptr_t)out % 16 == 0 && (uintptr_t)pool % 16 == 0,
                "attention: %d query heads over %d kv heads of %d, rows of %d and %d floats, %d sequences of up to %d tokens", nq, nkv, hd,
                q_stride, out_stride, R, max_new);
    ZLM_REQUIRE(window >= 0 && chunk >= 0, "attention: window=%d, chunk=%d", window, chunk);
    const dim3 grid(nq, (max_new + AT_Q - 1) / AT_Q, R);
#define ZLM_AT(HD) launch_f32_tile<HD>(grid, st, out, out_stride, q, q_stride, pool, block_table, table_stride, cu_seqlens, seq_slot, \
                                       seq_start, nq, nkv, scale, window, sink, chunk, sinks)
    return hd == 64 ? ZLM_AT(64) : hd == 96 ? ZLM_AT(96) : ZLM_AT(128);
#undef ZLM_AT
}

ZLM_TRANSLATION_UNIT(attention_generic)
