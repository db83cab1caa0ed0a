// Retention: linear attention with one fixed decay per head, no softmax and no denominator.
//
//   q_t, k_t = rot(q_t), rot(k_t) * k_scale      rotation of the first n_rot coordinates of a head, coordinate i
//                                                with i + n_rot/2, by the angle pos * inv_freq[i]
//   S_t = decay_h * S_(t-1) + k_t v_t^T          [dim][vdim] per head and sequence, fp32, kept in the sequence's state
//   o_t = S_t^T q_t                              fp32
//
// q, k, v are columns of one fused projection [T][ld] in the compute element type; everything after the
// projection (angles, rotated q and k, the decay, the state, o) is fp32 in both element types.
//
// The columns of the state are independent: a thread holds DPT rows of four columns in registers, the `ds`
// threads that share the columns are neighbouring lanes and add their parts of o by shuffles.  A block takes
// 4 * 128 / ds columns of one head of one sequence and walks the sequence's tokens in order, RT_CHUNK at a time:
// the chunk's rotated q and k and its v columns are staged in shared memory by the whole block.
//
// Long prompts, three kernels (retention_parts): the sequence is cut into pieces of `piece` tokens; in bfloat16 with heads of up
// to 128 rotated coordinates as products on the tensor cores (further down), otherwise
//   1. every piece runs the recurrence from a zero state (the same code): its local outputs, and the state
//      it would leave, A_c
//   2. the pieces' states are chained: S_c = decay^len_c * S_(c-1) + A_c   (S_(-1) is the sequence's state)
//   3. every piece adds what the state before it contributes: o_t += decay^(t - t0 + 1) * S_(c-1)^T q_t
// so that the pieces run side by side; the sums are the same up to their order.
#include "split_mma.cuh"

#define RT_THREADS 128
#define RT_CHUNK 64          // tokens staged at a time, at most (a piece of a long prompt)

// MODE 0: the whole recurrence from the sequence's state (reads and writes `state`).
// MODE 1: a piece from a zero state; its final state goes to part_state [pieces][H][D][V].
// MODE 2: o += decay^(j+1) * S_before^T q for a piece, S_before from chain [pieces][H][D][V] (the state before piece c).
//
// A thread holds a tile of DPT rows x RT_CPT columns of the state, so that a staged q or k value is used for
// RT_CPT columns and a v value for DPT rows (one column a thread had every thread read all of q and k from shared
// memory for every token, and the shared-memory pipe, not the arithmetic, set the time).  The `ds` threads that
// share a tile's columns are neighbouring lanes; their segments of a staged row lie DPT + 4 floats apart, so that
// their 16-byte reads fall into different banks.
#define RT_CPT 4
template <typename TA, int DPT, int MODE>
__global__ void __launch_bounds__(RT_THREADS)
retention_kernel(float* __restrict__ o, const TA* __restrict__ proj, int ld, int q_off, int k_off, int v_off,
                 const float* __restrict__ inv_freq, int n_rot, const float* __restrict__ decay, float* __restrict__ state,
                 const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                 int maxp, int piece, int H, int D, int V,
                 int ds, float k_scale, const float* __restrict__ table, int T, int chunk) {
    extern __shared__ __align__(16) float sm[];
    const int DP = ds * (DPT + 4);           // a staged row: ds segments of DPT values, 4 floats of padding after each
    float* qs = sm;                          // [chunk][DP]
    float* ks = qs + chunk * DP;             // [chunk][DP]
    const int cols = RT_THREADS / ds * RT_CPT;
    float* vs = ks + chunk * DP;             // [chunk][cols]
    pdl_launch_dependents();
    const int tid = threadIdx.x, h = blockIdx.y;
    const int grp = tid / ds, part = tid % ds;
    const int col0 = blockIdx.x * cols + grp * RT_CPT;
    pdl_wait();
    int r, first, n;                          // sequence, first token of this block's run within the step, tokens
    if (MODE == 0) {
        r = blockIdx.z;
        first = 0;
        n = cu_seqlens[r + 1] - cu_seqlens[r];
    } else {
        // piece blockIdx.z % maxp of sequence blockIdx.z / maxp (maxp: the pieces of the step's longest sequence)
        r = blockIdx.z / maxp;
        first = (blockIdx.z % maxp) * piece;
        n = min(piece, cu_seqlens[r + 1] - cu_seqlens[r] - first);
        if (n <= 0) return;
    }
    const int row0 = cu_seqlens[r] + first, pos0 = seq_start[r] + first;
    const float d = decay[h];
    // the tile, two neighbouring rows a register pair (packed fp32 arithmetic: the pairs of q and k come straight
    // from their 16-byte reads)
    float2 S[DPT / 2][RT_CPT];
    float* sp = nullptr;
    if (MODE == 0) sp = state + ((size_t)seq_slot[r] * H + h) * D * V;
    else sp = state + ((size_t)blockIdx.z * H + h) * D * V;       // MODE 1: part_state (written); MODE 2: chain (read)
    const bool v4 = (V & 3) == 0 && col0 + RT_CPT <= V;             // the tile's columns as one 16-byte access
#pragma unroll
    for (int jj = 0; jj < DPT / 2; ++jj) {
        float t[2][RT_CPT];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = part * DPT + 2 * jj + e;
#pragma unroll
            for (int c = 0; c < RT_CPT; ++c) t[e][c] = 0.f;
            if (MODE == 1 || i >= D) continue;
            const float* src = sp + (size_t)i * V + col0;
            if (v4 && ZLM_CHK(src, 16)) {
                const float4 a = *(const float4*)src;
                t[e][0] = a.x; t[e][1] = a.y; t[e][2] = a.z; t[e][3] = a.w;
            } else {
#pragma unroll
                for (int c = 0; c < RT_CPT; ++c)
                    if (col0 + c < V && ZLM_CHK(src + c, 4)) t[e][c] = src[c];
            }
        }
#pragma unroll
        for (int c = 0; c < RT_CPT; ++c) S[jj][c] = make_float2(t[0][c], t[1][c]);
    }
    float dp = d;                              // MODE 2: decay^(j+1)
    const int half = n_rot >> 1;
    for (int c0 = 0; c0 < n; c0 += chunk) {
        const int cn = min(chunk, n - c0);
        __syncthreads();
        // the chunk's q and k, rotated: a thread turns a pair (f, f + half) of a token at a time, so that the pair and
        // its cosine and sine are read once; the loads of several pairs are in flight together
#pragma unroll 8
        for (int idx = tid; idx < cn * half; idx += RT_THREADS) {
            const int tt = idx / half, f = idx % half;
            const int rowi = row0 + c0 + tt;
            const TA* row = proj + (size_t)rowi * ld + (size_t)h * D;
            if (!ZLM_CHK(row + q_off, (size_t)D * sizeof(TA)) || !ZLM_CHK(row + k_off, (size_t)D * sizeof(TA))) continue;
            float sn, cs;
            if (table) {
                cs = table[(size_t)f * T + rowi];
                sn = table[(size_t)(half + f) * T + rowi];
            } else {
                sincosf((float)(pos0 + c0 + tt) * inv_freq[f], &sn, &cs);
            }
            const int i1 = f + half;
            const int a0 = tt * DP + (f / DPT) * (DPT + 4) + f % DPT, a1 = tt * DP + (i1 / DPT) * (DPT + 4) + i1 % DPT;
            const float qu = to_f32(row[q_off + f]), qv = to_f32(row[q_off + i1]);
            qs[a0] = qu * cs - qv * sn;
            qs[a1] = qv * cs + qu * sn;
            if (MODE != 2) {
                const float ku = to_f32(row[k_off + f]), kv = to_f32(row[k_off + i1]);
                ks[a0] = (ku * cs - kv * sn) * k_scale;
                ks[a1] = (kv * cs + ku * sn) * k_scale;
            }
        }
        // what lies beyond the rotated coordinates passes as it is
#pragma unroll 4
        for (int idx = tid; idx < cn * (D - n_rot); idx += RT_THREADS) {
            const int tt = idx / (D - n_rot), i = n_rot + idx % (D - n_rot);
            const TA* row = proj + (size_t)(row0 + c0 + tt) * ld + (size_t)h * D;
            if (!ZLM_CHK(row + q_off + i, sizeof(TA)) || !ZLM_CHK(row + k_off + i, sizeof(TA))) continue;
            const int at = tt * DP + (i / DPT) * (DPT + 4) + i % DPT;
            qs[at] = to_f32(row[q_off + i]);
            if (MODE != 2) ks[at] = to_f32(row[k_off + i]) * k_scale;
        }
        // rows of the tiles beyond the head's own stay zero: the walk below asks no row whether it exists
        for (int idx = tid; idx < cn * (ds * DPT - D); idx += RT_THREADS) {
            const int tt = idx / (ds * DPT - D), i = D + idx % (ds * DPT - D);
            const int at = tt * DP + (i / DPT) * (DPT + 4) + i % DPT;
            qs[at] = 0.f;
            ks[at] = 0.f;
        }
        if (MODE != 2) {
#pragma unroll 8
            for (int idx = tid; idx < cn * cols; idx += RT_THREADS) {
                const int tt = idx / cols, cc = idx % cols, gc = blockIdx.x * cols + cc;
                const TA* vp = proj + (size_t)(row0 + c0 + tt) * ld + v_off + (size_t)h * V + gc;
                vs[tt * cols + cc] = (gc < V && ZLM_CHK(vp, sizeof(TA))) ? to_f32(*vp) : 0.f;
            }
        } else {
            // the outputs that the pieces' own walks left, to which this pass adds: staged like the values, so that the
            // walk below does not wait for global memory at every token
#pragma unroll 8
            for (int idx = tid; idx < cn * cols; idx += RT_THREADS) {
                const int tt = idx / cols, cc = idx % cols, gc = blockIdx.x * cols + cc;
                const float* op = o + (size_t)(row0 + c0 + tt) * H * V + (size_t)h * V + gc;
                vs[tt * cols + cc] = (gc < V && ZLM_CHK(op, 4)) ? *op : 0.f;
            }
        }
        __syncthreads();
        for (int tt = 0; tt < cn; ++tt) {
            float2 acc2[RT_CPT];
            float2 vv[RT_CPT];
#pragma unroll
            for (int c = 0; c < RT_CPT; ++c) acc2[c] = vv[c] = make_float2(0.f, 0.f);
            const float* qr = qs + tt * DP + part * (DPT + 4);
            const float* kr = ks + tt * DP + part * (DPT + 4);
            if (MODE != 2) {
                const float4 a = *(const float4*)(vs + tt * cols + grp * RT_CPT);
                vv[0] = make_float2(a.x, a.x); vv[1] = make_float2(a.y, a.y);
                vv[2] = make_float2(a.z, a.z); vv[3] = make_float2(a.w, a.w);
            }
            const float2 d2 = make_float2(d, d);
            // S = d S + k v and o += S q, two rows an instruction (each element rounded as fmaf and a product would
            // round it); acc2 holds the sums over a thread's even and odd rows
#pragma unroll
            for (int j = 0; j < DPT; j += 4) {
                const float4 qa = *(const float4*)(qr + j);
                const float2 q2[2] = {make_float2(qa.x, qa.y), make_float2(qa.z, qa.w)};
                float2 k2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                if (MODE != 2) {
                    const float4 ka = *(const float4*)(kr + j);
                    k2[0] = make_float2(ka.x, ka.y);
                    k2[1] = make_float2(ka.z, ka.w);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int c = 0; c < RT_CPT; ++c) {
                        if (MODE != 2) S[j / 2 + e][c] = __ffma2_rn(d2, S[j / 2 + e][c], __fmul2_rn(k2[e], vv[c]));
                        acc2[c] = __ffma2_rn(S[j / 2 + e][c], q2[e], acc2[c]);
                    }
            }
            float acc[RT_CPT];
#pragma unroll
            for (int c = 0; c < RT_CPT; ++c) acc[c] = (acc2[c].x + acc2[c].y) * (MODE == 2 ? dp : 1.0f);
            if (MODE == 2) dp *= d;
            // the ds lanes of a tile add up their parts; while they do, the columns are dealt out among them (half of
            // the lanes go on with columns 0-1, half with 2-3, then one column each), so that the sums cost 4 shuffles
            // where 4 x log2(ds) would be the plain way.  `mine` is the first column a lane ends up with, `have` how many.
            int mine = 0, have = RT_CPT;
            if (ds >= 2) {
                const int off = ds >> 1;
                const bool up = (part & off) != 0;
                const float s0 = up ? acc[0] : acc[2], s1 = up ? acc[1] : acc[3];
                const float r0 = __shfl_xor_sync(0xffffffffu, s0, off), r1 = __shfl_xor_sync(0xffffffffu, s1, off);
                acc[0] = (up ? acc[2] : acc[0]) + r0;
                acc[1] = (up ? acc[3] : acc[1]) + r1;
                mine = up ? 2 : 0;
                have = 2;
            }
            if (ds >= 4) {
                const int off = ds >> 2;
                const bool up = (part & off) != 0;
                const float r0 = __shfl_xor_sync(0xffffffffu, up ? acc[0] : acc[1], off);
                acc[0] = (up ? acc[1] : acc[0]) + r0;
                mine += up ? 1 : 0;
                have = 1;
                for (int o2 = ds >> 3; o2 > 0; o2 >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o2);
            }
            // the lanes whose lower bits are zero write
            const bool writer = ds < 8 || (part & ((ds >> 2) - 1)) == 0;
            float* op = o + (size_t)(row0 + c0 + tt) * H * V + (size_t)h * V + col0 + mine;
            if (writer) {
#pragma unroll
                for (int c = 0; c < RT_CPT; ++c)
                    if (c < have && col0 + mine + c < V && ZLM_CHK(op + c, 4))
                        op[c] = MODE == 2 ? vs[tt * cols + grp * RT_CPT + mine + c] + acc[c] : acc[c];
            }
        }
    }
    if (MODE != 2) {
#pragma unroll
        for (int jj = 0; jj < DPT / 2; ++jj)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = part * DPT + 2 * jj + e;
                if (i >= D) continue;
                float* dst = sp + (size_t)i * V + col0;
                const float t[RT_CPT] = {e ? S[jj][0].y : S[jj][0].x, e ? S[jj][1].y : S[jj][1].x, e ? S[jj][2].y : S[jj][2].x,
                                         e ? S[jj][3].y : S[jj][3].x};
                if (v4 && ZLM_CHK(dst, 16)) {
                    *(float4*)dst = make_float4(t[0], t[1], t[2], t[3]);
                } else {
#pragma unroll
                    for (int c = 0; c < RT_CPT; ++c)
                        if (col0 + c < V && ZLM_CHK(dst + c, 4)) dst[c] = t[c];
                }
            }
    }
}

// ---------------------------------------------------------------------------- the pieces as products on the tensor cores
// bfloat16 projections, heads of up to 128 rotated coordinates: with w_i = decay^i, a piece of n tokens from state S is
//   state    S' = w_n S + sum_l w_(n-1-l) k_l v_l^T                                  one product (keys^T values)
//   outputs  o_j = sum_(l <= j) w_(j-l) (q_j . k_l) v_l + w_(j+1) S^T q_j            scores, weights times values, queries times state
// All of it stays fp32: rotated queries and keys, weights and states are cut into three bfloat16 pieces (split_mma.cuh).
// The token-by-token walk of the same pieces issues two packed FMAs and two shared-memory reads for 8 numbers of the state and
// waits for itself: 303 us with the chain, the heads' norm and gate for 2,048 tokens of 16 heads of 128 x 128, 87 us as products
// (states 22, chain 11, outputs 58 one by one; the tensor pipe 32 % and the issue slots 35 % busy in the outputs, bound by a block's
// phases between barriers at 16 warps an SM; 20 bytes of spills), and no
// further from 64-bit sums (outputs 2.4e-7 of their norm before, 1.7e-7 now; states 2.4e-7 and 2.0e-7).  Pieces of 64 tokens:
// the states of longer ones are fewer, but scores and weights grow with the square.
#define RM_THREADS 256

// rotated and scaled coordinates of the piece's tokens into pieces [SM_L][128] (zeros beyond n tokens and D coordinates): a
// thread turns eight neighbouring pairs (f, f + half) of one token's q and k with the same cosines and sines
struct RmRot {
    const float* inv_freq; const float* table;        // table [2][half][T], or null
    int n_rot, T;
};
template <bool Q>
__device__ __forceinline__ void rm_stage(__nv_bfloat16* qt, __nv_bfloat16* kt, const __nv_bfloat16* q, const __nv_bfloat16* k,
                                         size_t stride, int row0, int pos0, int n, int D, const RmRot& rot, float k_scale,
                                         const float* k_weight, int tid) {
    const int half = rot.n_rot >> 1, pairs = half >> 3, items = (D >> 3) - pairs;       // items: pairs of groups, then single groups
    struct Item { uint4 a[2], b[2]; float cs[8], sn[8]; };
    auto fetch = [&](int x, Item& t) {
        const int l = x % SM_L, it = x / SM_L;
        const bool turn = it < pairs, live = l < n;
        const int f0 = turn ? it * 8 : rot.n_rot + (it - pairs) * 8, f1 = f0 + half;
#pragma unroll
        for (int y = Q ? 0 : 1; y < 2; ++y) {
            const __nv_bfloat16* p = (y ? k : q) + (size_t)l * stride;
            t.a[y] = t.b[y] = make_uint4(0, 0, 0, 0);
            if (live && ZLM_CHK(p + f0, 16)) t.a[y] = *(const uint4*)(p + f0);
            if (turn && live && ZLM_CHK(p + f1, 16)) t.b[y] = *(const uint4*)(p + f1);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            t.cs[e] = 1.f;
            t.sn[e] = 0.f;
            if (!turn || !live) continue;
            if (rot.table) {
                const float* c = rot.table + (size_t)(f0 + e) * rot.T + row0 + l;
                const float* s = c + (size_t)half * rot.T;
                if (ZLM_CHK(c, 4)) t.cs[e] = *c;
                if (ZLM_CHK(s, 4)) t.sn[e] = *s;
            } else {
                if (ZLM_CHK(rot.inv_freq + f0 + e, 4)) sincosf((float)(pos0 + l) * rot.inv_freq[f0 + e], &t.sn[e], &t.cs[e]);
            }
        }
    };
    auto put = [&](int x, const Item& t) {
        const int l = x % SM_L, it = x / SM_L;
        const bool turn = it < pairs;
        const int f0 = turn ? it * 8 : rot.n_rot + (it - pairs) * 8, f1 = f0 + half;
        const float kw = k_scale * (k_weight ? k_weight[l] : 1.f);
#pragma unroll
        for (int y = Q ? 0 : 1; y < 2; ++y) {
            __nv_bfloat16* dst = y ? kt : qt;
            float u[8], v[8], r[8];
            widen8(t.a[y], u);
            widen8(t.b[y], v);
#pragma unroll
            for (int e = 0; e < 8; ++e) r[e] = (turn ? u[e] * t.cs[e] - v[e] * t.sn[e] : u[e]) * (y ? kw : 1.f);
            split8(dst, SM_L * 128, tile_off<128>(l, f0 >> 3), r);
            if (turn) {
#pragma unroll
                for (int e = 0; e < 8; ++e) r[e] = (v[e] * t.cs[e] + u[e] * t.sn[e]) * (y ? kw : 1.f);
                split8(dst, SM_L * 128, tile_off<128>(l, f1 >> 3), r);
            }
        }
    };
    // (two items' loads on their way at a time: the stores into shared memory let no later load past them)
    for (int x = tid; x < items * SM_L; x += 2 * RM_THREADS) {
        Item t0, t1;
        const bool two = x + RM_THREADS < items * SM_L;
        fetch(x, t0);
        if (two) fetch(x + RM_THREADS, t1);
        put(x, t0);
        if (two) put(x + RM_THREADS, t1);
    }
}
// decay^0 .. decay^64, each rounded once
__device__ __forceinline__ void rm_powers(float* pw, float d, int tid) {
    if (tid > SM_L) return;
    double p = 1.0, q = d;
    for (int i = tid; i; i >>= 1, q *= q)
        if (i & 1) p *= q;
    pw[tid] = (float)p;
}

// grid (R * maxp, H, ceil(V / 128))
__global__ void __launch_bounds__(RM_THREADS, 2)
retention_piece_state_kernel(float* __restrict__ part, const __nv_bfloat16* __restrict__ proj, int ld, int k_off, int v_off,
                             RmRot rot, const float* __restrict__ decay, const int* __restrict__ cu_seqlens,
                             const int* __restrict__ seq_start, int maxp, int H, int D, int V, float k_scale) {
    extern __shared__ __align__(128) __nv_bfloat16 rm_smem[];
    __nv_bfloat16* kt = rm_smem;                     // [3][SM_L][128]
    __nv_bfloat16* vt = kt + 3 * SM_L * 128;         // [SM_L][128]
    __shared__ float pw[SM_L + 1], kw[SM_L];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, c0 = blockIdx.z * 128;
    const int r = blockIdx.x / maxp, first = (blockIdx.x % maxp) * SM_L;
    // (ahead of pdl_wait(): the decays are weights, and the step's integer arrays are copied in ahead of its first kernel; no
    // kernel of a step may write them)
    if (!ZLM_CHK(cu_seqlens + r, 8) || !ZLM_CHK(seq_start + r, 4) || !ZLM_CHK(decay + h, 4)) return;
    const int n = min(SM_L, cu_seqlens[r + 1] - cu_seqlens[r] - first);
    if (n <= 0) return;
    rm_powers(pw, decay[h], tid);
    __syncthreads();
    if (tid < SM_L) kw[tid] = tid < n ? pw[n - 1 - tid] : 0.f;
    __syncthreads();
    const int row0 = cu_seqlens[r] + first;
    pdl_wait();
    const __nv_bfloat16* rows = proj + (size_t)row0 * ld;
    sm_stage_values(vt, rows + v_off + (size_t)h * V, ld, n, c0, V, tid);
    rm_stage<false>(nullptr, kt, nullptr, rows + k_off + (size_t)h * D, ld, row0, seq_start[r] + first, n, D, rot, k_scale, kw, tid);
    dec_wait<0>();
    __syncthreads();
    const int d0 = warp * 16;
    if (d0 >= D) return;
#pragma unroll 1
    for (int n0 = 0; n0 < 128 && c0 + n0 < V; n0 += 64) {
        SmSum<8> acc;
        acc.zero();
        sm_piece_state(acc, kt, vt, d0, n0, lane);
        sm_write_state(part + ((size_t)blockIdx.x * H + h) * D * V, acc, d0, c0 + n0, V, lane);
    }
}

// grid (R * maxp, H, ceil(V / 128)); a warp owns 16 queries and 64 value columns
__global__ void __launch_bounds__(RM_THREADS, 2)
retention_piece_out_kernel(SmOut out, const __nv_bfloat16* __restrict__ proj, int ld, int q_off, int k_off, int v_off,
                           RmRot rot, const float* __restrict__ decay, const float* __restrict__ before,
                           const int* __restrict__ cu_seqlens, const int* __restrict__ seq_start, int maxp, int H, int D, int V,
                           float k_scale) {
    extern __shared__ __align__(128) __nv_bfloat16 rm_smem[];
    __nv_bfloat16* qt = rm_smem;                     // [3][SM_L][128]
    __nv_bfloat16* kt = qt + 3 * SM_L * 128;         // [3][SM_L][128], later the weights and the state's rows:
    __nv_bfloat16* pt = kt;                          // [3][SM_L][SM_L]
    __nv_bfloat16* st = pt + 3 * SM_L * SM_L;        // [3][32][128], later the gate's columns
    __nv_bfloat16* vt = kt + 3 * SM_L * 128;         // [SM_L][128]
    __shared__ float pw[SM_L + 1], red[SM_L][2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, c0 = blockIdx.z * 128;
    const int r = blockIdx.x / maxp, first = (blockIdx.x % maxp) * SM_L;
    // (ahead of pdl_wait(): the decays are weights, and the step's integer arrays are copied in ahead of its first kernel; no
    // kernel of a step may write them)
    if (!ZLM_CHK(cu_seqlens + r, 8) || !ZLM_CHK(seq_start + r, 4) || !ZLM_CHK(decay + h, 4)) return;
    const int n = min(SM_L, cu_seqlens[r + 1] - cu_seqlens[r] - first);
    if (n <= 0) return;
    rm_powers(pw, decay[h], tid);
    const int row0 = cu_seqlens[r] + first;
    pdl_wait();
    const __nv_bfloat16* rows = proj + (size_t)row0 * ld;
    sm_stage_values(vt, rows + v_off + (size_t)h * V, ld, n, c0, V, tid);
    rm_stage<true>(qt, kt, rows + q_off + (size_t)h * D, rows + k_off + (size_t)h * D, ld, row0, seq_start[r] + first, n, D, rot,
                   k_scale, nullptr, tid);
    const float* S = before + ((size_t)blockIdx.x * H + h) * D * V;
    SmRows next = sm_fetch_state(S, 0, D, V, c0, tid);
    dec_wait<0>();
    const bool taken = __syncthreads_or(sm_clean_values(vt, tid));
    const int r0 = (warp >> 1) * 16, part = warp & 1;
    SmSum<4> dots;
    sm_scores(dots, qt, kt, r0, part * 32, D, lane);
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = r0 + (lane >> 2) + 8 * (e >> 1), l = part * 32 + i * 8 + (lane & 3) * 2 + (e & 1);
            s[i][e] = l <= j ? dots.get(i, e) * pw[l <= j ? j - l : 0] : 0.f;
        }
    __syncthreads();                                 // (the keys are read: weights and the state take their place)
    sm_put_weights(pt, s, r0, part * 32, lane);
    SmSum<8> acc;
    acc.zero();
    for (int d0 = 0; d0 < D; d0 += 32) {
        sm_put_state(st, next, tid);
        if (d0 + 32 < D) next = sm_fetch_state(S, d0 + 32, D, V, c0, tid);
        __syncthreads();
        sm_read_state(acc, qt, st, r0, part * 64, d0, D, lane);
        __syncthreads();
    }
    if (out.y) sm_stage_values(st, out.g + (size_t)row0 * out.g_stride + (size_t)h * V, out.g_stride, n, 0, V, tid);      // (the state is read)
    const float keep0 = pw[r0 + (lane >> 2) + 1], keep8 = pw[r0 + (lane >> 2) + 9];
    acc.scale(keep0, keep8);
    sm_read_values(acc, pt, vt, r0, part * 64, lane);
    sm_mend_out(acc, SmSeen{qt, pt, vt, S + c0, rows + v_off + (size_t)h * V + c0, (size_t)ld, D, V, 0.f}, keep0, keep8, taken, n, V - c0, r0,
                part * 64, lane);
    sm_write(acc, 1.f, 1.f, out, st, red, row0, n, h, H, V, c0, r0, part, lane);
}

// what the tensor-core form takes: 16-byte reads of 8 neighbouring coordinates (also of the halves of a rotation)
extern "C" int zlm_retention_products(int dtype, int ld, int q_off, int k_off, int v_off, int n_rot, int D, int V) {
    return dtype == ZLM_DTYPE_BF16 && D > 0 && D % 16 == 0 && D <= 128 && V > 0 && V % 8 == 0 && (V + 127) / 128 <= 65535 &&
           n_rot % 16 == 0 && ld % 8 == 0 && q_off % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0;
}

// chains the pieces' states of one sequence: before[c] = S_(c-1), S_c = decay^len_c * S_(c-1) + part[c]; the last S
// becomes the sequence's state.  A thread owns VEC neighbouring numbers; grid (ceil(D*V / (128 VEC)), H, R); the pieces of
// sequence r are r * maxp .. and `part_state` is overwritten in place by `before`.
template <int VEC>
__global__ void __launch_bounds__(128)
retention_chain_kernel(float* __restrict__ part_state, float* __restrict__ state, const float* __restrict__ decay,
                       const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slot, int maxp, int piece, int H,
                       int DV) {
    struct alignas(4 * VEC) Num { float v[VEC]; };
    pdl_launch_dependents();
    const int e = (blockIdx.x * 128 + threadIdx.x) * VEC, h = blockIdx.y, r = blockIdx.z;
    pdl_wait();
    if (e >= DV) return;
    const int n = cu_seqlens[r + 1] - cu_seqlens[r];
    const int np = (n + piece - 1) / piece;
    Num* sp = (Num*)(state + ((size_t)seq_slot[r] * H + h) * DV + e);
    if (!ZLM_CHK(sp, 4 * VEC)) return;
    Num S = *sp;
    const float d = decay[h];
    const float dl = powf(d, (float)piece);            // every piece but the last is whole
    const float dn = n == np * piece ? dl : powf(d, (float)(n - (np - 1) * piece));
    const size_t step = (size_t)H * DV;
    float* pp = part_state + ((size_t)r * maxp * H + h) * DV + e;
    for (int c0 = 0; c0 < np; c0 += 8, pp += 8 * step) {
        // eight pieces' states at a time: their loads do not wait for each other
        Num a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c0 + u < np && ZLM_CHK(pp + u * step, 4 * VEC)) a[u] = *(const Num*)(pp + u * step);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (c0 + u >= np) break;
            if (ZLM_CHK(pp + u * step, 4 * VEC)) *(Num*)(pp + u * step) = S;
            const float f = c0 + u == np - 1 ? dn : dl;
#pragma unroll
            for (int x = 0; x < VEC; ++x) S.v[x] = fmaf(f, S.v[x], a[u].v[x]);
        }
    }
    *sp = S;
}
static void launch_chain(float* part_state, float* state, const float* decay, const int* cu_seqlens, const int* seq_slot, int R, int maxp,
                         int piece, int H, int DV, cudaStream_t st) {
    if (DV % 4 == 0 && (uintptr_t)state % 16 == 0 && (uintptr_t)part_state % 16 == 0)
        zlm_launch(retention_chain_kernel<4>, dim3((DV + 511) / 512, H, R), dim3(128), 0, st, part_state, state, decay, cu_seqlens,
                   seq_slot, maxp, piece, H, DV);
    else
        zlm_launch(retention_chain_kernel<1>, dim3((DV + 127) / 128, H, R), dim3(128), 0, st, part_state, state, decay, cu_seqlens,
                   seq_slot, maxp, piece, H, DV);
}

static int retention_dpt(int D, int* ds) {
    // rows of the state a thread holds (times four columns, all in registers): 16 where 32 lanes of 16 hold a head's
    // rows (about 110 registers a thread: four blocks an SM), else 32; heads of more than 1024 rows are refused
    int dpt = D <= 512 ? 16 : 32;
    int n = (D + dpt - 1) / dpt, p = 1;
    while (p < n) p <<= 1;
    *ds = p;
    return dpt;
}

template <typename TA, int MODE>
static int launch_retention(dim3 grid, size_t smem, cudaStream_t st, int dpt, float* o, const void* proj, int ld, int q_off,
                            int k_off, int v_off, const float* inv_freq, int n_rot, const float* decay, float* state,
                            const int* cu_seqlens, const int* seq_slot, const int* seq_start, int maxp, int piece, int H, int D,
                            int V, int ds, float k_scale, const float* table, int T, int chunk) {
#define ZLM_RT_LAUNCH(DPT)                                                                                                \
    {                                                                                                                     \
        auto kern = retention_kernel<TA, DPT, MODE>;                                                                      \
        static bool attr_set_dev[64] = {}; bool& attr_set = attr_set_dev[zlm_device_index()];                             \
        if (!attr_set) {                                                                                                  \
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);          \
            if (e != cudaSuccess) {                                                                                       \
                zlm_set_error("retention: cannot reserve shared memory: %s", cudaGetErrorString(e));                      \
                return ZLM_ERR_CUDA;                                                                                      \
            }                                                                                                             \
            attr_set = true;                                                                                              \
        }                                                                                                                 \
        zlm_launch(kern, grid, dim3(RT_THREADS), smem, st, o, (const TA*)proj, ld, q_off, k_off, v_off, inv_freq, n_rot,   \
                   decay, state, cu_seqlens, seq_slot, seq_start, maxp, piece, H, D, V, ds, k_scale,                      \
                   table, T, chunk);                                                                                      \
    }
    if (dpt == 32) ZLM_RT_LAUNCH(32)
    else ZLM_RT_LAUNCH(16)
#undef ZLM_RT_LAUNCH
    return ZLM_OK;
}

static int retention_check(int H, int D, int V, int n_rot, int R) {
    ZLM_REQUIRE(H > 0 && H <= 65535 && D > 0 && D <= 1024 && V > 0 && R <= 65535, "retention: %d heads of %d x %d, %d sequences", H, D, V, R);
    ZLM_REQUIRE(n_rot >= 0 && n_rot % 2 == 0 && n_rot <= D, "retention: %d rotated coordinates of %d", n_rot, D);
    return ZLM_OK;
}

// o [T][H*V] fp32; proj [T][ld] with q at column q_off (H heads of D), k at k_off, v at v_off (H heads of V);
// state [slots][H][D][V] fp32 (zero for a new sequence); table: the step's cosines and sines [2][n_rot/2][T] if they were
// computed beforehand (else the kernel forms them from inv_freq)
extern "C" int zlm_retention(float* o, const void* proj, int ld, int q_off, int k_off, int v_off, int dtype,
                             const float* inv_freq, int n_rot, const float* decay, float* state, const int* cu_seqlens,
                             const int* seq_slot, const int* seq_start, int R, int H, int D, int V, float k_scale,
                             const float* table, int T, int max_new, cudaStream_t st) {
    if (R == 0) return ZLM_OK;
    int rc = retention_check(H, D, V, n_rot, R);
    if (rc) return rc;
    int ds;
    const int dpt = retention_dpt(D, &ds);
    const int cols = RT_THREADS / ds * RT_CPT;
    // tokens staged at a time: as many as fit in about 56 KB (four blocks an SM), at least 4
    const size_t row_bytes = (size_t)(2 * ds * (dpt + 4) + cols) * sizeof(float);
    int chunk = (int)((56 * 1024) / row_bytes);
    chunk = chunk > RT_CHUNK ? RT_CHUNK : (chunk < 4 ? 4 : chunk);
    if (max_new > 0 && chunk > max_new) chunk = max_new;          // (the longest sequence of the step: a decode step stages one token)
    const size_t smem = (size_t)chunk * row_bytes;
    const dim3 grid((V + cols - 1) / cols, H, R);
    if (dtype == ZLM_DTYPE_F32)
        rc = launch_retention<float, 0>(grid, smem, st, dpt, o, proj, ld, q_off, k_off, v_off, inv_freq, n_rot, decay, state,
                                        cu_seqlens, seq_slot, seq_start, 0, 0, H, D, V, ds, k_scale, table, T, chunk);
    else if (dtype == ZLM_DTYPE_BF16)
        rc = launch_retention<__nv_bfloat16, 0>(grid, smem, st, dpt, o, proj, ld, q_off, k_off, v_off, inv_freq, n_rot, decay,
                                                state, cu_seqlens, seq_slot, seq_start, 0, 0, H, D, V, ds, k_scale, table, T, chunk);
    else
        ZLM_REQUIRE(false, "retention: unsupported dtype %d", dtype);
    if (rc) return rc;
    return zlm_check_launch("retention");
}

// The same for long prompts, in pieces of `piece` tokens that run side by side: maxp pieces a sequence (those of the
// step's longest one; a shorter sequence's last pieces are empty); part_state is scratch of R * maxp * H * D * V floats.
// y (null: none; where zlm_retention_products says yes, heads of up to 128 value columns): [T][y_stride] bfloat16 receives, in
// the place of o, every head divided by its root mean square times silu (act 1) or sigmoid (0) of g [T][g_stride].
extern "C" int zlm_retention_parts(float* o, const void* proj, int ld, int q_off, int k_off, int v_off, int dtype,
                                   const float* inv_freq, int n_rot, const float* decay, float* state,
                                   const int* cu_seqlens, const int* seq_slot, const int* seq_start, int R, int maxp, int piece,
                                   float* part_state, int H, int D, int V, float k_scale, const float* table, int T,
                                   void* y, int y_stride, const void* g, int g_stride, float eps, int act, cudaStream_t st) {
    if (R == 0 || maxp == 0) return ZLM_OK;
    const long long pieces = (long long)R * maxp;
    int rc = retention_check(H, D, V, n_rot, R);
    if (rc) return rc;
    ZLM_REQUIRE(piece > 0 && pieces <= 65535 && part_state, "retention: %lld pieces of %d tokens", pieces, piece);
    const bool products = zlm_retention_products(dtype, ld, q_off, k_off, v_off, n_rot, D, V) && piece == SM_L &&
                          (uintptr_t)proj % 16 == 0 && (uintptr_t)part_state % 16 == 0 && (uintptr_t)o % 8 == 0;
    ZLM_REQUIRE(!y || (products && V <= 128 && y_stride % 8 == 0 && g_stride % 8 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)g % 16 == 0),
                "retention: heads of %d x %d do not take their gate along", D, V);
    if (products) {
        const size_t smem1 = (size_t)4 * SM_L * 128 * sizeof(__nv_bfloat16), smem2 = (size_t)7 * SM_L * 128 * sizeof(__nv_bfloat16);
        static bool attr_set_dev[64] = {};
        bool& attr_set = attr_set_dev[zlm_device_index()];
        if (!attr_set) {
            cudaError_t e1 = cudaFuncSetAttribute(retention_piece_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
            cudaError_t e2 = cudaFuncSetAttribute(retention_piece_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
            if (e1 != cudaSuccess || e2 != cudaSuccess) {
                zlm_set_error("retention: cannot reserve shared memory");
                return ZLM_ERR_CUDA;
            }
            attr_set = true;
        }
        const dim3 grid((unsigned)pieces, H, (V + 127) / 128);
        const RmRot rot{inv_freq, table, n_rot, T};
        zlm_launch(retention_piece_state_kernel, grid, dim3(RM_THREADS), smem1, st, part_state, (const __nv_bfloat16*)proj, ld, k_off,
                   v_off, rot, decay, cu_seqlens, seq_start, maxp, H, D, V, k_scale);
        launch_chain(part_state, state, decay, cu_seqlens, seq_slot, R, maxp, piece, H, D * V, st);
        zlm_launch(retention_piece_out_kernel, grid, dim3(RM_THREADS), smem2, st, SmOut{o, (__nv_bfloat16*)y, y_stride, (const __nv_bfloat16*)g, g_stride, VecW{nullptr, 0}, 0, eps, act},
                   (const __nv_bfloat16*)proj, ld, q_off, k_off, v_off, rot, decay, (const float*)part_state, cu_seqlens, seq_start, maxp, H, D, V, k_scale);
        return zlm_check_launch("retention_products");
    }
    int ds;
    const int dpt = retention_dpt(D, &ds);
    const int cols = RT_THREADS / ds * RT_CPT;
    // tokens staged at a time: as many as fit in about 56 KB (four blocks an SM), at least 4
    const size_t row_bytes = (size_t)(2 * ds * (dpt + 4) + cols) * sizeof(float);
    int chunk = (int)((56 * 1024) / row_bytes);
    chunk = chunk > RT_CHUNK ? RT_CHUNK : (chunk < 4 ? 4 : chunk);
    if (chunk > piece) chunk = piece;
    const size_t smem = (size_t)chunk * row_bytes;
    const dim3 grid((V + cols - 1) / cols, H, (unsigned)pieces);
    for (int mode = 1; mode <= 2; ++mode) {
        if (dtype == ZLM_DTYPE_F32) {
            rc = mode == 1 ? launch_retention<float, 1>(grid, smem, st, dpt, o, proj, ld, q_off, k_off, v_off, inv_freq, n_rot, decay,
                                                        part_state, cu_seqlens, seq_slot, seq_start, maxp, piece,
                                                        H, D, V, ds, k_scale, table, T, chunk)
                           : launch_retention<float, 2>(grid, smem, st, dpt, o, proj, ld, q_off, k_off, v_off, inv_freq, n_rot, decay,
                                                        part_state, cu_seqlens, seq_slot, seq_start, maxp, piece,
                                                        H, D, V, ds, k_scale, table, T, chunk);
        } else if (dtype == ZLM_DTYPE_BF16) {
            rc = mode == 1 ? launch_retention<__nv_bfloat16, 1>(grid, smem, st, dpt, o, proj, ld, q_off, k_off, v_off, inv_freq,
                                                                n_rot, decay, part_state, cu_seqlens, seq_slot, seq_start,
                                                                maxp, piece, H, D, V, ds, k_scale, table, T, chunk)
                           : launch_retention<__nv_bfloat16, 2>(grid, smem, st, dpt, o, proj, ld, q_off, k_off, v_off, inv_freq,
                                                                n_rot, decay, part_state, cu_seqlens, seq_slot, seq_start,
                                                                maxp, piece, H, D, V, ds, k_scale, table, T, chunk);
        } else {
            ZLM_REQUIRE(false, "retention: unsupported dtype %d", dtype);
        }
        if (rc) return rc;
        rc = zlm_check_launch("retention_parts");
        if (rc) return rc;
        if (mode == 1) {
            launch_chain(part_state, state, decay, cu_seqlens, seq_slot, R, maxp, piece, H, D * V, st);
            rc = zlm_check_launch("retention_chain");
            if (rc) return rc;
        }
    }
    return ZLM_OK;
}

ZLM_TRANSLATION_UNIT(retention)
