// Products of fp32 numbers on the bfloat16 tensor cores without giving up fp32: an operand is cut into three bfloat16
// pieces, hi + mid + lo, which together hold all 24 bits of it (each piece rounds what the pieces before it left), and the
// pieces' products that matter are added up: hi*hi, hi*mid, mid*hi, hi*lo, lo*hi, mid*mid where both operands are cut (what is
// left out is below 2^-25 of the product), three products where the other one is bfloat16 as it is.
// The tensor cores cut off what their accumulator cannot hold instead of rounding, which adds up along a chain (one
// accumulator for all products: 1.1e-6 of a retention's outputs against 2.4e-7 of the FFMA chain that this stands in for).  So
// the products of 16 terms start from zero each time, the small ones first, and are added by the rounding FADD: 1.8e-7.
// The helpers work on tiles in shared memory, one tile for each piece, rows swizzled as tile_off says.
#pragma once
#include "attn_common.cuh"

#define SM_L 64                      // tokens of a piece of a long prompt

// the three pieces of two neighbouring numbers
struct Split2 { unsigned p[3]; };
__device__ __forceinline__ Split2 split2(float a, float b) {
    Split2 s;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        s.p[x] = pack_bf16(a, b);
        a -= __uint_as_float(s.p[x] << 16);
        b -= __uint_as_float(s.p[x] & 0xffff0000u);
    }
    return s;
}
// eight neighbouring numbers into the three tiles at element offset `off`
__device__ __forceinline__ void split8(__nv_bfloat16* tile, int tile_elems, int off, const float* f) {
    unsigned u[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const Split2 s = split2(f[2 * e], f[2 * e + 1]);
#pragma unroll
        for (int x = 0; x < 3; ++x) u[x][e] = s.p[x];
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) *(uint4*)(tile + (size_t)x * tile_elems + off) = make_uint4(u[x][0], u[x][1], u[x][2], u[x][3]);
}
__device__ __forceinline__ void widen8(const uint4& u, float* f) {
    f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
    f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
    f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
}

// where a lane reads, for the four 8 x 8 matrices of an ldmatrix:
//   A of a product from rows of A (16 rows from r0, 16 columns from c0)
template <int HD> __device__ __forceinline__ const __nv_bfloat16* sm_a_rows(const __nv_bfloat16* t, int r0, int c0, int lane) {
    return t + tile_off<HD>(r0 + (lane & 15), (c0 >> 3) + (lane >> 4));
}
//   A from rows of A^T (16 rows of A^T from c0, 16 columns from r0), transposed on the way
template <int HD> __device__ __forceinline__ const __nv_bfloat16* sm_a_cols(const __nv_bfloat16* t, int r0, int c0, int lane) {
    return t + tile_off<HD>(c0 + (lane & 7) + ((lane >> 4) << 3), (r0 >> 3) + ((lane >> 3) & 1));
}
//   B of two neighbouring tiles of 8 outputs from rows of B^T (an output a row)
template <int HD> __device__ __forceinline__ const __nv_bfloat16* sm_b_rows(const __nv_bfloat16* t, int n0, int k0, int lane) {
    return t + tile_off<HD>(n0 + (lane & 7) + ((lane >> 4) << 3), (k0 >> 3) + ((lane >> 3) & 1));
}
//   the same from rows of B (an output a column), transposed on the way
template <int HD> __device__ __forceinline__ const __nv_bfloat16* sm_b_cols(const __nv_bfloat16* t, int n0, int k0, int lane) {
    return t + tile_off<HD>(k0 + (lane & 15), (n0 >> 3) + (lane >> 4));
}

// d = a b
__device__ __forceinline__ void sm_mma_zero(float* d, const unsigned* a, unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// NP pairs of neighbouring tiles of 16 x 8 sums += A B, 16 terms, both operands in pieces.  (The products of one tile wait for
// each other; those of the 2 NP tiles take turns.)
template <int NP> __device__ __forceinline__ void sm_mma6(float (*acc)[4], const unsigned (&a)[3][4], const unsigned (&b)[NP][3][4]) {
    constexpr int ia[6] = {1, 0, 2, 0, 1, 0}, ib[6] = {1, 2, 0, 1, 0, 0};
    float d[2 * NP][4];
#pragma unroll
    for (int x = 0; x < 6; ++x)
#pragma unroll
        for (int t = 0; t < 2 * NP; ++t) {
            const unsigned* p = b[t / 2][ib[x]] + (t & 1) * 2;
            if (x == 0) sm_mma_zero(d[t], a[ia[x]], p[0], p[1]);
            else dec_mma(d[t], a[ia[x]], p[0], p[1]);
        }
#pragma unroll
    for (int t = 0; t < 2 * NP; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[t][e] += d[t][e];
}
// the same with B in bfloat16 as it is
template <int NP> __device__ __forceinline__ void sm_mma3(float (*acc)[4], const unsigned (&a)[3][4], const unsigned (&b)[NP][4]) {
    float d[2 * NP][4];
#pragma unroll
    for (int x = 2; x >= 0; --x)
#pragma unroll
        for (int t = 0; t < 2 * NP; ++t) {
            const unsigned* p = b[t / 2] + (t & 1) * 2;
            if (x == 2) sm_mma_zero(d[t], a[x], p[0], p[1]);
            else dec_mma(d[t], a[x], p[0], p[1]);
        }
#pragma unroll
    for (int t = 0; t < 2 * NP; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[t][e] += d[t][e];
}
// the same with A in bfloat16 as it is and B in pieces
template <int NP> __device__ __forceinline__ void sm_mma3b(float (*acc)[4], const unsigned (&a)[4], const unsigned (&b)[NP][3][4]) {
    float d[2 * NP][4];
#pragma unroll
    for (int x = 2; x >= 0; --x)
#pragma unroll
        for (int t = 0; t < 2 * NP; ++t) {
            const unsigned* p = b[t / 2][x] + (t & 1) * 2;
            if (x == 2) sm_mma_zero(d[t], a, p[0], p[1]);
            else dec_mma(d[t], a, p[0], p[1]);
        }
#pragma unroll
    for (int t = 0; t < 2 * NP; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[t][e] += d[t][e];
}
// sums of NT tiles of 16 x 8
template <int NT> struct SmSum {
    float v[NT][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) v[n][e] = 0.f;
    }
    // times a factor by row (of a lane's two rows)
    __device__ __forceinline__ void scale(float r0, float r8) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) v[n][e] *= e < 2 ? r0 : r8;
    }
    __device__ __forceinline__ float get(int n, int e) const { return v[n][e]; }
};

// ---------------------------------------------------------------------------- numbers that are not finite
// Cut into pieces, an infinity leaves infinity - infinity = NaN behind, and a tile's zero weights make NaN of it in rows that do
// not see it (0 x infinity).  So what is not finite among the values is taken out of their tile before the products (one
// pass over the thread's own copies; a later token's values then leave the rows of earlier ones alone, to the bit), and sums
// that still come out not finite (keys, queries, states) are formed again as FFMA chains of the whole numbers, with the
// values that were taken out: infinities keep their signs and reach what sees them, as in a walk over the tokens.  Chosen
// over a second kernel that a flag would wake: that costs every call a launch.
__device__ __forceinline__ bool sm_odd(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }
// whether one of a thread's sums is not finite (zero times it is not zero)
template <int NT> __device__ __forceinline__ bool sm_any_odd(const SmSum<NT>& s) {
    float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) t[e] = fmaf(s.v[n][e], 0.f, t[e]);
    return (t[0] + t[1]) + (t[2] + t[3]) != 0.f;
}
// the thread's copies of sm_stage_values, between dec_wait<0>() and the barrier; true where something was taken out
__device__ __forceinline__ bool sm_clean_values(__nv_bfloat16* vt, int tid) {
    unsigned top = 0;
#pragma unroll
    for (int y = 0; y < SM_L * 16 / 256; ++y) {
        const int x = tid + y * 256;
        const uint4 u = *(const uint4*)(vt + tile_off<128>(x >> 4, x & 15));
        top = __vmaxu2(__vmaxu2(__vmaxu2(top, u.x & 0x7fff7fffu), __vmaxu2(u.y & 0x7fff7fffu, u.z & 0x7fff7fffu)), u.w & 0x7fff7fffu);
    }
    if ((top & 0xffffu) < 0x7f80u && (top >> 16) < 0x7f80u) return false;
    for (int x = tid; x < SM_L * 16; x += 256) {
        unsigned* p = (unsigned*)(vt + tile_off<128>(x >> 4, x & 15));
        for (int e = 0; e < 4; ++e) {
            if ((p[e] & 0x7f80u) == 0x7f80u) p[e] &= 0xffff0000u;
            if ((p[e] & 0x7f800000u) == 0x7f800000u) p[e] &= 0xffffu;
        }
    }
    return true;
}
// number c of a row of a tile in pieces of `elems` elements
template <int HD> __device__ __forceinline__ float sm_whole(const __nv_bfloat16* t, int elems, int row, int c) {
    const __nv_bfloat16* p = t + tile_off<HD>(row, c >> 3) + (c & 7);
    const float hi = to_f32(p[0]);
    return sm_odd(hi) ? hi : hi + (to_f32(p[elems]) + to_f32(p[2 * elems]));
}
// (calls, so that the kernels' own code stays short: their loops are unrolled, and inlined chains cost them 3 to 6 %)
// scores that are not finite: row by row of both tiles, in pieces [SM_L][128]
static __device__ __noinline__ void sm_mend_scores(float (*s)[4], const __nv_bfloat16* qt, const __nv_bfloat16* kt, int r0, int n0, int dim,
                                                   int lane) {
    for (int i = 0; i < 4; ++i)
        for (int e = 0; e < 4; ++e) {
            const int j = r0 + (lane >> 2) + 8 * (e >> 1), l = n0 + i * 8 + (lane & 3) * 2 + (e & 1);
            if (!sm_odd(s[i][e])) continue;
            float t = 0.f;
            for (int c = 0; c < dim; ++c) t = fmaf(sm_whole<128>(qt, SM_L * 128, j, c), sm_whole<128>(kt, SM_L * 128, l, c), t);
            s[i][e] = t;
        }
}
// numbers of a state that are not finite: columns of the weighted keys times columns of the values
static __device__ __noinline__ void sm_mend_state(float (*s)[4], const __nv_bfloat16* kt, const __nv_bfloat16* vt, int d0, int n0, int lane) {
    for (int i = 0; i < 8; ++i)
        for (int e = 0; e < 4; ++e) {
            const int d = d0 + (lane >> 2) + 8 * (e >> 1), c = n0 + i * 8 + (lane & 3) * 2 + (e & 1);
            if (!sm_odd(s[i][e])) continue;
            float t = 0.f;
            for (int l = 0; l < SM_L; ++l)
                t = fmaf(sm_whole<128>(kt, SM_L * 128, l, d), to_f32(vt[tile_off<128>(l, c >> 3) + (c & 7)]), t);
            s[i][e] = t;
        }
}
// what an output is made of: S the state's column of the head's value column c0 + c, v the piece's values of that column;
// q_scale: 0 where the queries' tile holds pieces, else the factor of queries that are bfloat16 as they are
struct SmSeen {
    const __nv_bfloat16 *qt, *pt, *vt;
    const float* S;
    const __nv_bfloat16* v;
    size_t stride;
    int D, V;
    float q_scale;
};
static __device__ __noinline__ void sm_mend_outputs(float (*acc)[4], const SmSeen& s, float keep0, float keep8, bool taken, int n, int cols,
                                                    int r0, int n0, int lane) {
    for (int i = 0; i < 8; ++i)
        for (int e = 0; e < 4; ++e) {
            const int j = r0 + (lane >> 2) + 8 * (e >> 1), c = n0 + i * 8 + (lane & 3) * 2 + (e & 1);
            if (j >= n || c >= cols) continue;
            float x = acc[i][e];
            if (sm_odd(x)) {
                x = 0.f;
                for (int d = 0; d < s.D; ++d) {
                    const float* p = s.S + (size_t)d * s.V + c;
                    const float q = s.q_scale == 0.f ? sm_whole<128>(s.qt, SM_L * 128, j, d) : to_f32(s.qt[tile_off<128>(j, d >> 3) + (d & 7)]);
                    if (ZLM_CHK(p, 4)) x = fmaf(q, *p, x);
                }
                x *= e < 2 ? keep0 : keep8;            // (the queries' factor among them)
                for (int l = 0; l <= j; ++l)
                    x = fmaf(sm_whole<SM_L>(s.pt, SM_L * SM_L, j, l), to_f32(s.vt[tile_off<128>(l, c >> 3) + (c & 7)]), x);
            }
            for (int l = 0; taken && l <= j; ++l) {
                const __nv_bfloat16* p = s.v + (size_t)l * s.stride + c;
                const float v = ZLM_CHK(p, 2) ? to_f32(*p) : 0.f;
                if (sm_odd(v)) x = fmaf(sm_whole<SM_L>(s.pt, SM_L * SM_L, j, l), v, x);
            }
            acc[i][e] = x;
        }
}
// a warp's outputs (16 rows of the piece's n from r0, 64 columns from n0 of the block's `cols`); queries, weights and the cleaned
// values still in their tiles; taken: sm_clean_values took something out somewhere in the block
__device__ __forceinline__ void sm_mend_out(SmSum<8>& acc, const SmSeen& s, float keep0, float keep8, bool taken, int n, int cols, int r0,
                                            int n0, int lane) {
    if (!taken && !sm_any_odd(acc)) return;
    SmSum<8> t = acc;                                // (a copy, so that the sums themselves stay in registers)
    sm_mend_outputs(t.v, s, keep0, keep8, taken, n, cols, r0, n0, lane);
    acc = t;
}

// ---------------------------------------------------------------------------- a piece of 64 tokens, one head, 128 value columns
// Blocks of 256 threads.  What a piece adds to a state:
//   acc += (keys)^T (values): the warp's 16 rows of the state from d0 on, 64 columns from n0 on;
//   kt: the weighted keys [SM_L][128] in pieces, vt: the values [SM_L][128]
__device__ __forceinline__ void sm_piece_state(SmSum<8>& acc, const __nv_bfloat16* kt, const __nv_bfloat16* vt, int d0, int n0, int lane) {
#pragma unroll
    for (int k0 = 0; k0 < SM_L; k0 += 16) {
        unsigned a[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) dec_ldsm4t(a[x][0], a[x][1], a[x][2], a[x][3], sm_a_cols<128>(kt + x * SM_L * 128, d0, k0, lane));
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            unsigned b[2][4];
#pragma unroll
            for (int y = 0; y < 2; ++y) dec_ldsm4t(b[y][0], b[y][1], b[y][2], b[y][3], sm_b_cols<128>(vt, n0 + n * 8 + y * 16, k0, lane));
            sm_mma3<2>(acc.v + n, a, b);
        }
    }
    if (!sm_any_odd(acc)) return;
    SmSum<8> t = acc;
    sm_mend_state(t.v, kt, vt, d0, n0, lane);
    acc = t;
}
// 16 rows from d0, 64 columns from c of a state [..][V]
__device__ __forceinline__ void sm_write_state(float* S, const SmSum<8>& acc, int d0, int c, int V, int lane) {
    float* dst = S + (size_t)(d0 + (lane >> 2)) * V + c + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float* p = dst + (size_t)8 * e * V + i * 8;
            if (c + i * 8 < V && ZLM_CHK(p, 8)) *(float2*)p = make_float2(acc.get(i, 2 * e), acc.get(i, 2 * e + 1));
        }
}
// Scores of 16 queries (rows r0 on) against 32 keys (rows n0 on), `dim` coordinates, both in pieces [SM_L][128]; where
// all 32 keys come after the last query the scores stay zero
__device__ __forceinline__ void sm_scores(SmSum<4>& s, const __nv_bfloat16* qt, const __nv_bfloat16* kt, int r0, int n0, int dim, int lane) {
    s.zero();
    if (n0 > r0 + 15) return;
    for (int k0 = 0; k0 < dim; k0 += 16) {
        unsigned a[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) dec_ldsm4(a[x][0], a[x][1], a[x][2], a[x][3], sm_a_rows<128>(qt + x * SM_L * 128, r0, k0, lane));
        unsigned b[2][3][4];
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 3; ++x)
                dec_ldsm4(b[y][x][0], b[y][x][1], b[y][x][2], b[y][x][3], sm_b_rows<128>(kt + x * SM_L * 128, n0 + y * 16, k0, lane));
        sm_mma6<2>(s.v, a, b);
    }
    if (!sm_any_odd(s)) return;
    SmSum<4> t = s;
    sm_mend_scores(t.v, qt, kt, r0, n0, dim, lane);
    s = t;
}
// the same of queries and keys that are bfloat16 as they are [SM_L][128]: their products are exact, and what is not finite
// comes out as from FFMA chains
__device__ __forceinline__ void sm_scores_plain(SmSum<4>& s, const __nv_bfloat16* qt, const __nv_bfloat16* kt, int r0, int n0, int dim, int lane) {
    s.zero();
    if (n0 > r0 + 15) return;
    for (int k0 = 0; k0 < dim; k0 += 16) {
        unsigned a[4], b[2][4];
        dec_ldsm4(a[0], a[1], a[2], a[3], sm_a_rows<128>(qt, r0, k0, lane));
#pragma unroll
        for (int y = 0; y < 2; ++y) dec_ldsm4(b[y][0], b[y][1], b[y][2], b[y][3], sm_b_rows<128>(kt, n0 + y * 16, k0, lane));
        float d[4][4];
#pragma unroll
        for (int t = 0; t < 4; ++t) sm_mma_zero(d[t], a, b[t / 2][(t & 1) * 2], b[t / 2][(t & 1) * 2 + 1]);
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) s.v[t][e] += d[t][e];
    }
}
// 32 rows of the state, 128 columns: fetched into registers (a thread's four float4), then cut into pieces [32][128]
struct SmRows { float4 f[4]; };
__device__ __forceinline__ SmRows sm_fetch_state(const float* S, int d0, int dim, int V, int c0, int tid) {
    SmRows r;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int row = d0 + (tid >> 4) + 16 * x, c = c0 + (tid & 15) * 8;
        const float* p = S + (size_t)row * V + c;
        const bool ok = row < dim && c < V && ZLM_CHK(p, 32);
        r.f[2 * x] = ok ? *(const float4*)p : make_float4(0.f, 0.f, 0.f, 0.f);
        r.f[2 * x + 1] = ok ? *(const float4*)(p + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return r;
}
__device__ __forceinline__ void sm_put_state(__nv_bfloat16* st, const SmRows& r, int tid) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const float f[8] = {r.f[2 * x].x, r.f[2 * x].y, r.f[2 * x].z, r.f[2 * x].w, r.f[2 * x + 1].x, r.f[2 * x + 1].y, r.f[2 * x + 1].z, r.f[2 * x + 1].w};
        split8(st, 32 * 128, tile_off<128>((tid >> 4) + 16 * x, tid & 15), f);
    }
}
// acc (16 queries from r0, 64 columns from n0) += queries, coordinates d0 .. d0 + 31, times the state's pieces [32][128]
__device__ __forceinline__ void sm_read_state(SmSum<8>& acc, const __nv_bfloat16* qt, const __nv_bfloat16* st, int r0, int n0, int d0, int dim, int lane) {
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 16) {
        if (d0 + k0 >= dim) return;
        unsigned a[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) dec_ldsm4(a[x][0], a[x][1], a[x][2], a[x][3], sm_a_rows<128>(qt + x * SM_L * 128, r0, d0 + k0, lane));
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            unsigned b[2][3][4];
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    dec_ldsm4t(b[y][x][0], b[y][x][1], b[y][x][2], b[y][x][3], sm_b_cols<128>(st + x * 32 * 128, n0 + n * 8 + y * 16, k0, lane));
            sm_mma6<2>(acc.v + n, a, b);
        }
    }
}
// the same with queries that are bfloat16 as they are
__device__ __forceinline__ void sm_read_state_plain(SmSum<8>& acc, const __nv_bfloat16* qt, const __nv_bfloat16* st, int r0, int n0, int d0, int dim,
                                                    int lane) {
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 16) {
        if (d0 + k0 >= dim) return;
        unsigned a[4];
        dec_ldsm4(a[0], a[1], a[2], a[3], sm_a_rows<128>(qt, r0, d0 + k0, lane));
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            unsigned b[2][3][4];
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    dec_ldsm4t(b[y][x][0], b[y][x][1], b[y][x][2], b[y][x][3], sm_b_cols<128>(st + x * 32 * 128, n0 + n * 8 + y * 16, k0, lane));
            sm_mma3b<2>(acc.v + n, a, b);
        }
    }
}
// the weights of 16 queries (from r0) on 32 keys (from n0) into pieces [SM_L][SM_L]
__device__ __forceinline__ void sm_put_weights(__nv_bfloat16* pt, const float (&s)[4][4], int r0, int n0, int lane) {
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const Split2 w = split2(s[n][2 * i], s[n][2 * i + 1]);
            const int row = r0 + (lane >> 2) + 8 * i;
#pragma unroll
            for (int x = 0; x < 3; ++x)
                *(unsigned*)(pt + x * SM_L * SM_L + tile_off<SM_L>(row, (n0 >> 3) + n) + (lane & 3) * 2) = w.p[x];
        }
}
// acc (16 queries from r0, 64 columns from n0) += weights times values [SM_L][128]; keys after the queries are skipped
__device__ __forceinline__ void sm_read_values(SmSum<8>& acc, const __nv_bfloat16* pt, const __nv_bfloat16* vt, int r0, int n0, int lane) {
#pragma unroll
    for (int k0 = 0; k0 < SM_L; k0 += 16) {
        if (k0 > r0) return;
        unsigned a[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) dec_ldsm4(a[x][0], a[x][1], a[x][2], a[x][3], sm_a_rows<SM_L>(pt + x * SM_L * SM_L, r0, k0, lane));
#pragma unroll
        for (int n = 0; n < 8; n += 4) {
            unsigned b[2][4];
#pragma unroll
            for (int y = 0; y < 2; ++y) dec_ldsm4t(b[y][0], b[y][1], b[y][2], b[y][3], sm_b_cols<128>(vt, n0 + n * 8 + y * 16, k0, lane));
            sm_mma3<2>(acc.v + n, a, b);
        }
    }
}
// the values of a piece, 128 columns from c0 (zeros beyond the piece's tokens and the head's columns), by asynchronous copies
__device__ __forceinline__ void sm_stage_values(__nv_bfloat16* vt, const __nv_bfloat16* v, size_t stride, int n, int c0, int V, int tid) {
#pragma unroll
    for (int y = 0; y < SM_L * 16 / 256; ++y) {
        const int x = tid + y * 256, l = x >> 4, c = x & 15;
        __nv_bfloat16* dst = vt + tile_off<128>(l, c);
        if (l < n && c0 + c * 8 < V) dec_cp_async16(dst, v + (size_t)l * stride + c0 + c * 8);
        else *(uint4*)dst = make_uint4(0, 0, 0, 0);
    }
    dec_commit();
}
// `dim` columns (up to 128) of the piece's rows, times a factor, into pieces [SM_L][128]; zeros beyond n rows
__device__ __forceinline__ void sm_stage_rows(__nv_bfloat16* t, const __nv_bfloat16* p, size_t stride, int n, int dim, float scale, int tid) {
    const int groups = dim >> 3;
    uint4 u[4];                                       // (up to 16 groups of 64 rows: all of them on their way at once)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        const int x = tid + y * 256, l = x / groups, c = x - l * groups;
        u[y] = make_uint4(0, 0, 0, 0);
        if (l < n && ZLM_CHK(p + (size_t)l * stride + c * 8, 16)) u[y] = *(const uint4*)(p + (size_t)l * stride + c * 8);
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        const int x = tid + y * 256, l = x / groups, c = x - l * groups;
        if (l >= SM_L) continue;
        float f[8];
        widen8(u[y], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= scale;
        split8(t, SM_L * 128, tile_off<128>(l, c), f);
    }
}

// ---------------------------------------------------------------------------- what leaves the kernels of a piece
// The outputs as they are (o [T][H * V] fp32), or what follows them in the mixers (y): every head divided by its root mean
// square, times a weight where there is one, times silu (act 1) or sigmoid (0) of a gate's columns, in bfloat16.
struct SmOut {
    float* o;
    __nv_bfloat16* y;                // null: o
    int y_stride;
    const __nv_bfloat16* g;
    int g_stride;
    VecW w;                          // null, or [w_rows ? H : 1][V]
    int w_rows;
    float eps;
    int act;
};
// a warp's 16 rows (of the piece's n) by 64 columns, times a factor for each of a lane's two rows; red [SM_L][2] in shared
// memory.  The gated form wants all of a head's columns in the block (V <= 128) and every thread of it here; gt is its tile
// of the gate's columns [SM_L][128], on the way by sm_stage_values, which the results pass through on their way out
__device__ __forceinline__ void sm_write(const SmSum<8>& acc, float f0, float f8, const SmOut& out, __nv_bfloat16* gt, float (*red)[2],
                                         int row0, int n, int h, int H, int V, int c0, int r0, int half, int lane) {
    const int c = c0 + half * 64 + (lane & 3) * 2;
    if (!out.y) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int j = r0 + (lane >> 2) + 8 * e;
                float* p = out.o + ((size_t)(row0 + j) * H + h) * V + c + i * 8;
                const float f = e ? f8 : f0;
                if (j < n && c + i * 8 < V && ZLM_CHK(p, 8)) *(float2*)p = make_float2(acc.get(i, 2 * e) * f, acc.get(i, 2 * e + 1) * f);
            }
        return;
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        float ss = 0.f;                                  // (columns beyond V are zero)
        const float f = e ? f8 : f0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float a = acc.get(i, 2 * e) * f, b = acc.get(i, 2 * e + 1) * f;
            ss = fmaf(a, a, fmaf(b, b, ss));
        }
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if ((lane & 3) == 0) red[r0 + (lane >> 2) + 8 * e][half] = ss;
    }
    // the weights, then (once they have arrived) the gate's logits of a row into registers before anything is written where
    // they stand: otherwise every exponential waits for the one before it (9,200 cycles of a block's 45,000)
    float2 w[8];
    if (out.w.p) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = (out.w_rows ? h * V : 0) + c + i * 8;
            w[i] = c + i * 8 < V && out.w.ok(at, 2) ? make_float2(out.w[at], out.w[at + 1]) : make_float2(0.f, 0.f);
        }
    }
    dec_wait<0>();
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int j = r0 + (lane >> 2) + 8 * e;
        const float f = (e ? f8 : f0) / sqrtf((red[j][0] + red[j][1]) / (float)V + out.eps);
        unsigned z[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] = *(const unsigned*)(gt + tile_off<128>(j, half * 8 + i) + (lane & 3) * 2);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float v[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float zz = __uint_as_float(x ? z[i] & 0xffff0000u : z[i] << 16), sg = 1.0f / (1.0f + expf(-zz));
                v[x] = acc.get(i, 2 * e + x) * f * (out.act == 1 ? zz * sg : sg);
                if (out.w.p) v[x] *= x ? w[i].y : w[i].x;
            }
            z[i] = pack_bf16(v[0], v[1]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) *(unsigned*)(gt + tile_off<128>(j, half * 8 + i) + (lane & 3) * 2) = z[i];
    }
    __syncthreads();
    for (int x = threadIdx.x; x < n * 16; x += 256) {
        __nv_bfloat16* yp = out.y + (size_t)(row0 + (x >> 4)) * out.y_stride + (size_t)h * V + (x & 15) * 8;
        if ((x & 15) * 8 < V && ZLM_CHK(yp, 16)) *(uint4*)yp = *(const uint4*)(gt + tile_off<128>(x >> 4, x & 15));
    }
}
