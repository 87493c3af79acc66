// Integer causal attention for short sequences (T <= 128) and heads of 4: one CTA per (sequence, head), one thread per token.  This is
// the shape of the reference's own model (64 heads of 4, T = 128), where a head's whole problem - 128 x 128 scores over a 4-wide
// contraction - is too small to tile: the tiled kernels of atencao.cuh spend their time in launches, tile set-up and the cross-CTA
// maxima of the backward.  The operands of a head live in shared memory, a thread walks its query row (or, in the last pass of the
// backward, its key column), the two matrix-wide maxima of the backward are CTA-level reductions, and forward and backward are one
// launch each.
//
// The bound is instruction issue, so the arithmetic is chosen for few instructions:
//   * |q . k| <= 4 * 2032^2 < 2^24: a score-like product is exact in fp32, two keys at a time (f32x2), and rounds to even at 2^-s through
//     one f32x2 FMA against 1.5 * 2^23 (valid for |x 2^-s| <= 2^22; the result is read from the bit pattern);
//   * P is exactly zero where the score lies 2130 or more below the maximum, which the slope makes the case of most keys: four keys of a
//     warp's 32 rows at a time are skipped when none of them counts (exponentials, P.V and, from the bytes of P, everything in the backward
//     but the first maximum);
//   * the exponentials of the row sum are kept (16 bits, shared memory) for P.
// 16 sequences of 128 tokens, 64 heads: forward 62 -> 31 us, backward 68 -> 51 us (both at 60 % of the issue slots).
//
// Specification and layouts as in atencao.cuh (jatai_cuda/ops.py:186-258; jatai_cuda/jatai_cuda.cu:822-1006): QKV [Bt*T, 3D]
// block tensor, P uint8 [Bt*H][j][i] with explicit zeros for j > i, raw outputs.
#pragma once
#include "comum.cuh"
#include "atencao.cuh"

namespace jt {
namespace atp {

constexpr int TMAX = 128, HD = 4;
constexpr float DOIS23 = 8388608.0f;

// N per-thread values -> their CTA-wide maxima (blockDim.x a multiple of 32, <= 128; red is [N][4])
template <int N>
__device__ __forceinline__ void max_cta(int (&v)[N], int* red, int tid) {
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = __reduce_max_sync(FULL, v[k]);
    __syncthreads();
    if ((tid & 31) == 0)
#pragma unroll
        for (int k = 0; k < N; k++) red[4 * k + (tid >> 5)] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) {
        v[k] = red[4 * k];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) v[k] = max(v[k], red[4 * k + w]);
    }
}
// four columns of a head, aligned with GA guard bits (ops.py:186-192)
__device__ __forceinline__ int4 alinha(uint32_t w, int s, int GA) {
    return make_int4(rnd_d((int)(int8_t)w << GA, s), rnd_d((int)(int8_t)(w >> 8) << GA, s), rnd_d((int)(int8_t)(w >> 16) << GA, s), rnd_d((int)(int8_t)(w >> 24) << GA, s));
}
// token i's row into the pair layout [T/2][4 columns][2 tokens] of floats
__device__ __forceinline__ void guarda_par(float* d, int i, int4 v) {
    d += (i >> 1) * 8 + (i & 1);
    d[0] = (float)v.x; d[2] = (float)v.y; d[4] = (float)v.z; d[6] = (float)v.w;
}
// the products of one row with the two tokens of pair n
__device__ __forceinline__ uint64_t ponto2(const uint64_t (&a)[4], const float* p, int n) {
    const ulonglong2 x = reinterpret_cast<const ulonglong2*>(p)[2 * n], y = reinterpret_cast<const ulonglong2*>(p)[2 * n + 1];
    return ffma2(a[3], y.y, ffma2(a[2], y.x, ffma2(a[1], x.y, fmul2(a[0], x.x))));
}
__device__ __forceinline__ void grava_cru(int* acc, int16_t* e, size_t p, const int (&o)[4], int ex) {
    const uint32_t e2 = (uint32_t)(ex & 0xffff) | ((uint32_t)ex << 16);
    *reinterpret_cast<int4*>(acc + p) = make_int4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<uint2*>(e + p) = make_uint2(e2, e2);
}

// -------------------------------------------------------------------------------------------------- forward
// ops.py:198-219.  grid Bt*H, T threads (thread = query row).  Row maximum; exponentials and their sum; P (key-major, the threads of a
// warp write consecutive bytes) and O = P . V.
// Dynamic shared memory: k pairs [T][4] | v [T][4] | exponentials, [warp w][8 (w + 1) groups of 4 keys][32 rows] of 4 x 16 bits.
//
// A shift of the scores below 2 (or left, or above 31) leaves the range of the float rounding: such a head, which no trained model has, goes
// the general way, key by key.
__device__ __noinline__ void frente_geral(int i, int* k_s, const int* v_s, int4 q, int s_u, int incl, int kid, long long idx, uint8_t* Pc, int T, int (&o)[4]) {
    auto score = [&](int j) {
        const int4 k = reinterpret_cast<const int4*>(k_s)[j];
        return rnd(q.x * k.x + q.y * k.y + q.z * k.z + q.w * k.w, s_u, kid, idx) - ((i - j) << incl);
    };
    int m = U_MIN;
    for (int j = 0; j <= i; j++) m = max(m, score(j));
    int soma = 0;
    for (int j = 0; j <= i; j++) soma += exp3_dif(m, score(j));
    if (soma <= 0) { reporta(E_DIV, kid, idx, soma, 0); soma = 1; }
    const int inv = (1 << 28) / soma;
    for (int j = 0; j < T; j++) {
        int p = 0;
        if (j <= i) {
            p = min((exp3_dif(m, score(j)) * inv + (1 << 19)) >> 20, 255);
            const int4 v = reinterpret_cast<const int4*>(v_s)[j];
            o[0] += p * v.x; o[1] += p * v.y; o[2] += p * v.z; o[3] += p * v.w;
        }
        Pc[(size_t)j * T] = (uint8_t)p;
    }
}
__global__ void __launch_bounds__(TMAX, 7) k_atencao_peq(const int8_t* __restrict__ qm, const int8_t* __restrict__ qE, int* __restrict__ Oacc,
                                                         int16_t* __restrict__ Oe, uint8_t* __restrict__ P, int T, int H, int D, int GA, int blk, int kid) {
    extern __shared__ __align__(16) unsigned char sm[];
    float* k_s = reinterpret_cast<float*>(sm);
    int* v_s = reinterpret_cast<int*>(sm + T * 16);
    __shared__ int red[12];
    // the warp of the last rows has the most to do and warp n of a block sits on the SM's scheduler n & 3: the rows turn with the block
    const int lane = threadIdx.x & 31, w = ((threadIdx.x >> 5) + blockIdx.x) % (T >> 5), i = 32 * w + lane;
    const int bh = blockIdx.x, b = bh / H, h = bh % H, ld = 3 * D, ldb = ld / blk;
    uint2* ex_s = reinterpret_cast<uint2*>(sm + T * 32 + 1024 * w * (w + 1)) + lane;
    const size_t lin = (size_t)b * T + i;
    pdl_espera();
    pdl_solta();
    const int eq = qE[lin * ldb + (h * HD) / blk], ek = qE[lin * ldb + (D + h * HD) / blk], ev = qE[lin * ldb + (2 * D + h * HD) / blk];
    const uint32_t mq = *reinterpret_cast<const uint32_t*>(qm + lin * ld + h * HD), mk = *reinterpret_cast<const uint32_t*>(qm + lin * ld + D + h * HD),
                   mv = *reinterpret_cast<const uint32_t*>(qm + lin * ld + 2 * D + h * HD);
    int em[3] = {eq, ek, ev};
    max_cta<3>(em, red, threadIdx.x);
    const int4 q = alinha(mq, em[0] - eq, GA), kk = alinha(mk, em[1] - ek, GA);
    const int s_u = -((em[0] - GA) + (em[1] - GA) - 1 + 8), incl = at::incl_alibi(h);
    const bool rapido = s_u >= 2 && s_u <= 31;                     // the same for the whole CTA
    if (rapido) guarda_par(k_s, i, kk);
    else reinterpret_cast<int4*>(k_s)[i] = kk;
    reinterpret_cast<int4*>(v_s)[i] = alinha(mv, em[2] - ev, GA);
    __syncthreads();
    const long long idx = (long long)lin * D + h * HD;
    uint8_t* Ph = P + (size_t)bh * T * T;
    int o[4] = {0, 0, 0, 0};
    if (rapido) {
        const uint64_t qp[4] = {par_f((float)q.x, (float)q.x), par_f((float)q.y, (float)q.y), par_f((float)q.z, (float)q.z), par_f((float)q.w, (float)q.w)};
        const uint64_t esc = par_f(pot2(-s_u), pot2(-s_u)), mag = par_f(MAGIA_F, MAGIA_F);
        const float I = (float)(1 << incl);
        // scores of the pair n: rounded product (biased by 1.5 * 2^23) minus bias and slope; the sums stay below 2^24
        const uint64_t n0 = par_f(-MAGIA_F - (float)i * I, -MAGIA_F - (float)(i - 1) * I), passo = par_f(2 * I, 2 * I), passo2 = par_f(4 * I, 4 * I);
        uint64_t nb = n0;
        auto escores = [&](int n, uint64_t nn) { return fadd2(ffma2(ponto2(qp, k_s, n), esc, mag), nn); };
        float m = -3.0e38f;
#pragma unroll 4
        for (int n = 0; n < 16 * w; n++, nb = fadd2(nb, passo)) {
            const uint64_t u = escores(n, nb);
            m = fmaxf(m, fmaxf(f_lo(u), f_hi(u)));
        }
#pragma unroll 4
        for (int n = 0; n < 16; n++, nb = fadd2(nb, passo)) {      // the diagonal: key 32 w + 2 n (+ 1) counts up to row 32 w + lane
            const uint64_t u = escores(16 * w + n, nb);
            m = fmaxf(m, fmaxf(2 * n <= lane ? f_lo(u) : -3.0e38f, 2 * n < lane ? f_hi(u) : -3.0e38f));
        }
        // m - u + 2^23, exact below 2^24 and no smaller than that beyond: the low bits are the difference once it is cut at 6000
        const uint64_t mm = par_f(m + DOIS23, m + DOIS23), menos = par_f(-1.0f, -1.0f);
        int soma = 0;
        unsigned vivos = 0;                                        // groups of 4 keys with a non-zero exponential in this warp
        nb = n0;
#pragma unroll 1
        for (int g = 0; g < 8 * (w + 1); g++) {
            const uint64_t da = ffma2(escores(2 * g, nb), menos, mm), db = ffma2(escores(2 * g + 1, fadd2(nb, passo)), menos, mm);
            nb = fadd2(nb, passo2);
            float d[4] = {f_lo(da), f_hi(da), f_lo(db), f_hi(db)};
            if (g >= 8 * w) {
                const int c = 4 * (g - 8 * w);
#pragma unroll
                for (int k = 0; k < 4; k++) d[k] = c + k <= lane ? d[k] : 2 * DOIS23;
            }
            // 2130 below the maximum and beyond, exp >> 3 is 0 (p < 2^15, shifted by 12 + 3)
            if (!__any_sync(FULL, fminf(fminf(d[0], d[1]), fminf(d[2], d[3])) < DOIS23 + 2130.0f)) continue;
            vivos |= 1u << g;
            uint32_t e[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                e[k] = (uint32_t)exp3_t(__float_as_uint(fminf(d[k], DOIS23 + 6000.0f)) * 23637u + ((13u << 22) - 0x4B000000u * 23637u));
                soma += (int)e[k];
            }
            ex_s[g * 32] = make_uint2(e[0] | e[1] << 16, e[2] | e[3] << 16);
        }
        if (soma <= 0) { reporta(E_DIV, kid, idx, soma, 0); soma = 1; }
        const int inv = (1 << 28) / soma;
#pragma unroll 1
        for (int g = 0; g < T / 4; g++) {
            if (!(vivos >> g & 1)) {                               // 4 key rows x 32 bytes of zeros
                if (lane < 8) *reinterpret_cast<uint4*>(Ph + (size_t)(4 * g + (lane >> 1)) * T + 32 * w + 16 * (lane & 1)) = make_uint4(0, 0, 0, 0);
                continue;
            }
            const uint2 e = ex_s[g * 32];
            const uint32_t ee[4] = {e.x & 0xffff, e.x >> 16, e.y & 0xffff, e.y >> 16};
            uint8_t* Pc = Ph + (size_t)(4 * g) * T + i;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int p = min(((int)ee[k] * inv + (1 << 19)) >> 20, 255);
                const int4 v = reinterpret_cast<const int4*>(v_s)[4 * g + k];
                o[0] += p * v.x; o[1] += p * v.y; o[2] += p * v.z; o[3] += p * v.w;
                Pc[(size_t)k * T] = (uint8_t)p;
            }
        }
    } else
        frente_geral(i, reinterpret_cast<int*>(k_s), v_s, q, s_u, incl, kid, idx, Ph + i, T, o);
    grava_cru(Oacc, Oe, lin * D + h * HD, o, (em[2] - GA) - 8);
}
inline size_t smem_frente_peq(int T) { return (size_t)T * 32 + 1024 * (T / 32) * (T / 32 + 1); }

// -------------------------------------------------------------------------------------------------- backward
// ops.py:221-258.  grid Bt*H, T threads.  Passes (thread = query row unless stated): max |gP| (or, upper-bound variant, the operand
// norms); s_lin; max |dS|; dS' and gq; then thread = key column: gk and gv.  P of the head sits in shared memory from the diagonal on:
// block b of 32 key rows holds the queries from 32 b, row pitch T - 32 b + 4 bytes (an odd number of words).  What a hand-made P has
// beyond the diagonal is dropped while it is loaded.
// Dynamic shared memory: v pairs [T][4] | k | q | g [T][4] | g pairs [T][4] | s_lin + 1.5 * 2^23's bits [T] | P.
__device__ __forceinline__ int pk_passo(int T, int bl) { return T - 32 * bl + 4; }
__device__ __forceinline__ int pk_base(int T, int bl) { return 32 * bl * (T + 4) - 512 * bl * (bl - 1); }      // sum of 32 (T + 4 - 32 b') over b' < bl

__global__ void __launch_bounds__(TMAX, 7) k_atencao_back_peq(const int8_t* __restrict__ gom, const int8_t* __restrict__ goE, const int8_t* __restrict__ qm,
                                                              const int8_t* __restrict__ qE, const uint8_t* __restrict__ P, int* __restrict__ Gacc,
                                                              int16_t* __restrict__ Ge, int T, int H, int D, int GA, int blk, int limite, int kid) {
    extern __shared__ __align__(16) unsigned char sm[];
    float* v_s = reinterpret_cast<float*>(sm);
    int4* k_s = reinterpret_cast<int4*>(sm + T * 16);
    int4* q_s = k_s + T;
    int4* g_s = q_s + T;
    float* gf_s = reinterpret_cast<float*>(g_s + T);
    int* sl_s = reinterpret_cast<int*>(gf_s + 4 * T);
    uint8_t* P_s = reinterpret_cast<uint8_t*>(sl_s + T);
    __shared__ int red[16];
    // the warp of the last rows has the most to do and warp n of a block sits on the SM's scheduler n & 3: the rows turn with the block
    const int lane = threadIdx.x & 31, w = ((threadIdx.x >> 5) + blockIdx.x) % (T >> 5), i = 32 * w + lane;
    const int bh = blockIdx.x, b = bh / H, h = bh % H, ld = 3 * D, ldb = ld / blk;
    const size_t lin = (size_t)b * T + i;
    pdl_espera();
    pdl_solta();
    const int eg = goE[lin * (D / blk) + (h * HD) / blk], eq = qE[lin * ldb + (h * HD) / blk], ek = qE[lin * ldb + (D + h * HD) / blk],
              ev = qE[lin * ldb + (2 * D + h * HD) / blk];
    const uint32_t mg = *reinterpret_cast<const uint32_t*>(gom + lin * D + h * HD), mq = *reinterpret_cast<const uint32_t*>(qm + lin * ld + h * HD),
                   mk = *reinterpret_cast<const uint32_t*>(qm + lin * ld + D + h * HD), mv = *reinterpret_cast<const uint32_t*>(qm + lin * ld + 2 * D + h * HD);
    int mp = 0;
    {
        const uint4* Pg = reinterpret_cast<const uint4*>(P + (size_t)bh * T * T);
#pragma unroll 1
        for (int bl = 0; bl < T / 32; bl++) {
            const int n16 = T / 16 - 2 * bl;                       // 16-byte pieces of a row from the diagonal block on
            for (int t = i; t < 32 * n16; t += T) {
                const int r = t / n16, c = t % n16, j = 32 * bl + r;
                const uint4 x = Pg[(size_t)j * (T / 16) + 2 * bl + c];
                uint32_t y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int fora = r - 16 * c - 4 * k;           // queries before the key
                    if (fora > 0) y[k] = fora >= 4 ? 0 : y[k] >> (8 * fora) << (8 * fora);
                    reinterpret_cast<uint32_t*>(P_s + pk_base(T, bl) + r * pk_passo(T, bl) + 16 * c)[k] = y[k];
                    if (limite) mp = max(max(mp, (int)(y[k] & 0xff)), max(max((int)(y[k] >> 8 & 0xff), (int)(y[k] >> 16 & 0xff)), (int)(y[k] >> 24)));
                }
            }
        }
    }
    int em[4] = {eg, eq, ek, ev};
    max_cta<4>(em, red, threadIdx.x);
    const int emg = em[0], emq = em[1], emk = em[2], emv = em[3];
    const int4 g = alinha(mg, emg - eg, GA), v = alinha(mv, emv - ev, GA);
    guarda_par(v_s, i, v);
    k_s[i] = alinha(mk, emk - ek, GA);
    q_s[i] = alinha(mq, emq - eq, GA);
    g_s[i] = g;
    guarda_par(gf_s, i, g);
    __syncthreads();
    const uint64_t gp[4] = {par_f((float)g.x, (float)g.x), par_f((float)g.y, (float)g.y), par_f((float)g.z, (float)g.z), par_f((float)g.w, (float)g.w)};
    // shift of gP (to 15 bits): from its exact maximum over j <= i, or from the bounds of the upper-bound variant (ops.py:231-235)
    int sh;
    if (limite) {
        int mx[2] = {max(max(abs(g.x), abs(g.y)), max(abs(g.z), abs(g.w))), abs(v.x) + abs(v.y) + abs(v.z) + abs(v.w)};
        max_cta<2>(mx, red, threadIdx.x);
        sh = max(bitlen(mx[0] * mx[1]) - 15, 0);
    } else {
        float mx = 0.0f;
#pragma unroll 4
        for (int n = 0; n < 16 * w; n++) {
            const uint64_t x = ponto2(gp, v_s, n);
            mx = fmaxf(mx, fmaxf(fabsf(f_lo(x)), fabsf(f_hi(x))));
        }
#pragma unroll 4
        for (int n = 0; n < 16; n++) {
            const uint64_t x = ponto2(gp, v_s, 16 * w + n);
            mx = fmaxf(mx, fmaxf(2 * n <= lane ? fabsf(f_lo(x)) : 0.0f, 2 * n < lane ? fabsf(f_hi(x)) : 0.0f));
        }
        int m1[1] = {(int)mx};
        max_cta<1>(m1, red, threadIdx.x);
        sh = max(bitlen(m1[0]) - 15, 0);
    }
    const uint64_t esc = par_f(pot2(-sh), pot2(-sh)), mag = par_f(MAGIA_F, MAGIA_F);
    // bit patterns of gP' + 1.5 * 2^23 for 4 keys (|gP'| <= 2^15; the sums below wrap like the specification's, so the bias comes off at the end)
    auto gpl4 = [&](const uint64_t (&um)[4], const float* outro, int n, uint32_t (&x)[4]) {
        const uint64_t a = ffma2(ponto2(um, outro, 2 * n), esc, mag), c = ffma2(ponto2(um, outro, 2 * n + 1), esc, mag);
        x[0] = (uint32_t)a; x[1] = (uint32_t)(a >> 32); x[2] = (uint32_t)c; x[3] = (uint32_t)(c >> 32);
    };
    auto gpl = [&](int n, uint32_t (&x)[4]) { gpl4(gp, v_s, n, x); };
    // s_lin of this row, then the maxima that give the shift of dS (to 12 bits) (ops.py:236-244)
    uint32_t s = 0, sp = 0;
    unsigned vivos = 0;                                            // groups of 4 keys in which this warp has a non-zero P
#pragma unroll 1
    for (int bl = 0; bl <= w; bl++) {
        const int pp = pk_passo(T, bl);
        const uint8_t* p = P_s + pk_base(T, bl) + i - 32 * bl;
        uint32_t soma[8];
#pragma unroll
        for (int n = 0; n < 8; n++) {
            soma[n] = (uint32_t)p[(4 * n) * pp] + p[(4 * n + 1) * pp] + p[(4 * n + 2) * pp] + p[(4 * n + 3) * pp];
            sp += soma[n];
        }
#pragma unroll
        for (int n = 0; n < 8; n++) vivos |= (__any_sync(FULL, soma[n] != 0) ? 1u : 0u) << (8 * bl + n);
    }
    // f(first key of the group, the four P of this row, the four gP') over those groups
    auto anda = [&](auto f) {
#pragma unroll 2
        for (unsigned m = vivos; m; m &= m - 1) {
            const int n = __ffs(m) - 1, bl = n >> 3, pp = pk_passo(T, bl);
            const uint8_t* p = P_s + pk_base(T, bl) + i - 32 * bl + 4 * (n & 7) * pp;
            const uint32_t pv[4] = {p[0], p[pp], p[2 * pp], p[3 * pp]};
            uint32_t x[4];
            gpl(n, x);
            f(4 * n, pv, x);
        }
    };
    anda([&](int, const uint32_t (&p)[4], const uint32_t (&x)[4]) {
#pragma unroll
        for (int k = 0; k < 4; k++) s += p[k] * x[k];
    });
    const int sl = rnd_d((int)(s - MAGIA * sp), 8);
    const uint32_t tira = MAGIA + (uint32_t)sl;
    sl_s[i] = (int)tira;
    int sh2;
    {
        int mds = 0;
        anda([&](int, const uint32_t (&p)[4], const uint32_t (&x)[4]) {
#pragma unroll
            for (int k = 0; k < 4; k++) mds = max(mds, abs((int)(p[k] * (x[k] - tira))));
        });
        if (limite) {
            int mgq = 0;
            for (int n = 0; n < 8 * (w + 1); n++) {
                uint32_t x[4];
                gpl(n, x);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (4 * n + k <= i) mgq = max(mgq, abs((int)(x[k] - MAGIA)));
            }
            int mx[3] = {mp, mgq, abs(sl)};
            max_cta<3>(mx, red, threadIdx.x);
            sh2 = max(bitlen(mx[0] * (mx[1] + mx[2])) - 12, 0);
        } else {
            int mx[1] = {mds};
            max_cta<1>(mx, red, threadIdx.x);
            sh2 = max(bitlen(mx[0]) - 12, 0);
        }
    }
    const int eds = (emg - GA) + (emv - GA) + sh - 9 + sh2;
    const Arred arred2(sh2);
    // gq of this row
    int o[4] = {0, 0, 0, 0};
    anda([&](int j, const uint32_t (&p)[4], const uint32_t (&x)[4]) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int ds = arred2((int)(p[k] * (x[k] - tira)));
            const int4 y = k_s[j + k];
            o[0] += ds * y.x; o[1] += ds * y.y; o[2] += ds * y.z; o[3] += ds * y.w;
        }
    });
    grava_cru(Gacc, Ge, lin * 3 * D + h * HD, o, eds + (emk - GA));
    // (max_cta had the whole CTA past the writes of sl_s)
    // thread = key j = i: gk[j] = sum_{r >= j} dS'[r][j] q[r], gv[j] = sum_{r >= j} P[r][j] dO[r]
    int gk[4] = {0, 0, 0, 0}, gv[4] = {0, 0, 0, 0};
    const uint32_t* pk = reinterpret_cast<const uint32_t*>(P_s + pk_base(T, w) + lane * pk_passo(T, w));
    unsigned vivas = 0;                                            // groups of 4 queries in which this warp's keys have a non-zero P
#pragma unroll 8
    for (int n = 8 * w; n < T / 4; n++) vivas |= (__any_sync(FULL, pk[n - 8 * w] != 0) ? 1u : 0u) << n;
    const uint64_t vp[4] = {par_f((float)v.x, (float)v.x), par_f((float)v.y, (float)v.y), par_f((float)v.z, (float)v.z), par_f((float)v.w, (float)v.w)};
#pragma unroll 2
    for (unsigned m = vivas; m; m &= m - 1) {
        const int n = __ffs(m) - 1;
        const uint32_t p4 = pk[n - 8 * w];
        uint32_t x[4];
        gpl4(vp, gf_s, n, x);
        const int4 sl4 = reinterpret_cast<const int4*>(sl_s)[n];
        const int tl[4] = {sl4.x, sl4.y, sl4.z, sl4.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int p = (int)__byte_perm(p4, 0, 0x4440 + k);
            const int4 y = g_s[4 * n + k], z = q_s[4 * n + k];
            const int ds = arred2(p * ((int)x[k] - tl[k]));
            gv[0] += p * y.x; gv[1] += p * y.y; gv[2] += p * y.z; gv[3] += p * y.w;
            gk[0] += ds * z.x; gk[1] += ds * z.y; gk[2] += ds * z.z; gk[3] += ds * z.w;
        }
    }
    grava_cru(Gacc, Ge, lin * 3 * D + D + h * HD, gk, eds + (emq - GA));
    grava_cru(Gacc, Ge, lin * 3 * D + 2 * D + h * HD, gv, (emg - GA) - 8);
}
inline size_t smem_back_peq(int T) {
    const int nb = T / 32;
    return (size_t)T * 84 + 32 * nb * (T + 4) - 512 * nb * (nb - 1);
}

}  // namespace atp

static bool atp_serve(int blk, int T, int H, int D, int GA) {
    return D == H * atp::HD && T % 32 == 0 && T <= atp::TMAX && D % blk == 0 && GA >= 0 && GA <= 4;
}

static int atencao_frente_peq(int blk, const int8_t* qm, const int8_t* qE, int* Oacc, int16_t* Oe, uint8_t* P, int Bt, int T, int H, int D, int GA,
                              int kid, cudaStream_t st) {
    lanca_pdl(atp::k_atencao_peq, dim3(Bt * H), dim3(T), atp::smem_frente_peq(T), st, qm, qE, Oacc, Oe, P, T, H, D, GA, blk, kid);
    return (int)cudaGetLastError();
}
static int atencao_tras_peq(int blk, const int8_t* gom, const int8_t* goE, const int8_t* qm, const int8_t* qE, const uint8_t* P, int* Gacc, int16_t* Ge,
                            int Bt, int T, int H, int D, int GA, int limite, int kid, cudaStream_t st) {
    lanca_pdl(atp::k_atencao_back_peq, dim3(Bt * H), dim3(T), atp::smem_back_peq(T), st, gom, goE, qm, qE, P, Gacc, Ge, T, H, D, GA, blk, limite, kid);
    return (int)cudaGetLastError();
}

}  // namespace jt
