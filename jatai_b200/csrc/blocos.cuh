// Bandwidth-bound block kernels: quant, soma, relu2(+back), momento, peso, embed, um_quente, transpoe,
// rms(+back), softmax_ce.  One pass over HBM each, 128-bit accesses.
//
// Work decomposition (all kernels): one thread owns 16 consecutive elements of a row = one 128-bit load of
// int8 mantissas; GL = BLK/16 neighbouring lanes own one exponent block and reduce with xor-shuffles.
// Arithmetic: the int64 specification of the reference (jatai_cuda/ops.py, cited per kernel) in int32.
#pragma once
#include "comum.cuh"

namespace jt {

#define JT_FIO16                                                                         \
    const long long t_ = (long long)blockIdx.x * blockDim.x + threadIdx.x;               \
    const bool ativo = t_ < n16;                                                         \
    const long long t16 = ativo ? t_ : 0;   /* idle lanes recompute thread 0, store nothing */ \
    const long long o = t16 * 16;                                                        \
    const long long w = o / BLK;                                                         \
    const bool lider = ativo && (t16 % (BLK / 16) == 0);

// raw (acc int32, e int16 per element) -> block.  ops.py:125-126
template <int BLK>
__global__ void __launch_bounds__(256, 4) k_quant(const int* __restrict__ acc, const int16_t* __restrict__ e, int8_t* __restrict__ m,
                                               int8_t* __restrict__ E, long long n16, int kid) {
    JT_FIO16
    int v[16], ee[16], q[16];
    le16_i32(acc + o, v);
    le16_i16(e + o, ee);
    {
        // fp32 path (a whole warp or none): every |v| <= 2^24 is exact in fp32, v * 2^(e - largest exponent of a non-zero value
        // of the block) is an exact scaling while the exponents are at most 100 apart, and the fp32 quantiser then gives the
        // bits of the integer one (the block's top bit and the one-more-bit retry depend on the largest scaled magnitude alone)
        int eref = -32768, big = 0;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            big |= (v[i] > (1 << 24)) | (v[i] < -(1 << 24));
            if (v[i] != 0) eref = max(eref, ee[i]);
        }
        eref = grupo_max<BLK / 16>(eref);
#pragma unroll
        for (int i = 0; i < 16; i++) big |= (v[i] != 0) & (eref - ee[i] > 100);
        if (__all_sync(FULL, big == 0)) {
            float f[16];
#pragma unroll
            for (int i = 0; i < 16; i++) f[i] = (float)v[i] * __int_as_float((127 + max(min(ee[i] - eref, 0), -100)) << 23);
            uint4 pac;
            const int Eo = quant_f32<BLK / 16>(f, eref, pac, kid, o);
            if (ativo) *reinterpret_cast<uint4*>(m + o) = pac;
            if (lider) E[w] = (int8_t)Eo;
            return;
        }
    }
    // blocks whose elements all carry one exponent (attention outputs: one exponent per head) take the cheaper
    // uniform quantiser; the choice is made per block, the lanes of a block always agree
    int dif = 0;
#pragma unroll
    for (int i = 1; i < 16; i++) dif |= ee[i] ^ ee[0];
    dif |= ee[0] ^ __shfl_sync(FULL, ee[0], (threadIdx.x & 31) & ~(BLK / 16 - 1));
    dif = grupo_or<BLK / 16>(dif);
    const unsigned m_uni = __ballot_sync(FULL, dif == 0);
    int Eo;
    if (dif == 0) Eo = quant_uniforme<16, BLK / 16>(v, ee[0], q, kid, o, m_uni);
    else Eo = quant_geral<16, BLK / 16>(v, ee, q, kid, o, ~m_uni);
    if (ativo) grava16(m + o, q);
    if (lider) E[w] = (int8_t)Eo;
}

// ---- several 16-element chunks per thread --------------------------------------------------------------
// A thread issues the 128-bit loads of U chunks (one every gridDim*blockDim chunks, so lane groups stay aligned)
// before it touches any of them: with one chunk per thread the ~1300 resident threads of an SM keep only ~20 KB in
// flight, far less than the ~45 KB that HBM latency x bandwidth asks for.
#define JT_PEDACO(k)                                                                      \
    const long long tk_ = t0_ + (long long)(k) * nth_;                                    \
    const bool ativo = tk_ < n16;                                                         \
    const long long t16 = ativo ? tk_ : 0;                                                \
    const long long o = t16 * 16;                                                         \
    const long long w = o / BLK;                                                          \
    const bool lider = ativo && (t16 % (BLK / 16) == 0);
#define JT_MULTI                                                                          \
    const long long nth_ = (long long)gridDim.x * blockDim.x;                             \
    const long long t0_ = (long long)blockIdx.x * blockDim.x + threadIdx.x;

// One 16-element chunk of z = x + y (see k_soma below for the arithmetic); the GL lanes of a block call together.
// Returns the block exponent, `pac` receives the 16 mantissas.
template <int GL, int ST = 1>
__device__ __forceinline__ int soma16(const int (&xv)[16], int ex, const int (&yv)[16], int ey, uint4& pac, int kid, long long o) {
    const bool x_maior = ex >= ey;
    const int eH = x_maior ? ex : ey, d = x_maior ? ex - ey : ey - ex;
    const int dl = min(d, 21), s2 = d - dl;                         // s2 > 0: the far operand is rounded first
    int hi[16], lo[16], wv[16];
#pragma unroll
    for (int i = 0; i < 16; i++) { hi[i] = x_maior ? xv[i] : yv[i]; lo[i] = x_maior ? yv[i] : xv[i]; }
    int mx = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        wv[i] = (hi[i] << dl) + rnd_d(lo[i], s2);
        mx = max(mx, wv[i] < 0 ? -wv[i] : wv[i]);
    }
    mx = grupo_max<GL, ST>(mx);
    int s = bitlen(mx) - 7;
    if (desloca(mx, s) > 127) s += 1;
    const int E = eH - dl + s;
    pac = make_uint4(0, 0, 0, 0);
    int Eo = E_ZERO;
    if (mx != 0 && E >= -126) {
        if (E > 126) reporta(E_EXP, kid, o, E, eH);
        Eo = E;
        int q[16];
        if (s > 0) {
            const int c = (1 << (s - 1)) - 1;
#pragma unroll
            for (int i = 0; i < 16; i++) q[i] = (wv[i] + c + ((wv[i] >> s) & 1)) >> s;
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) q[i] = wv[i] << (-s);
        }
        pac.x = junta4(q[0], q[1], q[2], q[3]);
        pac.y = junta4(q[4], q[5], q[6], q[7]);
        pac.z = junta4(q[8], q[9], q[10], q[11]);
        pac.w = junta4(q[12], q[13], q[14], q[15]);
    }
    return Eo;
}

// One lane's 16 elements of the sum of two block tensors, in fp32 where the exponents are at most 16 apart (k_soma has the reasons)
template <int GL, int ST = 1>
__device__ __forceinline__ int soma16_misto(const uint4& rx, int ex, const uint4& ry, int ey, uint4& pac, int kid, long long o) {
    const bool x_maior = ex >= ey;
    const int eH = x_maior ? ex : ey, eL = x_maior ? ey : ex;
    const uint4 rl = x_maior ? ry : rx;
    const int d = (eL == E_ZERO && (rl.x | rl.y | rl.z | rl.w) == 0) ? 0 : eH - eL;
    if (__all_sync(FULL, d <= 16)) {
        float fx[16], fy[16];
        bytes_para_float(rx, fx);
        bytes_para_float(ry, fy);
        const float a = x_maior ? __int_as_float((127 + d) << 23) : 1.f, b = x_maior ? 1.f : __int_as_float((127 + d) << 23);
#pragma unroll
        for (int i = 0; i < 16; i++) fx[i] = fmaf(fx[i], a, fy[i] * b);
        return quant_f32<GL, ST>(fx, eH - d, pac, kid, o);
    }
    int xv[16], yv[16];
    desempacota16(rx, xv);
    desempacota16(ry, yv);
    return soma16<GL, ST>(xv, ex, yv, ey, pac, kid, o);
}

// z = x + y.  ops.py:128-132: ec = max(xE, yE) - 21; v = rnd(x, ec - xE) + rnd(y, ec - yE); quant(v, ec).
// With hi / lo = the operand of larger / smaller exponent and d their distance, v = 2^(21-dl) * w where dl = min(d, 21),
// w = hi * 2^dl + lo' and lo' = lo (d <= 21) or rnd(lo, d - 21) (the specification rounds the far operand first).
// The quantiser is invariant under the common power of two, so the block is quant(w, e_hi - dl): the same bits with
// 28-bit instead of 30-bit intermediates, one code path for every d, and rounding shifts shared by the block.
template <int BLK, int U = 4>
__global__ void __launch_bounds__(256, 3) k_soma(const int8_t* __restrict__ xm, const int8_t* __restrict__ xE, const int8_t* __restrict__ ym,
                                              const int8_t* __restrict__ yE, int8_t* __restrict__ zm, int8_t* __restrict__ zE,
                                              long long n16, int kid) {
    constexpr int GL = BLK / 16;
    JT_MULTI
    uint4 rx[U], ry[U];
    int ex[U], ey[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
        JT_PEDACO(k)
        rx[k] = *reinterpret_cast<const uint4*>(xm + o);
        ry[k] = *reinterpret_cast<const uint4*>(ym + o);
        ex[k] = xE[w];
        ey[k] = yE[w];
        (void)lider;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
        JT_PEDACO(k)
        uint4 pac;
        int Eo;
        // fp32 path: with the exponents at most 16 apart w = hi * 2^d + lo is below 2^24, exact in fp32, and the fp32 quantiser
        // gives the bits of the integer one; an all-zero block on either side leaves the other operand alone.  Taken by a
        // whole warp or not at all (the quantisers shuffle inside the lane groups of a block).
        Eo = soma16_misto<GL>(rx[k], ex[k], ry[k], ey[k], pac, kid, o);
        if (ativo) *reinterpret_cast<uint4*>(zm + o) = pac;
        if (lider) zE[w] = (int8_t)Eo;
    }
}

// a = max(h, 0)^2.  ops.py:134-137.  fp32 path: h^2 <= 16129 is exact
template <int BLK, int U = 4>
__global__ void __launch_bounds__(256) k_relu2(const int8_t* __restrict__ hm, const int8_t* __restrict__ hE, int8_t* __restrict__ am,
                                               int8_t* __restrict__ aE, long long n16, int kid) {
    JT_MULTI
    uint4 rh[U];
    int eh[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
        JT_PEDACO(k)
        rh[k] = *reinterpret_cast<const uint4*>(hm + o);
        eh[k] = hE[w];
        (void)lider;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
        JT_PEDACO(k)
        float f[16];
        bytes_para_float(rh[k], f);
#pragma unroll
        for (int i = 0; i < 16; i++) { const float r = fmaxf(f[i], 0.f); f[i] = r * r; }
        uint4 pac;
        const int Eo = quant_f32<BLK / 16>(f, 2 * eh[k], pac, kid, o);
        if (ativo) *reinterpret_cast<uint4*>(am + o) = pac;
        if (lider) aE[w] = (int8_t)Eo;
    }
}

// gh = g * 2 * max(h, 0).  ops.py:139-141.  fp32 path: |g h 2| <= 32258 is exact
template <int BLK, int U = 4>
__global__ void __launch_bounds__(256) k_relu2_back(const int8_t* __restrict__ gm, const int8_t* __restrict__ gE, const int8_t* __restrict__ hm,
                                                    const int8_t* __restrict__ hE, int8_t* __restrict__ om, int8_t* __restrict__ oE,
                                                    long long n16, int kid) {
    JT_MULTI
    uint4 rg[U], rh[U];
    int ee[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
        JT_PEDACO(k)
        rg[k] = *reinterpret_cast<const uint4*>(gm + o);
        rh[k] = *reinterpret_cast<const uint4*>(hm + o);
        ee[k] = (int)gE[w] + (int)hE[w];
        (void)lider;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
        JT_PEDACO(k)
        float g[16], h[16];
        bytes_para_float(rg[k], g);
        bytes_para_float(rh[k], h);
#pragma unroll
        for (int i = 0; i < 16; i++) g[i] = g[i] * fmaxf(h[i], 0.f) * 2.f;
        uint4 pac;
        const int Eo = quant_f32<BLK / 16>(g, ee[k], pac, kid, o);
        if (ativo) *reinterpret_cast<uint4*>(om + o) = pac;
        if (lider) oE[w] = (int8_t)Eo;
    }
}

// momentum, in place: m <- quant(rnd(7 m, ec - em) + rnd(g, ec - eg), ec), em = ME - 3,
// per element ec = max(em + 10, eg + bitlen(g)) - 28.  ops.py:273-278.  The 16 elements of a lane, in double precision: the two roundings are
// fused multiply-adds (the second sum leaves v + 1.5 * 2^52), the bit lengths exponent fields, the quantiser's rounding a third one.
// Returns the block exponent; `pac` receives the mantissas.  (All int before: 72 instructions per element, a third of them at the
// quarter rate of clz: 65 us at 16384 x 1024, now 36; the traffic's floor is 21.)
template <int GL>
__device__ __forceinline__ int momento16(const uint4& m4, int em, const int (&g)[16], const int (&eg)[16], uint4& pac, int kid, long long o) {
    const uint32_t mw[4] = {m4.x, m4.y, m4.z, m4.w};
    int v[16], ec[16], topo = SEM_TOPO, blmax = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const double gd = int_para_d(g[i]);
        const int bl = bitlen_d(gd);
        blmax = max(blmax, bl);
        ec[i] = max(em + 10, eg[i] + bl) - 28;
        const double a = fma(gd, pot2_d(eg[i] - ec[i]), MAGIA_D), b = fma(int_para_d(byte_s(mw[i >> 2], i & 3) * 7), pot2_d(em - ec[i]), MAGIA_D);
        const double t = (a - MAGIA_D) + b;
        v[i] = __double2loint(t);
        const int bv = (__double2hiint(t - MAGIA_D) >> 20) & 0x7ff;
        topo = max(topo, bv == 0 ? SEM_TOPO : bv - 1022 + ec[i]);
    }
    if (blmax > 30) {                                              // (cold) a gradient at or beyond 2^30
#pragma unroll
        for (int i = 0; i < 16; i++)
            if (g[i] >= LIM || g[i] <= -LIM) reporta(E_ACUM, kid, o + i, g[i], eg[i]);
    }
    topo = grupo_max<GL>(topo);
    pac = make_uint4(0, 0, 0, 0);
    if (topo == SEM_TOPO) topo = -10000;
    int E = topo - 7;
    uint32_t q[16];
    int qm = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        q[i] = (uint32_t)__double2loint(fma(int_para_d(v[i]), pot2_d(ec[i] - E), MAGIA_D));
        qm = max(qm, abs((int)q[i]));
    }
    if (grupo_max<GL>(qm) > 127) {
        E += 1;
#pragma unroll
        for (int i = 0; i < 16; i++) q[i] = (uint32_t)__double2loint(fma(int_para_d(v[i]), pot2_d(ec[i] - E), MAGIA_D));
    }
    if (E < -126) return E_ZERO;
    if (E > 126) reporta(E_EXP, kid, o, E, topo);
    pac = junta16(q);
    return E;
}

// weight step with error feedback: W <- quant(W - M 2^-k + R), R <- quant(what that rounding lost).  ops.py:280-290.  The exponents are
// those of the blocks, so the three alignments are multiplications by one power of two each (an operand 2^20 below the
// largest or less is rounded first: cold), and the residual, below 2^23, goes through the fp32 quantiser.
// (57 us at 16384 x 1024 with integer shifts throughout, now 24 on its own, 28 behind the momentum.)
template <int GL>
__device__ __forceinline__ void peso16(const uint4& w4, int ew, const uint4& m4, int em, const uint4& r4, int er, bool ef, uint4& pw, int& Ew, uint4& pr, int& Er,
                                       int kid, long long o) {
    const uint32_t ww[4] = {w4.x, w4.y, w4.z, w4.w}, mw[4] = {m4.x, m4.y, m4.z, m4.w}, rw[4] = {r4.x, r4.y, r4.z, r4.w};
    const int ec = max(max(ew + 7, em + 7), er + 7) - 27;
    const int dw = ew - ec, dm = em - ec, dr = ef ? er - ec : -100;          // at most 20
    auto fator = [](int d) { return d >= 0 ? 1 << d : 0; };
    auto certo = [](int d) { return d >= 0 || d <= -8; };                    // a mantissa is below 2^7: 8 places down it rounds to 0
    int v[16], mx = 0;
    if (__all_sync(FULL, certo(dw) && certo(dm) && certo(dr))) {
        const int fw = fator(dw), fm = -fator(dm), fr = fator(dr);
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = byte_s(ww[i >> 2], i & 3) * fw + byte_s(mw[i >> 2], i & 3) * fm + byte_s(rw[i >> 2], i & 3) * fr;
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++)
            v[i] = desloca(byte_s(ww[i >> 2], i & 3), -dw) - desloca(byte_s(mw[i >> 2], i & 3), -dm) + (ef ? desloca(byte_s(rw[i >> 2], i & 3), -dr) : 0);
    }
#pragma unroll
    for (int i = 0; i < 16; i++) mx = max(mx, abs(v[i]));
    mx = grupo_max<GL>(mx);
    int sh = bitlen(mx) - 7;
    if (desloca(mx, sh) > 127) sh += 1;
    const int E = ec + sh;
    uint32_t q[16];
    pw = pr = make_uint4(0, 0, 0, 0);
    Ew = Er = E_ZERO;
    if (mx != 0 && E >= -126) {
        if (E > 126) reporta(E_EXP, kid, o, E, ec);
        Ew = E;
        if (sh > 0) {
            const int c = (1 << (sh - 1)) - 1;
#pragma unroll
            for (int i = 0; i < 16; i++) q[i] = (uint32_t)((v[i] + c + ((v[i] >> sh) & 1)) >> sh);
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) q[i] = (uint32_t)(v[i] << (-sh));
        }
        pw = junta16(q);
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) q[i] = 0;
        sh = 0;
    }
    if (!ef) return;
    // what the rounding lost: v - q 2^sh, at most 2^(sh - 1) <= 2^22, or (a block flushed to zero) v itself
    float f[16];
    bool cabe = true;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        v[i] -= sh > 0 ? (int)q[i] << sh : (int)q[i] >> -sh;
        f[i] = (float)v[i];
        cabe = cabe && abs(v[i]) <= (1 << 24);
    }
    if (__all_sync(FULL, cabe)) Er = quant_f32<GL>(f, ec, pr, kid, o);
    else {
        int r[16];
        Er = quant_uniforme<16, GL>(v, ec, r, kid, o);
#pragma unroll
        for (int i = 0; i < 16; i++) q[i] = (uint32_t)r[i];
        pr = junta16(q);
    }
}

template <int BLK>
__global__ void __launch_bounds__(128, 5) k_momento(const int* __restrict__ gacc, const int16_t* __restrict__ ge, int8_t* __restrict__ Mm,
                                                 int8_t* __restrict__ ME, long long n16, int kid) {
    JT_FIO16
    int g[16], eg[16];
    const uint4 m4 = *reinterpret_cast<const uint4*>(Mm + o);
    le16_i32(gacc + o, g);
    le16_i16(ge + o, eg);
    uint4 pac;
    const int Eo = momento16<BLK / 16>(m4, (int)ME[w] - 3, g, eg, pac, kid, o);
    if (ativo) *reinterpret_cast<uint4*>(Mm + o) = pac;
    if (lider) ME[w] = (int8_t)Eo;
}

template <int BLK>
__global__ void __launch_bounds__(256) k_peso(int8_t* __restrict__ Wm, int8_t* __restrict__ WE, const int8_t* __restrict__ Mm,
                                              const int8_t* __restrict__ ME, int8_t* __restrict__ Rm, int8_t* __restrict__ RE, int k_lr, int ef,
                                              long long n16, int kid) {
    JT_FIO16
    const uint4 w4 = *reinterpret_cast<const uint4*>(Wm + o), m4 = *reinterpret_cast<const uint4*>(Mm + o);
    const uint4 r4 = ef ? *reinterpret_cast<const uint4*>(Rm + o) : make_uint4(0, 0, 0, 0);
    uint4 pw, pr;
    int Ew, Er;
    peso16<BLK / 16>(w4, WE[w], m4, (int)ME[w] - k_lr, r4, ef ? (int)RE[w] : E_ZERO, ef != 0, pw, Ew, pr, Er, kid, o);
    if (ativo) *reinterpret_cast<uint4*>(Wm + o) = pw;
    if (lider) WE[w] = (int8_t)Ew;
    if (!ef) return;
    if (ativo) *reinterpret_cast<uint4*>(Rm + o) = pr;
    if (lider) RE[w] = (int8_t)Er;
}

// momentum and weight step of the same 16 elements in one launch (the optimiser of a weight is always this pair):
// k_momento followed by k_peso on the momentum just written, which stays in registers.
template <int BLK>
__global__ void __launch_bounds__(128, 5) k_momento_peso(const int* __restrict__ gacc, const int16_t* __restrict__ ge, int8_t* __restrict__ Mm,
                                                      int8_t* __restrict__ ME, int8_t* __restrict__ Wm, int8_t* __restrict__ WE,
                                                      int8_t* __restrict__ Rm, int8_t* __restrict__ RE, int k_lr, int ef, long long n16, int kid) {
    pdl_espera();
    pdl_solta();
    JT_FIO16
    int g[16], eg[16];
    uint4 m4 = *reinterpret_cast<const uint4*>(Mm + o);
    le16_i32(gacc + o, g);
    le16_i16(ge + o, eg);
    const int em = (int)ME[w] - 3, ew = WE[w], er = ef ? (int)RE[w] : E_ZERO;
    const uint4 w4 = *reinterpret_cast<const uint4*>(Wm + o);
    const uint4 r4 = ef ? *reinterpret_cast<const uint4*>(Rm + o) : make_uint4(0, 0, 0, 0);
    const int Em = momento16<BLK / 16>(m4, em, g, eg, m4, kid, o);
    if (ativo) *reinterpret_cast<uint4*>(Mm + o) = m4;
    if (lider) ME[w] = (int8_t)Em;
    uint4 pw, pr;
    int Ew, Er;
    peso16<BLK / 16>(w4, ew, m4, (int)(int8_t)Em - k_lr, r4, er, ef != 0, pw, Ew, pr, Er, kid, o);
    if (ativo) *reinterpret_cast<uint4*>(Wm + o) = pw;
    if (lider) WE[w] = (int8_t)Ew;
    if (!ef) return;
    if (ativo) *reinterpret_cast<uint4*>(Rm + o) = pr;
    if (lider) RE[w] = (int8_t)Er;
}

// row gather of the embedding table; an out-of-range token zeroes the row and records E_ARG.  ops.py:143-145
template <int BLK>
__global__ void __launch_bounds__(256) k_embed(const int8_t* __restrict__ Wm, const int8_t* __restrict__ WE, const int* __restrict__ tok,
                                               int8_t* __restrict__ Xm, int8_t* __restrict__ XE, int M, int D, int V, int kid) {
    pdl_espera();
    pdl_solta();
    const int por_linha = D / 16;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)M * por_linha) return;
    const int lin = (int)(t / por_linha), c = (int)(t % por_linha) * 16;
    const int tk = tok[lin];
    const bool ok = tk >= 0 && tk < V;
    if (!ok && c == 0) reporta(E_ARG, kid, (long long)lin * D, tk, V);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (ok) v = *reinterpret_cast<const uint4*>(Wm + (size_t)tk * D + c);
    *reinterpret_cast<uint4*>(Xm + (size_t)lin * D + c) = v;
    if (c % BLK == 0) XE[(size_t)lin * (D / BLK) + c / BLK] = ok ? WE[(size_t)tk * (D / BLK) + c / BLK] : (int8_t)E_ZERO;
}

// one-hot rows with exponent 0 (the embedding gradient is a GEMM on them).  ops.py:147-151
template <int BLK>
__global__ void __launch_bounds__(256) k_um_quente(const int* __restrict__ tok, int8_t* __restrict__ U, int8_t* __restrict__ UE, int M, int V,
                                                   int kid) {
    pdl_espera();
    pdl_solta();
    const int por_linha = V / 16;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)M * por_linha) return;
    const int lin = (int)(t / por_linha), c = (int)(t % por_linha) * 16;
    const int tk = tok[lin];
    if ((tk < 0 || tk >= V) && c == 0) reporta(E_ARG, kid, (long long)lin * V, tk, V);
    uint32_t u[4] = {0, 0, 0, 0};
    if (tk >= c && tk < c + 16) u[(tk - c) >> 2] = 1u << (8 * ((tk - c) & 3));
    *reinterpret_cast<uint4*>(U + (size_t)lin * V + c) = make_uint4(u[0], u[1], u[2], u[3]);
    if (c % BLK == 0) UE[(size_t)lin * (V / BLK) + c / BLK] = 0;
}

// per-byte signed maximum into a 4-byte-aligned word of an int8 array
__device__ __forceinline__ void max4_atomico(int8_t* p, uint32_t meu) {
    unsigned* w = reinterpret_cast<unsigned*>(p);
    unsigned visto = *w;
    for (;;) {
        const unsigned novo = __vmaxs4(visto, meu);
        if (novo == visto) return;
        const unsigned antes = atomicCAS(w, visto, novo);
        if (antes == visto) return;
        visto = antes;
    }
}

// [R,C] blocked along C -> [C,R] blocked along R; the new blocks span BLK rows of one column, so every element brings its own exponent and the
// block is quantised again.  ops.py:121-123
//
// A warp takes 32 rows x 128 columns straight from global memory: a lane loads the word of its 4 columns in every row (32 coalesced 128-byte
// loads in flight per warp, no shared memory, no barrier), which is four 32-element columns; the exponents, a row per lane, travel by
// shuffles.  The quantiser runs in fp32, exactly: a mantissa times 2^(e - eref) is exact, the largest magnitude gives
// top = max(e + bitlen(v)) through its exponent field, and one FFMA against 1.5*2^23 rounds v * 2^(e - E) half to even
// (|result| <= 127, inside the window).  A transposed block can never need the "one more bit" retry (|m| <= 127 going in).  Rows whose
// exponents are more than 100 apart take integers.  Block 128: the four warps of a CTA (128 rows) exchange their columns' tops first.
// Block 32: where the exponents lie at most 24 apart, two rows at a time in halves, which are as exact there (4 instructions an element instead of 11; the
// rows' factors go through shared memory as halves).  16384 x (4096 + 1024) 65.7 -> 59.5 us, 2048 x (512 + 2048) 7.4 -> 6.95: what is left is the
// latency of a warp's 32 loads at 16 warps an SM (128 registers, for the fp32 form).
// CPT = 4: a lane does its 4 columns; CPT = 1, for matrices that would leave SMs idle: four warps share the 32 x 128 piece, a column each.
// (Tiles staged in shared memory before, two shared loads per element: 16384 x (4096 + 1024) 95 -> 66 us, block 128 154 -> 50 us; 128 x 128
// 6.4 -> 2.1 us.)
struct ArgsTransp { const int8_t* X; const int8_t* EX; int8_t* Y; int8_t* EY; int C; int8_t* RM; };

// (cold) the 32 rows of one column in integers, read again: e + bitlen of the largest / the mantissas for the exponent Eo
__device__ __noinline__ int transpoe_topo_lento(const int8_t* X, const int8_t* E, int C, int nbx) {
    int topo = SEM_TOPO;
    for (int i = 0; i < 32; i++)
        if (X[(size_t)i * C] != 0) topo = max(topo, (int)E[(size_t)i * nbx] + bitlen(X[(size_t)i * C]));
    return topo;
}
__device__ __noinline__ void transpoe_grava_lento(const int8_t* X, const int8_t* E, int C, int nbx, int Eo, int8_t* dst) {
    for (int i = 0; i < 32; i++) {
        const int v = X[(size_t)i * C];
        dst[i] = (int8_t)(Eo == E_ZERO || v == 0 ? 0 : desloca(v, Eo - (int)E[(size_t)i * nbx]));
    }
}

template <bool B> struct SimNao { static constexpr bool v = B; };
template <int BLK, int CPT>
__device__ __forceinline__ void transpoe_corpo(const ArgsTransp& A, int r0, int c0, int R, int kid) {
    pdl_espera();
    pdl_solta();
    __shared__ int topos[BLK == 128 ? 4 : 1][BLK == 128 ? 128 : 1];
    // block 32: a CTA is 32 rows (CPT = 1) or 128; block 128 always 128, its four 32-row groups belong together
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rg = CPT == 1 && BLK == 32 ? 0 : wid & 3, k0 = CPT == 1 ? (BLK == 32 ? wid : wid >> 2) : 0;
    const int C = A.C, nbx = C / BLK, nby = R / BLK, col0 = c0 + 4 * lane, lin0 = r0 + rg * 32;
    const bool dentro = col0 < C;
    // lane r: the exponents of row r, one byte per 32-column block of the piece (block 128: the same byte four times)
    uint32_t ew;
    {
        const int8_t* pe = A.EX + (size_t)(lin0 + lane) * nbx + c0 / BLK;
        if (BLK == 128) ew = (uint32_t)(uint8_t)pe[0] * 0x01010101u;
        else if ((nbx & 3) == 0 && ((uintptr_t)A.EX & 3) == 0) ew = *reinterpret_cast<const uint32_t*>(pe);
        else {
            ew = 0;
#pragma unroll
            for (int b = 0; b < 4; b++) ew |= (uint32_t)(uint8_t)(c0 / 32 + b < nbx ? pe[b] : (int8_t)E_ZERO) << (8 * b);
        }
    }
    uint32_t w[32];                                                // sign bits flipped: byte b stands for b + 128
    {
        const int8_t* px = A.X + (size_t)lin0 * C + (dentro ? col0 : 0);
#pragma unroll
        for (int i = 0; i < 32; i++, px += C) w[i] = *reinterpret_cast<const uint32_t*>(px) ^ 0x80808080u;
    }
    uint32_t mx4;
    if (BLK == 128) mx4 = (uint32_t)(uint8_t)(int8_t)__reduce_max_sync(FULL, (int)(int8_t)ew) * 0x01010101u;
    else {
        mx4 = 0;
#pragma unroll
        for (int b = 0; b < 4; b++) mx4 |= (uint32_t)(uint8_t)(int8_t)__reduce_max_sync(FULL, (int)(int8_t)(ew >> (8 * b))) << (8 * b);
    }
    // how far below the largest exponent of its block this row's are (0..254); beyond 100, all-zero blocks (-127) apart, fp32 does not reach
    uint32_t d4 = __vsub4(mx4, ew);
    const uint32_t longe = __reduce_or_sync(FULL, __vcmpgtu4(d4, 0x64646464u) & ~__vcmpeq4(ew, 0x81818181u));
    const int bl = lane >> 3, eref = (int)(int8_t)(mx4 >> (8 * bl));
    const bool largo = (longe >> (8 * bl)) & 1;
    uint32_t emax4 = 0x80808080u;                                  // the new exponents of this lane's columns, -128 where it has none
    if constexpr (BLK == 32) {
        // In halves, two rows at a time: with exponents at most 24 apart (all-zero blocks apart) a mantissa times 2^(e - eref) is exact, the largest gives the
        // block's exponent, and one fused multiply-add against 1.5 * 2^10 rounds half to even.  Its factor is at most 2^15: a column whose largest element lies
        // further below the largest exponent of its 32-column block (2^30 at most) is multiplied by 2^15 first, which is exact, where a lane has one column.  (Left to
        // fp32, the whole warp, such columns cost 4 to 6 % more than without halves: 2048 x 512 with few small elements 3.44 us, 3.30 without halves, 3.17 so.
        // With four columns a lane, fp32: the second form of the output there costs every other input 1.5 %, 16384 x 4096 45.8 -> 46.7.)
        // An all-zero block's row may lie anywhere below; beyond 24 its factor is 0.  Should its mantissas not be cleared, that is what they come to where
        // the column's new exponent is -119 or more: at least eref - 15 >= -117 with one factor, eref - 30 >= -110 with two from eref = -80 on, and fp32 below that.
        __shared__ __align__(16) uint16_t esc_s[4][4][32];         // per warp and block: the rows' factors
        const bool perto = __reduce_or_sync(FULL, __vcmpgtu4(d4, 0x18181818u) & ~__vcmpeq4(ew, 0x81818181u)) == 0;
        if (perto) {
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int d = (d4 >> (8 * b)) & 0xff;
                esc_s[wid][b][lane] = d <= 14 ? (uint16_t)((15 - d) << 10) : d <= 24 ? (uint16_t)(1 << (24 - d)) : (uint16_t)0;      // 2^-d
            }
            __syncwarp();
            uint32_t he[16], t[CPT][16], mx[CPT];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint4 x = reinterpret_cast<const uint4*>(esc_s[wid][bl])[j];
                he[4 * j] = x.x; he[4 * j + 1] = x.y; he[4 * j + 2] = x.z; he[4 * j + 3] = x.w;
            }
#pragma unroll
            for (int c = 0; c < CPT; c++) mx[c] = 0;
            const uint32_t qual = CPT == 1 ? (uint32_t)(k0 | (k0 + 4) << 4) : 0x5140u;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                uint32_t hb, x[2];
                asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(hb) : "r"(he[j]), "r"(0xE480E480u));                  // -1152 of them
                x[0] = __byte_perm(w[2 * j], w[2 * j + 1], qual);
                if (CPT > 1) x[1] = __byte_perm(w[2 * j], w[2 * j + 1], 0x7362);
#pragma unroll
                for (int c = 0; c < CPT; c++) {
                    const uint32_t a = __byte_perm(x[c >> 1], 0x64646464u, c & 1 ? 0x4342 : 0x4140);       // 1152 + m
                    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(t[c][j]) : "r"(a), "r"(he[j]), "r"(hb));
                    asm("max.f16x2 %0, %0, %1;" : "+r"(mx[c]) : "r"(t[c][j] & 0x7FFF7FFFu));
                }
            }
            int Eo[CPT];
            bool serve = true;                                     // the factors of this lane's columns are 2^15 at most
#pragma unroll
            for (int c = 0; c < CPT; c++) {
                const uint32_t m = max(mx[c] & 0xFFFFu, mx[c] >> 16);                                       // (not negative: ordered like their bits)
                float f;
                asm("{\n .reg .b16 h;\n cvt.u16.u32 h, %1;\n cvt.f32.f16 %0, h;\n}" : "=f"(f) : "r"(m));
                Eo[c] = m == 0 ? SEM_TOPO : eref + (__float_as_int(f) >> 23) - 126 - 7;
                serve = serve && (m == 0 || eref - Eo[c] <= 15);
            }
            auto grava = [&](auto longe15) {                       // longe15: some factor is beyond 2^15
#pragma unroll
                for (int c = 0; c < CPT; c++) {
                    const int k = k0 + c;
                    const size_t col = (size_t)col0 + k;
                    const bool morto = Eo[c] < -126;
                    if (dentro && Eo[c] > 126) reporta(E_EXP, kid, (long long)col * R + lin0, Eo[c], eref);
                    int kB = eref - Eo[c];                                                                  // 2^kB
                    if constexpr (decltype(longe15)::v) {
                        const uint32_t A2 = kB > 15 ? 0x78007800u : 0x3C003C00u;                            // 2^15 (an empty column's zeros too) or 1
#pragma unroll
                        for (int j = 0; j < 16; j++) asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(t[c][j]) : "r"(A2));
                        if (kB > 15) kB -= 15;
                    }
                    const uint32_t B = morto ? 0u : (uint32_t)(15 + kB) << 10, B2 = B | B << 16;
                    if (morto) Eo[c] = E_ZERO;
                    if (dentro) {
                        uint32_t q[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(q[j]) : "r"(t[c][j]), "r"(B2), "r"(0x66006600u));
                        uint4* dst = reinterpret_cast<uint4*>(A.Y + col * R + lin0);
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            dst[h] = make_uint4(__byte_perm(q[8 * h], q[8 * h + 1], 0x6420), __byte_perm(q[8 * h + 2], q[8 * h + 3], 0x6420),
                                                __byte_perm(q[8 * h + 4], q[8 * h + 5], 0x6420), __byte_perm(q[8 * h + 6], q[8 * h + 7], 0x6420));
                        A.EY[col * nby + lin0 / BLK] = (int8_t)Eo[c];
                    }
                    emax4 = (emax4 & ~(0xffu << (8 * k))) | ((uint32_t)(uint8_t)(int8_t)Eo[c] << (8 * k));
                }
                if (A.RM != nullptr && dentro) max4_atomico(A.RM + col0, emax4);
            };
            if (__all_sync(FULL, serve)) {
                grava(SimNao<false>());
                return;
            }
            if (CPT == 1 && !__any_sync(FULL, !serve && eref < -80)) {
                grava(SimNao<true>());
                return;
            }
        }
    }
    d4 = __vminu4(d4, 0x7f7f7f7fu);
    float fa[32];                                                  // 2^(e - eref)
#pragma unroll
    for (int i = 0; i < 32; i++) fa[i] = __int_as_float(0x3f800000 - (int)((__shfl_sync(FULL, d4, i) >> (8 * bl)) & 0xff) * 0x800000);
    auto valor = [&](int i, int k) {                               // element (row i, column k) times 2^(e - eref), exact
        return (__uint_as_float(__byte_perm(w[i], 0x4B400000u, 0x7650 + k)) - 12583040.0f) * fa[i];
    };
    auto topo_de = [&](float mx) { return mx == 0.f ? SEM_TOPO : eref + (__float_as_int(mx) >> 23) - 126; };       // e + bitlen of the largest
    const int8_t *px0 = A.X + (size_t)lin0 * C + (dentro ? col0 : 0), *pe0 = A.EX + (size_t)lin0 * nbx + (dentro ? col0 : 0) / BLK;      // (cold path)
    if (BLK == 128) {
        float mx[CPT];
#pragma unroll
        for (int kk = 0; kk < CPT; kk++) mx[kk] = 0.f;
#pragma unroll
        for (int i = 0; i < 32; i++)
#pragma unroll
            for (int kk = 0; kk < CPT; kk++) mx[kk] = fmaxf(mx[kk], fabsf(valor(i, k0 + kk)));
#pragma unroll
        for (int kk = 0; kk < CPT; kk++) topos[rg][4 * lane + k0 + kk] = largo ? transpoe_topo_lento(px0 + k0 + kk, pe0, C, nbx) : topo_de(mx[kk]);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 32; i++) asm volatile("" : "+r"(w[i]));          // the values are computed again below rather than kept: 128 registers
    }
#pragma unroll
    for (int kk = 0; kk < CPT; kk++) {
        const int k = k0 + kk;
        float t[32];
        int topo;
        if (BLK == 128) {
            topo = max(max(topos[0][4 * lane + k], topos[1][4 * lane + k]), max(topos[2][4 * lane + k], topos[3][4 * lane + k]));
#pragma unroll
            for (int i = 0; i < 32; i++) t[i] = valor(i, k);
        } else {
            float mx = 0.f;
#pragma unroll
            for (int i = 0; i < 32; i++) { t[i] = valor(i, k); mx = fmaxf(mx, fabsf(t[i])); }
            topo = topo_de(mx);
            if (largo) topo = transpoe_topo_lento(px0 + k, pe0, C, nbx);
        }
        const size_t col = (size_t)col0 + k;
        int Eo = topo - 7;
        const bool morto = Eo < -126;
        if (dentro && Eo > 126) reporta(E_EXP, kid, (long long)col * R + lin0, Eo, eref);
        const float B = morto ? 0.f : __int_as_float((127 + max(min(eref - Eo, 127), -120)) << 23);
        if (morto) Eo = E_ZERO;
        if (dentro) {
            int8_t* dst = A.Y + col * R + lin0;
            if (largo) transpoe_grava_lento(px0 + k, pe0, C, nbx, Eo, dst);
            else {
                uint32_t a[16], b[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    a[i] = (uint32_t)__float_as_int(fmaf(t[i], B, 12582912.0f));
                    b[i] = (uint32_t)__float_as_int(fmaf(t[16 + i], B, 12582912.0f));
                }
                reinterpret_cast<uint4*>(dst)[0] = junta16(a);
                reinterpret_cast<uint4*>(dst)[1] = junta16(b);
            }
            if (BLK == 32 || rg == 0) A.EY[col * nby + lin0 / BLK] = (int8_t)Eo;
        }
        emax4 = (emax4 & ~(0xffu << (8 * k))) | ((uint32_t)(uint8_t)(int8_t)Eo << (8 * k));
    }
    // row maxima of the transposed tensor (what a GEMM aligns its rows to): the caller pre-set RM to -128
    if (A.RM != nullptr && dentro) max4_atomico(A.RM + col0, emax4);
}

// one or two matrices with the same number of rows (the operands of a weight-gradient GEMM) in one launch: CTAs 0 .. n0-1 take the first
template <int BLK, int CPT>
__global__ void __launch_bounds__(CPT == 1 && BLK == 128 ? 512 : 128, CPT == 1 && BLK == 128 ? 1 : 4) k_transpoe(const ArgsTransp a0, const ArgsTransp a1, int n0, int R, int kid) {
    constexpr int TR = CPT == 1 && BLK == 32 ? 32 : 128;           // rows of a CTA
    const bool segunda = (int)blockIdx.x >= n0;
    const ArgsTransp A = segunda ? a1 : a0;
    const int t = (int)blockIdx.x - (segunda ? n0 : 0), nx = (A.C + 127) / 128;
    transpoe_corpo<BLK, CPT>(A, t / nx * TR, t % nx * 128, R, kid);
}

// RMSNorm without gain, one warp per row, NP*512 >= D columns held in registers.  ops.py:153-165
//   ss = sum_b rnd(sq_b << G, 2 (emax - e_b));  r = isqrt(ss >> log2D);  k = bitlen(r) + 10;  inv = 2^k / r
//   y = quant(x * inv, e_b - k - emax + G/2);  cache = (r, emax)
template <int BLK, int NP>
__global__ void __launch_bounds__(256) k_rms(const int8_t* __restrict__ Xm, const int8_t* __restrict__ XE, int8_t* __restrict__ Ym,
                                             int8_t* __restrict__ YE, int* __restrict__ cr, int* __restrict__ cemax, int M, int D, int log2D, int G,
                                             int kid) {
    pdl_espera();
    pdl_solta();
    constexpr int GL = BLK / 16;
    const int lane = threadIdx.x & 31;
    const long long lin_ = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    const bool linha_ok = lin_ < M;
    const long long lin = linha_ok ? lin_ : 0;
    const int nb = D / BLK;
    int x[NP][16], eb[NP];
    bool tem[NP];
    int emax = -128;
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int c = (p * 32 + lane) * 16;
        tem[p] = c < D;
        if (tem[p]) {
            le16(Xm + lin * D + c, x[p]);
            eb[p] = XE[lin * nb + c / BLK];
            emax = max(emax, eb[p]);
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) x[p][i] = 0;
            eb[p] = E_ZERO;
        }
    }
    emax = warp_max(emax);
    int ss = 0;
#pragma unroll
    for (int p = 0; p < NP; p++) {
        int sq = 0;
#pragma unroll
        for (int i = 0; i < 16; i++) sq += x[p][i] * x[p][i];
#pragma unroll
        for (int o = GL / 2; o; o >>= 1) sq += __shfl_xor_sync(FULL, sq, o);      // whole block on every lane of the group
        if ((lane % GL) == 0 && tem[p]) ss += rnd_d(sq << G, 2 * (emax - eb[p]));
    }
    ss = warp_sum(ss);
    const int r = isqrt_i(ss >> log2D);
    const int k = bitlen(r) + 10;
    const int inv = (1 << k) / r;
    const float invf = (float)inv;                   // inv <= 2^11 and |x| <= 127: x * inv < 2^18 is exact in fp32
#pragma unroll
    for (int p = 0; p < NP; p++) {
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; i++) f[i] = (float)x[p][i] * invf;
        const int c = (p * 32 + lane) * 16;
        uint4 pac;
        const int Eo = quant_f32<GL>(f, eb[p] - k - emax + G / 2, pac, kid, lin * D + c);
        if (tem[p] && linha_ok) {
            *reinterpret_cast<uint4*>(Ym + lin * D + c) = pac;
            if ((lane % GL) == 0) YE[lin * nb + c / BLK] = (int8_t)Eo;
        }
    }
    if (lane == 0 && linha_ok) { cr[lin] = r; cemax[lin] = emax; }
}

// RMSNorm backward: dx = (g - y * mean(g y)) / rms with two shrink steps (15 and 18 bits).  ops.py:167-184
// SOMA: the result is added to the block tensor x (the residual gradient) before it is stored: soma(x, rms_back(...)).
//
// In floating point, exactly.  The terms of the mean are products below 2^14 with one shift per block: a product and a fused multiply-add
// against 1.5 * 2^23 each, whose bit patterns are added.  The bracket is done in double precision: its two terms are rounded by fused
// multiply-adds against 1.5 * 2^52 (their difference is the integer), adding 1.5 * 2^(35 + exponent) and taking it off again rounds that to
// 18 significant bits, half to even, and what is left - the scale stays in the number, so all elements of a block share one
// exponent, and 18 bits fit the high word alone - is multiplied by 2^k / rms and rounded to the mantissa by one more.
// (Integer shifts and the general quantiser before: 113 instructions per element, 98 us at 16384 x 1024, now 25.)
template <int BLK, int NP, bool SOMA>
__device__ __forceinline__ void rms_back_corpo(const int8_t* __restrict__ gm, const int8_t* __restrict__ gE, const int8_t* __restrict__ ym,
                                               const int8_t* __restrict__ yE, const int* __restrict__ cr, const int* __restrict__ cemax,
                                               const int8_t* __restrict__ xm, const int8_t* __restrict__ xE, int8_t* __restrict__ om,
                                               int8_t* __restrict__ oE, int M, int D, int log2D, int G, int GB, int kid) {
    pdl_espera();
    pdl_solta();
    constexpr int GL = BLK / 16;
    const int lane = threadIdx.x & 31;
    const long long lin_ = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    const bool linha_ok = lin_ < M;
    const long long lin = linha_ok ? lin_ : 0;
    const int nb = D / BLK;
    uint4 g4[NP], y4[NP], x4[NP];
    int eg[NP], ey[NP], ex[NP];
    bool tem[NP];
    int smax = -100000;
    const int r = cr[lin], emax = cemax[lin];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int c = (p * 32 + lane) * 16;
        tem[p] = c < D;
        g4[p] = y4[p] = x4[p] = make_uint4(0, 0, 0, 0);
        eg[p] = ey[p] = ex[p] = E_ZERO;
        if (tem[p]) {
            g4[p] = *reinterpret_cast<const uint4*>(gm + lin * D + c);
            y4[p] = *reinterpret_cast<const uint4*>(ym + lin * D + c);
            eg[p] = gE[lin * nb + c / BLK];
            ey[p] = yE[lin * nb + c / BLK];
            if (SOMA) {
                x4[p] = *reinterpret_cast<const uint4*>(xm + lin * D + c);
                ex[p] = xE[lin * nb + c / BLK];
            }
            smax = max(smax, eg[p] + ey[p]);
        }
    }
    smax = warp_max(smax);
    int S = 0;
    if (GB <= 8) {
#pragma unroll
        for (int p = 0; p < NP; p++) {
            const float esc = __int_as_float((127 + GB - min(smax - (eg[p] + ey[p]), 60)) << 23);      // |g y 2^GB| <= 127^2 * 2^8 < 2^22
            float gf[16], yf[16];
            bytes_para_float(g4[p], gf);
            bytes_para_float(y4[p], yf);
#pragma unroll
            for (int i = 0; i < 16; i++) S += __float_as_int(fmaf(gf[i] * yf[i], esc, 12582912.0f)) - 0x4B400000;
        }
    } else {
#pragma unroll
        for (int p = 0; p < NP; p++) {
            int gi[16], yi[16];
            desempacota16(g4[p], gi);
            desempacota16(y4[p], yi);
#pragma unroll
            for (int i = 0; i < 16; i++) S += rnd_d((gi[i] * yi[i]) << GB, smax - (eg[p] + ey[p]));
        }
    }
    S = warp_sum(S);
    int eS = smax - GB - log2D;
    const int sh = max(bitlen(S) - 15, 0);
    S = rnd_d(S, sh);
    eS += sh;
    const int k = bitlen(r) + 10;
    const double inv = (double)((1 << k) / max(r, 1)), Sd = (double)S;
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int c = (p * 32 + lane) * 16;
        const long long o = lin * D + c;
        // ec >= eg + 7 - 28 and ec >= ey + eS + 22 - 28: the 7-bit g moves up by at most 21, the 22-bit y S by at most 6
        const int ec = max(eg[p] + 7, ey[p] + eS + 22) - 28;
        const double eg_d = pot2_d(eg[p] - ec), ey_d = Sd * pot2_d(ey[p] + eS - ec);
        const uint32_t gw[4] = {g4[p].x, g4[p].y, g4[p].z, g4[p].w}, yw[4] = {y4[p].x, y4[p].y, y4[p].z, y4[p].w};
        int d[16], dmax = 0;                                       // high words of the bracket's 18-bit values; their low words are 0
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const double dentro = fma(int_para_d(byte_s(gw[i >> 2], i & 3)), eg_d, MAGIA_D) - fma(int_para_d(byte_s(yw[i >> 2], i & 3)), ey_d, MAGIA_D);
            const double m18 = __hiloint2double((__double2hiint(dentro) & 0x7ff00000) + (35 << 20) + 0x80000, 0);
            d[i] = __double2hiint((dentro + m18) - m18);
            dmax = max(dmax, d[i] & 0x7fffffff);
        }
        dmax = grupo_max<GL>(dmax);
        const int e0 = ec - k - (emax - G / 2);
        const double vmax = __hiloint2double(dmax, 0) * inv;
        int E = bitlen_d(vmax) + e0 - 7, Eo = E_ZERO;
        double esc = inv * pot2_d(e0 - E);
        if ((int)(uint32_t)__double2loint(fma(__hiloint2double(dmax, 0), esc, MAGIA_D)) > 127) { E += 1; esc *= 0.5; }
        uint4 pac = make_uint4(0, 0, 0, 0);
        if (dmax != 0 && E >= -126) {
            if (E > 126) reporta(E_EXP, kid, o, E, e0);
            Eo = E;
            uint32_t q[16];
#pragma unroll
            for (int i = 0; i < 16; i++) q[i] = (uint32_t)__double2loint(fma(__hiloint2double(d[i], 0), esc, MAGIA_D));
            pac = junta16(q);
        }
        if (SOMA) Eo = soma16_misto<GL>(x4[p], ex[p], pac, (int)(int8_t)Eo, pac, kid, o);
        if (tem[p] && linha_ok) {
            *reinterpret_cast<uint4*>(om + o) = pac;
            if ((lane % GL) == 0) oE[lin * nb + c / BLK] = (int8_t)Eo;
        }
    }
}
template <int BLK, int NP>
__global__ void __launch_bounds__(256) k_rms_back(const int8_t* __restrict__ gm, const int8_t* __restrict__ gE, const int8_t* __restrict__ ym,
                                                  const int8_t* __restrict__ yE, const int* __restrict__ cr, const int* __restrict__ cemax,
                                                  int8_t* __restrict__ om, int8_t* __restrict__ oE, int M, int D, int log2D, int G, int GB, int kid) {
    rms_back_corpo<BLK, NP, false>(gm, gE, ym, yE, cr, cemax, nullptr, nullptr, om, oE, M, D, log2D, G, GB, kid);
}
template <int BLK, int NP>
__global__ void __launch_bounds__(256) k_rms_back_soma(const int8_t* __restrict__ gm, const int8_t* __restrict__ gE, const int8_t* __restrict__ ym,
                                                       const int8_t* __restrict__ yE, const int* __restrict__ cr, const int* __restrict__ cemax,
                                                       const int8_t* __restrict__ xm, const int8_t* __restrict__ xE, int8_t* __restrict__ om,
                                                       int8_t* __restrict__ oE, int M, int D, int log2D, int G, int GB, int kid) {
    rms_back_corpo<BLK, NP, true>(gm, gE, ym, yE, cr, cemax, xm, xE, om, oE, M, D, log2D, G, GB, kid);
}

// integer softmax + cross-entropy gradient, LL lanes (a warp; half a warp for V <= 256: 16384 x 256 21.4 -> 12.7 us) per row of raw logits.
// ops.py:260-271
//   u = rnd(acc, -(e + 8)); ex = exp(-(umax - u)/256) >> 3; s = sum ex; v = (ex * (2^28 / s) + 2^15) >> 16;
//   v[target] -= 4096; g = quant(v, -12 - log2M); also d_alvo = umax - u[target] and s for the loss report.
template <int BLK, int NP, int LL = 32>
__global__ void __launch_bounds__(256) k_softmax_ce(const int* __restrict__ acc, const int16_t* __restrict__ e, const int* __restrict__ alvo,
                                                    int8_t* __restrict__ gm, int8_t* __restrict__ gE, int* __restrict__ d_alvo, int* __restrict__ soma,
                                                    int M, int V, int log2M, int kid) {
    pdl_espera();
    pdl_solta();
    constexpr int GL = BLK / 16;
    const int lane = threadIdx.x & 31;
    const int ll = lane & (LL - 1);                                 // lane within the row
    const long long lin_ = (long long)blockIdx.x * (256 / LL) + threadIdx.x / LL;
    const bool linha_ok = lin_ < M;
    const long long lin = linha_ok ? lin_ : 0;
    int u[NP][16];
    bool tem[NP];
    int umax = U_MIN;
    const int tk = alvo[lin];
    if (ll == 0 && linha_ok && (tk < 0 || tk >= V)) reporta(E_ARG, kid, lin * V, tk, V);
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int c = (p * 32 + ll) * 16;
        tem[p] = c < V;
        int a[16], ee[16], emx = -100000;
        if (tem[p]) {
            le16_i32(acc + lin * V + c, a);
            le16_i16(e + lin * V + c, ee);
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) { a[i] = 0; ee[i] = -100; }
        }
#pragma unroll
        for (int i = 0; i < 16; i++) emx = max(emx, ee[i]);
        if (__all_sync(FULL, emx <= -8)) {                          // right shifts only, the usual case: one fused multiply-add in double precision rounds
#pragma unroll
            for (int i = 0; i < 16; i++) u[p][i] = __double2loint(fma(int_para_d(a[i]), pot2_d(ee[i] + 8), MAGIA_D));
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) u[p][i] = rnd(a[i], -(ee[i] + 8), kid, lin * V + c + i);
        }
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if (!tem[p]) u[p][i] = U_MIN;
            umax = max(umax, u[p][i]);
        }
    }
    umax = grupo_max<LL>(umax);
    int s = 0, ut = U_MIN;
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int c = (p * 32 + ll) * 16;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if (c + i == tk) ut = u[p][i];
            u[p][i] = tem[p] ? exp3_dif(umax, u[p][i]) : 0;              // u now holds ex
            s += u[p][i];
        }
    }
#pragma unroll
    for (int d = LL / 2; d; d >>= 1) s += __shfl_xor_sync(FULL, s, d);
    ut = grupo_max<LL>(ut);
    if (s <= 0) { if (ll == 0 && linha_ok) reporta(E_DIV, kid, lin * V, s, 0); s = 1; }
    const int inv = (1 << 28) / s;
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int c = (p * 32 + ll) * 16;
        float f[16];                                                       // |v| <= 2^12 + 2^15: exact in fp32
#pragma unroll
        for (int i = 0; i < 16; i++) f[i] = (float)(((u[p][i] * inv + (1 << 15)) >> 16) - (c + i == tk ? 4096 : 0));
        uint4 pac;
        const int Eo = quant_f32<GL>(f, -12 - log2M, pac, kid, lin * V + c);
        if (tem[p] && linha_ok) {
            *reinterpret_cast<uint4*>(gm + lin * V + c) = pac;
            if ((lane % GL) == 0) gE[lin * (V / BLK) + c / BLK] = (int8_t)Eo;
        }
    }
    if (ll == 0 && linha_ok) { d_alvo[lin] = umax - ut; soma[lin] = s; }
}

// loss of every row of softmax_ce's outputs, d / 256 + log(s / 4096) in double precision (report only)
__global__ void __launch_bounds__(256) k_perda(const int* __restrict__ d, const int* __restrict__ s, double* __restrict__ saida, int M) {
    pdl_espera();
    pdl_solta();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < M) saida[i] = (double)d[i] / 256 + log((double)s[i] / 4096);
}

}  // namespace jt
