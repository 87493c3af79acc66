// C ABI of the B200 library: the jt_* entry points the reference's ctypes launcher binds
// (jatai_cuda/jatai_cuda.cu:1061-1201; jatai_cuda/ops.py:299-324), plus jt_blk / jt_gemm_via / jt_gemm_ext.
// Declarations with the per-function reference citations: include/jatai_b200.h.
//
// Conventions (as in the reference): raw device pointers, C ints, the last argument of every operation is
// the launch id `kid`; the return value is the cudaError_t of the launch (0 = ok, invalid arguments give
// cudaErrorInvalidValue without launching); nothing here synchronises except jt_erro_le / jt_sincroniza;
// every launch goes to the stream set with jt_stream (NULL = legacy default stream).
//
// Build: nvcc -O3 -gencode arch=compute_100a,code=sm_100a -lineinfo -shared -Xcompiler -fPIC jatai_b200.cu -o libjatai_b200.so
#include <cstdio>
#include <cstring>
#include <cuda.h>
#include <cuda_runtime.h>

#include "comum.cuh"
#include "blocos.cuh"
#include "gemm_comum.cuh"
#include "gemm_simt.cuh"
#include "gemm_tc.cuh"
#include "gemm_h.cuh"
#include "atencao.cuh"
#include "atencao_tc.cuh"
#include "atencao_peq.cuh"

using namespace jt;

// ---------------------------------------------------------------------------------------------- host state
static cudaStream_t g_stream = 0;
static bool g_ao_lado = false;       // the launches to come run beside another chain of launches (jt_stream_ao_lado)
static int g_blk = 32;               // exponent block length: 32 (native) or 128 (the reference's format)
static int g_via = 0;                // GEMM path: 0 automatic | 1 tensor core (forced) | 2 CUDA cores | 3 tensor core, rounding by conversion | 4 half-precision tensor pipe (forced)
static int g_alvo_ctas = 148;        // split-K of raw GEMMs aims at this many CTAs
static int g_at_via = 0;             // attention path: 0 automatic (tensor cores; one CTA per head for short sequences of heads of 4) | 1 the tiled CUDA-core kernels
static int g_tn = 0;                 // tile width of the tensor-core GEMM: 0 automatic | 64 | 128
static int g_somas = 0;              // products whose blocks look for tiles that add up in tensor memory: 0 automatic | 1 none | 2 every one that can

static int fim() { return (int)cudaGetLastError(); }
static unsigned nblocos16(long long n16) { return (unsigned)((n16 + 255) / 256); }
static unsigned nblocos_128(long long n16) { return (unsigned)((n16 + 127) / 128); }
static unsigned nblocos16u(long long n16, int U) { return (unsigned)((n16 + 256LL * U - 1) / (256LL * U)); }      // U chunks per thread

template <int BLK, int MODO, int VIA, int TNv, bool SO = false>
static int lanca_tc(const CUtensorMap& mA, const CUtensorMap& mB, const int8_t* EA, const int8_t* EB, const int8_t* RA, const int8_t* RB,
                    const SaidaGemm& S, int M, int N, int K, int partes, int kid) {
    static bool feito[64];                 // kernel attributes are per device
    using C_ = tc::Cfg<TNv, VIA, SO>;
    auto k = tc::k_gemm_tc<BLK, MODO, VIA, TNv, SO>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    bool& pronto = feito[dev];
    if (!pronto) {
        cudaError_t c = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C_::SMEM_BYTES);
        if (c != cudaSuccess) return (int)c;
        // shared memory for the resident CTAs and no more: what is left of the 256 KB serves the L1 (register spills)
        c = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)((C_::SMEM_BYTES + 1024) * C_::CTAS_SM * 100 / (228 * 1024)) + 1);
        if (c != cudaSuccess) return (int)c;
        pronto = true;
    }
    const dim3 grade(N / TNv, M / tc::TM, partes);
    lanca_pdl(k, grade, dim3(C_::N_THR), C_::SMEM_BYTES, g_stream, mA, mB, EA, EB, RA, RB, S, M, N, K, (K / tc::KC) / partes, kid);
    return fim();
}

template <int BLK, int MODO>
static int lanca_simt(const int8_t* A, const int8_t* EA, const int8_t* B, const int8_t* EB, const int8_t* RA, const int8_t* RB,
                      const SaidaGemm& S, int M, int N, int K, int partes, int kid) {
    const dim3 grade(N / TN, M / 64, partes);
    k_gemm_simt<BLK, MODO><<<grade, 256, SIMT_SMEM, g_stream>>>(A, EA, B, EB, RA, RB, S, M, N, K, (K / 32) / partes, kid);
    return fim();
}

// Beside another chain (jt_stream_ao_lado): most blocks of a product that has more of them than 128 x 128 tiles (64-column tiles, K ranges).
constexpr int N_LADO = 48;
// Whether the 8-bit kernel takes 64-column tiles (block 32 only) for a product of t 128 x 128 ones.  Up to 148 of them have an SM each and 16 drain warps: a tile takes
// 0.6 to 0.8 of a 128-column one (2048 x 512 x 512 7.9 us against 10.8, K = 2048 20.6 against 29.8).  From 75 to 148 128-column tiles these have an SM
// each, where two 64-column ones on an SM take longer (2048 x 768 x 512 12.0 us against 10.9, K = 2048 35.1 against 29.8).  Beyond, the pairs run without
// wave boundaries (about 1.03 t/148 + 0.3 rounds of a 128-column tile) against ceil(t/148) whole rounds: 160 tiles, K = 512 17.9 us against 20.0,
// 256 tiles 22.3 against 20.5.
static bool estreito_i8(long long t) {
    if (g_ao_lado && 2 * t > N_LADO) return false;
    return 2 * t <= N_SM || (t > N_SM && 1.03 * (double)t / N_SM + 0.3 < (double)((t + N_SM - 1) / N_SM));
}
// K ranges of a raw product of block 128, estimated in microseconds: a 64-element chunk of one wave of tiles takes the 8-bit kernel 0.345 and the half-precision one 0.20,
// clearing the output and adding the ranges atomically 10 and 0.6 for every MB that is added.  8-bit kernel: 256 x 256 x 2048 17.2 in one range, 22.7 in two,
// K = 4096 28.1 in one, 19.0 in sixteen; half precision: 1024 x 512 x 4096 25.6 in one, 34.4 in two, 512 x 512 x 16384 70 in one, 40 in eight.
constexpr double I8_B128 = 0.345, H_B128 = 0.20;
static double soma_partes(int M, int N, int partes) { return partes > 1 ? 10.0 + (double)M * N * partes / 4.2e5 : 0.0; }
static int partes_b128(int M, int N, int K, double pedaco, bool iguais) {
    const long long t = (long long)(N / 128) * ((M + 127) / 128);
    const double n = (K + 63) / 64;
    int melhor = 1;
    // Beside another chain none: a step of 6 layers with 4096 tokens x 256 columns took 1368 us with up to 48 blocks of them, 1342 without.
    if (g_ao_lado) return 1;
    for (int p = 2; t * p <= g_alvo_ctas && K / 128 >= 2 * p && (!iguais || K / 128 % p == 0); p *= 2)      // (two blocks at least; of equal length for the 8-bit kernel)
        if (n / p * pedaco + soma_partes(M, N, p) < n / melhor * pedaco + soma_partes(M, N, melhor)) melhor = p;
    return melhor;
}
template <int BLK>
static int gemm_blk(const int8_t* A, const int8_t* EA, const int8_t* B, const int8_t* EB, const int8_t* RA, const int8_t* RB,
                    const SaidaGemm& S, int M, int N, int K, int modo, int kid) {
    if (M <= 0 || N <= 0 || K <= 0 || M % 64 || N % TN || K % BLK || K % 32 || modo < 0 || modo > 4) return (int)cudaErrorInvalidValue;
    const bool alinhado = (((uintptr_t)A | (uintptr_t)B) & 15) == 0 && (((uintptr_t)EA | (uintptr_t)EB) & 3) == 0;
    bool usa_tc = g_via != 2 && M % tc::TM == 0 && K % tc::KC == 0 && alinhado;
    const bool estreito = BLK == 32 && usa_tc && g_tn != 128 && (g_tn == 64 || estreito_i8((long long)(N / TN) * (M / tc::TM)));
    const int tn = estreito ? 64 : TN;
    CUtensorMap mA, mB;
    // a shape the tensor-core kernel takes never falls back silently: a tensor map that can not be encoded is an error
    if (usa_tc && !(faz_mapa(&mA, A, M, K) && faz_mapa(&mB, B, N, K, tn))) return (int)cudaErrorInvalidValue;
    if (!usa_tc && g_via != 0 && g_via != 2) return (int)cudaErrorInvalidValue;     // nor does a forced tensor-core path on a shape it can not take
    // split-K (raw output only): powers of two while the grid stays below the target and the K range divides evenly.  Clearing the output and
    // adding atomically cost 6 to 9 us, a unit of the tensor-core kernel takes 1.2: a part keeps at least 8 (512 x 256 x 256: 13.8 us in
    // two parts, 6.8 in one).
    // Block 128 takes what partes_b128 finds best.
    const int unidades = usa_tc ? K / tc::KC : K / BLK;            // indivisible K units of the chosen kernel
    const long long tiles = usa_tc ? (long long)(N / tn) * (M / tc::TM) : (long long)(N / TN) * (M / 64);
    int partes = 1;
    const int alvo = g_ao_lado && g_alvo_ctas > N_LADO ? N_LADO : g_alvo_ctas;
    if (modo == 1 && BLK == 128 && usa_tc) partes = partes_b128(M, N, K, I8_B128, true);
    else if (modo == 1)
        while (partes * (usa_tc ? 16 : 2) <= unidades && tiles * partes * 2 <= alvo && unidades % (partes * 2) == 0) partes *= 2;
    const bool so = estreito && tiles * partes <= N_SM;
    if (partes > 1) {
        cudaError_t c = cudaMemsetAsync(S.C32, 0, (size_t)M * N * sizeof(int), g_stream);
        if (c != cudaSuccess) return (int)c;
    }
    if (usa_tc) {
        // block 32: FMA rounding with its range check (exact), or the conversion when asked for (jt_gemm_via(3)); block 128: conversion
#define JT_TC(MD)                                                                                                    \
    case MD:                                                                                                         \
        if constexpr (BLK == 32) {                                                                                   \
            if (estreito) {                                                                                          \
                if (g_via == 3) return lanca_tc<32, MD, 2, 64>(mA, mB, EA, EB, RA, RB, S, M, N, K, partes, kid);     \
                if (so) return lanca_tc<32, MD, 1, 64, true>(mA, mB, EA, EB, RA, RB, S, M, N, K, partes, kid);       \
                return lanca_tc<32, MD, 1, 64>(mA, mB, EA, EB, RA, RB, S, M, N, K, partes, kid);                     \
            }                                                                                                        \
            if (g_via == 3) return lanca_tc<32, MD, 2, 128>(mA, mB, EA, EB, RA, RB, S, M, N, K, partes, kid);        \
            return lanca_tc<32, MD, 1, 128>(mA, mB, EA, EB, RA, RB, S, M, N, K, partes, kid);                        \
        }                                                                                                            \
        return lanca_tc<BLK, MD, 2, 128>(mA, mB, EA, EB, RA, RB, S, M, N, K, partes, kid);
        switch (modo) { JT_TC(0) JT_TC(1) JT_TC(2) JT_TC(3) JT_TC(4) }
#undef JT_TC
    }
#define JT_SI(MD) case MD: return lanca_simt<BLK, MD>(A, EA, B, EB, RA, RB, S, M, N, K, partes, kid);
    switch (modo) { JT_SI(0) JT_SI(1) JT_SI(2) JT_SI(3) JT_SI(4) }
#undef JT_SI
    return (int)cudaErrorInvalidValue;
}

// ---- the half-precision path (gemm_h.cuh): operands prepared in a workspace of the caller
struct EspacoH { size_t A, B, RA, RB, nA, nB, total; };
static EspacoH espaco_h(int M, int N, int K) {
    auto ar = [](size_t x) { return (x + 1023) & ~(size_t)1023; };
    EspacoH e;
    e.A = 0;
    e.B = e.A + ar((size_t)M * K * 2);
    e.RA = e.B + ar((size_t)N * K * 2);
    e.RB = e.RA + ar(M);
    e.nA = e.RB + ar(N);
    e.nB = e.nA + ar((size_t)((M + 31) / 32) * (K / 32) * 4);
    e.total = e.nB + ar((size_t)(N / 32) * (K / 32) * 4);
    return e;
}
static bool forma_gemm(int blk, int M, int N, int K, int modo) {
    return M > 0 && N > 0 && K > 0 && M % 64 == 0 && N % TN == 0 && K % blk == 0 && K % 32 == 0 && modo >= 0 && modo <= 4;
}
// Estimated times of the GEMM kernels in microseconds (measured at 64..16384 rows, 128..4096 columns, K = 64..16384): waves of tiles
// times (64-element chunks of K x time per chunk + the start and end of a tile).  They place the lines between the kernels: against the
// kernels forced one by one at 70 sizes the choice loses more than 3 % (3.1 to 5) at ten where every tile rounds, because it looks for sums (2048 x 1536 x 512
// 16.6 us against 16.0, 16384 x 4096 x 1024 with ReLU^2 258 against 250; where none rounds they are worth 16.4 -> 13.8 and 257 -> 169), and at 2048 x 1024 x 1024
// where none rounds, since 128 tiles do not look (15.2 against 14.1).  Outside of these sizes: K = 256 with 160 to 192 tiles that round (13.2 against 12.7 with the
// 8-bit kernel), 256 tiles of K = 128 (11.9 and 11.4), and, block 128, 2048 x 1024 x 16384 raw (109 and 103).
struct Custos { double i8, h64, h128; int grupo; };                  // grupo: blocks of a cluster per 64-wide tile
static Custos custos_gemm(int blk, int M, int N, int K, int modo) {
    const bool cru = modo == 1;
    const double n = (K + 63) / 64;
    const long long t128 = (long long)(N / 128) * ((M + 127) / 128), t64 = 2 * t128;
    auto ondas = [](long long t, int vagas) { return (double)((t + vagas - 1) / vagas); };
    const double prep = 4.0 + (double)(M + N) * K * 3 / (blk == 32 ? 4.8e6 : 5.3e6);    // k_prep_h: a launch, and 3 bytes per element at 4.8 TB/s (block 128: 5.3)
    // What a raw output, or the backward of ReLU^2, costs a wave of tiles more than a block output does.  With it, short K is where the lines lie for products of more tiles than
    // 64-wide ones have SMs: 2048 x 1536 x 128 9.8 us with the 8-bit kernel and 11.5 with the half-precision one, raw 13.0 and 16.5, 2048 x 640 x 256
    // 7.8 and 8.7; 2048 x 1536 x 256 12.8 and 13.1, or 11.5 with exponents that round nothing.
    auto saida = [&](double crua, double relu2_back) { return cru ? crua : modo == 4 ? relu2_back : 0.0; };
    Custos c;
    c.grupo = 1;
    // 64-wide tiles read 1.5 times as much for an output element.  With all SMs at it, or operands beyond 48 MB, they wait for the cache
    // (0.26 to 0.30 us a chunk): 4096 x 4096 x 4096 263 us, 183 with 128-wide ones.  So they have one wave or none.
    // Beside another chain (jt_stream_ao_lado) it is the SMs' time that counts: as many 64-wide tiles as fill the chip, and K ranges over clusters, are
    // done sooner but hold more SMs (2048 x 512 x 2048 raw 17.3 us on 128 SMs or 22.8 on 64).  A third of the chip is free for them (a short step's
    // chains are long ones), in the half-precision kernel and in the 8-bit one: N_LADO blocks.  Steps with 24, 36 or 48: 6 layers of
    // 512 columns 1184, 1194, 1193 us with 1024 tokens (1259 before the 8-bit kernel kept to it), 1027, 1016, 1017 with 512; 6 layers of 4096 tokens x 256
    // columns 1388, 1410, 1416; 12 layers of 2048 x 512 3120 each.
    const int vagas = g_ao_lado ? N_LADO : N_SM;
    const double p64 = (double)(M + N) * K * 2 > 48e6 ? 0.28 : 0.18;
    c.h64 = blk == 32 && t64 <= vagas ? prep + n * p64 + 2.9 : 1e9;
    if (blk == 32) {
        int partes = 1;                                                                 // (gemm_h: raw outputs of few 128-wide tiles, clearing and atomic additions 15 us)
        while (cru && !g_ao_lado && t128 * partes * 2 <= N_SM && n >= partes * 64) partes *= 2;
        c.h128 = prep + 1.0 + ondas(t128 * partes, N_SM) * (n / partes * 0.31 + 2.4 + saida(2.6, 1.5)) + (partes > 1 ? 15.0 : 0.0);
    } else {
        // (several waves of tiles wait for the cache: 0.25 a chunk.  12288 x 640 x 11136 raw 295 us, 275 with the 8-bit kernel; 8192 x 2048 x 2048 99.5 and 121.5)
        const int partes = cru ? partes_b128(M, N, K, H_B128, false) : 1;
        c.h128 = prep + (t128 <= N_SM ? 3.4 + n / partes * H_B128 + soma_partes(M, N, partes) + (cru ? 1.9 : 0.0) : 1.7 + ondas(t128, N_SM) * (n * 0.25 + (cru ? 4.2 : 1.7)));
    }
    // K ranges over a cluster while every block has an SM for itself (132 blocks in clusters of 4, 120 in clusters of 8 are at work at once) and keeps 4 chunks
    for (int g = 2; blk == 32 && g <= 8 && t64 * g <= vagas && t64 * g <= (g == 8 ? 120 : g == 4 ? 132 : N_SM) && n >= 4 * g; g *= 2) {
        const double x = prep + n / g * p64 + 3.9;
        if (x < c.h64) { c.h64 = x; c.grupo = g; }
    }
    if (M % tc::TM || K % tc::KC) c.i8 = 1e9;                                           // whole tiles only
    else if (blk == 32 && estreito_i8(t128)) c.i8 = t64 <= N_SM ? n * 0.55 + 3.4 : ondas(t64, 2 * N_SM) * (n * 0.76 + 3.4 + saida(1.75, 0.9));
    else if (blk == 32) c.i8 = 0.5 + ondas(t128, N_SM) * (n * 0.79 + 4.0 + saida(2.2, 1.25));
    else {
        const int partes = cru ? partes_b128(M, N, K, I8_B128, true) : 1;
        c.i8 = t128 > N_SM ? 2.5 + ondas(t128, N_SM) * (cru ? n * 0.365 + 5.0 : n * 0.41 + 3.0) : cru ? 6.3 + n / partes * I8_B128 + soma_partes(M, N, partes) : 4.6 + n * 0.375;
    }
    return c;
}
// whether a caller with a workspace takes the half-precision path
static bool usa_h(int M, int N, int K, int modo) {
    if (g_via != 0) return g_via == 4;
    const Custos c = custos_gemm(g_blk, M, N, K, modo);
    return (c.h64 < c.h128 ? c.h64 : c.h128) < c.i8;
}
template <int BLK, int MODO, int TNv, bool GRUPO, bool SOMA = false>
static int lanca_h(const CUtensorMap& mA, const CUtensorMap& mB, const int8_t* RA, const int8_t* RB, const uint32_t* nA, const uint32_t* nB, const SaidaGemm& S,
                   int M, int N, int K, const th::Grade& G, int kid) {
    using C_ = th::CfgH<TNv, BLK>;
    auto k = th::k_gemm_h<BLK, MODO, TNv, GRUPO, SOMA>;
    cudaError_t c = at_smem(k, C_::SMEM_BYTES);
    if (c != cudaSuccess) return (int)c;
    const int tiles = G.nx * G.ny * G.partes;
    if (GRUPO) lanca_cluster(k, dim3(tiles), dim3(C_::N_THR), C_::SMEM_BYTES, g_stream, G.partes, mA, mB, RA, RB, nA, nB, S, M, N, K, G, kid);
    else lanca_pdl(k, dim3(tiles > N_SM ? N_SM : tiles), dim3(C_::N_THR), C_::SMEM_BYTES, g_stream, mA, mB, RA, RB, nA, nB, S, M, N, K, G, kid);
    return fim();
}
template <int BLK>
static int gemm_h(const int8_t* A, const int8_t* EA, const int8_t* B, const int8_t* EB, const int8_t* RA, const int8_t* RB, const SaidaGemm& S, int M, int N,
                  int K, int modo, unsigned char* ws, int kid) {
    const EspacoH e = espaco_h(M, N, K);
    uint16_t *Ah = (uint16_t*)(ws + e.A), *Bh = (uint16_t*)(ws + e.B);
    int8_t *RAw = (int8_t*)(ws + e.RA), *RBw = (int8_t*)(ws + e.RB);
    uint32_t *nA = (uint32_t*)(ws + e.nA), *nB = (uint32_t*)(ws + e.nB);
    const int nfx = (K + 511) / 512, ctasA = (M + 31) / 32 * nfx, ctasB = N / 32 * nfx;
    th::ArgsPrepH P = {{A, B}, {EA, EB}, {RA, RB}, {Ah, Bh}, {RAw, RBw}, {nA, nB}, {M, N}, ctasA, K};
    const Custos c = custos_gemm(BLK, M, N, K, modo);
    const bool estreito = BLK == 32 && g_tn != 128 && (g_tn == 64 || c.h64 < c.h128);
    const int tn = estreito ? 64 : TN;
    CUtensorMap mA, mB;
    if (!(faz_mapa_h(&mA, Ah, M, K, tc::TM) && faz_mapa_h(&mB, Bh, N, K, tn))) return (int)cudaErrorInvalidValue;
    const int nped = (K + th::KH - 1) / th::KH, uni = BLK / 64 > 1 ? BLK / 64 : 1;
    const long long tiles = (long long)(N / tn) * ((M + 127) / 128);
    const bool grupo = estreito && c.grupo > 1;
    int partes = grupo ? c.grupo : 1;
    if (modo == 1 && BLK == 128) partes = partes_b128(M, N, K, H_B128, false);
    else if (modo == 1 && !grupo && !g_ao_lado)
        while (tiles * partes * 2 <= g_alvo_ctas && nped >= partes * 2 * 32) partes *= 2;
    const int ppp = ((nped + partes - 1) / partes + uni - 1) / uni * uni;
    if (!grupo) partes = (nped + ppp - 1) / ppp;                   // (in a cluster a block without chunks adds zeros)
    const th::Grade G = {N / tn, (M + 127) / 128, partes, ppp};
    // Whether tiles may add up in tensor memory where nothing is rounded.  It depends on the data, which the host does not see: each block looks at its
    // tiles (k_gemm_h).  K <= 1024: the bounds of a tile are one word per lane.  With more than one tile per SM the gain where tiles qualify is 15 to 35 %
    // (2048 x 1536 x 512 16.4 -> 13.8 us, 4096 x 1024 x 1024 24.3 -> 20.2, 16384 x 4096 x 1024 with ReLU^2 257 -> 169; K <= 128 3 to 12 %), the price where
    // none does 1 to 5 % (16.0 -> 16.6, 23.4 -> 24.3, 250 -> 258).  With fewer both are about 5 % (4096 x 512 x 512 11.4 -> 10.8, 11.0 -> 11.7; 2048 x 1024 x 1024 15.2 -> 14.1,
    // 14.9 -> 15.3).  Larger K and raw outputs are not measured.
    const bool soma = BLK == 32 && modo != 1 && !estreito && K <= 1024 && partes == 1 && tiles <= (long long)th::N_PLANOS * N_SM && (g_somas == 2 || (g_somas == 0 && tiles > N_SM));
    // The bounds with the shift serve every product.  Long rows are prepared faster without it (4096 x 1024 x 16384 raw 271 -> 267 us, the preparation
    // 55.2 -> 51.5), shorter ones with it (1536 x 512 x 4096 raw 42.8 against 43.0 us, 2048 x 512 x 2048 20.7 against 20.9).
    lanca_pdl(soma || K < 8192 ? th::k_prep_h<BLK, BLK == 32> : th::k_prep_h<BLK, false>, dim3(ctasA + ctasB), dim3(256), 0, g_stream, P);
    if (partes > 1 && !grupo) {
        cudaError_t c = cudaMemsetAsync(S.C32, 0, (size_t)M * N * sizeof(int), g_stream);
        if (c != cudaSuccess) return (int)c;
    }
#define JT_H(MD)                                                                                                                            \
    case MD:                                                                                                                                \
        if constexpr (BLK == 32)                                                                                                            \
            if (estreito)                                                                                                                   \
                return grupo ? lanca_h<32, MD, 64, true>(mA, mB, RAw, RBw, nA, nB, S, M, N, K, G, kid)                                      \
                             : lanca_h<32, MD, 64, false>(mA, mB, RAw, RBw, nA, nB, S, M, N, K, G, kid);                                    \
        if constexpr (BLK == 32 && MD != 1)                                                                                                 \
            if (soma) return lanca_h<32, MD, 128, false, true>(mA, mB, RAw, RBw, nA, nB, S, M, N, K, G, kid);                               \
        return lanca_h<BLK, MD, 128, false>(mA, mB, RAw, RBw, nA, nB, S, M, N, K, G, kid);
    switch (modo) { JT_H(0) JT_H(1) JT_H(2) JT_H(3) JT_H(4) }
#undef JT_H
    return (int)cudaErrorInvalidValue;
}

// a workspace of the caller: the kernels' widest access to one is a TMA box of 128-byte rows (PyTorch's allocator gives multiples of 512)
static bool ws_serve(const void* ws) { return ws && ((uintptr_t)ws & 127) == 0; }

#define JT_POR_BLK(EXPR32, EXPR128) (g_blk == 32 ? (EXPR32) : (EXPR128))

extern "C" {

// ---------------------------------------------------------------------------------------------- control
// Where the error record was last cleared: that happens in the order of one stream, and a launch on another one must not come before it.
static struct { cudaEvent_t ev[64]; int dev; cudaStream_t onde, esperam[16]; int n; bool pendente; } g_limpa;
static void espera_limpeza(cudaStream_t st) {
    if (!g_limpa.pendente || st == g_limpa.onde) return;
    for (int i = 0; i < g_limpa.n; i++)
        if (g_limpa.esperam[i] == st) return;
    // (launches that are being captured run when the graph is launched, on a stream of its caller's choice)
    int dev = -1;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != g_limpa.dev || cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return;
    }
    if (g_limpa.n == 16) {                 // more streams than there is room for: wait here
        if (cudaEventSynchronize(g_limpa.ev[dev]) == cudaSuccess) g_limpa.pendente = false;
        return;
    }
    if (cudaStreamWaitEvent(st, g_limpa.ev[dev], 0) == cudaSuccess) g_limpa.esperam[g_limpa.n++] = st;
}
int jt_erro_le(long long* out) {
    Erro e;
    // the launches and the clearing before this call are on the stream set with jt_stream or ordered before it
    (void)cudaStreamSynchronize(g_stream);
    cudaError_t c = cudaMemcpyFromSymbol(&e, g_erro, sizeof(Erro));
    if (c != cudaSuccess) return -(int)c;
    out[0] = e.n; out[1] = e.codigo; out[2] = e.kid; out[3] = e.idx; out[4] = e.valor; out[5] = e.aux;
    return e.n;
}
// Limit of every bounded wait of the tensor-core kernels, in SM clock cycles (<= 0: back to the default of about 2 s).
int jt_espera_limite(long long ciclos) {
    const long long v = ciclos > 0 ? ciclos : tc::LIMITE_CICLOS;
    return (int)cudaMemcpyToSymbol(tc::g_limite_espera, &v, sizeof(v));
}
// Test switch: with 1 the tensor-core GEMM issues no operand load, so its MMA warp's first wait runs out after the limit in
// force, the CTA records code 7, raises its abort flag and every warp leaves through the normal exit (outputs undefined).
int jt_gemm_sem_cargas(int ligado) {
    const int v = ligado ? 1 : 0;
    return (int)cudaMemcpyToSymbol(tc::g_sem_cargas, &v, sizeof(v));
}
// Self-test of the bounded wait: one warp waits on a barrier nothing completes and must give up after the limit in force
// (set a short one first).  *saiu (device int) becomes 2 when it gave up; the error record then holds code 7, place 99.
int jt_teste_espera(int* saiu, int kid) {
    tc::k_teste_espera<<<1, 32, 0, g_stream>>>(kid, saiu);
    return fim();
}
// Programmatic dependent launch of the kernels that support it (0 = plain stream order).
int jt_pdl(int ligado) { pdl_ligado() = ligado ? 1 : 0; return 0; }
// Clears the error record, in the order of the launches: on the stream set with jt_stream, and before the launches that follow on any other one
// it is set to.  A step that begins does not wait for the GPU.
int jt_erro_limpa() {
    static void* onde[64];                 // address of the record, per device
    int dev = 0;
    cudaError_t c = cudaGetDevice(&dev);
    if (c != cudaSuccess) return (int)c;
    if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    if (!onde[dev] && (c = cudaGetSymbolAddress(&onde[dev], g_erro)) != cudaSuccess) return (int)c;
    if ((c = cudaMemsetAsync(onde[dev], 0, sizeof(Erro), g_stream)) != cudaSuccess) return (int)c;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    g_limpa.pendente = cudaStreamIsCapturing(g_stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
    if (!g_limpa.pendente) return 0;
    if (!g_limpa.ev[dev] && (c = cudaEventCreateWithFlags(&g_limpa.ev[dev], cudaEventDisableTiming)) != cudaSuccess) return (int)c;
    g_limpa.dev = dev;
    g_limpa.onde = g_stream;
    g_limpa.n = 0;
    return (int)cudaEventRecord(g_limpa.ev[dev], g_stream);
}
int jt_sincroniza() { return (int)cudaDeviceSynchronize(); }
void jt_stream(void* st) {
    g_ao_lado = false;
    g_stream = (cudaStream_t)st;
    espera_limpeza(g_stream);
}
// jt_stream for a chain of launches that runs beside another one, until the next jt_stream: a product of either tensor-core kernel then has a block for each of its
// 128 x 128 tiles at most, or N_LADO.  The results are the same.
void jt_stream_ao_lado(void* st) {
    jt_stream(st);
    g_ao_lado = true;
}
void* jt_stream_atual() { return (void*)g_stream; }
void jt_gemm_split(int alvo) { g_alvo_ctas = alvo > 0 ? alvo : 148; }
void jt_gemm_bm(int) {}
void jt_atencao_linhas(int) {}
int jt_res_estocastico(int ligado) { return ligado ? (int)cudaErrorNotSupported : 0; }
int jt_blk(int blk) {
    if (blk != 32 && blk != 128) return (int)cudaErrorInvalidValue;
    g_blk = blk;
    return 0;
}
int jt_blk_atual() { return g_blk; }
int jt_gemm_tn(int tn) {
    if (tn != 0 && tn != 64 && tn != 128) return (int)cudaErrorInvalidValue;
    g_tn = tn;
    return 0;
}
int jt_gemm_somas(int quando) {
    if (quando < 0 || quando > 2) return (int)cudaErrorInvalidValue;
    g_somas = quando;
    return 0;
}
int jt_gemm_via(int via) {
    if (via < 0 || via > 4) return (int)cudaErrorInvalidValue;
    g_via = via;
    return 0;
}

// ---------------------------------------------------------------------------------------------- GEMM
int jt_gemm_ext(const void* A, const void* EA, const void* B, const void* EB, void* Cm, void* CE, void* C32, void* Ce, const void* Xm,
                const void* XE, void* Om2, void* OE2, const void* RA, const void* RB, int M, int N, int K, int modo, int kid) {
    SaidaGemm S = {(int8_t*)Cm, (int8_t*)CE, (int*)C32, (int16_t*)Ce, (const int8_t*)Xm, (const int8_t*)XE, (int8_t*)Om2, (int8_t*)OE2};
    if (modo == 1 ? (!C32 || !Ce) : (!Cm || !CE)) return (int)cudaErrorInvalidValue;
    if ((modo == 2 || modo == 4) && (!Xm || !XE)) return (int)cudaErrorInvalidValue;
    if (modo == 3 && (!Om2 || !OE2)) return (int)cudaErrorInvalidValue;
    return JT_POR_BLK(gemm_blk<32>((const int8_t*)A, (const int8_t*)EA, (const int8_t*)B, (const int8_t*)EB, (const int8_t*)RA, (const int8_t*)RB, S, M, N, K, modo, kid),
                      gemm_blk<128>((const int8_t*)A, (const int8_t*)EA, (const int8_t*)B, (const int8_t*)EB, (const int8_t*)RA, (const int8_t*)RB, S, M, N, K, modo, kid));
}
int jt_gemm_f(const void* A, const void* EA, const void* B, const void* EB, void* Cm, void* CE, void* C32, void* Ce, const void* Xm,
              const void* XE, void* Om2, void* OE2, int M, int N, int K, int modo, int kid) {
    return jt_gemm_ext(A, EA, B, EB, Cm, CE, C32, Ce, Xm, XE, Om2, OE2, nullptr, nullptr, M, N, K, modo, kid);
}
int jt_gemm(const void* A, const void* EA, const void* B, const void* EB, void* Cm, void* CE, void* C32, void* Ce, int M, int N, int K,
            int modo, int kid) {
    return jt_gemm_ext(A, EA, B, EB, Cm, CE, C32, Ce, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, M, N, K, modo, kid);
}
// Workspace of jt_gemm_ws for these sizes, in bytes; 0: the call would not use one (jt_gemm_ext is the same).
long long jt_gemm_ws_bytes(int M, int N, int K, int modo) {
    if (!forma_gemm(g_blk, M, N, K, modo) || !usa_h(M, N, K, modo)) return 0;
    return (long long)espaco_h(M, N, K).total;
}
// jt_gemm_ext with a workspace of at least jt_gemm_ws_bytes bytes (128-byte aligned, private to this call until its kernels are done)
int jt_gemm_ws(const void* A, const void* EA, const void* B, const void* EB, void* Cm, void* CE, void* C32, void* Ce, const void* Xm, const void* XE,
               void* Om2, void* OE2, const void* RA, const void* RB, void* ws, int M, int N, int K, int modo, int kid) {
    const bool alinhado = (((uintptr_t)A | (uintptr_t)B) & 15) == 0;
    if (!ws_serve(ws) || !alinhado || !forma_gemm(g_blk, M, N, K, modo) || !usa_h(M, N, K, modo))
        return jt_gemm_ext(A, EA, B, EB, Cm, CE, C32, Ce, Xm, XE, Om2, OE2, RA, RB, M, N, K, modo, kid);
    SaidaGemm S = {(int8_t*)Cm, (int8_t*)CE, (int*)C32, (int16_t*)Ce, (const int8_t*)Xm, (const int8_t*)XE, (int8_t*)Om2, (int8_t*)OE2};
    if (modo == 1 ? (!C32 || !Ce) : (!Cm || !CE)) return (int)cudaErrorInvalidValue;
    if ((modo == 2 || modo == 4) && (!Xm || !XE)) return (int)cudaErrorInvalidValue;
    if (modo == 3 && (!Om2 || !OE2)) return (int)cudaErrorInvalidValue;
    return JT_POR_BLK(gemm_h<32>((const int8_t*)A, (const int8_t*)EA, (const int8_t*)B, (const int8_t*)EB, (const int8_t*)RA, (const int8_t*)RB, S, M, N, K, modo, (unsigned char*)ws, kid),
                      gemm_h<128>((const int8_t*)A, (const int8_t*)EA, (const int8_t*)B, (const int8_t*)EB, (const int8_t*)RA, (const int8_t*)RB, S, M, N, K, modo, (unsigned char*)ws, kid));
}
// row-maximum exponents of a block tensor [R, C] (int8 per row): what a data-parallel rank exchanges before a
// weight-gradient GEMM so that all ranks align their partial sums to the same exponents
int jt_max_linha(const void* E, void* R8, int linhas, int nb, int kid) {
    (void)kid;
    if (linhas <= 0 || nb <= 0) return (int)cudaErrorInvalidValue;
    k_max_linha<<<(linhas + 255) / 256, 256, 0, g_stream>>>((const int8_t*)E, (int8_t*)R8, linhas, nb);
    return fim();
}

// ---------------------------------------------------------------------------------------------- block ops
#define JT_N16 (nblocos * (long long)g_blk / 16)
int jt_quant(const void* acc, const void* e, void* m, void* E, long long nblocos, int kid) {
    const long long n16 = JT_N16;
    if (g_blk == 32) k_quant<32><<<nblocos16(n16), 256, 0, g_stream>>>((const int*)acc, (const int16_t*)e, (int8_t*)m, (int8_t*)E, n16, kid);
    else k_quant<128><<<nblocos16(n16), 256, 0, g_stream>>>((const int*)acc, (const int16_t*)e, (int8_t*)m, (int8_t*)E, n16, kid);
    return fim();
}
int jt_soma(const void* xm, const void* xE, const void* ym, const void* yE, void* zm, void* zE, long long nblocos, int kid) {
    const long long n16 = JT_N16;
#define ARGS (const int8_t*)xm, (const int8_t*)xE, (const int8_t*)ym, (const int8_t*)yE, (int8_t*)zm, (int8_t*)zE, n16, kid
    if (g_blk == 32) k_soma<32><<<nblocos16u(n16, 4), 256, 0, g_stream>>>(ARGS);
    else k_soma<128><<<nblocos16u(n16, 4), 256, 0, g_stream>>>(ARGS);
#undef ARGS
    return fim();
}
int jt_relu2(const void* hm, const void* hE, void* am, void* aE, long long nblocos, int kid) {
    const long long n16 = JT_N16;
    if (g_blk == 32) k_relu2<32><<<nblocos16u(n16, 4), 256, 0, g_stream>>>((const int8_t*)hm, (const int8_t*)hE, (int8_t*)am, (int8_t*)aE, n16, kid);
    else k_relu2<128><<<nblocos16u(n16, 4), 256, 0, g_stream>>>((const int8_t*)hm, (const int8_t*)hE, (int8_t*)am, (int8_t*)aE, n16, kid);
    return fim();
}
int jt_relu2_back(const void* gm, const void* gE, const void* hm, const void* hE, void* om, void* oE, long long nblocos, int kid) {
    const long long n16 = JT_N16;
#define ARGS (const int8_t*)gm, (const int8_t*)gE, (const int8_t*)hm, (const int8_t*)hE, (int8_t*)om, (int8_t*)oE, n16, kid
    if (g_blk == 32) k_relu2_back<32><<<nblocos16u(n16, 4), 256, 0, g_stream>>>(ARGS);
    else k_relu2_back<128><<<nblocos16u(n16, 4), 256, 0, g_stream>>>(ARGS);
#undef ARGS
    return fim();
}
int jt_momento(const void* gacc, const void* ge, void* Mm, void* ME, long long nblocos, int kid) {
    const long long n16 = JT_N16;
    if (g_blk == 32) k_momento<32><<<nblocos_128(n16), 128, 0, g_stream>>>((const int*)gacc, (const int16_t*)ge, (int8_t*)Mm, (int8_t*)ME, n16, kid);
    else k_momento<128><<<nblocos_128(n16), 128, 0, g_stream>>>((const int*)gacc, (const int16_t*)ge, (int8_t*)Mm, (int8_t*)ME, n16, kid);
    return fim();
}
int jt_peso(void* Wm, void* WE, const void* Mm, const void* ME, void* Rm, void* RE, int k_lr, int ef, long long nblocos, int kid) {
    const long long n16 = JT_N16;
#define ARGS (int8_t*)Wm, (int8_t*)WE, (const int8_t*)Mm, (const int8_t*)ME, (int8_t*)Rm, (int8_t*)RE, k_lr, ef, n16, kid
    if (g_blk == 32) k_peso<32><<<nblocos16(n16), 256, 0, g_stream>>>(ARGS);
    else k_peso<128><<<nblocos16(n16), 256, 0, g_stream>>>(ARGS);
#undef ARGS
    return fim();
}
int jt_momento_peso(const void* gacc, const void* ge, void* Mm, void* ME, void* Wm, void* WE, void* Rm, void* RE, int k_lr, int ef,
                    long long nblocos, int kid) {
    const long long n16 = JT_N16;
#define ARGS (const int*)gacc, (const int16_t*)ge, (int8_t*)Mm, (int8_t*)ME, (int8_t*)Wm, (int8_t*)WE, (int8_t*)Rm, (int8_t*)RE, k_lr, ef, n16, kid
    if (g_blk == 32) lanca_pdl(k_momento_peso<32>, dim3(nblocos_128(n16)), dim3(128), 0, g_stream, ARGS);
    else lanca_pdl(k_momento_peso<128>, dim3(nblocos_128(n16)), dim3(128), 0, g_stream, ARGS);
#undef ARGS
    return fim();
}
}  // extern "C"
static int transpoe_impl(const ArgsTransp& a0, const ArgsTransp& a1, int R, int kid) {
    auto pecas = [&](const ArgsTransp& a) { return a.X ? (a.C + 127) / 128 * (R / 128) : 0; };
    const int n0 = pecas(a0), n = n0 + pecas(a1);              // 128 x 128 pieces
    // fewer than three (block 128: two) per SM: four warps share the columns of every 32 rows
    const bool poucas = n < (g_blk == 32 ? 3 : 2) * N_SM;
    if (g_blk == 32) {
        if (poucas) lanca_pdl(k_transpoe<32, 1>, dim3(4 * n), dim3(128), 0, g_stream, a0, a1, 4 * n0, R, kid);
        else lanca_pdl(k_transpoe<32, 4>, dim3(n), dim3(128), 0, g_stream, a0, a1, n0, R, kid);
    } else {
        if (poucas) lanca_pdl(k_transpoe<128, 1>, dim3(n), dim3(512), 0, g_stream, a0, a1, n0, R, kid);
        else lanca_pdl(k_transpoe<128, 4>, dim3(n), dim3(128), 0, g_stream, a0, a1, n0, R, kid);
    }
    return fim();
}
extern "C" {
int jt_transpoe(const void* X, const void* EX, void* Y, void* EY, int R, int C, int kid) {
    if (R <= 0 || C <= 0 || R % 128 || C % 64 || C % g_blk) return (int)cudaErrorInvalidValue;
    return transpoe_impl({(const int8_t*)X, (const int8_t*)EX, (int8_t*)Y, (int8_t*)EY, C, nullptr}, {}, R, kid);
}
// the pair of transpositions; RM1 / RM2 (optional, both or none): int8 [C1] / [C2], pre-set to -128 by the caller, receive the
// row maxima of the exponents of Y1 / Y2 (what jt_max_linha would compute from EY1 / EY2)
static int transpoe2_impl(const void* X1, const void* EX1, void* Y1, void* EY1, const void* X2, const void* EX2, void* Y2, void* EY2, int C1, int C2,
                          int R, void* RM1, void* RM2, int kid) {
    if (R <= 0 || C1 <= 0 || C2 <= 0 || R % 128 || C1 % 64 || C2 % 64 || C1 % g_blk || C2 % g_blk) return (int)cudaErrorInvalidValue;
    const bool com_max = RM1 != nullptr || RM2 != nullptr;
    if (com_max && (RM1 == nullptr || RM2 == nullptr || (((uintptr_t)RM1 | (uintptr_t)RM2) & 3) != 0)) return (int)cudaErrorInvalidValue;
    if (com_max && (g_blk != 32 || C1 % 256 || C2 % 256)) return (int)cudaErrorNotSupported;
    return transpoe_impl({(const int8_t*)X1, (const int8_t*)EX1, (int8_t*)Y1, (int8_t*)EY1, C1, (int8_t*)RM1},
                         {(const int8_t*)X2, (const int8_t*)EX2, (int8_t*)Y2, (int8_t*)EY2, C2, (int8_t*)RM2}, R, kid);
}
int jt_transpoe2(const void* X1, const void* EX1, void* Y1, void* EY1, const void* X2, const void* EX2, void* Y2, void* EY2, int C1, int C2,
                 int R, int kid) {
    return transpoe2_impl(X1, EX1, Y1, EY1, X2, EX2, Y2, EY2, C1, C2, R, nullptr, nullptr, kid);
}
int jt_transpoe2_max(const void* X1, const void* EX1, void* Y1, void* EY1, const void* X2, const void* EX2, void* Y2, void* EY2, void* RM1,
                     void* RM2, int C1, int C2, int R, int kid) {
    if (RM1 == nullptr || RM2 == nullptr) return (int)cudaErrorInvalidValue;
    return transpoe2_impl(X1, EX1, Y1, EY1, X2, EX2, Y2, EY2, C1, C2, R, RM1, RM2, kid);
}
int jt_embed(const void* Wm, const void* WE, const void* tok, void* Xm, void* XE, int M, int D, int V, int kid) {
    if (M <= 0 || D <= 0 || D % g_blk) return (int)cudaErrorInvalidValue;
    const unsigned g = (unsigned)(((long long)M * (D / 16) + 255) / 256);
#define ARGS (const int8_t*)Wm, (const int8_t*)WE, (const int*)tok, (int8_t*)Xm, (int8_t*)XE, M, D, V, kid
    if (g_blk == 32) lanca_pdl(k_embed<32>, dim3(g), dim3(256), 0, g_stream, ARGS);
    else lanca_pdl(k_embed<128>, dim3(g), dim3(256), 0, g_stream, ARGS);
#undef ARGS
    return fim();
}
int jt_um_quente(const void* tok, void* U, void* UE, int M, int V, int kid) {
    if (M <= 0 || V <= 0 || V % g_blk) return (int)cudaErrorInvalidValue;
    const unsigned g = (unsigned)(((long long)M * (V / 16) + 255) / 256);
    if (g_blk == 32) lanca_pdl(k_um_quente<32>, dim3(g), dim3(256), 0, g_stream, (const int*)tok, (int8_t*)U, (int8_t*)UE, M, V, kid);
    else lanca_pdl(k_um_quente<128>, dim3(g), dim3(256), 0, g_stream, (const int*)tok, (int8_t*)U, (int8_t*)UE, M, V, kid);
    return fim();
}

// one warp per row; NP = number of 512-column passes a row needs
#define JT_LINHA(KERN, COLS, ...)                                                                    \
    do {                                                                                             \
        const unsigned g_ = (unsigned)((M + 7) / 8);                                                 \
        const int np_ = ((COLS) + 511) / 512;                                                        \
        if (g_blk == 32) {                                                                           \
            if (np_ == 1) lanca_pdl(KERN<32, 1>, dim3(g_), dim3(256), 0, g_stream, __VA_ARGS__);                        \
            else if (np_ == 2) lanca_pdl(KERN<32, 2>, dim3(g_), dim3(256), 0, g_stream, __VA_ARGS__);                   \
            else lanca_pdl(KERN<32, 4>, dim3(g_), dim3(256), 0, g_stream, __VA_ARGS__);                                 \
        } else {                                                                                     \
            if (np_ == 1) lanca_pdl(KERN<128, 1>, dim3(g_), dim3(256), 0, g_stream, __VA_ARGS__);                       \
            else if (np_ == 2) lanca_pdl(KERN<128, 2>, dim3(g_), dim3(256), 0, g_stream, __VA_ARGS__);                  \
            else lanca_pdl(KERN<128, 4>, dim3(g_), dim3(256), 0, g_stream, __VA_ARGS__);                                \
        }                                                                                            \
    } while (0)

int jt_rms(const void* Xm, const void* XE, void* Ym, void* YE, void* cr, void* cemax, int M, int D, int log2D, int G, int kid) {
    if (M <= 0 || D <= 0 || D % g_blk || D > 2048 || (1 << log2D) != D) return (int)cudaErrorInvalidValue;
    JT_LINHA(k_rms, D, (const int8_t*)Xm, (const int8_t*)XE, (int8_t*)Ym, (int8_t*)YE, (int*)cr, (int*)cemax, M, D, log2D, G, kid);
    return fim();
}
int jt_rms_back(const void* gm, const void* gE, const void* ym, const void* yE, const void* cr, const void* cemax, void* om, void* oE, int M,
                int D, int log2D, int G, int GB, int kid) {
    if (M <= 0 || D <= 0 || D % g_blk || D > 2048 || (1 << log2D) != D) return (int)cudaErrorInvalidValue;
    JT_LINHA(k_rms_back, D, (const int8_t*)gm, (const int8_t*)gE, (const int8_t*)ym, (const int8_t*)yE, (const int*)cr, (const int*)cemax,
             (int8_t*)om, (int8_t*)oE, M, D, log2D, G, GB, kid);
    return fim();
}
int jt_rms_back_soma(const void* gm, const void* gE, const void* ym, const void* yE, const void* cr, const void* cemax, const void* xm,
                     const void* xE, void* om, void* oE, int M, int D, int log2D, int G, int GB, int kid) {
    if (M <= 0 || D <= 0 || D % g_blk || D > 2048 || (1 << log2D) != D || !xm || !xE) return (int)cudaErrorInvalidValue;
    JT_LINHA(k_rms_back_soma, D, (const int8_t*)gm, (const int8_t*)gE, (const int8_t*)ym, (const int8_t*)yE, (const int*)cr, (const int*)cemax,
             (const int8_t*)xm, (const int8_t*)xE, (int8_t*)om, (int8_t*)oE, M, D, log2D, G, GB, kid);
    return fim();
}
int jt_softmax_ce(const void* acc, const void* e, const void* alvo, void* gm, void* gE, void* d_alvo, void* soma, int M, int V, int log2M,
                  int kid) {
    if (M <= 0 || V <= 0 || V % g_blk || V > 2048) return (int)cudaErrorInvalidValue;
    if (V <= 256) {                        // 16 lanes take a row: with 32 half of a warp would have nothing
        lanca_pdl(g_blk == 32 ? k_softmax_ce<32, 1, 16> : k_softmax_ce<128, 1, 16>, dim3((M + 15) / 16), dim3(256), 0, g_stream, (const int*)acc,
                  (const int16_t*)e, (const int*)alvo, (int8_t*)gm, (int8_t*)gE, (int*)d_alvo, (int*)soma, M, V, log2M, kid);
        return fim();
    }
    JT_LINHA(k_softmax_ce, V, (const int*)acc, (const int16_t*)e, (const int*)alvo, (int8_t*)gm, (int8_t*)gE, (int*)d_alvo, (int*)soma, M, V,
             log2M, kid);
    return fim();
}

int jt_perda(const void* d_alvo, const void* soma, void* perda, int M, int kid) {
    (void)kid;
    if (M <= 0) return (int)cudaErrorInvalidValue;
    lanca_pdl(k_perda, dim3((M + 255) / 256), dim3(256), 0, g_stream, (const int*)d_alvo, (const int*)soma, (double*)perda, M);
    return fim();
}

// ---------------------------------------------------------------------------------------------- attention
}  // extern "C"
// What the accesses of the kernels ask of the addresses: the tensor-core path reads mantissas 8 bytes and P 16 bytes (and by TMA) at a time, the
// one-CTA-per-head kernels mantissas 4 and P 16 bytes.  A tensor that starts elsewhere in a larger buffer goes to the general
// kernels, which take heads of 4 at any multiple of 4 and P anywhere.
static bool p_alinhado(const void* P) { return ((uintptr_t)P & 15) == 0; }
static bool usa_atc(int Bt, int T, int H, int D, int GA, bool tras) { return g_at_via == 0 && Bt > 0 && H > 0 && atc_serve(g_blk, T, H, D, GA, tras); }
static bool usa_atc(const void* qm, const void* gom, const void* P, int Bt, int T, int H, int D, int GA, bool tras) {
    return (((uintptr_t)qm | (uintptr_t)gom) & 7) == 0 && p_alinhado(P) && usa_atc(Bt, T, H, D, GA, tras);
}
extern "C" {
// Workspace of jt_atencao_ws (tras = 0) / jt_atencao_back_ws (1) for these sizes, in bytes; 0: the call would not use one.
long long jt_atencao_ws_bytes(int Bt, int T, int H, int D, int GA, int tras) {
    return usa_atc(Bt, T, H, D, GA, tras != 0) ? (long long)atc_ws_bytes(Bt, H, T, tras != 0) : 0;
}
// jt_atencao, or (Om, OE instead of Oacc, Oe) jt_atencao_quant, with a workspace of the caller: at least jt_atencao_ws_bytes bytes, 128-byte
// aligned, private to this call until its kernels are done.  Without one that serves, the raw form is jt_atencao, the other is not supported.
int jt_atencao_ws(const void* qm, const void* qE, void* Oacc, void* Oe, void* Om, void* OE, void* P, void* ws, int Bt, int T, int H, int D, int GA, int kid) {
    const bool tc = ws_serve(ws) && usa_atc(qm, nullptr, P, Bt, T, H, D, GA, false);
    if (Om ? !tc || g_blk != 32 || D != 64 * H : !Oacc || !Oe) return (int)(Om ? cudaErrorNotSupported : cudaErrorInvalidValue);
    if (tc)
        return atencao_frente_tc(g_blk, (const int8_t*)qm, (const int8_t*)qE, (int*)Oacc, (int16_t*)Oe, (int8_t*)Om, (int8_t*)OE, (uint8_t*)P, Bt, T, H, D, GA,
                                 kid, g_stream, (unsigned char*)ws);
    if (g_at_via == 0 && Bt > 0 && atp_serve(g_blk, T, H, D, GA) && p_alinhado(P))
        return atencao_frente_peq(g_blk, (const int8_t*)qm, (const int8_t*)qE, (int*)Oacc, (int16_t*)Oe, (uint8_t*)P, Bt, T, H, D, GA, kid, g_stream);
    return atencao_frente(g_blk, (const int8_t*)qm, (const int8_t*)qE, (int*)Oacc, (int16_t*)Oe, (uint8_t*)P, Bt, T, H, D, GA, kid, g_stream);
}
int jt_atencao_back_ws(const void* gom, const void* goE, const void* qm, const void* qE, const void* P, void* Gacc, void* Ge, void* Gm, void* GE, void* ws,
                       int Bt, int T, int H, int D, int GA, int limite, int kid) {
    const bool tc = ws_serve(ws) && usa_atc(qm, gom, P, Bt, T, H, D, GA, true);
    if (Gm ? !tc || g_blk != 32 || D != 64 * H : !Gacc || !Ge) return (int)(Gm ? cudaErrorNotSupported : cudaErrorInvalidValue);
    if (tc)
        return atencao_tras_tc(g_blk, (const int8_t*)gom, (const int8_t*)goE, (const int8_t*)qm, (const int8_t*)qE, (const uint8_t*)P, (int*)Gacc,
                               (int16_t*)Ge, (int8_t*)Gm, (int8_t*)GE, Bt, T, H, D, GA, limite, kid, g_stream, (unsigned char*)ws);
    if (g_at_via == 0 && Bt > 0 && atp_serve(g_blk, T, H, D, GA) && p_alinhado(P))
        return atencao_tras_peq(g_blk, (const int8_t*)gom, (const int8_t*)goE, (const int8_t*)qm, (const int8_t*)qE, (const uint8_t*)P, (int*)Gacc,
                                (int16_t*)Ge, Bt, T, H, D, GA, limite, kid, g_stream);
    return atencao_tras(g_blk, (const int8_t*)gom, (const int8_t*)goE, (const int8_t*)qm, (const int8_t*)qE, (const uint8_t*)P, (int*)Gacc,
                        (int16_t*)Ge, Bt, T, H, D, GA, limite, kid, g_stream);
}
// Without a workspace of the caller the library takes one for the length of the call; where there is none to be had, the raw forms go to the
// general kernels, which need none (forward) or little (backward).
int jt_atencao(const void* qm, const void* qE, void* Oacc, void* Oe, void* P, int Bt, int T, int H, int D, int GA, int kid) {
    Espaco ws(g_stream);
    if (usa_atc(qm, nullptr, P, Bt, T, H, D, GA, false)) (void)ws.toma(atc_ws_bytes(Bt, H, T, false));
    return jt_atencao_ws(qm, qE, Oacc, Oe, nullptr, nullptr, P, ws.p, Bt, T, H, D, GA, kid);
}
int jt_atencao_back(const void* gom, const void* goE, const void* qm, const void* qE, const void* P, void* Gacc, void* Ge, int Bt, int T,
                    int H, int D, int GA, int limite, int kid) {
    Espaco ws(g_stream);
    if (usa_atc(qm, gom, P, Bt, T, H, D, GA, true)) (void)ws.toma(atc_ws_bytes(Bt, H, T, true));
    return jt_atencao_back_ws(gom, goE, qm, qE, P, Gacc, Ge, nullptr, nullptr, ws.p, Bt, T, H, D, GA, limite, kid);
}
// jt_quant(jt_atencao(...)) and jt_quant(jt_atencao_back(...)) in the attention kernels' own output stage: block tensors [Bt*T, D] and
// [Bt*T, 3D] come out directly.  Served by the tensor-core path at head dimension 64 and block length 32; elsewhere
// cudaErrorNotSupported, and the caller composes the two operations.
int jt_atencao_quant(const void* qm, const void* qE, void* Om, void* OE, void* P, int Bt, int T, int H, int D, int GA, int kid) {
    if (!Om || g_blk != 32 || D != 64 * H || !usa_atc(qm, nullptr, P, Bt, T, H, D, GA, false)) return (int)cudaErrorNotSupported;
    Espaco ws(g_stream);
    if (!ws.toma(atc_ws_bytes(Bt, H, T, false))) return (int)cudaErrorMemoryAllocation;
    return jt_atencao_ws(qm, qE, nullptr, nullptr, Om, OE, P, ws.p, Bt, T, H, D, GA, kid);
}
int jt_atencao_back_quant(const void* gom, const void* goE, const void* qm, const void* qE, const void* P, void* Gm, void* GE, int Bt, int T, int H,
                          int D, int GA, int limite, int kid) {
    if (!Gm || g_blk != 32 || D != 64 * H || !usa_atc(qm, gom, P, Bt, T, H, D, GA, true)) return (int)cudaErrorNotSupported;
    Espaco ws(g_stream);
    if (!ws.toma(atc_ws_bytes(Bt, H, T, true))) return (int)cudaErrorMemoryAllocation;
    return jt_atencao_back_ws(gom, goE, qm, qE, P, nullptr, nullptr, Gm, GE, ws.p, Bt, T, H, D, GA, limite, kid);
}
// The largest workspace the library takes for a call, in bytes (0: no limit) / returns what its pool of the current device keeps between calls.
int jt_espaco_limite(long long bytes) {
    if (bytes < 0) return (int)cudaErrorInvalidValue;
    g_espaco_limite = bytes;
    return 0;
}
int jt_espaco_libera() {
    int dev = 0;
    cudaError_t c = cudaGetDevice(&dev);
    if (c != cudaSuccess) return (int)c;
    std::lock_guard<std::mutex> l(g_pool_trava);
    return dev < 0 || dev >= AT_MAX_DEV || !g_pool[dev] ? 0 : (int)cudaMemPoolTrimTo(g_pool[dev], 0);
}
int jt_atencao_via(int via) {
    if (via < 0 || via > 1) return (int)cudaErrorInvalidValue;
    g_at_via = via;
    return 0;
}

// Attention backward for callers that must not allocate device memory: a process that runs under a fixed memory
// budget carved up before start-up, a host thread inside a callback where allocation is not
// permitted, or an embedding runtime that forbids the library to touch the allocator at all.  jt_atencao_back
// takes a workspace for the length of the call; this variant keeps the workspace (statistics + one s_lin per
// query row = Bt*H*(8+T) ints) in the fixed array below instead, and calls no allocating routine.
//   * limit: Bt*H*(8+T) <= JT_FIXO_INTS (2^20 ints = 4 MiB, resident on every GPU that loads the library until
//     the process exits); larger problems are refused with cudaErrorInvalidValue and a message on stderr;
//   * the first call on each device looks up the array's device address (cudaGetSymbolAddress, with that device
//     current) and remembers it; make that first call outside any stream capture;
//   * every call shares the one array: the statistics slots are cleared at the start of each call, the s_lin
//     slots are overwritten before they are read; two calls that overlap on the GPU (different streams) race.
constexpr size_t JT_FIXO_INTS = (size_t)1 << 20;
static __device__ __align__(256) int g_at_fixo[JT_FIXO_INTS];
static int* g_at_fixo_end[64];          // device address of g_at_fixo, per device ordinal (host-side cache)

int jt_atencao_back_fixo(const void* gom, const void* goE, const void* qm, const void* qE, const void* P, void* Gacc, void* Ge, int Bt,
                         int T, int H, int D, int GA, int limite, int kid) {
    if (Bt <= 0 || T <= 0 || H <= 0) return (int)cudaErrorInvalidValue;
    const size_t precisa = (size_t)Bt * H * (at::N_EST + T);
    if (precisa > JT_FIXO_INTS) {
        fprintf(stderr, "jt_atencao_back_fixo: Bt*H*(8+T) = %zu ints exceeds the fixed workspace of %zu ints; use jt_atencao_back\n",
                precisa, JT_FIXO_INTS);
        return (int)cudaErrorInvalidValue;
    }
    int dev = 0;
    cudaError_t c = cudaGetDevice(&dev);
    if (c != cudaSuccess) return (int)c;
    if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    if (!g_at_fixo_end[dev]) {
        void* p = nullptr;
        c = cudaGetSymbolAddress(&p, g_at_fixo);      // the symbol name is a host-side handle, not a device pointer
        if (c != cudaSuccess) return (int)c;
        g_at_fixo_end[dev] = static_cast<int*>(p);
    }
    return atencao_tras_ws(g_blk, (const int8_t*)gom, (const int8_t*)goE, (const int8_t*)qm, (const int8_t*)qE, (const uint8_t*)P, (int*)Gacc,
                           (int16_t*)Ge, Bt, T, H, D, GA, limite, kid, g_stream, g_at_fixo_end[dev],
                           precisa + (size_t)Bt * H * T * T <= JT_FIXO_INTS);      // room for the T x T matrices too, or the phases recompute
}

// The 16-bit residual stream of the reference (jt_para16 / jt_para8 / jt_soma16) is an opt-in ablation without an
// int64 specification; it is not part of this library.  The symbols exist so that the reference launcher's
// restype loop (ops.py:301-304) finds them; calling one reports "not supported".
int jt_para16(const void*, const void*, void*, void*, long long, int) { return (int)cudaErrorNotSupported; }
int jt_para8(const void*, const void*, void*, void*, long long, int) { return (int)cudaErrorNotSupported; }
int jt_soma16(const void*, const void*, const void*, const void*, void*, void*, long long, int) { return (int)cudaErrorNotSupported; }

}  // extern "C"
