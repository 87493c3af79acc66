// Block GEMM on the half-precision tensor pipe (tcgen05.mma kind::f16, fp32 accumulators in tensor memory) with the exponent alignment
// folded into the operands.
//
//   C[M,N] = A[M,K] . B[N,K]^T, operands blocked along K (jatai_cuda/ops.py:95-108):
//   acc_ij = sum over K-blocks b of rnd(p_ijb << 4, (RA_i - ea_ib) + (RB_j - eb_jb)),  p = exact int8 dot product of the block.
//
// What has to be rounded is r = p 2^(4 - sa - sb) with sa = RA_i - ea_ib, sb = RB_j - eb_jb.  A mantissa times a power of two is exact in
// half precision over the range that matters, so a first kernel (k_prep_h) writes A' = a 2^(2 - sa) and B' = b 2^(2 - sb) as f16 and
// the tensor core's fp32 sum over one block IS r, exactly: all products of a block are whole multiples of 2^(4 - sa - sb) below
// 2^24 of them (|p| <= 32 * 127^2 < 2^19, block 128: < 2^21).  From sa = 27 on (or sb) |r| < 1/2 for every p, the rounded value is 0
// and the operand is written as 0 (a 2^(2 - 26) is the smallest subnormal that occurs).
//
// That leaves the CUDA cores ONE packed addition per two element-steps - r + 1.5 * 2^23 rounds half to even at integer granularity -
// and one three-input integer addition per two element-steps (two K-blocks at a time): no exponent table, no scaling, no int -> float
// conversion.  The rounding is exact while |r| < 2^22, i.e. |p| 2^-(sa+sb) < 2^18.  Block 32: k_prep_h leaves, per 32 rows and K-block,
// the largest squared norm of a block scaled by 4^-s; by Cauchy-Schwarz the bound holds for a warp's 32 x 32 outputs whenever the product
// of its two norms is below 2^36, which a warp evaluates for 32 K-blocks at once; where it does not hold, it rounds by conversion.  Block 128
// (a quarter of the drains): the results' exponent fields are checked, and a warp in which one has left the window converts.
//
// Where sa + sb <= 4 nothing is rounded at all: r is a whole number.  A tile in which that holds for every K-block (what a step multiplies by
// its weights nearly always is: normalised rows and weights have block exponents one or two apart) need not be drained K-block by
// K-block; its chunks add up in tensor memory, in fp32, exactly while the sum of the bounds stays below 2^24 last places.  Large
// products with K <= 1024 look for it, with the norms and the largest shift that k_prep_h leaves: 16384 x 4096 x 1024 with ReLU^2 256 -> 167 us,
// 16384 x 1024 x 1024 69 -> 50.5.  Drained once, a tile waits for nothing but its operands, its MMAs and the output stage of the one before.
#pragma once
#include "gemm_tc.cuh"
#include "gemm_h_ordem.cuh"

namespace jt {
namespace th {

using namespace tc;

constexpr int KH = 64;                                     // K elements per operand stage: 128 bytes of f16, one swizzle row
constexpr float LIM_NORMA = 68719000000.0f;               // just below 2^36 (the product of two fp32 roundings included)
constexpr float LIM_SOMA = 16770000.0f;                    // just below 2^24
constexpr int N_PLANOS = 2048;                             // tiles of a block whose plans are kept, a byte each

// ------------------------------------------------------------------------------------------ operand preparation
struct ArgsPrepH {
    const int8_t* m[2]; const int8_t* E[2]; const int8_t* Rext[2];      // A and B: mantissas, exponents, external row maxima or nullptr
    uint16_t* h[2]; int8_t* R[2]; uint32_t* nrm[2];                      // f16 operands, row maxima, bounds [ceil(rows/32)][K/32] (block 32)
    int linhas[2], ctas0;                                                // rows of each; CTAs of A (B's follow)
    int K;
};

// 4 mantissas (bytes) -> 4 halves, scaled: with its sign bit flipped a byte b is b + 128; under the bits of 1024 it reads as the half
// 1152 + b, and one fused multiply-add takes the 1152 off and scales, exactly (every result is representable)
__device__ __forceinline__ void bytes_para_h(uint32_t w, uint32_t esc, uint32_t tira, uint32_t& lo, uint32_t& hi) {
    const uint32_t u = w ^ 0x80808080u;
    const uint32_t a = __byte_perm(u, 0x64646464u, 0x4140), b = __byte_perm(u, 0x64646464u, 0x4342);
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(lo) : "r"(a), "r"(esc), "r"(tira));
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(hi) : "r"(b), "r"(esc), "r"(tira));
}
__device__ __forceinline__ uint32_t dois_h(float v) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %1;" : "=r"(r) : "f"(v));
    return r;
}

// A bound is one word per 32 rows and K-block: the largest squared norm of a block of the group, scaled by 4^-s, as a float.  With DESLOC (products
// that add up in tensor memory need it) it is rounded up to 18 bits of mantissa, and the five bits that leaves free are the largest s of a
// block that is not zero.  4096 + 1024 rows of 16384: 55.2 us with it, 51.5 without.
//
// One CTA of 256 threads: 32 rows x 512 columns of one operand; a warp takes 4 rows, a lane 16 consecutive elements of each.  Bound by
// memory (1 byte in, 2 out per element); the exponents of the whole row are read by every CTA of the row (K / 32 bytes, from L2).
template <int BLK, bool DESLOC>
__global__ void __launch_bounds__(256) k_prep_h(const ArgsPrepH P) {
    pdl_espera();
    pdl_solta();
    __shared__ float nrm_s[8][16];
    __shared__ int smax_s[DESLOC ? 8 : 1][16];
    const int q = (int)blockIdx.x >= P.ctas0, cta = (int)blockIdx.x - (q ? P.ctas0 : 0);
    const int K = P.K, nb = K / BLK, nfx = (K + 511) / 512, c0 = (cta % nfx) * 512, g32 = cta / nfx;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, c = c0 + lane * 16;
    const int8_t *m = q ? P.m[1] : P.m[0], *E = q ? P.E[1] : P.E[0], *Rx = q ? P.Rext[1] : P.Rext[0];
    const int linhas = q ? P.linhas[1] : P.linhas[0], l0 = g32 * 32 + wid * 4;
    uint16_t* h = q ? P.h[1] : P.h[0];
    const bool dentro = c < K;
    uint4 v[4];
    int e[4], r[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int l = min(l0 + i, linhas - 1);
        v[i] = dentro ? *reinterpret_cast<const uint4*>(m + (size_t)l * K + c) : make_uint4(0, 0, 0, 0);
        e[i] = dentro ? (int)E[(size_t)l * nb + c / BLK] : E_ZERO;
        r[i] = -128;
    }
    if (Rx) {
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = Rx[min(l0 + i, linhas - 1)];
    } else {
        if ((nb & 3) == 0 && ((uintptr_t)E & 3) == 0) {          // (an exponent tensor may start at any byte of a larger buffer)
            for (int b = lane * 4; b < nb; b += 128)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t w = *reinterpret_cast<const uint32_t*>(E + (size_t)min(l0 + i, linhas - 1) * nb + b);
                    const unsigned m1 = __vmaxs4(w, w >> 16 | w << 16), m2 = __vmaxs4(m1, m1 >> 8 | m1 << 24);
                    r[i] = max(r[i], (int)(int8_t)(m2 & 0xff));
                }
        } else {
            for (int b = lane; b < nb; b += 32)
#pragma unroll
                for (int i = 0; i < 4; i++) r[i] = max(r[i], (int)E[(size_t)min(l0 + i, linhas - 1) * nb + b]);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = __reduce_max_sync(FULL, r[i]);
    }
    float nmax = 0.f;
    int smax = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int s = r[i] - e[i];
        const float esc = s <= 26 ? pot2(2 - s) : 0.f;
        const uint32_t e2 = dois_h(esc), t2 = dois_h(-1152.0f * esc);
        uint32_t o[8];
        bytes_para_h(v[i].x, e2, t2, o[0], o[1]);
        bytes_para_h(v[i].y, e2, t2, o[2], o[3]);
        bytes_para_h(v[i].z, e2, t2, o[4], o[5]);
        bytes_para_h(v[i].w, e2, t2, o[6], o[7]);
        if (dentro && l0 + i < linhas) {
            uint4* d = reinterpret_cast<uint4*>(h + (size_t)(l0 + i) * K + c);
            d[0] = make_uint4(o[0], o[1], o[2], o[3]);
            d[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
        if (BLK == 32) {
            int n = __dp4a((int)v[i].x, (int)v[i].x, 0);
            n = __dp4a((int)v[i].y, (int)v[i].y, n);
            n = __dp4a((int)v[i].z, (int)v[i].z, n);
            n = __dp4a((int)v[i].w, (int)v[i].w, n);
            n += __shfl_xor_sync(FULL, n, 1);
            // (a block of zeros, or one so far down that its operand is zero, adds nothing)
            nmax = fmaxf(nmax, (float)n * (s <= 26 ? pot2(-2 * s) : 0.f));
            if (DESLOC) smax = max(smax, n != 0 && s <= 26 ? s : 0);
        }
    }
    if (c0 == 0 && lane < 4 && l0 + lane < linhas) {
        const int rr = lane == 0 ? r[0] : lane == 1 ? r[1] : lane == 2 ? r[2] : r[3];
        (q ? P.R[1] : P.R[0])[l0 + lane] = (int8_t)rr;
    }
    if (BLK == 32) {
        // (the low five bits of a norm rounded up are free for the shift)
        if ((lane & 1) == 0) {
            nrm_s[wid][lane >> 1] = nmax;
            if (DESLOC) smax_s[wid][lane >> 1] = smax;
        }
        __syncthreads();
        if (threadIdx.x < 16 && c0 / 32 + (int)threadIdx.x < nb) {
            float n = 0.f;
            int sm = 0;
#pragma unroll
            for (int w = 0; w < 8; w++) {
                n = fmaxf(n, nrm_s[w][threadIdx.x]);
                if (DESLOC) sm = max(sm, smax_s[w][threadIdx.x]);
            }
            (q ? P.nrm[1] : P.nrm[0])[(size_t)g32 * nb + c0 / 32 + threadIdx.x] = DESLOC ? ((__float_as_uint(n) + 31u) & ~31u) | (uint32_t)sm : __float_as_uint(n);
        }
    }
}

// ------------------------------------------------------------------------------------------ the product
// A CTA works through 128 x TNv tiles of C (each optionally one K range of it); 16 drain warps, one warp that loads and two that multiply.  One CTA per
// SM, persistent: while the drain warps put a tile out, the next one's operands are already being loaded and multiplied.
//   TNv 128: a drain warp has 32 rows x 32 columns, tensor memory two stages of a chunk
//   TNv 64, block 32: 32 rows x 16 columns, four stages.  For products of up to 148 such tiles; where these leave SMs without work, the K ranges of
//           a tile go to a cluster of 2 to 8 CTAs (512 x 512 x 2048 raw: 14.3 -> 11.2 us).  (Two CTAs of 8 drain warps x 32 columns on an SM before:
//           with two warps to a scheduler a chunk took 600 cycles, its instructions' latencies one after the other, now 310: 2048 x 512 x 2048
//           with the sum 20.8 -> 17.7 us, 2048 x 512 x 4096 raw 44.9 -> 26.8, in one K range instead of two that add atomically.)
// What bounds a rounded chunk is the drain warps' instructions: the stage they want is nearly always there (a wait takes 76 cycles when it is, 100 on
// average).  128 wide, 4096 x 4096 x 4096: 138 instructions a warp and chunk, of which 64 add, 790 cycles -> 110, 650.  What it took: the look at the norms
// once per 16 chunks instead of a test in each, and their loads 16 chunks ahead (834 -> 783 us for 16384 x 4096 x 4096); the multiplying warps
// look at the ring before the stage, so that what they wait for last is what comes last (-> 741); warp numbers known to be uniform and the
// two stages' addresses by one bit (-> 706 -> 684).  Measured and not kept: 8 columns of both K-blocks on their way while 8 are added (1030: twice
// the loads and waits); 8 drain warps of 64 columns with up to 232 registers, loads of 32 columns, the whole stage in registers at once or in halves
// (875 to 905: two warps to a scheduler); 16 warps with 112 registers and loads of 32 columns (835); a look at the next stage before the additions (750).
template <int TNv, int BLK>
struct CfgH {
    static constexpr int N_DW = 16, N_EPI = N_DW * 32;
    static constexpr int COLS = TNv / (N_DW / 4);                           // accumulator columns of a drain thread: 32 or 16
    static constexpr int G = BLK == 32 ? 2 : 1;                             // K-blocks handed over together
    static constexpr int NS = 512 / (G * TNv);                       // tensor-memory stages of G x TNv columns
    static constexpr int N_THR = N_EPI + 32 + 32 * N_MW;          // multiplying warps: each takes every N_MW-th stage
    static_assert(NS >= N_MW && (COLS == 32 || COLS == 16), "");
    static constexpr uint32_t B_BYTES = TNv * 128, STAGE_BYTES = A_BYTES + B_BYTES;
    // the staged accumulators have memory of their own: the loads of the next tile go on meanwhile
    static constexpr uint32_t ACC_BYTES = TM * (TNv + 4) * 4, OFF_ACC = NST * STAGE_BYTES;
    static constexpr uint32_t OFF_RA = OFF_ACC + ACC_BYTES, OFF_RB = OFF_RA + TM * 4, OFF_RBF = OFF_RB + TNv * 4,
                              OFF_RBM = OFF_RBF + TNv * 4;
    static constexpr uint32_t OFF_BAR = OFF_RBM + 32, OFF_MISC = OFF_BAR + (2 * NST + 2 * NS + 1) * 8;
    static constexpr uint32_t SMEM_BYTES = OFF_MISC + 16 + (TNv == 128 && BLK == 32 ? N_PLANOS : 0) + 1024;            // + slack to align the base to 1024 bytes
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of a CTA");
    static_assert(OFF_BAR % 16 == 0, "the drain warps turn from one stage's barrier to the other's by a bit of the address");
    // instruction descriptor kind::f16: D = f32, A = B = f16, both K-major, N = TNv, M = 128
    static constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(TNv >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
};
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acumula) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "r"(acumula) : "memory");
}
// 16 consecutive columns of this lane, asynchronous: the registers may be used after tmem_pronto on them
__device__ __forceinline__ void tmem_pede(uint32_t t, uint32_t (&d)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];" : JT_O16(d, 0) : "r"(t) : "memory");
}
#define JT_IO4(a, i) "+r"(a[i]), "+r"(a[i + 1]), "+r"(a[i + 2]), "+r"(a[i + 3])
#define JT_IO16(a, i) JT_IO4(a, i), JT_IO4(a, i + 4), JT_IO4(a, i + 8), JT_IO4(a, i + 12)
__device__ __forceinline__ void tmem_pronto(uint32_t (&a)[16]) { asm volatile("tcgen05.wait::ld.sync.aligned;" : JT_IO16(a, 0)::"memory"); }
// two fp32 additions in one instruction: r + 1.5 * 2^23, the rounding of the specification
__device__ __forceinline__ void soma_magia(uint32_t& a, uint32_t& b) {
    asm volatile("{\n .reg .b64 t;\n mov.b64 t, {%0, %1};\n add.rn.f32x2 t, t, %2;\n mov.b64 {%0, %1}, t;\n}" : "+r"(a), "+r"(b) : "l"(par(MAGIA, MAGIA)));
}
// acc += a + b in one three-input addition of the integer pipe.  (volatile: left to itself the compiler turns such sums into pairs of
// multiply-adds on the floating-point pipe, which the packed additions already fill)
__device__ __forceinline__ void soma3(int& acc, uint32_t a, uint32_t b) {
    asm volatile("add.s32 %0, %0, %1;\n add.s32 %0, %0, %2;" : "+r"(acc) : "r"(a), "r"(b));
}
// NV columns of two K-blocks onto the accumulators acc[o ...]
template <int NV, int NA>
__device__ __forceinline__ void junta_lote(uint32_t (&a)[NV], uint32_t (&b)[NV], int (&acc)[NA], int o) {
#pragma unroll
    for (int k = 0; k < NV; k += 2) {
        soma_magia(a[k], a[k + 1]);
        soma_magia(b[k], b[k + 1]);
        soma3(acc[o + k], a[k], b[k]);
        soma3(acc[o + k + 1], a[k + 1], b[k + 1]);
    }
}
// the same by conversion, exact for every value (K-blocks whose norm product reaches 2^36)
template <int NV, int NA>
__device__ __forceinline__ void converte_lote(const uint32_t (&a)[NV], const uint32_t (&b)[NV], int (&acc)[NA], int o) {
#pragma unroll
    for (int k = 0; k < NV; k++)
        acc[o + k] += __float2int_rn(__uint_as_float(a[k])) + __float2int_rn(__uint_as_float(b[k])) + (int)(2 * MAGIA);
}

__device__ __forceinline__ void grupo_barreira() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes at the same place of another block of the cluster
__device__ __forceinline__ int4 le_vizinho(uint32_t end, int bloco) {
    int4 v;
    asm volatile("{\n .reg .b32 t;\n mapa.shared::cluster.u32 t, %4, %5;\n ld.shared::cluster.v4.s32 {%0, %1, %2, %3}, [t];\n}"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(end), "r"(bloco) : "memory");
    return v;
}

template <bool B> struct Logico { static constexpr bool v = B; };
// a barrier of the first and last warps (not the loading one) that tells each whether any thread said yes
template <int N>
__device__ __forceinline__ bool barreira_ou(bool sim) {
    uint32_t r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred q, 2, %2, p;\n selp.u32 %0, 1, 0, q;\n}" : "=r"(r) : "r"((uint32_t)sim), "n"(N) : "memory");
    return r != 0;
}

// SOMA: tiles in which nothing is rounded add up in tensor memory (128-wide tiles of block 32; 64-wide ones, one tile to an SM, were not tried with
// it, and block 128 drains every four MMAs as it is).  The loops with and without sums are both in the kernel: with the second drain in
// them the loops that round come out up to 5 % slower.
template <int BLK, int MODO, int TNv, bool GRUPO, bool SOMA>
__global__ void __launch_bounds__(CfgH<TNv, BLK>::N_THR, 1) k_gemm_h(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                                                       const int8_t* __restrict__ RA, const int8_t* __restrict__ RB, const uint32_t* __restrict__ nA,
                                                       const uint32_t* __restrict__ nB, SaidaGemm S, int M, int N, int K, Grade Gr, int kid) {
    using C_ = CfgH<TNv, BLK>;
    constexpr int NS = C_::NS, COLS = C_::COLS, LV = 16, N_EPI = C_::N_EPI, N_DW = C_::N_DW;
    constexpr int CB = BLK == 32 ? 1 : 2;                                   // chunks per tensor-memory stage: two K-blocks of 32, or one of 128
    static_assert(!SOMA || (TNv == 128 && BLK == 32 && !GRUPO), "");
    extern __shared__ unsigned char smem_bruto[];
    unsigned char* smem = smem_bruto + ((1024u - (smem_u32(smem_bruto) & 1023u)) & 1023u);      // stays in the shared address space
    const uint32_t sbase = smem_u32(smem);
    int* acc_s = reinterpret_cast<int*>(smem + C_::OFF_ACC);
    int* RAs = reinterpret_cast<int*>(smem + C_::OFF_RA);
    int* RBs = reinterpret_cast<int*>(smem + C_::OFF_RB);
    float* RBf = reinterpret_cast<float*>(smem + C_::OFF_RBF);
    int* RBm = reinterpret_cast<int*>(smem + C_::OFF_RBM);
    const uint32_t bar_full = sbase + C_::OFF_BAR, bar_empty = bar_full + NST * 8, bar_tfull = bar_empty + NST * 8, bar_tempty = bar_tfull + NS * 8, bar_encontro = bar_tempty + NS * 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C_::OFF_MISC);
    volatile int* aborta = reinterpret_cast<volatile int*>(smem + C_::OFF_MISC + 4);
    unsigned char* planos = smem + C_::OFF_MISC + 16;
    const int tid = threadIdx.x, wid = __shfl_sync(FULL, tid >> 5, 0), lane = tid & 31;
    const int ntiles = Gr.nx * Gr.ny * Gr.partes, npedT = (K + KH - 1) / KH;
    // the tiles of this block: in a cluster the K ranges lie next to each other
    const Percurso Pc = {GRUPO ? (int)blockIdx.x / Gr.partes + (int)blockIdx.x % Gr.partes * (Gr.nx * Gr.ny) : (int)blockIdx.x, GRUPO ? ntiles : (int)gridDim.x, ntiles, npedT};

    if (tid == 0) {
        for (int i = 0; i < NST; i++) { mbar_init(bar_full + 8 * i, 1); mbar_init(bar_empty + 8 * i, 1); }
        for (int i = 0; i < NS; i++) { mbar_init(bar_tfull + 8 * i, 1); mbar_init(bar_tempty + 8 * i, N_DW); }
        mbar_init(bar_encontro, N_MW);
        *aborta = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (wid == N_DW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_antes();
    __syncthreads();
    tc_fence_depois();
    const uint32_t tmem = *tmem_slot;
    pdl_espera();                                  // everything above touches no global memory: it overlaps the predecessor's tail
    pdl_solta();

    // The plans of this block's tiles: how many chunks of K add up in tensor memory before a drain; 0: every K-block is drained and rounded.  Chunks
    // can add up where none of their products is rounded (shift <= 4) and their sums stay below 2^24 last places of the finest product,
    // 2^(4 - largest shift), by Cauchy-Schwarz for the whole tile.  A tile that fails anywhere is rounded throughout.  The drain warps make all
    // of them, a tile each at a time, while the first operands are on their way; a block without a tile that adds up takes the loops
    // without sums.  (Made by the loading warp tile by tile and waited for by everyone, they cost a tile up to 1000 cycles.  With the rounding loops of that
    // time, 138 instructions a chunk, and exponents that round: no sums at all / plans tile by tile / made here 75.6 / 79.2 / 74.6 us for 16384 x 1024 x 1024, 213 / 227 / 209 for
    // 16384 x 4096 x 512 with the sum, 289 / 305 / 293 for 16384 x 4096 x 1024 with ReLU^2.  With exponents that do not: 77 / 55 / 50.5, 214 / 143 / 137, 290 / 187 / 168.)
    bool somas = false;
    if (SOMA && wid != N_DW) {
        const int nb = K / 32, gA = (M + 31) / 32;
        for (int nt = wid, tile = Pc.tile0 + wid * Pc.passo; wid < N_DW && tile < ntiles; nt += N_DW, tile += N_DW * Pc.passo) {
            const int n0 = tile % Gr.nx * TNv, m0 = tile / Gr.nx * TM;       // (one K range, of at most 32 K-blocks: a lane each)
            uint32_t sa = 0, sb = 0;
            float ma = 0.f, mb = 0.f;
#pragma unroll
            for (int g = 0; g < 4; g++) {
                const uint32_t a = lane < nb ? nA[(size_t)min(m0 / 32 + g, gA - 1) * nb + lane] : 0u, b = lane < nb ? nB[(size_t)(n0 / 32 + g) * nb + lane] : 0u;
                sa = max(sa, a & 31u); ma = fmaxf(ma, __uint_as_float(a));
                sb = max(sb, b & 31u); mb = fmaxf(mb, __uint_as_float(b));
            }
            int sh = ma > 0.f && mb > 0.f ? (int)(sa + sb) : 0, junta = 0;
            float lim = sqrtf(ma) * sqrtf(mb) * 1.0001f;                     // of what the K-block adds to any sum, 2^-4
#pragma unroll
            for (int k = 0; k < 5; k++) {                                    // all aligned groups of 2^k chunks, from 2 on (single ones: the drain as it is)
                sh = max(sh, __shfl_xor_sync(FULL, sh, 1 << k));
                lim += __shfl_xor_sync(FULL, lim, 1 << k);
                if (!__all_sync(FULL, sh <= GG && lim * pot2(min(sh, GG)) < LIM_SOMA)) break;
                if (k) junta = 1 << k;
            }
            if (lane == 0) planos[nt] = (unsigned char)junta;
            somas |= junta != 0;
        }
        somas = barreira_ou<(N_DW + N_MW) * 32>(somas);
    }

    // The loading and the multiplying warps run their loops as whole warps, with one elected lane for the asynchronous instructions: the
    // addresses and descriptors then live in uniform registers.  They share their schedulers with busy drain warps, so what counts
    // is how few instructions a chunk takes them (with one lane in a divergent branch the multiplying warp took 680 cycles a chunk and
    // bounded the kernel).
    if (wid == N_DW) {
        // ------------------------------------------------------------------ loads
        struct {
            const CUtensorMap *mapA, *mapB;
            volatile int* aborta;
            Grade Gr;
            uint32_t sbase, bar_full, bar_empty;
            int kid;
            bool eleito;
            int n0, m0;                                                      // of the tile that is being loaded
            __device__ __forceinline__ bool vazio(int s, uint32_t fase) { return __all_sync(FULL, espera(bar_empty + 8 * s, fase, aborta, kid, 1)); }
            __device__ __forceinline__ void tile(int tile) { n0 = tile % Gr.nx * TNv; m0 = tile / Gr.nx % Gr.ny * TM; }
            __device__ __forceinline__ void carrega(int s, int c) {
                if (eleito) {
                    mbar_expect_tx(bar_full + 8 * s, C_::STAGE_BYTES);
                    tma_2d(sbase + s * C_::STAGE_BYTES, mapA, c * KH, m0, bar_full + 8 * s);
                    tma_2d(sbase + s * C_::STAGE_BYTES + A_BYTES, mapB, c * KH, n0, bar_full + 8 * s);
                }
            }
        } v = {&mapA, &mapB, aborta, Gr, sbase, bar_full, bar_empty, kid, elege()};
        if (*reinterpret_cast<volatile int*>(&g_sem_cargas) == 0) laco_cargas(v, Gr, Pc);
    } else if (wid > N_DW) {
        // ------------------------------------------------------------------ MMAs
        struct {
            volatile int* aborta;
            const unsigned char* planos;
            uint32_t tmem, bar_full, bar_empty, bar_tfull, bar_tempty, bar_encontro;
            uint64_t da0, db0;
            int kid;
            bool eleito;
            __device__ __forceinline__ void tile(int) {}
            __device__ __forceinline__ int plano(uint32_t nt) { return planos[nt]; }
            __device__ __forceinline__ bool encontra(uint32_t fase) {
                __syncwarp();
                if (eleito) mbar_arrive(bar_encontro);
                return __all_sync(FULL, espera(bar_encontro, fase, aborta, kid, 8));
            }
            __device__ __forceinline__ bool livre(int t, uint32_t fase) { return __all_sync(FULL, espera(bar_tempty + 8 * t, fase, aborta, kid, 3)); }
            __device__ __forceinline__ bool cheio(int s, uint32_t fase) {
                return __all_sync(FULL, espera(bar_full + 8 * s, fase, aborta, kid, 2));
            }
            __device__ __forceinline__ void arredonda(int s, int t, int j, bool certo, int) {
                tc_fence_depois();
                const uint64_t da = da0 + (uint32_t)(s * (C_::STAGE_BYTES >> 4)), db = db0 + (uint32_t)(s * (C_::STAGE_BYTES >> 4));
                const uint32_t d = tmem + t * (C_::G * TNv);
                if (!(eleito && certo)) return;
                if (BLK == 32) {
                    mma_f16(d, da, db, C_::IDESC, 0);                       // +32 bytes (16 elements of K) per instruction
                    mma_f16(d, da + 2, db + 2, C_::IDESC, 1);
                    mma_f16(d + TNv, da + 4, db + 4, C_::IDESC, 0);
                    mma_f16(d + TNv, da + 6, db + 6, C_::IDESC, 1);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++) mma_f16(d, da + 2 * q, db + 2 * q, C_::IDESC, j | q);
                }
                if (j == CB - 1) tc_commit(bar_tfull + 8 * t);
                tc_commit(bar_empty + 8 * s);
            }
            __device__ __forceinline__ void soma(int s, int t, int i, bool fim, bool certo, int) {
                tc_fence_depois();
                const uint64_t da = da0 + (uint32_t)(s * (C_::STAGE_BYTES >> 4)), db = db0 + (uint32_t)(s * (C_::STAGE_BYTES >> 4));
                const uint32_t d = tmem + t * (C_::G * TNv);
                if (!(eleito && certo)) return;
#pragma unroll
                for (int q = 0; q < 4; q++) mma_f16(d, da + 2 * q, db + 2 * q, C_::IDESC, i | q);
                if (fim) tc_commit(bar_tfull + 8 * t);
                tc_commit(bar_empty + 8 * s);
            }
        } v = {aborta, planos, tmem, bar_full, bar_empty, bar_tfull, bar_tempty, bar_encontro, desc_sw128(sbase), desc_sw128(sbase + A_BYTES), kid, elege()};
        if (SOMA && somas) laco_produtos<true, NS, CB>(v, Gr, Pc, wid - N_DW - 1);
        else laco_produtos<false, NS, CB>(v, Gr, Pc, wid - N_DW - 1);
    } else {
        // ------------------------------------------------------------------ drain + output stage
        const int quarto = wid & 3, cg = wid >> 2, lin = quarto * 32 + lane;
        const uint32_t base = tmem + ((uint32_t)(quarto * 32) << 16) + cg * COLS;
        auto drena = [&](auto misto) {
            constexpr bool MISTO = decltype(misto)::v;
            // the stage at hand: its columns, its barrier, the drains before it
            uint32_t ta = base, bt = bar_tfull, n_t = 0, nt = 0;
            // waits for the next stage (a wait that gives up makes all later ones return at once) / hands it back, its contents in registers
            auto recebe = [&]() {
                espera(bt, n_t / NS & 1, aborta, kid, 4);
                __syncwarp();
                tc_fence_depois();
            };
            auto devolve = [&]() {
                tc_fence_antes();
                __syncwarp();
                if (lane == 0) mbar_arrive(bt + (bar_tempty - bar_tfull));
                n_t++;
                if constexpr (NS == 2) {
                    ta ^= C_::G * TNv;
                    bt ^= 8;
                } else {
                    ta = base + n_t % NS * (C_::G * TNv);
                    bt = bar_tfull + n_t % NS * 8;
                }
            };
            // The next tile.  With the bounds in registers from above, or a signed step, the loop of raw products came out 3 % slower (4096 x 1024 x 16384
            // 268 -> 278 us, now 235); where there are sums it was the other way round (16384 x 4096 x 512 209 us against 213, now 196).
            auto seguinte = [&](int tile) -> int {
                if constexpr (SOMA) return tile + Pc.passo;
                else return (int)((uint32_t)tile + (GRUPO ? (uint32_t)ntiles : gridDim.x));
            };
            for (int tile = GRUPO || SOMA ? Pc.tile0 : (int)blockIdx.x; tile < ntiles; tile = seguinte(tile), nt++) {
                const int n0 = tile % Gr.nx * TNv, m0 = tile / Gr.nx % Gr.ny * TM, parte = tile / (Gr.nx * Gr.ny), ped0 = parte * Gr.ppp;
                const int nped = GRUPO ? max(min(Gr.ppp, npedT - ped0), 0) : min(Gr.ppp, npedT - ped0);
                // the row maxima, wanted by the output stage: read now, stored to shared memory after the main loop
                int ra = 0, rb = 0;
                if (tid < TM) ra = m0 + tid < M ? (int)RA[m0 + tid] : 0;
                if (tid < TNv) rb = RB[n0 + tid];
                constexpr int PITCHv = TNv + 4;
                // what the output stage needs goes to shared memory
                auto tabelas = [&]() {
                    if (!GRUPO && tile != (int)blockIdx.x) asm volatile("bar.sync 1, %0;" ::"n"(N_EPI) : "memory");      // the previous tile is out
                    if (tid < TM) RAs[tid] = ra;
                    if (tid < TNv) {
                        RBs[tid] = rb;
                        if (MODO != 1) {
                            // what the fp32 path of the output stage needs: each block's extreme column exponents and the column scales
                            int mn = __reduce_min_sync(FULL, rb), mx = __reduce_max_sync(FULL, rb);
                            if (lane == 0) { RBm[wid] = mn; RBm[4 + wid] = mx; }
                            if (BLK > 32) {                                          // one block over the four warps: place 0 gets its extremes
                                asm volatile("bar.sync 3, %0;" ::"n"(TNv) : "memory");
                                mn = min(min(RBm[0], RBm[1]), min(RBm[2], RBm[3]));
                                mx = max(max(RBm[4], RBm[5]), max(RBm[6], RBm[7]));
                                if (tid == 0) { RBm[0] = mn; RBm[4] = mx; }
                            }
                            RBf[tid] = pot2(min(rb - mn, 100));
                        }
                    }
                };
                const int junta = MISTO ? planos[nt] : 0;
                if (MISTO && junta) {
                    // Sums of whole numbers, straight to shared memory (and added there where a tile has several): with accumulators in registers
                    // this way in and the rounding one out of the loops share them, which costs the rounding loop 5 %.
                    tabelas();
                    for (int u = 0; u < nped / CB; u += junta) {
                        recebe();
                        const uint32_t te = ta;
#pragma unroll
                        for (int o = 0; o < COLS; o += LV) {
                            uint32_t a[LV], v[LV], fora = 0;
                            tmem_pede(te + o, a);
                            tmem_pronto(a);
                            if (o + LV == COLS) devolve();
                            // (the exponent field of every sum with the constant must be that of 1.5 * 2^23, else the warp converts)
#pragma unroll
                            for (int k = 0; k < LV; k += 2) {
                                v[k] = a[k]; v[k + 1] = a[k + 1];
                                soma_magia(v[k], v[k + 1]);
                                fora |= (v[k] ^ MAGIA) | (v[k + 1] ^ MAGIA);
                                v[k] -= MAGIA; v[k + 1] -= MAGIA;
                            }
                            if (__any_sync(FULL, (fora & 0xFF800000u) != 0)) {
#pragma unroll
                                for (int k = 0; k < LV; k++) v[k] = (uint32_t)__float2int_rn(__uint_as_float(a[k]));
                            }
                            uint4* d = reinterpret_cast<uint4*>(acc_s + lin * PITCHv + cg * COLS + o);
#pragma unroll
                            for (int k = 0; k < LV / 4; k++) {
                                uint4 w = make_uint4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                                if (u) { const uint4 z = d[k]; w.x += z.x; w.y += z.y; w.z += z.z; w.w += z.w; }
                                d[k] = w;
                            }
                        }
                    }
                } else {
                    int acc[COLS];
#pragma unroll
                    for (int j = 0; j < COLS; j++) acc[j] = 0;
                    if constexpr (BLK == 32) {
                        // the largest squared norms of this warp's 32 rows of A and of its columns' 32 of B, a lane per K-block, 16 chunks at a time
                        const int nb = K / 32, fb = min(nb, (ped0 + nped) * 2);
                        const uint32_t *pA = nA + (size_t)min(m0 / 32 + quarto, (M + 31) / 32 - 1) * nb, *pB = nB + (size_t)((n0 + cg * COLS) / 32) * nb;
                        float na = 0.f, nbm = 0.f;
                        auto normas = [&](int c0) {
                            const int f = (ped0 + c0) * 2 + lane;
                            na = nbm = 0.f;
                            if (f < fb) { na = __uint_as_float(pA[f]); nbm = __uint_as_float(pB[f]); }
                        };
                        normas(0);
                        for (int c0 = 0; c0 < nped; c0 += 16) {
                            unsigned suspeitos = __ballot_sync(FULL, na * nbm >= LIM_NORMA);      // bits 2 c, 2 c + 1: the K-blocks of chunk c may leave the exact window
                            const int cf = min(nped - c0, 16);
                            normas(c0 + 16);                                     // (on their way while these chunks are added: waited for here they cost 500 cycles)
                            if (suspeitos == 0) {
#pragma unroll 1
                                for (int c = 0; c < cf; c++) {
                                    recebe();
                                    const uint32_t te = ta;
#pragma unroll
                                    for (int o = 0; o < COLS; o += LV) {
                                        uint32_t a[LV], b[LV];
                                        tmem_pede(te + o, a);
                                        tmem_pede(te + TNv + o, b);
                                        tmem_pronto(a);
                                        tmem_pronto(b);
                                        if (o + LV == COLS) devolve();
                                        junta_lote(a, b, acc, o);
                                    }
                                }
                            } else {
#pragma unroll 1
                                for (int c = 0; c < cf; c++, suspeitos >>= 2) {
                                    recebe();
                                    const uint32_t te = ta;
                                    const bool certo = (suspeitos & 3u) == 0;
#pragma unroll
                                    for (int o = 0; o < COLS; o += LV) {
                                        uint32_t a[LV], b[LV];
                                        tmem_pede(te + o, a);
                                        tmem_pede(te + TNv + o, b);
                                        tmem_pronto(a);
                                        tmem_pronto(b);
                                        if (o + LV == COLS) devolve();
                                        if (certo) junta_lote(a, b, acc, o);
                                        else converte_lote(a, b, acc, o);
                                    }
                                }
                            }
                        }
                    } else {
                        for (int c = 0; c < nped / 2; c++) {
                            recebe();
                            const uint32_t te = ta;
#pragma unroll
                            for (int o = 0; o < COLS; o += LV) {
                                uint32_t a[LV], x[LV], fora = 0;
                                tmem_pede(te + o, a);
                                tmem_pronto(a);
                                if (o + LV == COLS) devolve();
                                // (the exponent field of every sum must be that of 1.5 * 2^23)
#pragma unroll
                                for (int k = 0; k < LV; k += 2) {
                                    x[k] = a[k]; x[k + 1] = a[k + 1];
                                    soma_magia(x[k], x[k + 1]);
                                    fora |= (x[k] ^ MAGIA) | (x[k + 1] ^ MAGIA);
                                }
                                if (__any_sync(FULL, (fora & 0xFF800000u) != 0)) {
#pragma unroll
                                    for (int k = 0; k < LV; k++) x[k] = (uint32_t)__float2int_rn(__uint_as_float(a[k])) + MAGIA;
                                }
#pragma unroll
                                for (int k = 0; k < LV; k++) acc[o + k] += (int)x[k];
                            }
                        }
                    }
                    const uint32_t vies = (uint32_t)(BLK == 32 ? nped * 2 : nped / 2) * MAGIA;
                    tabelas();
#pragma unroll
                    for (int j = 0; j < COLS; j += 4)
                        *reinterpret_cast<int4*>(acc_s + lin * PITCHv + cg * COLS + j) =
                            make_int4((int)((uint32_t)acc[j] - vies), (int)((uint32_t)acc[j + 1] - vies), (int)((uint32_t)acc[j + 2] - vies), (int)((uint32_t)acc[j + 3] - vies));
                }
                asm volatile("bar.sync 1, %0;" ::"n"(N_EPI) : "memory");
                if constexpr (!GRUPO) epilogo_tile<BLK, MODO, N_EPI, TNv>(acc_s, RAs, RBs, min(TM, M - m0), m0, n0, N, S, Gr.partes > 1, parte == 0, kid, tid, RBf, RBm);
                else {
                    grupo_barreira();                                            // every block's accumulators are there
                    const int lr = TM / Gr.partes, r0 = parte * lr;              // the rows this block puts out
                    for (int t = tid; t < lr * (TNv / 4); t += N_EPI) {
                        const int o = (r0 + t / (TNv / 4)) * PITCHv + t % (TNv / 4) * 4;
                        int4 v = *reinterpret_cast<const int4*>(acc_s + o);
                        for (int k = 1; k < Gr.partes; k++) {
                            const int4 x = le_vizinho(smem_u32(acc_s + o), (parte + k) % Gr.partes);
                            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
                        }
                        *reinterpret_cast<int4*>(acc_s + o) = v;                 // (only this block reads these rows of its own)
                    }
                    asm volatile("bar.sync 1, %0;" ::"n"(N_EPI) : "memory");
                    epilogo_tile<BLK, MODO, N_EPI, TNv>(acc_s + r0 * PITCHv, RAs + r0, RBs, min(lr, max(M - m0 - r0, 0)), m0 + r0, n0, N, S, false, true, kid, tid, RBf, RBm);
                }
            }
        };
        if (SOMA && somas) drena(Logico<SOMA>{});
        else drena(Logico<false>{});
    }
    if constexpr (GRUPO) {
        __syncwarp();
        if (wid >= N_DW) grupo_barreira();
        grupo_barreira();                                                    // nobody leaves while another reads its accumulators
    }
    tc_fence_antes();
    __syncthreads();
    if (wid == N_DW) {
        tc_fence_depois();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
    }
}

}  // namespace th
}  // namespace jt
