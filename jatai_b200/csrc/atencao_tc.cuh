// Integer causal attention with ALiBi on the tensor cores, head dimension 64, 16 or 4, every T that is a multiple of 32.
//
// Same specification and layouts as atencao.cuh (jatai_cuda/ops.py:186-258 generalised; jatai_cuda/jatai_cuda.cu:822-1006).  Every one of
// the six contractions - q.k^T, P.V, dO.v^T, dS'.k, dS'^T.q, P^T.dO - is an exact integer sum followed by ONE rounding, so (unlike the
// block GEMM) a whole contraction can accumulate in tensor memory.
//   * Scores and gP = dO.v^T: aligned operands have |a| <= 2032, which f16 holds exactly; the other side is split in two signed 6-bit
//     digits, b = 64 hi + lo, so that each of the two fp32 accumulators (kind::f16) is an exact integer below 2^22 (64 x 2032 x 32).
//   * The others take the token axis as K and reach further than 24 bits: two signed 8-bit digits v = 128 hi + lo (lo in [-64, 63]) on
//     kind::i8, hi.hi / hi.lo + lo.hi / lo.lo recombined with shifts (the final int32 wraps exactly like the specification's
//     int64 -> int32 truncation); P is uint8 and enters as it is.
//
// A preparation kernel aligns q, k, v (and dO) of every head to the head's maximum exponent once and writes what the MMAs read (all
// K-major, rows of 128 bytes, TMA with the 128-byte swizzle):
//     plain          [BH*T][64] f16                      token rows
//     digits         [2][BH*T][64] f16                   token rows of the hi digits, then of the lo digits
//     transposed     [BH*128][T] int8                    row = one digit of one column (hi rows 0..63, lo rows 64..127), over the tokens
// A head of 16 columns fills 16 of the 64 (and of each 64 digit rows); the rest is neither written nor multiplied into a result.  A head of 4
// has zeros behind it in the token rows, up to the 16 columns of one MMA.
//
// A query tile of 64 rows takes its keys in windows of 128 that end with the tile's last query and go back from there.  With the
// reference's slopes P is exactly zero a few dozen keys behind the diagonal, so one window is nearly always all there is: the forward
// works out after the first window how many it needs, the backward reads a map of the non-zero parts of P.  The one-window case keeps
// everything in registers between the passes (scores, exponentials, P); with more windows each pass computes the scores again.
// Between load, MMA and drain a block has little to overlap, so the overlap comes from three blocks per SM (k_ab_max: four).
//
// Orientation of every score-like product of a query tile: tensor-memory lane = key (M = 128 keys of a window), column = query; a
// thread of the drain owns one key and 32 queries.  Stored P is key-major, so that thread reads or writes 32 contiguous bytes of P.
// Products whose output is [token, column] are computed transposed: lane = digit row of the columns (hi rows 0..63, lo rows
// 64..127), column = token, and recombined through shared memory.
//
// Every mbarrier wait is bounded (sentinel 7, abort flag, normal exit with tensor memory freed), as in the block GEMM.
#pragma once
#include <cooperative_groups.h>
#include "comum.cuh"
#include "gemm_tc.cuh"
#include "gemm_h.cuh"
#include "atencao.cuh"

namespace jt {
namespace atc {

using namespace tc;

constexpr int NI = 64, TJ = 128;         // queries (or keys) of a tile, keys (or queries) of a window
constexpr int NTA = 256;                 // threads: 4 lane quarters x 2 halves of 32 columns
constexpr int SB = 2 * NI;               // columns of a score buffer in tensor memory: hi | lo
constexpr int GY = 65535;                // limit of a grid's y: heads beyond go to further launches (y0 = the first head of one)
constexpr uint32_t idesc(int n, bool b_sem_sinal) {       // kind::i8, D = s32, A = s8, B = s8 or u8, both K-major, M = 128
    return (2u << 4) | (1u << 7) | ((b_sem_sinal ? 0u : 1u) << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
constexpr uint32_t ID_S = idesc(SB, false), ID_PU = idesc(NI, true);
constexpr uint32_t ID_F16 = (1u << 4) | ((uint32_t)(SB >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);      // kind::f16, D = f32, N = 128, M = 128
constexpr uint32_t ID_F16N = (1u << 4) | ((uint32_t)(NI >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);     // the same with N = 64
constexpr uint32_t TILE_A = 128 * 128, TILE_N = NI * 128;

__device__ __forceinline__ void digitos(int v, int& hi, int& lo) {
    hi = (v + 64) >> 7;
    lo = v - (hi << 7);
}
// byte offset of (row, byte) inside a K-major tile of 128-byte rows with the 128-byte swizzle (8-row groups of 1024 bytes)
__device__ __forceinline__ uint32_t sw128(int linha, int byte) {
    return (uint32_t)((linha >> 3) * 1024 + (linha & 7) * 128 + ((((byte >> 4) ^ (linha & 7)) << 4) | (byte & 15)));
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_aloca(uint32_t* slot, int colunas) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(colunas) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_libera(uint32_t tmem, int colunas) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(colunas) : "memory");
}
// The MMAs of one score-like product, hd columns.  A = 128 token rows (plain), B = the 64 token rows of the hi digits and the 64 of the lo
// digits; or, digits on the A side, two products with the 64 token rows of B (plain).
__device__ __forceinline__ void mma_escores(uint32_t tm, uint64_t da, uint64_t db, int hd) {
    for (int q = 0; q < (hd + 15) / 16; q++) th::mma_f16(tm, da + 2 * q, db + 2 * q, ID_F16, q != 0);
}
__device__ __forceinline__ void mma_escores_a(uint32_t tm, uint64_t dah, uint64_t dal, uint64_t db, int hd) {
    for (int q = 0; q < (hd + 15) / 16; q++) {
        th::mma_f16(tm, dah + 2 * q, db + 2 * q, ID_F16N, q != 0);
        th::mma_f16(tm + NI, dal + 2 * q, db + 2 * q, ID_F16N, q != 0);
    }
}
// 16 scores of this lane from the two accumulators (hi at t, lo 64 columns on): 64 hi + lo, through the bit patterns of hi + 1.5 * 2^23 and
// lo + 1.5 * 2^23
__device__ __forceinline__ void escores16_cru(uint32_t t, uint32_t (&h)[16], uint32_t (&l)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : JT_O16(h, 0), JT_O16(l, 0)
        : "r"(t), "r"(t + NI)
        : "memory");
}
__device__ __forceinline__ void escores16(uint32_t t, int (&x)[16]) {
    uint32_t h[16], l[16];
    escores16_cru(t, h, l);
#pragma unroll
    for (int k = 0; k < 16; k += 2) {
        th::soma_magia(h[k], h[k + 1]);
        th::soma_magia(l[k], l[k + 1]);
        x[k] = (int)((h[k] << 6) + (l[k] - 65u * MAGIA));
        x[k + 1] = (int)((h[k + 1] << 6) + (l[k + 1] - 65u * MAGIA));
    }
}
// CTA-wide maximum of a non-negative per-thread value -> one atomicMax
__device__ __forceinline__ void max_cta(int v, int* destino, int* red, int tid) {
    v = __reduce_max_sync(FULL, v);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
        int r = red[0];
#pragma unroll
        for (int i = 1; i < NTA / 32; i++) r = max(r, red[i]);
        if (r > 0) atomicMax(destino, r);
    }
}
__device__ __forceinline__ int junta3(uint32_t hh, uint32_t cr, uint32_t ll) { return (int)((hh << 14) + (cr << 7) + ll); }

// Output of 8 consecutive columns of one row (the 4 lanes tid & 3 = 0..3 hold the 32 columns of one exponent block, all with the
// exponent e): raw (int32 + int16 exponent per element), or - the caller asked for the quantised form and the block length is 32 -
// straight to a block tensor, i.e. jt_quant of the raw output (ops.py:125-126) without the round trip through memory.
// All 32 lanes of a warp call it together (the quantiser shuffles); `grava` = false computes and stores nothing.
__device__ __forceinline__ void grava8(int* acc, int16_t* ex, int8_t* qm, int8_t* qE, size_t p, size_t pe, const int (&o)[8], int e, int kid, int tid,
                                       bool grava = true) {
    if (qm) {
        int q[8];
        const int E = quant_uniforme<8, 4>(o, e, q, kid, (long long)p);
        if (!grava) return;
        *reinterpret_cast<uint2*>(qm + p) = make_uint2(junta4(q[0], q[1], q[2], q[3]), junta4(q[4], q[5], q[6], q[7]));
        if ((tid & 3) == 0) qE[pe] = (int8_t)E;
        return;
    }
    if (!grava) return;
    const uint32_t e2 = (uint32_t)(e & 0xffff) | ((uint32_t)e << 16);
    *reinterpret_cast<int4*>(acc + p) = make_int4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<int4*>(acc + p + 4) = make_int4(o[4], o[5], o[6], o[7]);
    *reinterpret_cast<uint4*>(ex + p) = make_uint4(e2, e2, e2, e2);
}

// -------------------------------------------------------------------------------------------------- preparation
// z = 0 q, 1 k, 2 v (columns of QKV), 3 dO.  Per tensor: the layouts wanted (nullptr = not), of the combinations that k_at_prep lists.
struct ArgsPrep {
    const int8_t* qm; const int8_t* qE; const int8_t* gm; const int8_t* gE;
    uint16_t* plano[4]; uint16_t* dig[4]; int8_t* tra[4];
    int* em;                    // [BH][4] head-maximum exponents, indexed by z
    int* est;                   // backward: the statistics slots [BH][N_EST] to clear (nullptr in the forward)
    int* nrm;                   // forward: [BH][2][ceil(T/128)] largest sum of squares of an aligned row of q (0) / k (1) per 128 tokens
    int BH, T, H, D, GA, blk;
    int y0;                     // first group of this launch
};
__device__ __forceinline__ uint32_t par_h(uint64_t x) {            // two floats that halves hold exactly
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(f_hi(x)), "f"(f_lo(x)));
    return r;
}

// grid (pieces of 128 tokens, sequences x groups of 64 / hd heads, 3 or 4), 256 threads: 128 tokens of 64 columns - one head of 64, four
// of 16 or sixteen of 4 - of one tensor.  The pieces of a sequence are a cluster (at most 8), which exchanges the maximum exponents: reading a
// sequence's exponents in every block was half of the traffic to the cache.  The bound of a plain version (one element at a time in integers, digit bytes stored one by
// one) was instruction issue, three times the memory time.  So: a thread takes 4 tokens x 8 columns; pairs of elements in f32x2 (a byte
// becomes a float by its place in 2^23's mantissa; v 2^(GA - s) rounds to even in one FMA against 1.5 * 2^23, exactly rnd_d; the 6-bit
// digits are hi = round(r / 64), lo = r - 64 hi); the transposed digits of 4 tokens are packed into a word and cross shared memory in
// 16-byte pieces swapped by the column group, without bank conflicts.
// 16 x 1024 tokens, forward + backward: 16 heads of 64 218 -> 175 us, 16 heads of 16 196 -> 57 us.
template <int hd, bool PLANO, bool DIG, bool TRA, bool NRM>
__device__ __forceinline__ void prep_corpo(const ArgsPrep& A, uint16_t* dp, uint16_t* dg, int8_t* dt, int* red, uint32_t* tr) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, z = blockIdx.z, hpc = 64 / hd, gh = (A.H + hpc - 1) / hpc;
    const unsigned grupo = blockIdx.y + A.y0;
    const int b = grupo / gh, h0 = grupo % gh * hpc;               // first head of the group
    const int T = A.T, D = A.D, blk = A.blk, linha0 = b * T;
    const int8_t* m = z == 3 ? A.gm : A.qm;
    const int8_t* E = z == 3 ? A.gE : A.qE;
    const int ld = z == 3 ? D : 3 * D, col0 = (z == 3 ? 0 : z * D) + h0 * hd, ldb = ld / blk;
    const int cg = tid & 7, tg = tid >> 3;                         // columns 8 cg .. + 7, tokens 4 tg .. + 3 of a piece
    constexpr int NH = hd < 8 ? 8 / hd : 1;                        // heads of this thread
    const int h = h0 + 8 * cg / hd, ch = 8 * cg % hd, bh = b * A.H + h;
    const bool ha = h < A.H;                                       // (H is a multiple of 2 where a thread has two heads: D is one of 32)
    const size_t BHT = (size_t)A.BH * T;
    const int peca = blockIdx.x, t0 = peca * 128;
    const bool dentro = t0 + 4 * tg < T;                           // (T is a multiple of 32)
    uint2 w[4];
    int ex[4], em;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const size_t lin = (size_t)(linha0 + t0 + 4 * tg + k);
        w[k] = make_uint2(0, 0);
        ex[k] = -128;
        if (dentro && ha) {
            w[k] = *reinterpret_cast<const uint2*>(m + lin * ld + col0 + 8 * cg);
            ex[k] = E[lin * ldb + (col0 + 8 * cg) / blk];
        }
    }
    {
        // maximum exponents of the two halves of 32 columns (a head of 16 lies in one of them, a head of 64 in both), over the sequence:
        // the blocks of the cluster have the other tokens
        const int meu = max(max(ex[0], ex[1]), max(ex[2], ex[3]));
        int e0 = __reduce_max_sync(FULL, cg < 4 ? meu : -128), e1 = __reduce_max_sync(FULL, cg < 4 ? -128 : meu);
        if (lane == 0) { red[wid] = e0; red[8 + wid] = e1; }
        __syncthreads();
        if (tid < 2) {
            int e = red[8 * tid];
#pragma unroll
            for (int i = 1; i < 8; i++) e = max(e, red[8 * tid + i]);
            red[16 + tid] = e;
        }
        const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        cl.sync();
        if (tid < 32) {
            const int* r = cl.map_shared_rank(red, lane < (int)gridDim.x ? lane : 0);
            e0 = __reduce_max_sync(FULL, r[16]);
            e1 = __reduce_max_sync(FULL, r[17]);
            if (lane == 0) { red[18] = e0; red[19] = e1; }
        }
        __syncthreads();
        // (nobody leaves before everyone has read: the second half of this barrier is at the end)
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
        e0 = red[18]; e1 = red[19];
        em = hd == 64 ? max(e0, e1) : cg < 4 ? e0 : e1;
    }
    if (blockIdx.x == 0 && ch == 0 && ha)
#pragma unroll
        for (int k = 0; k < NH; k++) {
            if (tid < 8) A.em[(bh + k) * 4 + z] = em;
            if (A.est && z == 3 && tg < at::N_EST) A.est[(bh + k) * at::N_EST + tg] = 0;
        }
    const uint64_t mag = par_f(MAGIA_F, MAGIA_F), menos_mag = par_f(-MAGIA_F, -MAGIA_F), vies = par_f(-8388736.0f, -8388736.0f);      // 2^23 + 128
    const uint64_t um64 = par_f(0.015625f, 0.015625f), m64 = par_f(-64.0f, -64.0f);
    float norma[NH] = {};
    uint32_t u[4][8];                                          // 2 r + 128: hi digit in byte 1, 2 (lo + 64) in byte 0
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float f1 = pot2(A.GA - min(em - ex[k], 40));     // |v 2^GA| < 2^11: 0 from a shift of 13 on
        const uint64_t f = par_f(f1, f1);
        uint32_t pl[4], dh[4], dl[4];
        float nk[NH] = {};
#pragma unroll
        for (int c = 0; c < 4; c++) {                          // two columns at a time
            const uint32_t x = (c < 2 ? w[k].x : w[k].y) ^ 0x80808080u;
            const uint64_t v = fadd2(par(__byte_perm(x, 0x4B000000u, 0x7540 + 2 * (c & 1)), __byte_perm(x, 0x4B000000u, 0x7540 + 2 * (c & 1) + 1)), vies);
            const uint64_t r = ffma2(v, f, mag), rf = fadd2(r, menos_mag);
            u[k][2 * c] = 2 * (uint32_t)r + (128u - 2 * MAGIA);
            u[k][2 * c + 1] = 2 * (uint32_t)(r >> 32) + (128u - 2 * MAGIA);
            if (PLANO) pl[c] = par_h(rf);
            if (DIG) {
                const uint64_t hi = fadd2(ffma2(rf, um64, mag), menos_mag);
                dh[c] = par_h(hi);
                dl[c] = par_h(ffma2(hi, m64, rf));
            }
            if (NRM) nk[c * NH / 4] = fmaf(f_lo(rf), f_lo(rf), fmaf(f_hi(rf), f_hi(rf), nk[c * NH / 4]));
        }
        if (dentro && ha) {
            // a head's 8 columns or, of heads of 4, two times 4 columns and 12 zeros
            auto poe = [&](uint16_t* d, const uint32_t (&x)[4]) {
#pragma unroll
                for (int n = 0; n < NH; n++) {
                    uint4* q = reinterpret_cast<uint4*>(d + ((size_t)(bh + n) * T + t0 + 4 * tg + k) * 64 + ch);
                    q[0] = NH == 1 ? make_uint4(x[0], x[1], x[2], x[3]) : make_uint4(x[2 * n], x[2 * n + 1], 0, 0);
                    if (NH > 1) q[1] = make_uint4(0, 0, 0, 0);
                }
            };
            if (PLANO) poe(dp, pl);
            if (DIG) {
                poe(dg, dh);
                poe(dg + BHT * 64, dl);
            }
        }
        if (NRM) {                                                 // squared norm of a head's row: its 8 or 2 lanes are neighbours
#pragma unroll
            for (int n = 0; n < NH; n++) {
                if (hd > 8) nk[n] += __shfl_xor_sync(FULL, nk[n], 1);
                if (hd == 64) {
                    nk[n] += __shfl_xor_sync(FULL, nk[n], 2);
                    nk[n] += __shfl_xor_sync(FULL, nk[n], 4);
                }
                norma[n] = fmaxf(norma[n], nk[n]);
            }
        }
    }
    if (NRM) {
        // the largest of the 128 tokens, rounded up by more than the error of 64 fp32 additions (it only bounds products)
#pragma unroll
        for (int n = 0; n < NH; n++) {
            norma[n] = fmaxf(norma[n], __shfl_xor_sync(FULL, norma[n], 8));
            norma[n] = fmaxf(norma[n], __shfl_xor_sync(FULL, norma[n], 16));
            if (lane < 8) red[32 + (8 * n + wid) * 8 + lane] = __float2int_ru(norma[n] * 1.00002f);
        }
        __syncthreads();
        if (tid < 8 && ch == 0 && ha)
#pragma unroll
            for (int n = 0; n < NH; n++) {
                int mx = 0;
                for (int k = 0; k < 8; k++) mx = max(mx, red[32 + (8 * n + k) * 8 + cg]);
                A.nrm[((size_t)(bh + n) * 2 + z) * ((T + 127) / 128) + peca] = mx;
            }
    }
    if (TRA) {
        if (ha)
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const uint32_t lo = __byte_perm(__byte_perm(u[0][c], u[1][c], 0x0040), __byte_perm(u[2][c], u[3][c], 0x0040), 0x5410) >> 1 ^ 0x40404040u;
                const int q = (8 * cg + c) * 32 + (tg ^ 4 * cg);
                tr[q] = __byte_perm(__byte_perm(u[0][c], u[1][c], 0x0051), __byte_perm(u[2][c], u[3][c], 0x0051), 0x5410);
                tr[64 * 32 + q] = lo | (lo & 0x40404040u) << 1;      // 7 bits to a signed byte
            }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int linha = (tid >> 3) + 32 * q, c = tid & 7, cv = linha & 63, hh = h0 + cv / hd;      // digit row, virtual column, its head
            if (hh < A.H && t0 + 16 * c < T)
                *reinterpret_cast<uint4*>(dt + ((size_t)(b * A.H + hh) * 128 + (linha & 64) + cv % hd) * T + t0 + 16 * c) =
                    *reinterpret_cast<const uint4*>(tr + linha * 32 + 4 * (c ^ (linha >> 3 & 7)));
        }
    }
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}
template <int hd>
__global__ void __launch_bounds__(256, 4) k_at_prep(const ArgsPrep A) {
    __shared__ int red[32 + 2 * 8 * 8];
    __shared__ __align__(16) uint32_t tr[128 * 32];
    const int z = blockIdx.z;
    uint16_t* dp = z == 0 ? A.plano[0] : z == 1 ? A.plano[1] : z == 2 ? A.plano[2] : A.plano[3];
    uint16_t* dg = z == 0 ? A.dig[0] : z == 1 ? A.dig[1] : z == 2 ? A.dig[2] : A.dig[3];
    int8_t* dt = z == 0 ? A.tra[0] : z == 1 ? A.tra[1] : z == 2 ? A.tra[2] : A.tra[3];
    pdl_espera();
    pdl_solta();
    if (A.nrm) {                                                   // forward: q digits, k plain, v transposed
        if (dg) prep_corpo<hd, false, true, false, true>(A, dp, dg, dt, red, tr);
        else if (dp) prep_corpo<hd, true, false, false, true>(A, dp, dg, dt, red, tr);
        else prep_corpo<hd, false, false, true, false>(A, dp, dg, dt, red, tr);
    } else {                                                       // backward: q, k transposed, v plain, dO digits and transposed
        if (dg) prep_corpo<hd, false, true, true, false>(A, dp, dg, dt, red, tr);
        else if (dp) prep_corpo<hd, true, false, false, false>(A, dp, dg, dt, red, tr);
        else prep_corpo<hd, false, false, true, false>(A, dp, dg, dt, red, tr);
    }
}

struct Barras {
    uint32_t base;
    __device__ uint32_t operator[](int i) const { return base + 8 * i; }
};
// What every kernel below starts with: barriers, the abort flag, tensor memory.  The carve-up behind the operands (OFF): barriers, the
// tensor-memory address, the abort flag, then 128 bytes in, `n` words of the kernel's own.
struct Base {
    unsigned char* smem; uint32_t s, tmem; uint32_t* slot; volatile int* aborta; Barras bar;
};
__device__ __forceinline__ Base comeca(unsigned char* bruto, uint32_t off, int barras) {
    Base b;
    // (pointer arithmetic on the array keeps the shared address space: a round trip through an integer makes every access generic)
    b.smem = bruto + ((1024u - (smem_u32(bruto) & 1023u)) & 1023u);
    b.s = smem_u32(b.smem);
    b.bar.base = b.s + off;
    b.slot = reinterpret_cast<uint32_t*>(b.smem + off + 112);
    b.aborta = reinterpret_cast<volatile int*>(b.smem + off + 116);
    if (threadIdx.x == 0) {
        for (int i = 0; i < barras; i++) mbar_init(b.bar[i], 1);
        *b.aborta = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    return b;
}
// Tensor memory, once per block (it waits until the blocks beside it leave enough: 512 columns per SM).  The blocks that need one window take
// only the columns of the scores, so that three fit an SM; the output then goes over the scores, which everyone has read by then.
__device__ __forceinline__ void aloca(Base& b, int colunas) {
    if (threadIdx.x < 32) tmem_aloca(b.slot, colunas);
    tc_fence_antes();
    __syncthreads();
    tc_fence_depois();
    b.tmem = *b.slot;
}
__device__ __forceinline__ void termina(const Base& b, int colunas) {
    tc_fence_antes();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_depois();
        tmem_libera(b.tmem, colunas);
    }
}
// One thread: 32 n token rows of a token-major operand (the maps' boxes are 32 rows high).  With `gira`, the 32-row groups of a window are
// turned: group p of the tile, which the MMA puts into tensor-memory lanes 32 p .. 32 p + 31 and which the warps p and p + 4 drain, is
// group (p + gira) & 3 of the window.  Warp w sits on scheduler w & 3 of its SM and the groups near the diagonal have nearly all the
// work, so without the turn (by the block's number) the blocks of an SM would all lean on the same two schedulers.
__device__ __forceinline__ void linhas32(uint32_t dst, const CUtensorMap* m, int y, int n, int gira, uint32_t bar) {
    for (int p = 0; p < n; p++) tma_2d(dst + p * 4096, m, 0, y + 32 * (n == 4 ? (p + gira) & 3 : p), bar);
}
__device__ __forceinline__ void carrega(uint32_t dst, const CUtensorMap* m, int x, int y, uint32_t bytes, uint32_t bar) {
    mbar_expect_tx(bar, bytes);
    tma_2d(dst, m, x, y, bar);
}
__device__ __forceinline__ void carrega_janela(uint32_t dst, const CUtensorMap* m, int y, int gira, uint32_t bar) {
    mbar_expect_tx(bar, TILE_A);
    linhas32(dst, m, y, 4, gira, bar);
}
// the 64 hi and the 64 lo digit rows of a tile, token rows `lin` on (BHT rows to the lo digits)
__device__ __forceinline__ void carrega_dig(uint32_t dst, const CUtensorMap* m, int lin, int BHT, uint32_t bar) {
    mbar_expect_tx(bar, 2 * TILE_N);
    linhas32(dst, m, lin, 2, 0, bar);
    linhas32(dst + TILE_N, m, BHT + lin, 2, 0, bar);
}
// a warp writes zeros to rows q0 .. q0 + 31, bytes 32 kq .. 32 kq + 31 of a swizzled tile
__device__ __forceinline__ void zera_bloco(unsigned char* tile, int q0, int kq, int lane) {
#pragma unroll
    for (int k = 0; k < 2; k++) *reinterpret_cast<uint4*>(tile + sw128(q0 + (lane >> 1) + 16 * k, 32 * kq + 16 * (lane & 1))) = make_uint4(0, 0, 0, 0);
}
// 32 bytes as numbers
__device__ __forceinline__ int byte_u(const uint32_t (&w)[8], int k) { return (int)__byte_perm(w[k >> 2], 0, 0x4440 + (k & 3)); }

// Output of the columns of a tile's 64 rows (all threads of the block): valor(row, column) gives the integer, `lin` the token row of row 0,
// the rows from `fim` on are not stored; `col` of `ld` columns.
template <typename F>
__device__ __forceinline__ void grava_tile(F valor, int* acc, int16_t* ex, int8_t* qm, int8_t* qE, size_t lin, int fim, int ld, int col, int hd, int e, int kid, int tid) {
    if (hd == 4) {                                                 // (raw only)
        if (tid < fim) {
            const uint32_t e2 = (uint32_t)(e & 0xffff) | ((uint32_t)e << 16);
            const size_t p = (lin + tid) * ld + col;
            *reinterpret_cast<int4*>(acc + p) = make_int4(valor(tid, 0), valor(tid, 1), valor(tid, 2), valor(tid, 3));
            *reinterpret_cast<uint2*>(ex + p) = make_uint2(e2, e2);
        }
        return;
    }
    for (int t = tid; t < NI * hd / 8; t += NTA) {                 // (whole warps)
        const int r = t / (hd / 8), d0 = t % (hd / 8) * 8;
        int o[8];
#pragma unroll
        for (int k = 0; k < 8; k++) o[k] = valor(r, d0 + k);
        const size_t l = lin + min(r, fim - 1);
        grava8(acc, ex, qm, qE, l * ld + col + d0, l * (ld / 32) + (col + d0) / 32, o, e, kid, t, r < fim);
    }
}

// -------------------------------------------------------------------------------------------------- forward
// ops.py:198-219.  A CTA owns 64 queries of one head.  Three passes over the windows: row maxima; exponentials ex = exp(-(m - u)/256) >> 3
// and their row sums; P = min((ex * inv + 2^19) >> 20, 255), stored, put into an MMA tile, and O^T += V^T . P^T.  With one window the
// scores are computed once and stay in registers.
//
// How many windows.  |q_i . k_j| <= sqrt(|q_i|^2 |k_j|^2) (the preparation left the largest squared norms per 128 tokens), so with
// B >= (|x| >> s_u) + 1 every score is u_ij <= B - (i - j) 2^incl.  The exponential (>> 3) is exactly 0 from m - u = 2130 on (p < 2^15
// shifted by n + 3 >= 15), so with the maximum m_i of the first window (which holds the diagonal; the true maximum is no smaller) a key
// at distance (i - j) 2^incl >= 2130 + B - m_i adds nothing to the row sum, cannot be the maximum and has P = 0.  This holds on the
// right-shift path, the only one that occurs in earnest; any other shift takes every window and the general roundings.
//
// Shared: Q digits 16 KB | K window 16 KB | V^T window 16 KB | P tile 8 KB; the output staging goes over the first three.
// Tensor memory: scores 128 columns, O 64.
struct ArgsFrente {
    const int* em; const int* nrm;
    int* Oacc; int16_t* Oe; int8_t* Qm; int8_t* QE; uint8_t* P;   // Qm / QE: block output (head dimension 64, block length 32) instead of the raw one
    int BH, T, H, D, hd, GA, kid;
    int y0;                                                       // first head of this launch
};
constexpr uint32_t FR_K = 2 * TILE_N, FR_V = FR_K + TILE_A, FR_P = FR_V + TILE_A, FR_BAR = FR_P + TILE_N;
constexpr size_t SM_FRENTE = 1024 + FR_BAR + 128 + (6 * NI + 2) * 4;

__global__ void __launch_bounds__(NTA, 3) k_at_frente(const __grid_constant__ CUtensorMap mQ, const __grid_constant__ CUtensorMap mK,
                                                      const __grid_constant__ CUtensorMap mVt, const ArgsFrente A) {
    extern __shared__ unsigned char bruto[];
    enum { B_Q = 0, B_K = 1, B_V = 2, B_S = 3, B_O = 4 };
    Base S = comeca(bruto, FR_BAR, 5);
    int* r_s = reinterpret_cast<int*>(S.smem + FR_BAR + 128);      // [4 lane quarters][64] partial maxima, partial sums
    int* m_s = r_s + 4 * NI;                                       // [64] row maxima
    int* i_s = m_s + NI;                                           // [64] 2^28 / row sum
    int* n_s = i_s + NI;                                           // [2] windows needed, per 32 queries
    const int T = A.T, H = A.H, D = A.D, GA = A.GA, kid = A.kid, hd = A.hd;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, quarto = wid & 3, q0 = 32 * (wid >> 2), lt = 32 * quarto + lane;
    const int tile = gridDim.x - 1 - blockIdx.x, bh = blockIdx.y + A.y0, b = bh / H, h = bh % H, i0 = tile * NI, linha0 = b * T;
    const int gira = (tile + bh) & 3, kq = (quarto + gira) & 3, jl = 32 * kq + lane;      // this warp's keys of a window, this thread's key
    const int j00 = i0 + NI - TJ;                                  // first key of the first window (may lie before the sequence: such rows are masked)
    pdl_espera();
    pdl_solta();
    if (tid == 0) {
        carrega_dig(S.s, &mQ, bh * T + i0, A.BH * T, S.bar[B_Q]);
        carrega_janela(S.s + FR_K, &mK, bh * T + j00, gira, S.bar[B_K]);
        carrega(S.s + FR_V, &mVt, j00, bh * 128, TILE_A, S.bar[B_V]);
    }
    const int emq = A.em[bh * 4], emk = A.em[bh * 4 + 1], emv = A.em[bh * 4 + 2];
    const int s_u = -((emq - GA) + (emk - GA) - (hd == 64 ? 3 : hd == 16 ? 2 : 1) + 8), incl = at::incl_alibi(h);
    const bool direita = s_u > 0 && s_u < 31;
    const int nmax = (i0 + NI - 1) / TJ + 1;
    int B = 0;                                                     // bound of the products in the units of the scores
    if (direita) {
        const int nch = (T + TJ - 1) / TJ;
        const int nq = A.nrm[(size_t)bh * 2 * nch + i0 / TJ];
        int nk = lane <= min(i0 + NI - 1, T - 1) / TJ ? A.nrm[((size_t)bh * 2 + 1) * nch + lane] : 0;
        nk = __reduce_max_sync(FULL, nk);
        B = (__float2int_ru(__fsqrt_ru(__fmul_ru(__int2float_ru(nq), __int2float_ru(nk)))) >> s_u) + 2;
    }
    // (from the norms alone, u_ii >= -B: usually this already says one window)
    const bool talvez_mais = nmax > 1 && (!direita || 65 << incl < 2130 + 2 * B);
    const int colunas = talvez_mais ? 256 : SB;
    aloca(S, colunas);
    const uint32_t t_lane = S.tmem + ((uint32_t)(32 * quarto) << 16), t_o = talvez_mais ? SB : 0;
    // zeros of P outside the first window, while the loads are on their way (further windows overwrite their part)
    for (int t = tid; t < T * 4; t += NTA) {
        const int j = t >> 2, i = i0 + 16 * (t & 3);
        if ((j < j00 || j >= i0 + NI) && i < T) *reinterpret_cast<uint4*>(A.P + ((size_t)bh * T + j) * T + i) = make_uint4(0, 0, 0, 0);
    }
    int v[32];                                                     // this thread's 32 scores of the window at hand, then their exponentials
    int minha = U_MIN;                                             // query q0 + lane: maximum, then sum, over this warp's keys
    int n = 1, passo = 0;                                          // windows; score computations so far
    bool ok = true, tem_ex = false, sem_efeito = false;            // v holds exponentials; they are all zero
#pragma unroll 1
    for (int fase = 0; fase < 3; fase++) {
        if (fase == 1) minha = 0;
#pragma unroll 1
        for (int s = 0; s < n; s++) {
            const int j = j00 - s * TJ + jl, dj = i0 + q0 - j;     // dj + k = distance of query k to this key
            const bool ha = j >= 0 && j < T && i0 + q0 < T;
            const int kmin = ha ? -dj : 32;                        // the key counts for query k >= kmin
            // Nothing of this warp's 32 keys x 32 queries counts: all beyond the diagonal or outside the sequence, or all so far behind it
            // that u_ij <= B - d 2^incl stays 2130 below u_ii >= -B.
            const int perto = i0 + q0 - (j00 - s * TJ + 32 * kq + 31);      // the smallest distance (query minus key), 62 below the largest
            bool morto = j - lane + 31 < 0 || perto < -62 || i0 + q0 >= T || (direita && perto > 0 && perto << incl >= 2130 + 2 * B);
            if (fase == 0 || n > 1) {
                if (passo) { tc_fence_antes(); __syncthreads(); }   // everyone has read the previous scores
                if (tid == 0 && ok) {
                    if (passo) carrega_janela(S.s + FR_K, &mK, bh * T + j00 - s * TJ, gira, S.bar[B_K]);
                    else ok = espera(S.bar[B_Q], 0, S.aborta, kid, 20);
                    ok = ok && espera(S.bar[B_K], passo & 1, S.aborta, kid, 21);
                    if (ok) {
                        tc_fence_depois();
                        mma_escores(S.tmem, desc_sw128(S.s + FR_K), desc_sw128(S.s), hd);
                        tc_commit(S.bar[B_S]);
                    }
                }
                __syncwarp();
                ok = __all_sync(FULL, ok && espera(S.bar[B_S], passo & 1, S.aborta, kid, 22));
                tc_fence_depois();
                passo++;
                if (!morto)
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    int x[16];
                    escores16(t_lane + q0 + 16 * g, x);
                    if (direita) {
                        // rnd_d(x, s) = (x + 2^(s-1) - 1 + ((x >> s) & 1)) >> s
                        const int meio = (1 << (s_u - 1)) - 1;
#pragma unroll
                        for (int k = 0; k < 16; k++) {
                            const int u = ((x[k] + meio + ((x[k] >> s_u) & 1)) >> s_u) - ((dj + 16 * g + k) << incl);
                            v[16 * g + k] = 16 * g + k >= kmin ? u : U_MIN;
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 16; k++) {
                            const int kk = 16 * g + k;
                            v[kk] = U_MIN;
                            if (kk >= kmin) v[kk] = rnd(x[k], s_u, kid, (long long)(linha0 + i0 + q0 + kk) * D + h * hd) - ((dj + kk) << incl);
                        }
                    }
                }
            }
            if (fase == 0) {
                if (!morto)
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    const int r = __reduce_max_sync(FULL, v[k]);
                    minha = lane == k ? max(minha, r) : minha;
                }
                if (s == 0 || s == n - 1) {
                    r_s[quarto * NI + q0 + lane] = minha;
                    __syncthreads();
                    if (tid < NI) {
                        const int m = max(max(r_s[tid], r_s[NI + tid]), max(r_s[2 * NI + tid], r_s[3 * NI + tid]));
                        m_s[tid] = m;
                        int ni = talvez_mais ? nmax : 1;
                        if (direita && talvez_mais) {
                            // keys from distance `longe` on do not count; n windows leave out the distances tid + 65 + 128 (n - 1) and more
                            const int longe = max((2130 + B - m + (1 << incl) - 1) >> incl, 0);
                            ni = i0 + tid < T ? 1 + max((longe - (tid + 65) + TJ - 1) / TJ, 0) : 1;
                        }
                        ni = __reduce_max_sync(FULL, ni);
                        if (lane == 0) n_s[wid] = min(ni, nmax);
                    }
                    __syncthreads();
                    if (s == 0) n = max(n_s[0], n_s[1]);
                }
                continue;
            }
            if (!morto && !tem_ex) {
                int dmin = 6000;
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    const int m = m_s[q0 + k];                     // a key beyond the diagonal is infinitely far below
                    v[k] = k < kmin || v[k] <= m - 6000 ? 6000 : m - v[k];
                    dmin = min(dmin, v[k]);
                }
                if (__any_sync(FULL, dmin < 2130)) {
#pragma unroll
                    for (int k = 0; k < 32; k++) v[k] = exp3_t((uint32_t)v[k] * 23637u + (13u << 22));
                } else
                    sem_efeito = true;
                tem_ex = n == 1;
            }
            morto = morto || sem_efeito;
            if (n > 1) sem_efeito = false;
            if (fase == 1) {
                if (!morto)
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    const int r = __reduce_add_sync(FULL, v[k]);
                    minha += lane == k ? r : 0;
                }
                continue;
            }
            if (s) ok = __all_sync(FULL, ok && espera(S.bar[B_O], (s - 1) & 1, S.aborta, kid, 23));      // the P tile and the V stage are free again
            uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (morto) zera_bloco(S.smem + FR_P, q0, kq, lane);
            else
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    const int p = min((v[k] * i_s[q0 + k] + (1 << 19)) >> 20, 255);
                    w[k >> 2] = (k & 3) == 0 ? (uint32_t)p : w[k >> 2] | (uint32_t)p << (8 * (k & 3));
                    S.smem[FR_P + sw128(q0 + k, jl)] = (uint8_t)p;
                }
            if (ha) {
                uint4* d = reinterpret_cast<uint4*>(A.P + ((size_t)bh * T + j) * T + i0 + q0);
                d[0] = make_uint4(w[0], w[1], w[2], w[3]);
                d[1] = make_uint4(w[4], w[5], w[6], w[7]);
            }
            fence_async();                                         // the tile is read by the tensor core (async proxy)
            tc_fence_antes();
            __syncthreads();
            if (tid == 0 && ok) {
                if (s) carrega(S.s + FR_V, &mVt, j00 - s * TJ, bh * 128, TILE_A, S.bar[B_V]);
                ok = espera(S.bar[B_V], s & 1, S.aborta, kid, 24);
                if (ok) {
                    tc_fence_depois();
                    const uint64_t da = desc_sw128(S.s + FR_V), db = desc_sw128(S.s + FR_P);
#pragma unroll
                    for (int q = 0; q < 4; q++) tc_mma_i8(S.tmem + t_o, da + 2 * q, db + 2 * q, ID_PU, (s | q) != 0);
                    tc_commit(S.bar[B_O]);
                }
            }
            __syncwarp();
        }
        if (fase == 1) {
            r_s[quarto * NI + q0 + lane] = minha;
            __syncthreads();
            if (tid < NI) {
                int soma = r_s[tid] + r_s[NI + tid] + r_s[2 * NI + tid] + r_s[3 * NI + tid];
                if (soma <= 0 && i0 + tid < T) reporta(E_DIV, kid, (long long)(linha0 + i0 + tid) * D + h * hd, soma, 0);
                i_s[tid] = (1 << 28) / max(soma, 1);               // ops.py:215
            }
            __syncthreads();
        }
    }
    ok = __all_sync(FULL, ok && espera(S.bar[B_O], (n - 1) & 1, S.aborta, kid, 25));
    tc_fence_depois();
    int* o_s = reinterpret_cast<int*>(S.smem);                     // [128 digit rows][65] over the operands
    if (ok) {
        uint32_t d[32];
        tmem_le32(t_lane + t_o + q0, d);
#pragma unroll
        for (int k = 0; k < 32; k++) o_s[lt * 65 + q0 + k] = (int)d[k];
    }
    __syncthreads();
    grava_tile([&](int i, int d) { return (int)(((uint32_t)o_s[d * 65 + i] << 7) + (uint32_t)o_s[(64 + d) * 65 + i]); }, A.Oacc, A.Oe, A.Qm, A.QE,
               (size_t)linha0 + i0, min(NI, T - i0), D, h * hd, hd, (emv - GA) - 8, kid, tid);
    termina(S, colunas);
}

// -------------------------------------------------------------------------------------------------- backward
// ops.py:222-258.  Two matrix-wide maxima of a head lie between its phases (ops.py:235,244), hence three kernels:
//   k_ab_max     max |gP| over j <= i, and the map of the non-zero parts of P (blocks of their own in the same launch)
//   k_ab_soma    gP' = rnd(gP, sh); s_lin; max |dS|
//   k_ab_saida   dS' = rnd(P (gP' - s_lin), sh2); gq = dS' . k (query tiles), gk = dS'^T . q and gv = P^T . dO (key tiles)
// Each computes gP = dO . v^T again on the tensor core; nothing T x T is kept anywhere.
struct ArgsTras {
    const uint8_t* P; int* Gacc; int16_t* Ge; int* est; int* sl; const int* em;      // em: [BH][4] = q, k, v, dO
    int* zm;                                                                          // [BH][16]: per 64 keys, bit qt = P may have a non-zero among queries 64 qt .. 64 qt + 63
    int8_t* Gm; int8_t* GE;                                                           // block output [M, 3D] instead of the raw one, or nullptr
    int BH, T, H, D, hd, GA, limite, kid, blocos_mapa;
    int y0;                                                                           // first head of this launch (k_ab_soma, k_ab_saida)
};
// The windows of a query tile / of a key tile in which stored P may be non-zero: everywhere else dS and P contribute nothing.  The first
// window always counts; the bounded variant takes maxima over everything and keeps them all.
__device__ __forceinline__ unsigned janelas_consulta(const ArgsTras& A, int bh, int qt) {
    const int n = (qt * NI + NI - 1) / TJ + 1;
    unsigned vivas = 1u;
    for (int s = 1; s < n; s++) {                                  // keys of the tiles qt - 2 s - 1 and qt - 2 s
        const int kt = qt - 2 * s;
        int m = A.limite ? -1 : A.zm[bh * 16 + kt];
        if (kt > 0 && !A.limite) m |= A.zm[bh * 16 + kt - 1];
        if (m >> qt & 1) vivas |= 1u << s;
    }
    return vivas;
}
__device__ __forceinline__ unsigned janelas_chave(const ArgsTras& A, int bh, int kt) {
    const int n = (A.T - kt * NI + TJ - 1) / TJ;
    unsigned vivas = 1u;
    if (n > 1) {
        const int m = A.limite ? -1 : A.zm[bh * 16 + kt];
        for (int s = 1; s < n; s++)
            if (m >> (kt + 2 * s) & 3) vivas |= 1u << s;
    }
    return vivas;
}

// zm[bh][kt]: P (key-major, [BH*T][T]) from the query tile kt + 2 on; the two before it belong to the first window and count anyway.
// One block per (head, key tile); a warp reads 8 key rows, 512 bytes at a time.
__device__ void mapa_p(const ArgsTras& A, int bh, int kt, unsigned* ou) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, T = A.T;
    unsigned m = 3u << kt;
    if (tid == 0) *ou = 0;
    __syncthreads();
    for (int p = 4 * (kt + 2) + lane; p < T / 16; p += 32) {       // 16-byte pieces; piece p belongs to query tile p / 4
        uint4 x[8];
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int j = kt * NI + wid * 8 + r;                   // (a piece at or beyond the tile kt + 2 exists only if the whole key tile does)
            x[r] = *reinterpret_cast<const uint4*>(A.P + ((size_t)bh * T + j) * T + 16 * p);
        }
        uint32_t o = 0;
#pragma unroll
        for (int r = 0; r < 8; r++) o |= x[r].x | x[r].y | x[r].z | x[r].w;
        if (o) m |= 1u << (p >> 2);
    }
    m = __reduce_or_sync(FULL, m);
    if (lane == 0) atomicOr(ou, m);
    __syncthreads();
    if (tid == 0) A.zm[bh * 16 + kt] = (int)*ou;
}

// Shared: dO digits 16 KB | two V windows 16 KB each; tensor memory: the scores.  The load of the next window runs behind the drain, the rest
// overlaps among the four blocks of an SM.  Only the bit length of the maximum is used (ops.py:235), and 64 hi + lo rounded towards
// zero to fp32 has the bit length of the exact value: two instructions an element instead of seven.
constexpr uint32_t MX_V = 2 * TILE_N, MX_BAR = MX_V + 2 * TILE_A;
constexpr size_t SM_MAX = 1024 + MX_BAR + 128;
__global__ void __launch_bounds__(NTA, 4) k_ab_max(const __grid_constant__ CUtensorMap mV, const __grid_constant__ CUtensorMap mG, const ArgsTras A) {
    extern __shared__ unsigned char bruto[];
    __shared__ int red[NTA / 32];
    __shared__ unsigned ou;
    const int T = A.T, nt = (T + NI - 1) / NI;
    if ((int)blockIdx.x < A.blocos_mapa) {
        pdl_espera();
        pdl_solta();
        mapa_p(A, blockIdx.x / nt, blockIdx.x % nt, &ou);
        return;
    }
    enum { B_G = 0, B_V = 1, B_S = 3 };
    Base S = comeca(bruto, MX_BAR, 4);
    aloca(S, SB);
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, quarto = wid & 3, q0 = 32 * (wid >> 2), jl = 32 * quarto + lane, kid = A.kid;
    const int item = blockIdx.x - A.blocos_mapa, bh = item % A.BH, i0 = (nt - 1 - item / A.BH) * NI, j00 = i0 + NI - TJ, n = (i0 + NI - 1) / TJ + 1;
    const uint32_t t_lane = S.tmem + ((uint32_t)(32 * quarto) << 16);
    pdl_espera();
    pdl_solta();
    bool ok = true;
    if (tid == 0) {
        carrega_dig(S.s, &mG, bh * T + i0, A.BH * T, S.bar[B_G]);
        for (int s = 0; s < 2 && s < n; s++) carrega(S.s + MX_V + s * TILE_A, &mV, 0, bh * T + j00 - s * TJ, TILE_A, S.bar[B_V + s]);
        ok = espera(S.bar[B_G], 0, S.aborta, kid, 30);
    }
    float mx = 0.0f;
    for (int s = 0; s < n; s++) {
        if (tid == 0 && ok) {
            ok = espera(S.bar[B_V + (s & 1)], (s >> 1) & 1, S.aborta, kid, 31);
            if (ok) {
                tc_fence_depois();
                mma_escores(S.tmem, desc_sw128(S.s + MX_V + (s & 1) * TILE_A), desc_sw128(S.s), A.hd);
                tc_commit(S.bar[B_S]);
            }
        }
        __syncwarp();
        ok = __all_sync(FULL, ok && espera(S.bar[B_S], s & 1, S.aborta, kid, 32));
        tc_fence_depois();
        if (tid == 0 && ok && s + 2 < n)                           // this product is done: its V stage takes the window after next
            carrega(S.s + MX_V + (s & 1) * TILE_A, &mV, 0, bh * T + j00 - (s + 2) * TJ, TILE_A, S.bar[B_V + (s & 1)]);
        __syncwarp();
        const int j = j00 - s * TJ + jl, kmin = j >= 0 && i0 + q0 < T ? j - i0 - q0 : 32;
        if (kmin < 32 || s == 0)                                   // (s == 0: a mixed warp reads together)
#pragma unroll
        for (int g = 0; g < 2; g++) {
            uint32_t hi[16], lo[16];
            escores16_cru(t_lane + q0 + 16 * g, hi, lo);
            if (s) {
#pragma unroll
                for (int k = 0; k < 16; k++) mx = fmaxf(mx, fabsf(__fmaf_rz(__uint_as_float(hi[k]), 64.0f, __uint_as_float(lo[k]))));
            } else {
#pragma unroll
                for (int k = 0; k < 16; k++) {
                    const float x = fabsf(__fmaf_rz(__uint_as_float(hi[k]), 64.0f, __uint_as_float(lo[k])));
                    mx = fmaxf(mx, 16 * g + k >= kmin ? x : 0.0f);
                }
            }
        }
        tc_fence_antes();
        __syncthreads();                                           // everyone has read the scores: the next product may write them
    }
    max_cta((int)mx, A.est + bh * at::N_EST + at::S_GP, red, tid);
    termina(S, SB);
}

// Query tiles: s_lin and the maxima of dS.  With one live window gP' and P stay in registers between the two passes.
// Shared: dO digits 16 KB | V window 16 KB; tensor memory: the scores.
constexpr uint32_t SO_V = 2 * TILE_N, SO_BAR = SO_V + TILE_A;
constexpr size_t SM_SOMA = 1024 + SO_BAR + 128 + 5 * NI * 4;
__global__ void __launch_bounds__(NTA, 3) k_ab_soma(const __grid_constant__ CUtensorMap mV, const __grid_constant__ CUtensorMap mG, const ArgsTras A) {
    extern __shared__ unsigned char bruto[];
    __shared__ int red[NTA / 32];
    enum { B_G = 0, B_V = 1, B_S = 2 };
    Base S = comeca(bruto, SO_BAR, 3);
    aloca(S, SB);
    int* r_s = reinterpret_cast<int*>(S.smem + SO_BAR + 128);      // [4 lane quarters][64] partial sums
    int* sl_s = r_s + 4 * NI;                                      // [64]
    const int T = A.T, kid = A.kid, tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, quarto = wid & 3, q0 = 32 * (wid >> 2);
    const int qt = gridDim.x - 1 - blockIdx.x, bh = blockIdx.y + A.y0, i0 = qt * NI, j00 = i0 + NI - TJ;
    const int gira = (qt + bh) & 3, jl = 32 * ((quarto + gira) & 3) + lane;
    const uint32_t t_lane = S.tmem + ((uint32_t)(32 * quarto) << 16);
    int* est = A.est + bh * at::N_EST;
    pdl_espera();
    pdl_solta();
    if (tid == 0) {
        carrega_dig(S.s, &mG, bh * T + i0, A.BH * T, S.bar[B_G]);
        carrega_janela(S.s + SO_V, &mV, bh * T + j00, gira, S.bar[B_V]);
    }
    const unsigned vivas = janelas_consulta(A, bh, qt);
    const bool uma = vivas == 1u;
    const Arred arred(at::desl1(est, A.limite));
    int v[32], minha = 0, mgp = 0, mds = 0, mp = 0, passo = 0;
    uint32_t w[8];
    bool ok = true, morto = false;                                 // P is zero in this warp's 32 x 32 part of the window
#pragma unroll 1
    for (int fase = 0; fase < 2; fase++) {
#pragma unroll 1
        for (unsigned m = vivas; m; m &= m - 1) {
            const int s = __ffs(m) - 1, j = j00 - s * TJ + jl;
            if (fase == 0 || !uma) {
                const bool ha = j >= 0 && j < T && i0 + q0 < T;
                const int kmin = ha ? j - i0 - q0 : 32;            // the key counts for query k >= kmin
#pragma unroll
                for (int k = 0; k < 8; k++) w[k] = 0;
                if (ha) {
                    const uint4* p = reinterpret_cast<const uint4*>(A.P + ((size_t)bh * T + j) * T + i0 + q0);
                    const uint4 a = p[0], c = p[1];
                    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = c.x; w[5] = c.y; w[6] = c.z; w[7] = c.w;
                }
                morto = !A.limite && !__any_sync(FULL, (w[0] | w[1] | w[2] | w[3] | w[4] | w[5] | w[6] | w[7]) != 0);
                if (passo) { tc_fence_antes(); __syncthreads(); }   // everyone has read the previous scores
                if (tid == 0 && ok) {
                    if (passo) carrega_janela(S.s + SO_V, &mV, bh * T + j00 - s * TJ, gira, S.bar[B_V]);
                    else ok = espera(S.bar[B_G], 0, S.aborta, kid, 33);
                    ok = ok && espera(S.bar[B_V], passo & 1, S.aborta, kid, 34);
                    if (ok) {
                        tc_fence_depois();
                        mma_escores(S.tmem, desc_sw128(S.s + SO_V), desc_sw128(S.s), A.hd);
                        tc_commit(S.bar[B_S]);
                    }
                }
                __syncwarp();
                ok = __all_sync(FULL, ok && espera(S.bar[B_S], passo & 1, S.aborta, kid, 35));
                tc_fence_depois();
                passo++;
                if (!morto)
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    int x[16];
                    escores16(t_lane + q0 + 16 * g, x);
#pragma unroll
                    for (int k = 0; k < 16; k++) v[16 * g + k] = 16 * g + k >= kmin ? arred(x[k]) : 0;
                }
            }
            if (morto) continue;
            if (fase == 0) {
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    if (A.limite) mgp = max(mgp, abs(v[k]));
                    const int r = __reduce_add_sync(FULL, byte_u(w, k) * v[k]);
                    minha += lane == k ? r : 0;
                }
            } else {
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    const int p = byte_u(w, k);
                    mds = max(mds, abs(p * (v[k] - sl_s[q0 + k])));
                    if (A.limite) mp = max(mp, p);
                }
            }
        }
        if (fase == 0) {
            r_s[quarto * NI + q0 + lane] = minha;
            __syncthreads();
            if (tid < NI) {
                const int sl = rnd_d(r_s[tid] + r_s[NI + tid] + r_s[2 * NI + tid] + r_s[3 * NI + tid], 8);
                sl_s[tid] = sl;
                if (i0 + tid < T) A.sl[(size_t)bh * T + i0 + tid] = sl;
            }
            __syncthreads();
        }
    }
    max_cta(mds, est + at::S_DS, red, tid);
    if (A.limite) {
        max_cta(mp, est + at::S_P, red, tid);
        max_cta(mgp, est + at::S_GPQ, red, tid);
        max_cta(tid < NI && i0 + tid < T ? abs(sl_s[tid]) : 0, est + at::S_SL, red, tid);
    }
    termina(S, SB);
}

// The output kernel.  Three roles (blockIdx.z): 0 key tiles, gk; 1 query tiles, gq; 2 key tiles, gv.
//   gq, gk: scores (lane = the other side's token in the window, column = the tile's token), dS' as digits into an MMA tile
//           (hi rows 0..63, lo rows 64..127, 128 bytes of window), then D[digit row of k or q][hi | lo column] += X^T . dS'.
//   gv:     dO^T . P only, both operands straight from memory.
// A warp whose 32 x 32 part of P is zero (half of them or more near the diagonal) only writes zeros of dS'.
// Shared, query tiles: dO digits 16 KB | v window 16 KB | transposed window 16 KB; key tiles: v 8 KB, P tile 8 KB | dO digits of the window
// 32 KB | transposed window 16 KB.  The dS' digits (16 KB) go over the window, which the scores have used up by then, and the output
// staging over everything.  Tensor memory: scores 128 columns, output 128 over them or, with several windows, beside them.
constexpr uint32_t SA_P = TILE_N, SA_A = 2 * TILE_N, SA_D = SA_A, SA_X = SA_A + 2 * TILE_A, SA_BAR = 2 * 128 * 65 * 4;
static_assert(SA_X + TILE_A <= SA_BAR, "the barriers lie behind the operands and the staging");
constexpr size_t SM_SAIDA = 1024 + SA_BAR + 128 + NI * 4;

template <bool CHAVE>
__device__ __forceinline__ int ab_saida(Base& S, const CUtensorMap& mB, const CUtensorMap& mA, const CUtensorMap& mX, const CUtensorMap& mP,
                                         const ArgsTras& A, int bh, int tile) {
    enum { B_B = 0, B_A = 1, B_X = 2, B_S = 3, B_O = 4 };
    int* sl_s = reinterpret_cast<int*>(S.smem + SA_BAR + 128);     // [64], query tiles
    const int T = A.T, H = A.H, D = A.D, GA = A.GA, kid = A.kid, hd = A.hd;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, quarto = wid & 3, q0 = 32 * (wid >> 2), lt = 32 * quarto + lane;
    const int gira = (tile + bh) & 3, kq = (quarto + gira) & 3, jl = 32 * kq + lane;      // this thread's token of a window
    const int b = bh / H, h = bh % H, t0 = tile * NI, w0 = CHAVE ? t0 : t0 + NI - TJ, wp = CHAVE ? TJ : -TJ;      // window s starts at token w0 + s wp
    const int* est = A.est + bh * at::N_EST;
    auto janela = [&](int s) {                                     // one thread: the operands of window s
        const int t = w0 + s * wp;
        if (CHAVE) {
            mbar_expect_tx(S.bar[B_A], 2 * TILE_A);
            linhas32(S.s + SA_A, &mA, bh * T + t, 4, gira, S.bar[B_A]);
            linhas32(S.s + SA_A + TILE_A, &mA, (A.BH + bh) * T + t, 4, gira, S.bar[B_A]);
        } else
            carrega_janela(S.s + SA_A, &mA, bh * T + t, gira, S.bar[B_A]);
        mbar_expect_tx(S.bar[B_X], TILE_A + (CHAVE ? TILE_N : 0));
        tma_2d(S.s + SA_X, &mX, t, bh * 128, S.bar[B_X]);
        if (CHAVE) tma_2d(S.s + SA_P, &mP, t, bh * T + t0, S.bar[B_X]);
    };
    if (tid == 0) {
        if (CHAVE) {
            mbar_expect_tx(S.bar[B_B], TILE_N);
            linhas32(S.s, &mB, bh * T + t0, 2, 0, S.bar[B_B]);
        } else
            carrega_dig(S.s, &mB, bh * T + t0, A.BH * T, S.bar[B_B]);
        janela(0);
    }
    const int sh = at::desl1(est, A.limite), sh2 = at::desl2(est, A.limite);
    const Arred arred(sh), arred2(sh2);
    const unsigned vivas = CHAVE ? janelas_chave(A, bh, tile) : janelas_consulta(A, bh, tile);
    const int colunas = vivas == 1u ? SB : 2 * SB;
    if (!CHAVE && tid < NI) sl_s[tid] = A.sl[(size_t)bh * T + min(t0 + tid, T - 1)];
    aloca(S, colunas);
    const uint32_t t_lane = S.tmem + ((uint32_t)(32 * quarto) << 16), t_o = colunas - SB;
    int passo = 0;
    bool ok = true;
#pragma unroll 1
    for (unsigned m = vivas; m; m &= m - 1, passo++) {
        const int s = __ffs(m) - 1, t = w0 + s * wp + jl;          // this thread's token of the window
        if (passo) ok = __all_sync(FULL, ok && espera(S.bar[B_O], (passo - 1) & 1, S.aborta, kid, 36));      // every operand is free again
        if (tid == 0 && ok) {
            if (passo) janela(s);
            else ok = espera(S.bar[B_B], 0, S.aborta, kid, 37);
            ok = ok && espera(S.bar[B_A], passo & 1, S.aborta, kid, 38);
            if (ok) {
                tc_fence_depois();
                if (CHAVE) mma_escores_a(S.tmem, desc_sw128(S.s + SA_A), desc_sw128(S.s + SA_A + TILE_A), desc_sw128(S.s), hd);
                else mma_escores(S.tmem, desc_sw128(S.s + SA_A), desc_sw128(S.s), hd);
                tc_commit(S.bar[B_S]);
            }
        }
        uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        int sl = 0;
        if (CHAVE) sl = A.sl[(size_t)bh * T + min(t, T - 1)];      // (a query beyond T has P = 0, the fill value)
        else if (t >= 0 && t < T && t0 + q0 < T) {
            const uint4* p = reinterpret_cast<const uint4*>(A.P + ((size_t)bh * T + t) * T + t0 + q0);
            const uint4 a = p[0], c = p[1];
            w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = c.x; w[5] = c.y; w[6] = c.z; w[7] = c.w;
        }
        __syncwarp();
        ok = __all_sync(FULL, ok && (!CHAVE || espera(S.bar[B_X], passo & 1, S.aborta, kid, 39)));
        if (CHAVE) {                                               // only to see whether anything is there
            const uint4 a = *reinterpret_cast<const uint4*>(S.smem + SA_P + sw128(q0 + (lane >> 1), 32 * kq + 16 * (lane & 1))),
                        c = *reinterpret_cast<const uint4*>(S.smem + SA_P + sw128(q0 + 16 + (lane >> 1), 32 * kq + 16 * (lane & 1)));
            w[0] = a.x | a.y | a.z | a.w | c.x | c.y | c.z | c.w;
        }
        const bool morto = !__any_sync(FULL, (w[0] | w[1] | w[2] | w[3] | w[4] | w[5] | w[6] | w[7]) != 0);
        ok = __all_sync(FULL, ok && espera(S.bar[B_S], passo & 1, S.aborta, kid, 40));
        tc_fence_depois();
        if (morto) {
            zera_bloco(S.smem + SA_D, q0, kq, lane);
            zera_bloco(S.smem + SA_D + TILE_N, q0, kq, lane);
        }
        const int dist = CHAVE ? t - t0 - q0 : t0 + q0 - t;        // query minus key at column q0
        if (!morto)
#pragma unroll
        for (int g = 0; g < 2; g++) {
            int x[16];
            escores16(t_lane + q0 + 16 * g, x);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const int kk = 16 * g + k;
                const int p = CHAVE ? S.smem[SA_P + sw128(q0 + kk, jl)] : byte_u(w, kk);
                const int y = p * (arred(x[k]) - (CHAVE ? sl : sl_s[q0 + kk]));
                const int ds = (CHAVE ? kk <= dist : kk >= -dist) ? arred2(y) : 0;
                int hi, lo;
                digitos(ds, hi, lo);
                S.smem[SA_D + sw128(q0 + kk, jl)] = (uint8_t)hi;
                S.smem[SA_D + TILE_N + sw128(q0 + kk, jl)] = (uint8_t)lo;
            }
        }
        fence_async();
        tc_fence_antes();
        __syncthreads();
        if (tid == 0 && ok) {
            ok = CHAVE || espera(S.bar[B_X], passo & 1, S.aborta, kid, 41);
            if (ok) {
                tc_fence_depois();
                const uint64_t da = desc_sw128(S.s + SA_X), db = desc_sw128(S.s + SA_D);
#pragma unroll
                for (int q = 0; q < 4; q++) tc_mma_i8(S.tmem + t_o, da + 2 * q, db + 2 * q, ID_S, (passo | q) != 0);
                tc_commit(S.bar[B_O]);
            }
        }
        __syncwarp();
    }
    ok = __all_sync(FULL, ok && espera(S.bar[B_O], (passo - 1) & 1, S.aborta, kid, 42));
    tc_fence_depois();
    int* o_s = reinterpret_cast<int*>(S.smem);                     // [2: columns of the hi digits, of the lo digits][128 digit rows][65]
    if (ok) {
#pragma unroll
        for (int a = 0; a < 2; a++) {
            uint32_t d[32];
            tmem_le32(t_lane + t_o + NI * a + q0, d);
#pragma unroll
            for (int k = 0; k < 32; k++) o_s[(a * 128 + lt) * 65 + q0 + k] = (int)d[k];
        }
    }
    __syncthreads();
    const int emz = A.em[bh * 4 + (CHAVE ? 0 : 1)], emv = A.em[bh * 4 + 2], emg = A.em[bh * 4 + 3];
    const int e = (emg - GA) + (emv - GA) + sh - 9 + sh2 + (emz - GA), col = (CHAVE ? D : 0) + h * hd;
    grava_tile([&](int r, int d) {
        const int* p = o_s + d * 65 + r;
        return junta3((uint32_t)p[0], (uint32_t)p[64 * 65] + (uint32_t)p[128 * 65], (uint32_t)p[192 * 65]);
    }, A.Gacc, A.Ge, A.Gm, A.GE, (size_t)b * T + t0, min(NI, T - t0), 3 * D, col, hd, e, kid, tid);
    return colunas;
}
__device__ __forceinline__ void ab_valor(Base& S, const CUtensorMap& mX, const CUtensorMap& mP, const ArgsTras& A, int bh, int tile) {
    enum { B_X = 0, B_O = 2 };                                     // two stages
    constexpr uint32_t EST = TILE_A + TILE_N;
    const int T = A.T, H = A.H, D = A.D, GA = A.GA, kid = A.kid, hd = A.hd;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, quarto = wid & 3, q0 = 32 * (wid >> 2), jl = 32 * quarto + lane;
    const int b = bh / H, h = bh % H, t0 = tile * NI;
    const unsigned vivas = janelas_chave(A, bh, tile);
    const int n = __popc(vivas);
    bool ok = true;
    aloca(S, NI);
    if (tid == 0) {
        auto janela = [&](int passo) {
            const int t = t0 + ((int)__fns(vivas, 0, passo + 1)) * TJ;
            const uint32_t d = S.s + (passo & 1) * EST, f = S.bar[B_X + (passo & 1)];
            mbar_expect_tx(f, EST);
            tma_2d(d, &mX, t, bh * 128, f);
            tma_2d(d + TILE_A, &mP, t, bh * T + t0, f);
        };
        janela(0);
        if (n > 1) janela(1);
        for (int c = 0; c < n && ok; c++) {
            ok = espera(S.bar[B_X + (c & 1)], (c >> 1) & 1, S.aborta, kid, 43);
            if (!ok) break;
            tc_fence_depois();
            const uint64_t da = desc_sw128(S.s + (c & 1) * EST), db = desc_sw128(S.s + (c & 1) * EST + TILE_A);
#pragma unroll
            for (int q = 0; q < 4; q++) tc_mma_i8(S.tmem, da + 2 * q, db + 2 * q, ID_PU, (c | q) != 0);
            tc_commit(S.bar[B_O]);
            if (c + 1 < n) ok = espera(S.bar[B_O], c & 1, S.aborta, kid, 44);
            if (c + 2 < n && ok) janela(c + 2);
        }
    }
    __syncwarp();
    ok = __all_sync(FULL, ok);
    ok = __syncthreads_and(ok) && __all_sync(FULL, espera(S.bar[B_O], (n - 1) & 1, S.aborta, kid, 45));
    tc_fence_depois();
    int* o_s = reinterpret_cast<int*>(S.smem);                     // [128 digit rows][65]
    if (ok) {
        uint32_t d[32];
        tmem_le32(S.tmem + ((uint32_t)(32 * quarto) << 16) + q0, d);
#pragma unroll
        for (int k = 0; k < 32; k++) o_s[jl * 65 + q0 + k] = (int)d[k];
    }
    __syncthreads();
    const int e = A.em[bh * 4 + 3] - GA - 8, col = 2 * D + h * hd;
    grava_tile([&](int r, int d) { return (int)(((uint32_t)o_s[d * 65 + r] << 7) + (uint32_t)o_s[(64 + d) * 65 + r]); }, A.Gacc, A.Ge, A.Gm, A.GE,
               (size_t)b * T + t0, min(NI, T - t0), 3 * D, col, hd, e, kid, tid);
}
__global__ void __launch_bounds__(NTA, 3) k_ab_saida(const __grid_constant__ CUtensorMap mV, const __grid_constant__ CUtensorMap mGd,
                                                     const __grid_constant__ CUtensorMap mKt, const __grid_constant__ CUtensorMap mQt,
                                                     const __grid_constant__ CUtensorMap mGt, const __grid_constant__ CUtensorMap mP, const ArgsTras A) {
    extern __shared__ unsigned char bruto[];
    Base S = comeca(bruto, SA_BAR, 5);
    pdl_espera();
    pdl_solta();
    const int bh = blockIdx.y + A.y0;
    int colunas = NI;
    if (blockIdx.z == 0) colunas = ab_saida<true>(S, mV, mGd, mQt, mP, A, bh, blockIdx.x);
    else if (blockIdx.z == 1) colunas = ab_saida<false>(S, mGd, mV, mKt, mP, A, bh, gridDim.x - 1 - blockIdx.x);
    else ab_valor(S, mGt, mP, A, bh, blockIdx.x);
    termina(S, colunas);
}

}  // namespace atc

// -------------------------------------------------------------------------------------------------- host side
static size_t atc_arredonda(size_t x) { return (x + 1023) & ~(size_t)1023; }

// Head dimension 64, 16 or, on long sequences, 4; the aligned operands fit f16 exactly up to 4 guard bits (127 << 4 = 2032).  A head of 4 is
// cheap to multiply on the CUDA cores, so the forward of atencao.cuh stays ahead up to T = 256 (2 x 256 tokens, 32 heads: 24 us against
// 40; 2 x 512, 64 heads: 150 against 135; 1 x 1024: 408 against 199); its backward does not (2 x 256: 66 us against 40), and up to
// T = 128 the kernels of one CTA per head take both.
static bool atc_serve(int blk, int T, int H, int D, int GA, bool tras) {
    return (D == H * 64 || D == H * 16 || (D == H * 4 && T > (tras ? 128 : 256))) && T % 32 == 0 && T >= 32 && T <= 1024 && D % blk == 0 &&
           (blk == 32 || blk == 128) && GA >= 0 && GA <= 4;
}
// f(y0, n): one launch for up to GY of the `total` heads (or groups of heads) along a grid's y
template <typename F>
static void atc_lancamentos(int total, F f) {
    for (int y0 = 0; y0 < total; y0 += atc::GY) f(y0, total - y0 < atc::GY ? total - y0 : atc::GY);
}
static void atc_prep(atc::ArgsPrep A, int Bt, int hd, int z, cudaStream_t st) {
    const int np = (A.T + 127) / 128, hpc = 64 / hd;
    atc_lancamentos(Bt * ((A.H + hpc - 1) / hpc), [&](int y0, int n) {
        A.y0 = y0;
        lanca_cluster(hd == 64 ? atc::k_at_prep<64> : hd == 16 ? atc::k_at_prep<16> : atc::k_at_prep<4>, dim3(np, n, z), dim3(256), 0, st, np, A);
    });
}

// Workspace: what the preparation writes.  Forward: head-maximum exponents [BH][4] and the largest squared row norms of q and k per 128 tokens
// [BH][2][ceil(T/128)]; q digits, k plain, v transposed.  Backward: statistics, s_lin, exponents, map of P; v plain, dO digits, q, k, dO transposed.
static size_t atc_ws_em(size_t BH, int T, bool tras) {
    return atc_arredonda(tras ? BH * (at::N_EST + T + 4 + 16) * sizeof(int) : BH * 16 + BH * 2 * ((T + 127) / 128) * 4);
}
static size_t atc_ws_lin(size_t BH, int T) { return atc_arredonda(BH * T * 128); }
static size_t atc_ws_bytes(int Bt, int H, int T, bool tras) {
    const size_t BH = (size_t)Bt * H;
    return atc_ws_em(BH, T, tras) + (tras ? 6 : 4) * atc_ws_lin(BH, T);
}

// forward: preparation (q digits, k plain, v transposed), then the kernel; ws: atc_ws_bytes bytes
// Qm / QE: block output (jt_quant of the raw output) instead of Oacc / Oe, block length 32 and head dimension 64 only; nullptr = raw output
static int atencao_frente_tc(int blk, const int8_t* qm, const int8_t* qE, int* Oacc, int16_t* Oe, int8_t* Qm, int8_t* QE, uint8_t* P, int Bt, int T, int H,
                             int D, int GA, int kid, cudaStream_t st, unsigned char* ws) {
    if (Qm && (blk != 32 || !QE || D != H * 64)) return (int)cudaErrorInvalidValue;
    const int BH = Bt * H, hd = D / H;
    const size_t b_em = atc_ws_em(BH, T, false), b_lin = atc_ws_lin(BH, T);
    int* em = reinterpret_cast<int*>(ws);
    int* nrm = em + 4 * BH;
    uint16_t *Qd = reinterpret_cast<uint16_t*>(ws + b_em), *K = reinterpret_cast<uint16_t*>(ws + b_em + 2 * b_lin);
    int8_t* Vt = reinterpret_cast<int8_t*>(ws + b_em + 3 * b_lin);
    atc::ArgsPrep Pp = {qm, qE, nullptr, nullptr, {nullptr, K, nullptr, nullptr}, {Qd, nullptr, nullptr, nullptr}, {nullptr, nullptr, Vt, nullptr},
                        em, nullptr, nrm, BH, T, H, D, GA, blk, 0};
    atc_prep(Pp, Bt, hd, 3, st);
    CUtensorMap mQ, mK, mVt;
    if (!(faz_mapa_h(&mQ, Qd, 2 * BH * T, 64, 32) && faz_mapa_h(&mK, K, BH * T, 64, 32) && faz_mapa(&mVt, Vt, BH * 128, T, 128)))
        return (int)cudaErrorInvalidValue;
    cudaError_t c = at_smem(atc::k_at_frente, atc::SM_FRENTE);
    if (c != cudaSuccess) return (int)c;
    atc::ArgsFrente A = {em, nrm, Oacc, Oe, Qm, QE, P, BH, T, H, D, hd, GA, kid, 0};
    atc_lancamentos(BH, [&](int y0, int n) {
        A.y0 = y0;
        lanca_pdl(atc::k_at_frente, dim3((T + atc::NI - 1) / atc::NI, n), dim3(atc::NTA), atc::SM_FRENTE, st, mQ, mK, mVt, A);
    });
    return (int)cudaGetLastError();
}

// backward: preparation (v plain, dO digits; q, k, dO transposed), the maxima, the sums, the outputs
static int atencao_tras_tc(int blk, const int8_t* gom, const int8_t* goE, const int8_t* qm, const int8_t* qE, const uint8_t* P, int* Gacc, int16_t* Ge,
                           int8_t* Gm, int8_t* GE, int Bt, int T, int H, int D, int GA, int limite, int kid, cudaStream_t st, unsigned char* ws) {
    if (Gm && (blk != 32 || !GE || D != H * 64)) return (int)cudaErrorInvalidValue;
    const int BH = Bt * H, hd = D / H, nt = (T + atc::NI - 1) / atc::NI;
    const size_t b_est = atc_ws_em(BH, T, true), b_lin = atc_ws_lin(BH, T);
    int* est = reinterpret_cast<int*>(ws);
    int* sl = est + (size_t)BH * at::N_EST;
    int* em = sl + (size_t)BH * T;
    int* zm = em + (size_t)BH * 4;
    auto parte = [&](int n) { return ws + b_est + n * b_lin; };
    uint16_t *V = (uint16_t*)parte(0), *Gd = (uint16_t*)parte(1);
    int8_t *Qt = (int8_t*)parte(3), *Kt = (int8_t*)parte(4), *Gt = (int8_t*)parte(5);
    atc::ArgsPrep Pp = {qm, qE, gom, goE, {nullptr, nullptr, V, nullptr}, {nullptr, nullptr, nullptr, Gd}, {Qt, Kt, nullptr, Gt},
                        em, est, nullptr, BH, T, H, D, GA, blk, 0};
    atc_prep(Pp, Bt, hd, 4, st);
    CUtensorMap mV, mV128, mGd, mKt, mQt, mGt, mP;
    if (!(faz_mapa_h(&mV, V, BH * T, 64, 32) && faz_mapa_h(&mV128, V, BH * T, 64, 128) && faz_mapa_h(&mGd, Gd, 2 * BH * T, 64, 32) &&
          faz_mapa(&mKt, Kt, BH * 128, T, 128) && faz_mapa(&mQt, Qt, BH * 128, T, 128) && faz_mapa(&mGt, Gt, BH * 128, T, 128) &&
          faz_mapa(&mP, P, BH * T, T, atc::NI)))
        return (int)cudaErrorInvalidValue;
    // up to two key tiles the first window is all there is: no map
    atc::ArgsTras A = {P, Gacc, Ge, est, sl, em, zm, Gm, GE, BH, T, H, D, hd, GA, limite, kid, nt > 2 ? BH * nt : 0, 0};
    cudaError_t c;
    if (limite) {
        at::ArgsTras L = {gom, goE, qm, qE, P, Gacc, Ge, est, sl, nullptr, T, H, D, GA, blk, limite, kid};
        if (hd == 64) at::k_lim<64><<<BH, 256, 0, st>>>(L);
        else if (hd == 16) at::k_lim<16><<<BH, 256, 0, st>>>(L);
        else at::k_lim<4><<<BH, 256, 0, st>>>(L);
    } else {
        if ((c = at_smem(atc::k_ab_max, atc::SM_MAX)) != cudaSuccess) return (int)c;
        lanca_pdl(atc::k_ab_max, dim3(A.blocos_mapa + BH * nt), dim3(atc::NTA), atc::SM_MAX, st, mV128, mGd, A);
    }
    if ((c = at_smem(atc::k_ab_soma, atc::SM_SOMA)) != cudaSuccess) return (int)c;
    atc_lancamentos(BH, [&](int y0, int n) {
        A.y0 = y0;
        lanca_pdl(atc::k_ab_soma, dim3(nt, n), dim3(atc::NTA), atc::SM_SOMA, st, mV, mGd, A);
    });
    if ((c = at_smem(atc::k_ab_saida, atc::SM_SAIDA)) != cudaSuccess) return (int)c;
    atc_lancamentos(BH, [&](int y0, int n) {
        A.y0 = y0;
        lanca_pdl(atc::k_ab_saida, dim3(nt, n, 3), dim3(atc::NTA), atc::SM_SAIDA, st, mV, mGd, mKt, mQt, mGt, mP, A);
    });
    return (int)cudaGetLastError();
}

}  // namespace jt
