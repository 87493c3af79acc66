// The order of barriers in k_gemm_h: the loops of the warp that loads and of the warps that multiply.  They are written over an object that does what
// they ask for.  In the kernel (gemm_h.cuh) that is the barriers, the copies and the MMAs; the test of the order compiles the same loops
// for the host, over barriers that complete in any order the hardware may choose.
#pragma once
#ifdef __CUDACC__
#define JT_LACO __device__ __forceinline__
#define JT_DESENROLA _Pragma("unroll")
#else
#define JT_LACO inline
#define JT_DESENROLA
#endif

namespace jt {
namespace th {

constexpr int NST = 4, N_MW = 2;                                            // places of the operand ring, multiplying warps

// how the tiles are numbered: columns fastest, then rows, then K ranges
// With GRUPO the K ranges of a tile are the blocks of a cluster (one tile per block): each leaves its accumulators in shared memory, and each
// puts out 1 / partes of the rows, summed over the cluster.
struct Grade { int nx, ny, partes, ppp; };                                  // tiles per row and column, K ranges, 64-element chunks per range
struct Percurso { int tile0, passo, ntiles, npedT; };                       // a block's tiles: tile0, tile0 + passo, ...; chunks of the whole K

// first chunk of a tile and the one after its last
JT_LACO int ped_ini(const Grade& G, int tile) { return tile / (G.nx * G.ny) * G.ppp; }
JT_LACO int ped_fim(const Grade& G, const Percurso& P, int tile) { const int f = ped_ini(G, tile) + G.ppp; return f < P.npedT ? f : P.npedT; }

// ------------------------------------------------------------------------------------------ loads
// v: vazio(s, phase)  waits until place s of the operand ring has been read (false: given up)
//    tile(tile)          the tile whose chunks follow
//    carrega(s, c)       has its chunk c copied there
template <class V>
JT_LACO void laco_cargas(V& v, const Grade& G, const Percurso& P) {
    int s = 0;
    unsigned fase = 1;
    bool ok = true;
    for (int tile = P.tile0; tile < P.ntiles && ok; tile += P.passo) {
        v.tile(tile);
        const int cf = ped_fim(G, P, tile);
        for (int c = ped_ini(G, tile); c < cf; c++) {
            ok = v.vazio(s, fase);
            if (!ok) break;
            v.carrega(s, c);
            if (++s == NST) { s = 0; fase ^= 1; }
        }
    }
}

// ------------------------------------------------------------------------------------------ MMAs
// A chunk takes a warp ~500 cycles of waits and issue, its MMAs 256: two warps take the stages of a rounded tile in turn (every stage starts a
// sum of its own).  NS: tensor-memory stages; CB: chunks per stage that is rounded; eu: this warp's number.
// SOMA: with tiles that add up.  v: tile(tile)  the tile whose chunks follow
//    plano(nt)         chunks per sum of the block's nt-th tile, 0: it is rounded
//    livre(t, phase)   waits until tensor-memory stage t has been drained
//    cheio(s, phase)   waits until place s of the ring has been loaded
//    arredonda(s, t, j, certo, c) / soma(s, t, i, fim, certo, c)  if `certo`, issue the MMAs of chunk c onto stage t: chunk j of a stage that is rounded / chunk i of a sum,
//                      `fim` its last; each commits the ring's place, the last of a stage the stage too
//    encontra(phase)   arrives where the multiplying warps meet and waits for the other
// All waits return false when they have given up.
template <bool SOMA, int NS, int CB, class V>
JT_LACO void laco_produtos(V& v, const Grade& G, const Percurso& P, int eu) {
    int s = 0, t = 0, vez = eu;
    unsigned fase = 0, fase_t = 1, nt = 0, encontros = 0;
    bool ok = true, soma_antes = false;
    for (int tile = P.tile0; tile < P.ntiles && ok; tile += P.passo, nt++) {
        v.tile(tile);
        const int junta = SOMA ? v.plano(nt) : 0;
        // A phase is known by its parity, so a warp may look at a place of the ring only when it is known that the chunk NST before has been loaded, and
        // at a stage only when its drain before last is known.  Within rounded tiles a warp's own waits see to both: the places and the stages that
        // it takes are the same ones again and again, so it has itself waited for what was there before, in either order.  What comes last is waited for last:
        // for stages of one chunk the stage (the drain is slower than the loads), for stages of two, of which there are four, the place (block 128,
        // 4096 x 4096 x 4096: 147.3 us, 153.5 with the stage last; 2624 x 3072 x 8064 raw 184.6 and 191.3).  A tile that adds up is one warp's, which does not see what the other waits for: around one the warps
        // meet, and what the tiles before it waited for has then come for both.
        if (SOMA && (junta || soma_antes)) {
            ok = v.encontra(encontros++ & 1);
            if (!ok) break;
        }
        soma_antes = junta;
        const int c0 = ped_ini(G, tile), cf = ped_fim(G, P, tile), nped = cf > c0 ? cf - c0 : 0;
        if (SOMA && junta) {
            const int nuni = nped / CB, net = (nuni + junta - 1) / junta;
            if (eu == 0) {
                for (int u0 = 0; u0 < nuni && ok; u0 += junta) {
                    const int nc = (junta < nuni - u0 ? junta : nuni - u0) * CB;
                    ok = v.livre(t, fase_t);
                    for (int i = 0; i < nc && ok; i++) {
                        ok = v.cheio(s, fase);
                        v.soma(s, t, i, i == nc - 1, ok, c0 + u0 * CB + i);
                        if (++s == NST) { s = 0; fase ^= 1; }
                    }
                    if (++t == NS) { t = 0; fase_t ^= 1; }
                }
            } else {
                fase ^= (s + nped) / NST & 1;
                s = (s + nped) % NST;
                fase_t ^= (t + net) / NS & 1;
                t = (t + net) % NS;
            }
            continue;
        }
        for (int i = 0; i < nped && ok; i += CB) {
            const bool minha = vez == 0;
            vez = minha ? N_MW - 1 : vez - 1;
JT_DESENROLA
            for (int j = 0; j < CB; j++) {
                if (minha && ok) {
                    if (CB > 1 && j == 0) ok = v.livre(t, fase_t);
                    ok = ok && v.cheio(s, fase);
                    if (CB == 1 && j == 0) ok = ok && v.livre(t, fase_t);
                    v.arredonda(s, t, j, ok, c0 + i + j);
                }
                if (++s == NST) { s = 0; fase ^= 1; }
            }
            if (++t == NS) { t = 0; fase_t ^= 1; }
        }
    }
}

}  // namespace th
}  // namespace jt
