// The loops of jatai_b200/csrc/gemm_h_ordem.cuh over simulated barriers: loads complete in any order (each one's latency is drawn, some are very
// late), warps stall anywhere.  Each drawn schedule must multiply what was asked for, put every stage out once and end.
//   ordem_gemm_h KIND CHUNKS SCHEDULES      KIND: plain (the kernel that only rounds), plain64 / plain128 (its forms for 64-wide tiles / block 128), round, sum, mixed
// Exit 0: all schedules are right; 1: the first one that is not is printed.
#include <ucontext.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "gemm_h_ordem.cuh"

using namespace jt::th;

namespace {

constexpr int N_DW = 2;                                  // two drain warps stand for the kernel's sixteen
constexpr int N_TILES = 28;

struct Falha { const char* o_que; };

// ---------------------------------------------------------------------------------------------- events in virtual time, warps as fibres
struct Sim {
    std::mt19937_64 rng;
    double agora = 0;
    std::multimap<double, std::function<void()>> fila;
    struct Fibra { ucontext_t c; std::vector<char> pilha; std::function<void()> f; bool fim = false; };
    std::vector<std::unique_ptr<Fibra>> fibras;
    Fibra* atual = nullptr;
    ucontext_t mestre;
    const char* falha = nullptr;

    explicit Sim(unsigned long long s) : rng(s) {}
    double unif() { return std::uniform_real_distribution<double>(0, 1)(rng); }
    // around `base`, one in thirty up to a hundred times that
    double demora(double base) { const double d = base * (0.5 + unif()); return unif() < 1.0 / 30 ? d * (1 + 100 * unif()) : d; }
    void depois(double d, std::function<void()> f) { fila.emplace(agora + d, std::move(f)); }
    static Sim*& unica() { static Sim* s; return s; }
    static void entra() {
        Fibra* f = unica()->atual;
        try { f->f(); } catch (const Falha& e) { unica()->falha = e.o_que; }
        f->fim = true;
        swapcontext(&f->c, &unica()->mestre);
    }
    void nova(std::function<void()> f) {
        fibras.push_back(std::make_unique<Fibra>());
        Fibra* b = fibras.back().get();
        b->f = std::move(f);
        b->pilha.resize(64 << 10);
        getcontext(&b->c);
        b->c.uc_stack.ss_sp = b->pilha.data();
        b->c.uc_stack.ss_size = b->pilha.size();
        makecontext(&b->c, entra, 0);
        depois(demora(1), [this, b] { corre(b); });
    }
    void corre(Fibra* b) {
        atual = b;
        swapcontext(&mestre, &b->c);
        atual = nullptr;
    }
    void cede() { swapcontext(&atual->c, &mestre); }
    void passa(double d) {
        Fibra* b = atual;
        depois(d, [this, b] { corre(b); });
        cede();
    }
    void roda() {
        unica() = this;
        while (!fila.empty() && !falha) {
            auto it = fila.begin();
            agora = it->first;
            auto f = std::move(it->second);
            fila.erase(it);
            f();
        }
        for (auto& b : fibras)
            if (!falha && !b->fim) falha = "a wait that nothing ends";
    }
};

// an mbarrier: phases completed, arrivals missing
struct Barra {
    Sim* S = nullptr;
    int conta = 1, faltam = 1;
    long long feitas = 0;
    std::vector<Sim::Fibra*> dormem;
    void cria(Sim& s, int n) { S = &s; conta = faltam = n; }
    void chega() {
        if (--faltam) return;
        faltam = conta;
        feitas++;
        for (auto* b : dormem) { Sim* s = S; s->depois(s->demora(0.1), [s, b] { s->corre(b); }); }
        dormem.clear();
    }
    bool espera(unsigned par) {                          // true as soon as the phase of this parity is the last one completed
        S->passa(S->demora(0.1));
        while ((feitas & 1) == (par & 1)) { dormem.push_back(S->atual); S->cede(); }
        return true;
    }
};

// NS: tensor-memory stages, CB: chunks per stage that is rounded
template <int NS, int CB>
struct Bloco {
    Sim& S;
    const int n_ped;
    std::vector<int> planos;
    Grade G;
    Percurso P;
    Barra cheio[NST], vazio[NST], tcheio[NS], tlivre[NS], encontro_b;
    struct Lugar { int tile = -1, c = -1; bool vem = false; } anel[NST];
    struct Estagio { int tile = -1; std::vector<int> c; int le = 0; bool usado = false; } tmem[NS];
    std::vector<int> postos;                             // chunks put out, tile after tile
    double fim_mma = 0;

    Bloco(Sim& s, int ped, std::vector<int> pl) : S(s), n_ped(ped), planos(std::move(pl)) {
        const int n = (int)planos.size();
        G = {1, n, 1, ped};
        P = {0, 1, n, ped};
        for (auto& b : cheio) b.cria(S, 1);
        for (auto& b : vazio) b.cria(S, 1);
        for (auto& b : tcheio) b.cria(S, 1);
        for (auto& b : tlivre) b.cria(S, N_DW);
        encontro_b.cria(S, N_MW);
    }

    struct Carrega {
        Bloco& B;
        int t = 0;
        void tile(int x) { t = x; }
        bool vazio(int s, unsigned fase) { return B.vazio[s].espera(fase); }
        void carrega(int s, int c) {
            Lugar& l = B.anel[s];
            if (l.vem) throw Falha{"a place of the ring is loaded while its load is on the way"};
            l = {t, c, true};
            Bloco* b = &B;
            B.S.depois(B.S.demora(2), [b, s] { b->anel[s].vem = false; b->cheio[s].chega(); });
        }
    };
    // MMAs run in the order of their issue; a commit arrives when those before it are done
    void emite(int s, int t, bool primeiro, bool fim, int tile, int c) {
        const Lugar& l = anel[s];
        if (l.tile != tile || l.c != c) throw Falha{"an operand is multiplied that is another chunk's"};
        if (l.vem) throw Falha{"an operand is multiplied before it has been loaded"};
        Estagio& e = tmem[t];
        if (primeiro) {
            if (e.usado) throw Falha{"a tensor-memory stage is written before it has been drained"};
            e.tile = tile; e.c.clear(); e.le = 0; e.usado = true;
        }
        if (e.tile != tile) throw Falha{"a sum goes on in another tile's stage"};
        e.c.push_back(c);
        fim_mma = std::max(fim_mma, S.agora) + S.demora(0.3);
        S.depois(fim_mma - S.agora, [this, s] { vazio[s].chega(); });
        if (fim) S.depois(fim_mma - S.agora, [this, t] { tcheio[t].chega(); });
    }
    struct Multiplica {
        Bloco& B;
        int t = 0;
        char ultima = 0;                                 // the last wait: for a stage or for a place
        void tile(int x) { t = x; }
        int plano(unsigned nt) { return B.planos[nt]; }
        bool encontra(unsigned fase) { B.encontro_b.chega(); return B.encontro_b.espera(fase); }
        bool livre(int s, unsigned fase) { ultima = 'e'; return B.tlivre[s].espera(fase); }
        bool cheio(int s, unsigned fase) { ultima = 'l'; return B.cheio[s].espera(fase); }
        void arredonda(int s, int st, int j, bool, int c) {
            // (stages of one chunk are drained more slowly than chunks are loaded, four stages of two are not)
            if (ultima != (CB == 1 ? 'e' : 'l')) throw Falha{"the wait for what comes first is the last one"};
            B.emite(s, st, j == 0, j == CB - 1, t, c);
            B.S.passa(B.S.demora(0.2));
        }
        void soma(int s, int st, int i, bool fim, bool, int c) { B.emite(s, st, i == 0, fim, t, c); B.S.passa(B.S.demora(0.2)); }
    };
    template <bool SOMA>
    void drena(bool anota) {
        int t = 0;
        unsigned fase = 0;
        for (int tile = 0; tile < P.ntiles; tile++) {
            const int junta = SOMA ? planos[tile] : 0;
            for (int c = 0; c < n_ped; c += junta ? junta : CB) {
                tcheio[t].espera(fase);
                Estagio& e = tmem[t];
                const int n = std::min(junta ? junta : CB, n_ped - c);
                bool certo = e.tile == tile && (int)e.c.size() == n;
                for (int k = 0; certo && k < n; k++) certo = e.c[k] == c + k;
                if (!certo) throw Falha{"a stage is drained that does not hold its chunks"};
                if (anota) for (int k : e.c) postos.push_back(tile * n_ped + k);
                S.passa(S.demora(0.8));
                if (++e.le == N_DW) e.usado = false;
                tlivre[t].chega();
                if (++t == NS) { t = 0; fase ^= 1; }
            }
        }
    }
    template <bool SOMA>
    const char* roda() {
        Carrega vc{*this};
        std::vector<Multiplica> vm(N_MW, Multiplica{*this});
        S.nova([&] { laco_cargas(vc, G, P); });
        for (int w = 0; w < N_MW; w++) S.nova([&, w] { laco_produtos<SOMA, NS, CB>(vm[w], G, P, w); });
        for (int w = 0; w < N_DW; w++) S.nova([&, w] { drena<SOMA>(w == 0); });
        S.roda();
        if (S.falha) return S.falha;
        for (int k = 0; k < P.ntiles * n_ped; k++)
            if (k >= (int)postos.size() || postos[k] != k) return "a chunk is missing or out of its order";
        return nullptr;
    }
};

}  // namespace

int main(int argc, char** argv) {
    if (argc != 4) return 2;
    const std::string kind = argv[1];
    const int ped = atoi(argv[2]), n = atoi(argv[3]);
    for (int i = 0; i < n; i++) {
        Sim S(1000 + i);
        std::vector<int> planos(N_TILES);
        const double p = S.unif();
        const int parte = 2 << (S.rng() % 4);             // chunks per sum: 2 to 16
        for (int& x : planos) x = kind == "sum" || (kind == "mixed" && S.unif() < p) ? parte : 0;
        const char* erro = kind == "plain128" ? Bloco<4, 2>(S, ped, planos).roda<false>()
                           : kind == "plain64" ? Bloco<4, 1>(S, ped, planos).roda<false>()
                           : kind == "plain"  ? Bloco<2, 1>(S, ped, planos).roda<false>()
                                              : Bloco<2, 1>(S, ped, planos).roda<true>();
        if (erro) {
            printf("schedule %d, %d chunks a tile, plans", i, ped);
            for (int x : planos) printf(" %d", x);
            printf(": %s\n", erro);
            return 1;
        }
    }
    return 0;
}
