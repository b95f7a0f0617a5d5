// stop_join.cpp -- drives the rounds and contractions of stop_kernels.cu.
#include "stop_join.h"

#include <cstring>
#include <string>
#include <vector>

namespace nsat {

namespace {

// Rounds on a domain before it is contracted.  After one to five rounds a
// random function has kept 0.47, 0.32, 0.20, 0.11 and 0.06 of its states.
// While the table lies in L2 a round is cheap next to a contraction's passes
// and launches (2^24 entries, whole solve: contracted after 3 rounds 1068 us,
// after 4 979, after 5 873); beyond L2 a round is random HBM sectors (2^28
// entries: 31.4, 31.4 and 34.3 ms).
uint32_t first_rounds(uint64_t entries) { return entries * 4 <= (64ull << 20) ? 5 : 4; }
constexpr uint32_t kRoundsPerLevel = 3;   // on a contracted domain
// A contraction passes twice over the domain above it (mark, put back) and
// adds about ten launches and a wait for the host: it is worth it while half
// of the domain or less remains, for the tables whose rounds take longer than
// the launches.
constexpr double kKeepMost = 0.5;
constexpr uint64_t kContractLeast = 1ull << 20;     // of a contracted domain
constexpr uint64_t kTableLeast = 1ull << 22;        // of the table
constexpr uint64_t kSecondLook = 1ull << 24;
constexpr uint32_t kRoundsLeft = 5;       // fewer rounds than this do not pay for one
// Whether the table contracts is asked of a sample first (256 successors in
// 65536 are looked at), taken in an early round and read while the next ones
// run: bijections keep all their states in every round, and marking 2^24
// successors costs two rounds.  Round 1 tells a random function (0.47) from
// one that hardly shrinks; a large table is asked once more, later.
struct Look {
    uint32_t sample, contract;             // rounds
    double keep;                           // the most that may remain of the sample
};

struct Level {
    uint32_t count = 0;                    // domain size
    uint32_t round0 = 0;                   // rounds done when it was made
    uint32_t* states = nullptr;            // id -> position in the domain above
    uint32_t* ids = nullptr;               // position in the domain above -> id
    uint64_t* P[2] = {nullptr, nullptr};
    uint64_t* Q[2] = {nullptr, nullptr};
    uint32_t* start = nullptr;
};

struct Scratch {
    nsat_ctx* ctx;
    const std::function<void*(size_t)>& own;
    std::vector<void*> p;
    Scratch(nsat_ctx* c, const std::function<void*(size_t)>& o) : ctx(c), own(o) {}
    ~Scratch() { for (void* q : p) ctx_free(ctx, q); }
    template <typename T>
    bool get(T** out, uint64_t count) {
        void* q = nullptr;
        if (own) {
            q = own(count * sizeof(T));
            *out = static_cast<T*>(q);
            return q != nullptr;
        }
        if (ctx_alloc(ctx, &q, count * sizeof(T)) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        p.push_back(q);
        *out = static_cast<T*>(q);
        return true;
    }
};

// The words of nsat_stop_small and nsat_stop_grid.
int polled_answer(nsat_ctx* ctx, StopRun* x) {
    if (int rc = ctx_poll_words(ctx, 5)) return rc;
    const volatile uint64_t* w = ctx_words(ctx);
    x->polled = true;
    x->rounds = (uint32_t)w[0];
    x->start = (uint32_t)w[1];
    x->found = x->start != ~0u;
    x->entry = (uint32_t)w[2];
    x->steps_of = (uint32_t)w[3];
    x->ms = (uint32_t)w[4] * 1e-6;
    return NSAT_OK;
}

}  // namespace

#define JCK(call)                                                                              \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            return ctx_fail(ctx, NSAT_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)
#define JRUN(call)                                                                    \
    do {                                                                              \
        if ((call) != 0) return ctx_fail(ctx, NSAT_ECUDA, "doubling launch failed");  \
        x->launches++;                                                                \
    } while (0)

int stop_run(nsat_ctx* ctx, StopRun* x) {
    const uint32_t n = x->n, u = x->unknowns, mode = x->mode;
    const uint64_t N = 1ull << n;
    cudaStream_t st = ctx_stream(ctx);
    const int sms = ctx_sm_count(ctx);
    NsatStopState *d = nullptr, *h = nullptr;
    ctx_stop_state(ctx, &d, &h);
    x->found = false;
    x->launches = 0;
    bool answered = false;
    if (n <= NSAT_STOP_SMALL_BITS && n > 0) {
        const uint32_t seq = ctx_next_seq(ctx);
        JRUN(nsat_stop_small(x->a, n, u, mode, x->steps, x->steps ? nullptr : x->b, x->out64,
                             (uint64_t*)ctx_words(ctx), seq, st));
        if (int rc = polled_answer(ctx, x)) return rc;
        x->table = x->b;
        return NSAT_OK;
    }
    Scratch mem(ctx, x->scratch);
    uint32_t* dist = x->steps ? x->dist : nullptr;
    if (x->steps && !dist && !mem.get(&dist, N)) return NSAT_ENOMEM;
    uint32_t* keep = nullptr;
    if (n > NSAT_STOP_SMALL_BITS && n <= NSAT_STOP_GRID_BITS && mem.get(&keep, N)) {
        const uint32_t seq = ctx_next_seq(ctx);
        const int rc = nsat_stop_grid(x->a, x->b, keep, dist, n, u, mode, x->steps, x->out64, ctx_grid_state(ctx),
                                      ctx_grid_spins(ctx), (uint64_t*)ctx_words(ctx), seq, st);
        if (rc < 0) return ctx_fail(ctx, NSAT_ECUDA, "doubling launch failed");
        if (rc == 0) {
            x->launches++;
            if (int e = polled_answer(ctx, x)) return e;
            if (x->rounds != ~0u) {
                x->table = (x->rounds & 1) ? x->b : x->a;
                return NSAT_OK;
            }
            // the barrier gave up: a launch per round, from the table as built
            x->polled = false;
            ctx_grid_gave_up(ctx);
            JCK(cudaMemcpyAsync(x->a, keep, N * 4, cudaMemcpyDeviceToDevice, st));
        }
    }
    if (x->begin) JCK(cudaEventRecord(x->begin, st));
    memset(h, 0, sizeof(*h));
    memset(h->best, 0xff, sizeof(h->best));
    JCK(cudaMemcpyAsync(d, h, sizeof(*h), cudaMemcpyHostToDevice, st));

    uint32_t* T[2] = {x->a, x->b};
    std::vector<Level> lv;
    uint32_t* sample = nullptr;
    uint32_t* at_dist = nullptr;
    const uint32_t sample_words = N >= kTableLeast ? (uint32_t)(N >> 13) : 0;
    const Look looks[2] = {{1, first_rounds(N), 0.85}, {6, 8, kKeepMost}};
    uint32_t look = 0, contract_at = n + 1;
    if (!sample_words || !mem.get(&sample, sample_words)) look = 2;
    bool sampled = false;
    for (uint32_t r = 1; r <= n; r++) {
        if (lv.empty()) {
            const bool sampling = look < 2 && r == looks[look].sample && n > looks[look].contract + kRoundsLeft;
            if (sampling) {
                JCK(cudaMemsetAsync(sample, 0, (size_t)sample_words * 4, st));
                if (look) JCK(cudaMemsetAsync(&d->distinct, 0, 4, st));
            }
            JRUN(nsat_stop_join(T[(r - 1) & 1], T[r & 1], dist, n, u, r, mode, d, sampling ? sample : nullptr, sms, st));
            if (sampling) {
                JCK(cudaMemcpyAsync(&h->distinct, &d->distinct, 4, cudaMemcpyDeviceToHost, st));
                JCK(cudaEventRecord(ctx_stop_event(ctx), st));
                contract_at = looks[look].contract;
                sampled = true;
            }
        } else {
            Level& L = lv.back();
            const uint32_t k = r - 1 - L.round0;
            JRUN(nsat_stop_join_pq(L.P[k & 1], L.Q[k & 1], L.P[(k & 1) ^ 1], L.Q[(k & 1) ^ 1], L.start, L.count, n, r,
                                   mode, d, sms, st));
        }
        if (r != contract_at) continue;
        contract_at = n + 1;
        if (sampled) {       // the sample's copy was queued rounds ago: this hardly waits
            sampled = false;
            JCK(cudaEventSynchronize(ctx_stop_event(ctx)));
            const double keep = looks[look++].keep;
            if (256.0 * h->distinct > keep * (double)N) {
                if (N < kSecondLook) look = 2;
                continue;
            }
            look = 2;
        }
        // contract to the successors
        Level* L = lv.empty() ? nullptr : &lv.back();
        const uint64_t items = L ? L->count : N;
        Level nx;
        nx.round0 = r;
        const uint64_t bit_words = (items + 31) / 32;
        uint32_t* marked = nullptr;
        if (!mem.get(&marked, bit_words + (bit_words + 1023) / 1024)) continue;
        uint32_t* sums = marked + bit_words;
        JCK(cudaMemsetAsync(marked, 0, bit_words * 4, st));
        const uint64_t* upQ = L ? L->Q[(r - L->round0) & 1] : nullptr;
        const uint64_t* upP = L ? L->P[(r - L->round0) & 1] : nullptr;
        if (!L) JRUN(nsat_stop_mark32(T[r & 1], items, n, marked, r, mode, d, sms, st));
        else JRUN(nsat_stop_mark64(upQ, items, n, marked, r, mode, d, sms, st));
        JRUN(nsat_stop_rank(marked, items, sums, d, st));
        x->launches += 2;      // the rank's and the contraction's second kernels
        JCK(cudaMemcpyAsync(h, d, sizeof(*h), cudaMemcpyDeviceToHost, st));
        JCK(cudaStreamSynchronize(st));
        if (h->final_round || (h->best[r] != ~0u && (mode == 0 || h->best[r] == 0))) {
            if (!h->final_round) h->final_round = r;
            answered = true;
            break;
        }
        nx.count = h->count;
        if ((double)nx.count > kKeepMost * (double)items) continue;
        // ids of the positions above: those of level 0 go to the table's other buffer
        const uint64_t c = nx.count ? nx.count : 1;
        uint64_t* slab = nullptr;
        if (dist && !at_dist && !mem.get(&at_dist, N)) continue;
        if (!mem.get(&slab, 5 * c + (L ? (items + 1) / 2 : 0))) continue;
        nx.P[0] = slab;
        nx.P[1] = slab + c;
        nx.Q[0] = slab + 2 * c;
        nx.Q[1] = slab + 3 * c;
        nx.states = (uint32_t*)(slab + 4 * c);
        nx.start = nx.states + c;
        nx.ids = L ? (uint32_t*)(slab + 5 * c) : T[(r & 1) ^ 1];
        JRUN(nsat_stop_list(marked, items, sums, nx.states, nx.ids, st));
        if (!L)
            JRUN(nsat_stop_contract32(T[r & 1], dist, nx.states, nx.ids, nx.count, n, u, r, nx.P[0], nx.Q[0], nx.start,
                                      sms, st));
        else
            JRUN(nsat_stop_contract64(upP, upQ, L->start, L->count, nx.states, nx.ids, nx.count, n, nx.P[0], nx.Q[0],
                                      nx.start, sms, st));
        lv.push_back(nx);
        if (nx.count >= kContractLeast && n > r + kRoundsPerLevel + kRoundsLeft) contract_at = r + kRoundsPerLevel;
    }
    if (!answered) {
        JCK(cudaMemcpyAsync(h, d, sizeof(*h), cudaMemcpyDeviceToHost, st));
        JCK(cudaStreamSynchronize(st));
    }
    const uint32_t fr = h->final_round ? h->final_round : n;
    const uint32_t best = n ? h->best[fr] : ~0u;
    // the answers of every domain back to the one above it, then the table.  A
    // level made before the answering round has run at least one round.
    uint32_t last = fr;
    for (size_t l = lv.size(); l-- > 0;) {
        Level& L = lv[l];
        const uint64_t* q = L.Q[(last - L.round0) & 1];
        last = L.round0;
        if (l > 0) {
            Level& up = lv[l - 1];
            JRUN(nsat_stop_expand64(up.Q[(last - up.round0) & 1], up.count, q, L.states, L.ids, n, sms, st));
        } else {
            uint32_t* at = T[(last & 1) ^ 1];
            JRUN(nsat_stop_scatter(q, L.states, L.count, n, at, at_dist, sms, st));
            JRUN(nsat_stop_finish(T[last & 1], dist, at, at_dist, N, n, last, sms, st));
        }
    }
    uint32_t* table = T[last & 1];
    if (x->out64) JRUN(nsat_stop_widen(table, dist, N, n, fr, x->out64, sms, st));
    if (x->done) JCK(cudaEventRecord(x->done, st));
    if (best != ~0u) {
        JCK(cudaMemcpyAsync(&h->entry, table + best, 4, cudaMemcpyDeviceToHost, st));
        if (dist) JCK(cudaMemcpyAsync(&h->dist, dist + best, 4, cudaMemcpyDeviceToHost, st));
    }
    JCK(cudaStreamSynchronize(st));
    x->rounds = fr;
    x->table = table;
    x->found = best != ~0u;
    x->start = best;
    x->entry = best != ~0u ? h->entry : 0;
    x->steps_of = best != ~0u && dist ? h->dist : 0;
    return NSAT_OK;
}

}  // namespace nsat
