// lbm_batch.cu -- ensembles of independent lid-driven cavities on one GPU.
//
// An ensemble holds any number of cavities (lattices) of different sizes,
// parameters, storage types and step counts, each with its own step
// counter.  A tick advances every active cavity by k steps with one launch
// per chunk of a storage group and step (k_step / k_step2: each block reads
// its cavity's parity from the descriptor table), without waiting for the GPU,
// the chunks on streams of their own.  With kernel shape 3 a chunk of 16-bit
// cavities whose members are all at the same kind of step runs the
// staged-tile kernel instead, if its group is large enough (staged_pays).
// The static batch (lbm_cu_batch_*) runs a fixed
// ensemble to completion; the server (lbm_cu_server_*) admits queued solves
// between ticks under an HBM budget and retires finished ones (continuous
// batching).  Results of a cavity do not depend on the other members of its
// ensemble: every cavity is computed by the same per-cell arithmetic as a
// lone lattice.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <deque>
#include <memory>
#include <string>
#include <vector>

#include "lbm_internal.h"
#include "lbm_startup.cuh"

using namespace lbm;
using namespace lbm_rt;

namespace lbm_rt {

template <typename S, bool PAIR>
int launch_tick_t(bool les, const BatchArgs &a, int blocks, int j, int uni, Dep dep, cudaStream_t st) {
    if (blocks <= 0) return 0;
    if constexpr (PAIR) {
        return les ? launch_dep(dep, k_step2<S, true>, blocks, kBlock, 0, st, a, j)
                   : launch_dep(dep, k_step2<S, false>, blocks, kBlock, 0, st, a, j);
    } else if constexpr (sizeof(S) >= 4) {
        // float and double chunks whose cavities are all at the same kind of
        // step run that kind's kernel alone (its own launch bounds)
        if (uni == 1)
            return les ? launch_dep(dep, k_step<S, true, 1>, blocks, kBlock, 0, st, a, j)
                       : launch_dep(dep, k_step<S, false, 1>, blocks, kBlock, 0, st, a, j);
        if (uni == 2)
            return les ? launch_dep(dep, k_step<S, true, 2>, blocks, kBlock, 0, st, a, j)
                       : launch_dep(dep, k_step<S, false, 2>, blocks, kBlock, 0, st, a, j);
    }
    return les ? launch_dep(dep, k_step<S, true>, blocks, kBlock, 0, st, a, j)
               : launch_dep(dep, k_step<S, false>, blocks, kBlock, 0, st, a, j);
}

int launch_tick(int storage, bool pair, bool les, const BatchArgs &a, int blocks, int j, int uni, Dep dep, cudaStream_t st) {
    if (pair) {
        switch (storage) {
            case kF32: return launch_tick_t<float, true>(les, a, blocks, j, uni, dep, st);
            case kF16: return launch_tick_t<__half, true>(les, a, blocks, j, uni, dep, st);
            case kBF16: return launch_tick_t<__nv_bfloat16, true>(les, a, blocks, j, uni, dep, st);
            case kC16: return launch_tick_t<c16_t, true>(les, a, blocks, j, uni, dep, st);
        }
        return fail("the two-cell kernels need a float arithmetic type");
    }
    switch (storage) {
        case kF32: return launch_tick_t<float, false>(les, a, blocks, j, uni, dep, st);
        case kF64: return launch_tick_t<double, false>(les, a, blocks, j, uni, dep, st);
        case kF16: return launch_tick_t<__half, false>(les, a, blocks, j, uni, dep, st);
        case kBF16: return launch_tick_t<__nv_bfloat16, false>(les, a, blocks, j, uni, dep, st);
        case kC16: return launch_tick_t<c16_t, false>(les, a, blocks, j, uni, dep, st);
    }
    return fail("unknown storage type");
}

// Bytes a cavity holds on the device (populations, flags, optional u).
size_t cavity_bytes(const lbm_cavity &c, int store_v) {
    const int64_t n = (int64_t)c.nx * c.ny * c.nz;
    const int64_t ps = round_up(n, 256 / (int64_t)storage_bytes(c.storage));
    return (size_t)ps * 19 * storage_bytes(c.storage) + (size_t)round_up(n, 256) +
           (store_v ? (size_t)n * 3 * real_bytes(c.storage) : 0) + 4096;
}

int check_cavity(const lbm_cavity &c) {
    if (c.nx < 3 || c.ny < 3 || c.nz < 3) return fail("cavity edges must be at least 3 cells");
    if (c.storage < LBM_F32 || c.storage > LBM_C16) return fail("unknown storage type");
    if (!(c.tau0 > 0.5)) return fail("cavity tau0 must exceed 0.5");
    if (c.steps < 0) return fail("negative step count");
    return 0;
}

// The kernel arguments of a cavity: inv_tau = 1/tau0 in its arithmetic type.
lbm_params cavity_params(const lbm_cavity &c) {
    lbm_params p{};
    if (c.storage == LBM_F64) {
        p.inv_tau = 1.0 / c.tau0;
        p.tau0 = c.tau0;
    } else {
        const float t = (float)c.tau0;
        p.inv_tau = (double)(1.0f / t);
        p.tau0 = (double)t;
    }
    p.les_c = 18.0 * std::sqrt(2.0) * c.cs * c.cs;
    p.lid = c.lid;
    return p;
}

// A lid-driven cavity at step 0, asynchronously (k_cavity).
int cavity_reset(lbm_lattice *l, const lbm_cavity &c, cudaStream_t st) {
    const int g = grid_for(l->n);
    switch (l->storage) {
        case kF32: k_cavity<float><<<g, kBlock, 0, st>>>(l->h, c.seed, c.amp, l->store_v); break;
        case kF64: k_cavity<double><<<g, kBlock, 0, st>>>(l->h, c.seed, c.amp, l->store_v); break;
        case kF16: k_cavity<__half><<<g, kBlock, 0, st>>>(l->h, c.seed, c.amp, l->store_v); break;
        case kBF16: k_cavity<__nv_bfloat16><<<g, kBlock, 0, st>>>(l->h, c.seed, c.amp, l->store_v); break;
        case kC16: k_cavity<c16_t><<<g, kBlock, 0, st>>>(l->h, c.seed, c.amp, l->store_v); break;
    }
    CU(cudaGetLastError());
    return 0;
}

struct Ensemble {
    struct Slot {
        lbm_cavity spec{};
        lbm_lattice *lat = nullptr;
        void *block = nullptr;  // a server's device block under the lattice
        size_t block_bytes = 0;
        int64_t done = 0;
        bool active = false;
        int64_t id = -1;
    };
    // One launch per chunk of up to kBatchLattices members per step.
    struct Chunk {
        std::unique_ptr<BatchArgs> args;  // descriptors with this tick's parities
        std::unique_ptr<BatchArgs> sargs;  // the same numbered in staged tiles (staged groups)
        int blocks = 0;
        int tiles = 0;
        int parities = 0;  // bit p: some member's step counter has parity p
        bool les = false;
    };
    struct Group {
        int storage = 0;
        bool pair = false;
        bool staged = false;  // through the staged tiles where they apply (shape 3, 16-bit storage)
        std::vector<int> members;
        size_t per = 0;  // members of a chunk
        int64_t cells = 0;
        bool ragged = false;  // some row is not whole 16-byte units of half populations
        std::vector<Chunk> chunks;
    };
    std::vector<Slot> slots;
    std::vector<Group> groups;
    int store_v = 0;
    int shape = 1;
    bool dirty = true;
    static constexpr int kSideStreams = 3;
    cudaStream_t side_stream[kSideStreams] = {};
    cudaEvent_t forked = nullptr, joined[kSideStreams] = {};

    ~Ensemble() {
        for (cudaStream_t x : side_stream)
            if (x) cudaStreamDestroy(x);
        for (cudaEvent_t x : joined)
            if (x) cudaEventDestroy(x);
        if (forked) cudaEventDestroy(forked);
        for (auto &s : slots)
            if (s.lat) lbm_cu_destroy(s.lat);
    }
    // Member groups of the active cavities, one per (storage, shape).
    int build_groups() {
        groups.clear();
        for (size_t i = 0; i < slots.size(); i++) {
            const Slot &s = slots[i];
            if (!s.active) continue;
            const bool pair = shape == 2 && s.spec.storage != LBM_F64 && !(s.spec.nx & 1);
            const bool staged =
                shape == 3 && (s.spec.storage == LBM_F16 || s.spec.storage == LBM_BF16 || s.spec.storage == LBM_C16);
            Group *g = nullptr;
            for (auto &x : groups)
                if (x.storage == s.spec.storage && x.pair == pair) g = &x;
            if (!g) {
                groups.emplace_back();
                g = &groups.back();
                g->storage = s.spec.storage;
                g->pair = pair;
                g->staged = staged;
            }
            g->members.push_back((int)i);
        }
        for (auto &g : groups) {
            // an ensemble of one storage type runs as two chunks, so that there
            // are two to fill each other's last waves (20 half cavities 64.2k
            // -> 70.4k MLUPS, 20 float ones 40.2k -> 41.0k)
            const size_t n = g.members.size(), parts = groups.size() == 1 ? 2 : 1;
            g.per = std::min<size_t>(kBatchLattices, (n + parts - 1) / parts);
            g.chunks.resize((n + g.per - 1) / g.per);
            for (auto &c : g.chunks) {
                c.args.reset(new BatchArgs());
                if (g.staged) c.sargs.reset(new BatchArgs());
            }
        }
        dirty = false;
        return refresh_tables();
    }

    // Descriptors with the current step-counter parities (and block
    // numbering) into the launch arguments.
    int refresh_tables() {
        for (auto &g : groups) {
            const int per = cells_per_block(g.pair);
            g.cells = 0;
            g.ragged = false;
            for (size_t c = 0; c < g.chunks.size(); c++) {
                Chunk &ch = g.chunks[c];
                BatchArgs &a = *ch.args;
                memset(&a, 0, sizeof(a));
                const size_t k0 = c * g.per, k1 = std::min(g.members.size(), k0 + g.per);
                int first = 0, tile = 0;
                const int tcells = g.staged ? staged_cells(g.storage) : 0;
                if (g.staged) memset(ch.sargs.get(), 0, sizeof(BatchArgs));
                ch.les = false;
                ch.parities = 0;
                for (size_t k = k0; k < k1; k++) {
                    const Slot &s = slots[g.members[k]];
                    LatDesc h = s.lat->h;
                    h.first_block = first;
                    h.nblocks = (int)((h.n + per - 1) / per);
                    h.parity = (int)(s.done & 1);
                    first += h.nblocks;
                    g.cells += h.n;
                    g.ragged = g.ragged || h.nx % 8;
                    if (uses_les(h)) ch.les = true;
                    a.tab[k - k0] = h;
                    a.first[k - k0] = h.first_block;
                    ch.parities |= 1 << h.parity;
                    if (g.staged) {
                        h.first_block = tile;
                        h.nblocks = (int)((h.n + tcells - 1) / tcells);
                        tile += h.nblocks;
                        ch.sargs->tab[k - k0] = h;
                        ch.sargs->first[k - k0] = h.first_block;
                    }
                }
                a.ntab = (int)(k1 - k0);
                ch.blocks = first;
                if (g.staged) ch.sargs->ntab = a.ntab;
                ch.tiles = tile;
            }
        }
        return 0;
    }

    int launch_one(const Group &g, Chunk &ch, int j, bool store, Dep dep, cudaStream_t st) {
        const bool all_alpha = ch.parities == 1 << ((j + 1) & 1);
        const bool all_beta = ch.parities == 1 << (j & 1);
        if (g.staged && (all_alpha || all_beta) && staged_pays(all_beta, g.ragged, g.cells)) {
            // every member at the same kind of step: staged tiles.  The rule's
            // cells and rows are the whole group's, whose chunks run side by side
            // and fill the chip together.  By the chunk's own (half, 100 steps): 8 x
            // 73x73x72 4.40 -> 4.82 ms, 20 x 48^3 3.30 -> 3.53, 40 x 40^3 3.89 -> 4.22, 20
            // uneven cavities 7.22 -> 7.35; of 60 ensembles none was 1 % faster
            ch.sargs->store_v = store ? store_v : 0;
            ch.sargs->store_rho = 0;
            return launch_staged_batch(g.storage, all_beta, ch.les, *ch.sargs, ch.tiles, dep, st);
        }
        ch.args->store_v = store ? store_v : 0;
        ch.args->store_rho = 0;
        return launch_tick(g.storage, g.pair, ch.les, *ch.args, ch.blocks, j, all_alpha ? 1 : all_beta ? 2 : 0, dep, st);
    }

    // k steps launched one by one, the last one storing u.  The chunks
    // hold different cavities, so each runs its steps on a stream of its own
    // between a fork from `st` and a join with it: the blocks of one fill the
    // slots that the last blocks of another's step leave.  A launch with its 31
    // KB of descriptors takes the host about 3 us.  Measured against pairs of
    // steps replayed from a graph on one stream (half float, half half, us per
    // step): 4 cavities of 24^3 9.5 -> 5.6, 4 of 32^3 13.9 -> 6.0, 16 of 40^3
    // 27.9 -> 18.4, 2 of 96^3 41.7 -> 32.2.
    int launch_steps(int64_t k, cudaStream_t st) {
        std::vector<std::pair<Group *, Chunk *>> all;
        for (auto &g : groups)
            for (auto &ch : g.chunks) all.push_back({&g, &ch});
        const size_t side = std::min<size_t>(kSideStreams, all.size() - 1);
        for (size_t q = 0; q < side; q++) {
            if (!side_stream[q]) CU(cudaStreamCreateWithFlags(&side_stream[q], cudaStreamNonBlocking));
            if (!joined[q]) CU(cudaEventCreateWithFlags(&joined[q], cudaEventDisableTiming));
        }
        if (side) {
            if (!forked) CU(cudaEventCreateWithFlags(&forked, cudaEventDisableTiming));
            CU(cudaEventRecord(forked, st));
            for (size_t q = 0; q < side; q++) CU(cudaStreamWaitEvent(side_stream[q], forked, 0));
        }
        int rc = 0;
        for (int64_t j = 0; j < k && !rc; j++)
            for (size_t q = 0; q < all.size() && !rc; q++) {
                const size_t s = q % (side + 1);
                rc = launch_one(*all[q].first, *all[q].second, (int)(j & 1), j + 1 == k, Dep{}, s ? side_stream[s - 1] : st);
            }
        for (size_t q = 0; q < side; q++) {
            CU(cudaEventRecord(joined[q], side_stream[q]));
            CU(cudaStreamWaitEvent(st, joined[q], 0));
        }
        return rc;
    }

    int64_t active_count() const {
        int64_t n = 0;
        for (auto &s : slots) n += s.active;
        return n;
    }

    // Advance every active cavity by k steps; the last step writes u.
    int tick(int64_t k, cudaStream_t st) {
        if (k <= 0 || active_count() == 0) return 0;
        // nothing here waits for the GPU: descriptors travel with the launches
        if (dirty) {
            if (build_groups()) return -1;
        } else if (refresh_tables()) {
            return -1;
        }
        if (launch_steps(k, st)) return -1;
        for (auto &s : slots)
            if (s.active) s.done += k;
        return 0;
    }

    // Steps until the first active cavity completes.
    int64_t min_remaining() const {
        int64_t m = INT64_MAX;
        for (auto &s : slots)
            if (s.active) m = std::min(m, s.spec.steps - s.done);
        return m == INT64_MAX ? 0 : m;
    }

    // Cavities that reached their step count stop taking steps.
    void retire_finished() {
        for (auto &s : slots)
            if (s.active && s.done >= s.spec.steps) {
                s.active = false;
                dirty = true;
            }
    }
};

}  // namespace lbm_rt

struct lbm_batch {
    Ensemble e;
};

struct lbm_server {
    Ensemble e;
    double budget = 0;  // bytes of HBM the resident solves may hold
    double used = 0;
    // Device blocks, one per resident solve.  A released solve's block is
    // kept for a later one, at most an eighth of the budget of them and all
    // of them within it (cudaMalloc and cudaFree of a solve's fields took a
    // tenth of a burst's time).  No block is larger than its solve's share of
    // the budget (cavity_bytes), so that solves are admitted by `used` alone.
    // The device has finished with a block when it changes hands (release).
    // A tick that finds nothing to run gives the idle ones back (server_tick),
    // and so does the server's end.
    struct Block {
        void *p;
        size_t bytes;
    };
    std::vector<Block> idle;
    double held = 0, idle_bytes = 0;  // bytes of all blocks, of the idle ones

    ~lbm_server() {
        for (auto &sl : e.slots) {
            if (sl.lat) lbm_cu_destroy(sl.lat);
            sl.lat = nullptr;
            if (sl.block) cudaFree(sl.block);
        }
        while (!idle.empty()) drop_idle(0);
    }
    void drop_idle(size_t i) {
        cudaFree(idle[i].p);
        held -= (double)idle[i].bytes;
        idle_bytes -= (double)idle[i].bytes;
        idle.erase(idle.begin() + i);
    }
    // A block of `bytes` to `most` bytes: the smallest such idle one, else a
    // new one of `bytes`.
    int take(size_t bytes, size_t most, Block *out) {
        size_t best = idle.size();
        for (size_t i = 0; i < idle.size(); i++)
            if (idle[i].bytes >= bytes && idle[i].bytes <= most &&
                (best == idle.size() || idle[i].bytes < idle[best].bytes))
                best = i;
        if (best < idle.size()) {
            *out = idle[best];
            idle_bytes -= (double)idle[best].bytes;
            idle.erase(idle.begin() + best);
            return 0;
        }
        while (!idle.empty() && held + (double)bytes > budget) drop_idle(0);
        out->bytes = bytes;
        while (cudaMalloc(&out->p, bytes) != cudaSuccess) {
            cudaGetLastError();
            if (idle.empty()) return fail("cudaMalloc of a solve's fields failed");
            drop_idle(0);
        }
        held += (double)bytes;
        return 0;
    }
    void give(Block b) {
        idle.push_back(b);
        idle_bytes += (double)b.bytes;
        while (idle_bytes > budget / 8) drop_idle(0);
    }
    int max_active = 0;
    int64_t next_id = 0;
    struct Pending {
        int64_t id;
        lbm_cavity spec;
    };
    std::deque<Pending> queue;
    std::vector<int64_t> completed;  // finished since the last poll
    std::vector<int> free_slots;
    int64_t cell_updates = 0;
};

extern "C" {

// ---------------------------------------------------------------- one lattice
int lbm_cu_run(lbm_lattice *lat, int64_t first_step, int64_t steps, void *stream) {
    if (!lat) return fail("NULL lattice");
    // every step writes u and rho of the same cells, so only the last step's
    // can be read after the run (16 of a float cell's 168 bytes)
    for (int64_t t = 0; t < steps; t++)
        if (step_lattice(lat, (int)((first_step + t) & 1), t + 1 == steps, S(stream))) return -1;
    return 0;
}

// ------------------------------------------------------------------- batch
int lbm_cu_batch_create(const lbm_cavity *cav, int count, int store_velocity, lbm_batch **out) {
    if (!cav || !out || count < 0) return fail("bad argument");
    *out = nullptr;
    lbm_batch *b = new lbm_batch();
    b->e.store_v = store_velocity ? 1 : 0;
    for (int i = 0; i < count; i++) {
        if (check_cavity(cav[i])) {
            std::string m = "cavity " + std::to_string(i) + ": " + lbm_cu_last_error();
            delete b;
            return fail(m);
        }
        Ensemble::Slot s;
        s.spec = cav[i];
        s.id = i;
        if (lbm_cu_create(cav[i].nx, cav[i].ny, cav[i].nz, cav[i].storage, b->e.store_v, 0, &s.lat)) {
            std::string m = "cavity " + std::to_string(i) + ": " + lbm_cu_last_error();
            delete b;
            return fail(m);
        }
        const lbm_params p = cavity_params(cav[i]);
        if (lbm_cu_set_params(s.lat, &p)) {
            std::string m = lbm_cu_last_error();
            lbm_cu_destroy(s.lat);
            delete b;
            return fail(m);
        }
        b->e.slots.push_back(s);
    }
    *out = b;
    return 0;
}

int lbm_cu_batch_destroy(lbm_batch *b) {
    delete b;
    return 0;
}

int lbm_cu_batch_reset(lbm_batch *b, void *stream) {
    if (!b) return fail("NULL batch");
    for (auto &s : b->e.slots) {
        if (cavity_reset(s.lat, s.spec, S(stream))) return -1;
        s.done = 0;
        s.active = s.spec.steps > 0;
    }
    b->e.dirty = true;
    CU(cudaStreamSynchronize(S(stream)));  // a run may use another stream
    return 0;
}

int lbm_cu_batch_set_kernel_shape(lbm_batch *b, int cells_per_thread) {
    if (!b) return fail("NULL batch");
    if (cells_per_thread < 1 || cells_per_thread > 3) return fail("the ensemble kernel shape is 1, 2 or 3");
    b->e.shape = cells_per_thread;
    b->e.dirty = true;
    return 0;
}

int lbm_cu_batch_run(lbm_batch *b, int64_t max_steps, int use_graph, void *stream) {
    (void)use_graph;
    if (!b) return fail("NULL batch");
    int64_t budget = max_steps < 0 ? INT64_MAX : max_steps;
    b->e.retire_finished();
    while (budget > 0 && b->e.active_count() > 0) {
        const int64_t k = std::min(budget, b->e.min_remaining());
        if (b->e.tick(k, S(stream))) return -1;
        budget -= k;
        b->e.retire_finished();
    }
    CU(cudaStreamSynchronize(S(stream)));
    return 0;
}

int lbm_cu_batch_tune(lbm_batch *b, int trial_steps, int *cells_per_thread, double *ms_per_step, void *stream) {
    if (!b || trial_steps < 1) return fail("bad argument");
    cudaStream_t st = S(stream);
    cudaEvent_t e0, e1;
    CU(cudaEventCreate(&e0));
    CU(cudaEventCreate(&e1));
    double best_ms = 1e300;
    int best = 1;
    for (int shape = 1; shape <= 3; shape++) {
        b->e.shape = shape;
        b->e.dirty = true;
        if (lbm_cu_batch_reset(b, stream)) return -1;
        if (b->e.tick(2, st)) return -1;  // warm-up (and table build)
        CU(cudaEventRecord(e0, st));
        if (b->e.tick(trial_steps, st)) return -1;
        CU(cudaEventRecord(e1, st));
        CU(cudaEventSynchronize(e1));
        float ms = 0.f;
        CU(cudaEventElapsedTime(&ms, e0, e1));
        if (ms < best_ms) {
            best_ms = ms;
            best = shape;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    b->e.shape = best;
    b->e.dirty = true;
    if (lbm_cu_batch_reset(b, stream)) return -1;
    if (cells_per_thread) *cells_per_thread = best;
    if (ms_per_step) *ms_per_step = best_ms / trial_steps;
    return 0;
}

int lbm_cu_batch_status(const lbm_batch *b, int64_t *min_done, int *active) {
    if (!b) return fail("NULL batch");
    int64_t m = INT64_MAX;
    int a = 0;
    for (auto &s : b->e.slots) {
        m = std::min(m, s.done);
        a += s.active;
    }
    if (min_done) *min_done = m == INT64_MAX ? 0 : m;
    if (active) *active = a;
    return 0;
}

lbm_lattice *lbm_cu_batch_lattice(lbm_batch *b, int index) {
    if (!b || index < 0 || index >= (int)b->e.slots.size()) {
        fail("cavity index out of range");
        return nullptr;
    }
    return b->e.slots[index].lat;
}

// ------------------------------------------------------------------ server
int lbm_cu_server_create(double hbm_budget_bytes, int max_active, int store_velocity, lbm_server **out) {
    if (!out || !(hbm_budget_bytes > 0)) return fail("bad argument");
    lbm_server *s = new lbm_server();
    s->budget = hbm_budget_bytes;
    s->max_active = max_active > 0 ? max_active : 1 << 30;
    s->e.store_v = store_velocity ? 1 : 0;
    s->e.shape = 3;  // staged tiles for large parity-uniform 16-bit launches (measured the faster)
    *out = s;
    return 0;
}

int lbm_cu_server_destroy(lbm_server *s) {
    delete s;
    return 0;
}

int lbm_cu_server_set_kernel_shape(lbm_server *s, int cells_per_thread) {
    if (!s) return fail("NULL server");
    if (cells_per_thread < 1 || cells_per_thread > 3) return fail("the ensemble kernel shape is 1, 2 or 3");
    s->e.shape = cells_per_thread;
    s->e.dirty = true;
    return 0;
}

int lbm_cu_server_submit(lbm_server *s, const lbm_cavity *c, int64_t *id) {
    if (!s || !c) return fail("NULL argument");
    if (check_cavity(*c)) return -1;
    if (cavity_bytes(*c, s->e.store_v) > s->budget) return fail("solve does not fit the HBM budget");
    lbm_server::Pending p{s->next_id++, *c};
    s->queue.push_back(p);
    if (id) *id = p.id;
    return 0;
}

// Admit queued solves in arrival order while the budget and slot limit
// allow; returns the number admitted.
static int server_admit(lbm_server *s, cudaStream_t st) {
    int admitted = 0;
    while (!s->queue.empty()) {
        const lbm_server::Pending &p = s->queue.front();
        const size_t share = cavity_bytes(p.spec, s->e.store_v);
        const double need = (double)share;
        if (s->used + need > s->budget || s->e.active_count() >= s->max_active) break;
        Ensemble::Slot slot;
        slot.spec = p.spec;
        slot.id = p.id;
        lbm_server::Block blk{};
        const size_t bytes = lattice_block_bytes(p.spec.nx, p.spec.ny, p.spec.nz, p.spec.storage, s->e.store_v);
        if (s->take(bytes, share, &blk)) return -1;
        const lbm_params prm = cavity_params(p.spec);
        if (lattice_in_block(p.spec.nx, p.spec.ny, p.spec.nz, p.spec.storage, s->e.store_v, blk.p, &slot.lat) ||
            lbm_cu_set_params(slot.lat, &prm) || cavity_reset(slot.lat, p.spec, st)) {
            lbm_cu_destroy(slot.lat);
            s->give(blk);
            return -1;
        }
        slot.block = blk.p;
        slot.block_bytes = blk.bytes;
        slot.active = p.spec.steps > 0;
        if (!slot.active) s->completed.push_back(p.id);  // nothing to run
        if (!s->free_slots.empty()) {
            s->e.slots[s->free_slots.back()] = slot;
            s->free_slots.pop_back();
        } else {
            s->e.slots.push_back(slot);
        }
        s->used += need;
        s->queue.pop_front();
        s->e.dirty = true;
        admitted++;
    }
    return admitted;
}

int lbm_cu_server_tick(lbm_server *s, int64_t max_steps, int use_graph, int *admitted, void *stream) {
    (void)use_graph;
    if (!s) return fail("NULL server");
    cudaStream_t st = S(stream);
    const int adm = server_admit(s, st);
    if (adm < 0) return -1;
    if (admitted) *admitted = adm;
    if (s->queue.empty() && s->e.active_count() == 0)
        while (!s->idle.empty()) s->drop_idle(0);
    const int64_t k = std::min(max_steps > 0 ? max_steps : INT64_MAX, s->e.min_remaining());
    if (k > 0) {
        int64_t cells = 0;
        for (auto &sl : s->e.slots)
            if (sl.active) cells += sl.lat->n;
        if (s->e.tick(k, st)) return -1;
        s->cell_updates += cells * k;
    }
    for (auto &sl : s->e.slots)
        if (sl.active && sl.done >= sl.spec.steps) {
            sl.active = false;
            s->e.dirty = true;
            s->completed.push_back(sl.id);
        }
    CU(cudaStreamSynchronize(st));
    return 0;
}

int lbm_cu_server_poll(lbm_server *s, int64_t *ids, int capacity, int *count) {
    if (!s || !count) return fail("NULL argument");
    const int n = std::min<int>(capacity, (int)s->completed.size());
    for (int i = 0; i < n; i++) ids[i] = s->completed[i];
    s->completed.erase(s->completed.begin(), s->completed.begin() + n);
    *count = n;
    return 0;
}

// The lattice of a completed (or running) solve, for readback.
lbm_lattice *lbm_cu_server_lattice(lbm_server *s, int64_t id) {
    if (!s) return nullptr;
    for (auto &sl : s->e.slots)
        if (sl.lat && sl.id == id) return sl.lat;
    fail("no resident solve with this id");
    return nullptr;
}

// Free a completed solve's device memory and return its slot.
int lbm_cu_server_release(lbm_server *s, int64_t id) {
    if (!s) return fail("NULL server");
    for (size_t i = 0; i < s->e.slots.size(); i++) {
        auto &sl = s->e.slots[i];
        if (sl.lat && sl.id == id) {
            if (sl.active) return fail("solve is still running");
            // the caller's own work on the lattice, whatever its stream, ends before the block changes hands
            CU(cudaDeviceSynchronize());
            s->used -= (double)cavity_bytes(sl.spec, s->e.store_v);
            lbm_cu_destroy(sl.lat);
            s->give({sl.block, sl.block_bytes});
            sl = Ensemble::Slot();
            s->free_slots.push_back((int)i);
            return 0;
        }
    }
    return fail("no resident solve with this id");
}

int lbm_cu_server_status(const lbm_server *s, int *queued, int *active, double *hbm_used, int64_t *cell_updates) {
    if (!s) return fail("NULL server");
    if (queued) *queued = (int)s->queue.size();
    if (active) *active = (int)s->e.active_count();
    if (hbm_used) *hbm_used = s->used;
    if (cell_updates) *cell_updates = s->cell_updates;
    return 0;
}

}  // extern "C"
