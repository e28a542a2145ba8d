// The slot exchange's order (slot_order.h) run under a view-based model of release/acquire fences and relaxed
// accesses: a location is the list of its stores in coherence order; a relaxed load may return any store that is
// not older than what its thread knows of; a store carries what its thread knew at its last fence, and a thread
// learns what the stores it has read carry at its next fence.  A CTA is a coroutine with two lanes (of one warp) that
// know the same after a barrier; a seeded scheduler picks the next CTA after every access.
#include <ucontext.h>

#include <cstdint>
#include <cstring>
#include <random>
#include <vector>

#include "../../fastipc_gb300/csrc/slot_order.h"

namespace {

constexpr int CTAS = 3, LANES = 2, EPOCHS = 12, BUFFERS = 4, LOCS = (BUFFERS + 1) * CTAS, EMPTY = -1;
using View = std::vector<int>;
void join(View& a, const View& b) {
    for (int i = 0; i < LOCS; ++i) a[i] = a[i] > b[i] ? a[i] : b[i];
}
struct Store {
    int value;
    View view;
};
struct Lane {
    View cur = View(LOCS, 0), acq = View(LOCS, 0), rel = View(LOCS, 0);
};

struct Model {
    std::mt19937 rng;
    std::vector<Store> loc[LOCS];
    Lane lane[CTAS][LANES];
    ucontext_t main_ctx, ctx[CTAS];
    std::vector<char> stack[CTAS];
    bool over[CTAS] = {};
    int running = 0;
    bool wrong_sum = false, wrong_data = false;

    int slot(int buffer, int cta) const { return buffer * CTAS + cta; }
    int data(int cta) const { return BUFFERS * CTAS + cta; }
    void yield(int c) { swapcontext(&ctx[c], &main_ctx); }
    void store(int c, int l, int where, int v) {
        Lane& t = lane[c][l];
        View w = t.rel;
        t.cur[where] = (int)loc[where].size();
        w[where] = t.cur[where];
        join(t.acq, t.cur);
        loc[where].push_back({v, w});
        yield(c);
    }
    int load(int c, int l, int where, bool newest) {
        Lane& t = lane[c][l];
        const int last = (int)loc[where].size() - 1;
        const int i = newest ? last : std::uniform_int_distribution<int>(t.cur[where], last)(rng);
        t.cur[where] = i;
        join(t.acq, loc[where][i].view);
        const int v = loc[where][i].value;
        yield(c);
        return v;
    }
    void fence(int c, int l) {
        Lane& t = lane[c][l];
        join(t.cur, t.acq);
        t.acq = t.cur;
        t.rel = t.cur;
    }
    void barrier(int c) {
        View v = lane[c][0].cur;
        for (int l = 1; l < LANES; ++l) join(v, lane[c][l].cur);
        for (int l = 0; l < LANES; ++l) {
            join(lane[c][l].cur, v);
            join(lane[c][l].acq, v);
        }
    }
};

struct Slots {
    Model& m;
    int c, epoch;
    void fence() {
        for (int l = 0; l < LANES; ++l) m.fence(c, l);
    }
    void fence_posting() { m.fence(c, 0); }
    void post(int b) { m.store(c, 0, m.slot(b, c), epoch * 16 + c); }
    void clear(int b) { m.store(c, 0, m.slot(b, c), EMPTY); }
    bool poll(int b) {
        for (int k = 0; k < CTAS; ++k) {
            int v = EMPTY;
            for (int n = 0; v == EMPTY; ++n) v = m.load(c, k % LANES, m.slot(b, k), n > 20);
            if (v != epoch * 16 + k) m.wrong_sum = true;
        }
        return true;
    }
};

// 0: the product's order; orders that are wrong: 1 three buffers, the clear behind the last fence, the posting lanes
// alone in the first fence; 2 no fence before a post; 3 no fence after a poll
template <bool FENCE>
void run_exchange(int order, Slots& s, int e) {
    if (order == 0) {
        fipc::slot_exchange<FENCE>(s, e);
    } else if (order == 1) {
        if (FENCE) s.fence_posting();
        s.post(e % 3);
        s.poll(e % 3);
        if (FENCE) s.fence();
        s.clear((e + 2) % 3);
    } else {
        if (FENCE && order != 2) s.fence();
        s.post(e & 3);
        s.poll(e & 3);
        if (FENCE) {
            if (order != 3) s.fence();
        } else {
            s.clear((e - 1) & 3);
            s.clear((e - 2) & 3);
        }
    }
}

void cta(Model* m, int c, int order) {
    for (int e = 0; e < EPOCHS && !m->wrong_sum && !m->wrong_data; e += 2) {
        m->store(c, 1, m->data(c), e);   // a row, by a lane that does not post
        m->barrier(c);
        Slots s{*m, c, e};
        run_exchange<true>(order, s, e);
        m->barrier(c);
        for (int k = 0; k < CTAS; ++k)
            for (int l = 0; l < LANES; ++l)
                if (m->load(c, l, m->data(k), false) != e) m->wrong_data = true;
        m->barrier(c);
        s.epoch = e + 1;
        run_exchange<false>(order, s, e + 1);
        m->barrier(c);
    }
    m->over[c] = true;
    swapcontext(&m->ctx[c], &m->main_ctx);
}
void entry(uint32_t hi, uint32_t lo, int c, int order) { cta((Model*)(((uint64_t)hi << 32) | lo), c, order); }

}  // namespace

extern "C" {

// runs of the order over `seeds` schedules: bit 0: a poll took another epoch's value, bit 1: a row was not the one
// stored before the exchange, in any of them
int hc_slot_order(int order, int seeds) {
    int found = 0;
    for (int seed = 0; seed < seeds; ++seed) {
        Model m;
        m.rng.seed(seed);
        for (int i = 0; i < LOCS; ++i) m.loc[i] = {{EMPTY, View(LOCS, 0)}};
        for (int c = 0; c < CTAS; ++c) {
            m.stack[c].resize(1 << 16);
            getcontext(&m.ctx[c]);
            m.ctx[c].uc_stack.ss_sp = m.stack[c].data();
            m.ctx[c].uc_stack.ss_size = m.stack[c].size();
            m.ctx[c].uc_link = &m.main_ctx;
            const uint64_t p = (uint64_t)&m;
            makecontext(&m.ctx[c], (void (*)())entry, 4, (uint32_t)(p >> 32), (uint32_t)p, c, order);
        }
        for (;;) {
            int left[CTAS], n = 0;
            for (int c = 0; c < CTAS; ++c)
                if (!m.over[c]) left[n++] = c;
            if (!n || m.wrong_sum || m.wrong_data) break;
            const int c = left[m.rng() % n];
            swapcontext(&m.main_ctx, &m.ctx[c]);
        }
        found |= (m.wrong_sum ? 1 : 0) | (m.wrong_data ? 2 : 0);
    }
    return found;
}
}
