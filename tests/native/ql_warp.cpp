// A warp of 32 lanes on the host: each lane is a context of its own that runs
// to its next warp primitive before another lane goes on, in the order that
// the caller names.  Every order is one that a GPU may take.  An entry that a
// lane stores while another one reads or stores it, with no __syncwarp
// between, is counted as a race.

#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <vector>

#define __device__

namespace {

struct Warp {
    ucontext_t main, lane[32];
    std::vector<char> stack[32];
    bool done[32];
    int kind[32];  // primitive that the lane waits in: 1 syncwarp, 2 ballot
    bool vote[32];
    unsigned ballot;
    int current;
    bool diverged;
};
Warp* w;

void arrive(int kind, bool vote)
{
    const int me = w->current;
    w->kind[me] = kind;
    w->vote[me] = vote;
    swapcontext(&w->lane[me], &w->main);
}

// who touched an entry since the last __syncwarp
struct Entry {
    double value;
    unsigned readers, writers;
};
std::vector<Entry> entries;
long races;

struct Ref {
    Entry* e;
    operator double() const
    {
        const unsigned me = 1u << w->current;
        races += (e->writers & ~me) != 0;
        e->readers |= me;
        return e->value;
    }
    void operator=(double v)
    {
        const unsigned me = 1u << w->current;
        races += ((e->writers | e->readers) & ~me) != 0;
        e->writers |= me;
        e->value = v;
    }
};

struct Shared {
    Entry* p;
    Ref operator[](int i) const { return Ref{p + i}; }
};

void __syncwarp() { arrive(1, false); }

unsigned __ballot_sync(unsigned, bool vote)
{
    arrive(2, vote);
    return w->ballot;
}

int __ffs(unsigned v) { return __builtin_ffs(static_cast<int>(v)); }

double rsqrt(double x) { return 1.0 / std::sqrt(x); }

}  // namespace

#include "slq_ql.cuh"

namespace {

int g_k, g_status[32];

void lane_main()
{
    const int me = w->current;
    Entry* p = entries.data();
    g_status[me] = slq::ql_first_row(Shared{p}, Shared{p + g_k}, Shared{p + 2 * g_k}, g_k, me);
    w->done[me] = true;
    swapcontext(&w->lane[me], &w->main);
}

}  // namespace

// Lanes in the order order[0 .. 31].  Returns the warp's status, or -1 if the
// lanes met in different primitives or left at different ones.
extern "C" int ql_warp(double* d, double* e, double* z, int k, const int* order, long* raced)
{
    Warp warp;
    w = &warp;
    g_k = k;
    double* arrays[3] = {d, e, z};
    entries.clear();
    for (double* a : arrays)
        for (int i = 0; i < k; ++i) entries.push_back({a[i], 0, 0});
    races = 0;
    for (int i = 0; i < 32; ++i)
    {
        w->stack[i].resize(64 * 1024);
        w->done[i] = false;
        getcontext(&w->lane[i]);
        w->lane[i].uc_stack.ss_sp = w->stack[i].data();
        w->lane[i].uc_stack.ss_size = w->stack[i].size();
        w->lane[i].uc_link = &w->main;
        makecontext(&w->lane[i], lane_main, 0);
    }
    for (long rounds = 0; rounds < 4000000; ++rounds)
    {
        int finished = 0;
        for (int o = 0; o < 32; ++o)
        {
            const int i = order[o];
            w->current = i;
            swapcontext(&w->main, &w->lane[i]);
            finished += w->done[i];
        }
        if (finished == 32)
        {
            for (int i = 0; i < 3 * k; ++i) arrays[i / k][i % k] = entries[i].value;
            *raced = races;
            for (int i = 1; i < 32; ++i)
                if (g_status[i] != g_status[0]) return -1;
            return g_status[0];
        }
        if (finished) return -1;
        w->ballot = 0;
        for (int i = 0; i < 32; ++i)
        {
            if (w->kind[i] != w->kind[0]) return -1;
            if (w->vote[i]) w->ballot |= 1u << i;
        }
        if (w->kind[0] == 1)
            for (Entry& e : entries) e.readers = e.writers = 0;
    }
    return -1;
}
