// Streams, events and graphs as queues stepped in random order, over the pool of
// csrc/launch_slots.hpp.  Every launch clears its memory and later ends; the
// model fails when memory is cleared, freed or ended while another launch is
// between its clearing and its end.  argv: pool ("slots", or "ring": four slots
// in turn, remade when they are too small), seed, steps.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <random>

#include "launch_slots.hpp"

struct World {
    struct Op {
        int kind;  // 0 clear, 1 end, 2 record, 3 wait, 4 a graph's replay
        long arg, launch;  // (an event's launch: which of its records)
    };
    struct Graph {
        std::map<int, std::vector<Op>> chain;  // per captured stream
        std::vector<std::atomic<bool> *> held;
        bool alive = true;
        int pending = 0;  // replays enqueued or running
        bool running = false;
    };
    struct Replay {
        int graph;
        std::map<int, size_t> at;
    };
    std::vector<std::deque<Op>> stream;
    std::map<long, long> recorded, done;  // an event's records: enqueued, happened
    std::map<long, long> owner; // memory -> launch, while it is between clear and end
    std::map<long, size_t> size;
    std::vector<Graph> graphs;
    std::map<int, Replay> replay;  // running, by stream
    long next = 1, launches = 0;
    size_t live = 0;
    const char *fault = nullptr;

    void run(const Op &op) {
        if (op.kind == 0) {
            if (!size.count(op.arg)) fault = "freed memory cleared";
            if (owner.count(op.arg)) fault = "memory of a running launch cleared";
            owner[op.arg] = op.launch;
        } else if (op.kind == 1) {
            if (!size.count(op.arg)) fault = "a launch on freed memory";
            if (!owner.count(op.arg) || owner[op.arg] != op.launch) fault = "a launch lost its memory";
            owner.erase(op.arg);
        } else if (op.kind == 2) {
            done[op.arg] = op.launch;
        }
    }
    void drop_graph(Graph &g) {
        if (g.alive || g.pending) return;
        for (auto *f : g.held) f->store(false);
        g.held.clear();
    }
    // Advances stream k by one operation; false if it cannot.
    bool step(int k, std::mt19937 &rng) {
        if (stream[k].empty()) return false;
        const Op op = stream[k].front();
        if (op.kind == 3 && done[op.arg] < op.launch) return false;
        if (op.kind == 4) {
            Graph &g = graphs[op.arg];
            if (!replay.count(k)) {
                if (g.running) return false;  // an executable does not run beside itself
                g.running = true;
                replay[k] = {(int)op.arg, {}};
            }
            Replay &r = replay[k];
            std::vector<int> open;
            for (auto &c : g.chain)
                if (r.at[c.first] < c.second.size()) open.push_back(c.first);
            if (!open.empty()) {
                const int c = open[rng() % open.size()];
                run(g.chain[c][r.at[c]++]);
                return true;
            }
            g.running = false;
            --g.pending;
            replay.erase(k);
            drop_graph(g);
        } else {
            run(op);
        }
        stream[k].pop_front();
        return true;
    }
};

struct Model {
    typedef int Stream;
    typedef long Event;
    struct Capture {
        unsigned long long id = 0;
        int graph = -1;
    };
    World *w;
    std::mt19937 *rng;
    int alloc(size_t bytes, void **mem) {
        const long m = w->next++;
        w->size[m] = bytes;
        ++w->live;
        *mem = reinterpret_cast<void *>(m);
        return 0;
    }
    void dealloc(void *mem) {
        const long m = reinterpret_cast<long>(mem);
        if (w->owner.count(m)) w->fault = "memory of a running launch freed";
        w->size.erase(m);
        --w->live;
    }
    int make_event(Event *e) { return *e = w->next++, 0; }
    void drop_event(Event) {}
    int record(Event e, Stream s) {
        w->stream[s].push_back({2, e, ++w->recorded[e]});
        return 0;
    }
    bool happened(Event e) { return w->done[e] == w->recorded[e]; }
    int wait(Stream s, Event e) {
        w->stream[s].push_back({3, e, w->recorded[e]});
        return 0;
    }
    void sync(Event e) {
        while (!happened(e) && !w->fault)
            for (size_t k = 0; k < w->stream.size(); ++k) w->step((int)k, *rng);
    }
    int hold(int graph, std::atomic<bool> *flag) {
        w->graphs[graph].held.push_back(flag);
        return 0;
    }
    void emptied() {}
};

// Four slots in turn, all remade (freeing waits for the device) when too small.
struct Ring {
    struct Slot {
        void *mem = nullptr;
    } slot[4];
    size_t bytes = 0;
    unsigned next = 0;
    Model *api;
    Ring(Model *a, size_t) : api(a) {}
    int take(int, unsigned long long, const Model::Capture &, size_t need, Slot **out) {
        if (bytes < need) {
            bool busy = true;
            while (busy && !api->w->fault) {
                busy = false;
                for (size_t k = 0; k < api->w->stream.size(); ++k) busy |= api->w->step((int)k, *api->rng);
            }
            for (auto &s : slot) {
                if (s.mem) api->dealloc(s.mem);
                api->alloc(need, &s.mem);
            }
            bytes = need;
        }
        *out = &slot[next++ % 4];
        return 0;
    }
    int ended(Slot *, int) { return 0; }
    void release() {}
};

// kept: memory that the pool keeps for good.
template <class Pool>
int drive(unsigned seed, long steps, size_t kept) {
    std::mt19937 rng(seed);
    World w;
    w.stream.resize(8);
    Model api{&w, &rng};
    Pool pool(&api, 6);
    const bool grow = rng() % 2, captures = rng() % 2;
    const int threads = rng() % 2 ? 1 : 3;
    struct Pending {  // a host thread between take() and ended()
        typename Pool::Slot *slot = nullptr;
        int stream = 0, graph = -1;
        long launch = 0;
    } host[3];
    struct Open {
        int graph = -1;
        unsigned long long id = 0;
    } open;  // one capture at a time, over streams 6 and 7
    unsigned long long captures_made = 0;
    for (long n = 0; n < steps && !w.fault; ++n) {
        const int what = rng() % 16;
        if (what < 6) {
            Pending &h = host[rng() % threads];
            if (h.slot) {  // the launch, then its end
                World::Op op{1, reinterpret_cast<long>(h.slot->mem), h.launch};
                if (h.graph >= 0) w.graphs[h.graph].chain[h.stream].push_back(op);
                else w.stream[h.stream].push_back(op);
                pool.ended(h.slot, h.stream);
                h.slot = nullptr;
            } else {
                const int s = rng() % 8;
                Model::Capture cap;
                if (s >= 6 && open.id) cap.id = open.id, cap.graph = open.graph;
                const size_t bytes = grow ? 1 + rng() % 64 : 8;
                const unsigned long long id = s == 5 ? 0 : 100 + s;
                if (pool.take(s, id, cap, bytes, &h.slot)) return 2;
                h.stream = s;
                h.graph = cap.graph;
                h.launch = ++w.launches;
                World::Op op{0, reinterpret_cast<long>(h.slot->mem), h.launch};
                if (w.size[op.arg] < bytes) w.fault = "too small";
                if (h.graph >= 0) w.graphs[h.graph].chain[s].push_back(op);
                else w.stream[s].push_back(op);
            }
        } else if (what == 6 && captures) {
            bool busy = false;  // a capture ends when no thread is within it
            for (auto &h : host) busy |= h.slot && h.graph >= 0;
            if (!open.id) {
                w.graphs.emplace_back();
                open = {(int)w.graphs.size() - 1, ++captures_made};
            } else if (!busy) {
                open = Open();
            }
        } else if (what == 7 && !w.graphs.empty()) {
            const int g = rng() % w.graphs.size();
            if (w.graphs[g].alive && g != open.graph) {
                if (rng() % 4 == 0) {
                    w.graphs[g].alive = false;
                    w.drop_graph(w.graphs[g]);
                } else {
                    w.stream[rng() % 6].push_back({4, g, 0});
                    ++w.graphs[g].pending;
                }
            }
        } else if (what == 8 && rng() % 16 == 0) {
            pool.release();
        } else {
            for (int k = rng() % 6; k >= 0; --k) w.step(rng() % 8, rng);
        }
    }
    if (w.fault) {
        std::printf("seed %u: %s\n", seed, w.fault);
        return 1;
    }
    // idle, with every graph gone: release() leaves nothing
    for (auto &h : host)
        if (h.slot) return 0;
    for (auto &g : w.graphs)
        if (g.alive) g.alive = false, w.drop_graph(g);
    for (bool busy = true; busy;) {
        busy = false;
        for (int k = 0; k < 8; ++k) busy |= w.step(k, rng);
    }
    pool.release();
    return w.fault ? 1 : w.live > kept ? 3 : 0;
}

int main(int argc, char **argv) {
    if (argc != 4) return 9;
    const unsigned seed = std::strtoul(argv[2], nullptr, 10);
    const long steps = std::strtol(argv[3], nullptr, 10);
    return std::strcmp(argv[1], "ring") ? drive<st::SlotPool<Model>>(seed, steps, 0) : drive<Ring>(seed, steps, 4);
}
