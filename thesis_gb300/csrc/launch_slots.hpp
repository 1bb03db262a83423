// launch_slots.hpp -- device memory that a launch needs while it runs and that
// outlives no launch: the grid-barrier counter of a persistent kernel, the
// halo exchange buffer of the 2-D engine (launch_slots.cu).
//
// Who owns a slot, and until when:
//   * an eager launch: until the launch has ended, by an event recorded behind
//     it.  Later launches on the same stream take the slot again (they follow
//     it); one on another stream takes it only once the event has happened, or,
//     where every slot is in use, after making its stream wait for the one that
//     was given out first;
//   * a launch captured into a graph: the graph (and every executable made from
//     it) until it is destroyed, since a replay uses the same address at any
//     time.  The launches that one capture makes on one stream share a slot:
//     they follow one another in every replay, and the replays of one
//     executable follow one another;
//   * between take() and ended() the calling thread: another thread that
//     launches on the same stream in between gets another slot, so that nobody
//     clears memory between this launch's clearing and its kernel.
// A graph gives its slot back from a callback, which clears the slot's flag and
// touches nothing else.
//
// Api (Cuda in launch_slots.cu; a model of streams in the tests) has types
// Stream, Event and Capture {id (0: none), graph} and
//   int alloc(size_t, void **), void dealloc(void *),
//   int make_event(Event *), void drop_event(Event), int record(Event, Stream),
//   bool happened(Event), int wait(Stream, Event), void sync(Event),
//   int hold(graph, std::atomic<bool> *): clears the flag when the graph goes,
//   void emptied(): release() has left no slot.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <mutex>
#include <vector>

namespace st {

template <class Api>
class SlotPool {
   public:
    struct Slot {
        void *mem = nullptr;
        size_t bytes = 0;
        typename Api::Event done{};
        std::atomic<bool> graph{false};  // held by a graph
        bool leased = false;             // between take() and ended()
        bool used = false;               // done stands for a launch
        bool lost = false;               // its launch's end is unknown
        unsigned long long stream = 0;   // id of the last launch's stream (0: unknown)
        unsigned long long capture = 0;  // the capture of the last launch (0: none)
    };

    // At most `limit` slots beside those that graphs hold.
    SlotPool(Api *api, size_t limit) : api_(api), limit_(limit) {}

    // A slot of at least `bytes` for one launch on stream s, which `id` (0: none)
    // tells from every other stream of the process, or of the capture.  Every
    // take() that succeeds needs an ended().
    int take(typename Api::Stream s, unsigned long long id, const typename Api::Capture &cap, size_t bytes, Slot **out) {
        std::lock_guard<std::mutex> lock(mu_);
        Slot *best = nullptr;
        if (cap.id) {
            for (Slot *x : slots_)
                if (x->graph && !x->leased && x->capture == cap.id && id && x->stream == id && x->bytes >= bytes) best = x;
            if (best) return give(best, cap.id, out);
        } else if (id) {
            for (Slot *x : slots_)
                if (ours(x) && x->used && !x->capture && x->stream == id && x->bytes >= bytes) best = x;
            if (best) return give(best, 0, out);
        }
        size_t count = 0;
        for (Slot *x : slots_) count += !x->graph && !x->lost;
        for (Slot *x : slots_)  // given out longest ago first
            if (ours(x) && x->bytes >= bytes && (!x->used || api_->happened(x->done))) {
                best = x;
                break;
            }
        if (!best && !cap.id && count >= limit_) {
            for (Slot *x : slots_)
                if (ours(x) && x->bytes >= bytes) {
                    best = x;
                    break;
                }
            if (best) {
                if (int rc = api_->wait(s, best->done)) return rc;
            } else {
                for (Slot *x : slots_)  // none is large enough: a new one in the place of the oldest
                    if (ours(x)) {
                        drop(x);
                        break;
                    }
            }
        }
        if (!best) {
            Slot *x = new Slot;
            int rc = api_->alloc(bytes, &x->mem);
            if (!rc && (rc = api_->make_event(&x->done))) api_->dealloc(x->mem);
            if (rc) {
                delete x;
                return rc;
            }
            x->bytes = bytes;
            slots_.push_back(x);
            best = x;
        }
        if (cap.id) {
            best->graph = true;
            if (int rc = api_->hold(cap.graph, &best->graph)) {
                best->graph = false;
                return rc;
            }
        }
        best->stream = id;
        return give(best, cap.id, out);
    }

    // Behind the launch (or where it failed: the clearing may be under way).
    int ended(Slot *x, typename Api::Stream s) {
        std::lock_guard<std::mutex> lock(mu_);
        x->leased = false;
        if (x->capture) return 0;
        const int rc = api_->record(x->done, s);
        x->used = true;
        x->lost = rc != 0;
        return rc;
    }

    // Frees what no graph and no thread holds, once its launches have ended.
    void release() {
        std::lock_guard<std::mutex> lock(mu_);
        for (size_t k = slots_.size(); k-- > 0;)
            if (ours(slots_[k])) drop(slots_[k]);
        if (slots_.empty()) api_->emptied();
    }

    size_t count() {
        std::lock_guard<std::mutex> lock(mu_);
        return slots_.size();
    }

   private:
    static bool ours(const Slot *x) { return !x->graph && !x->leased && !x->lost; }

    int give(Slot *x, unsigned long long capture, Slot **out) {
        x->leased = true;
        x->capture = capture;
        slots_.erase(std::find(slots_.begin(), slots_.end(), x));
        slots_.push_back(x);
        *out = x;
        return 0;
    }

    void drop(Slot *x) {
        if (x->used) api_->sync(x->done);
        api_->drop_event(x->done);
        api_->dealloc(x->mem);
        slots_.erase(std::find(slots_.begin(), slots_.end(), x));
        delete x;
    }

    Api *api_;
    const size_t limit_;
    std::mutex mu_;
    std::vector<Slot *> slots_;  // given out longest ago first
};

}  // namespace st
