// What the host knows about the flow table without asking the device: no entry expires before floor(), at most live_most()
// are alive.  So a submit that records flows knows whether the sweep of expired ones (filter.go:202-208) could find any, and
// leaves its launch out where it could not.
//
// A submit with filter work widens both when it begins.  They are narrowed again by what the device reports behind a batch's
// work, but a report may have been taken before the work of another batch that was in flight with it, whatever the order
// in which the two are waited for.  Batches that overlap therefore form a group, and when the last one has been waited for
// the group's reports count together: the last of them, whichever that was, has seen every insert of the group, so the
// highest live count and the lowest floor among them (and what the group's lookups can have written behind it) hold.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <climits>
#include <mutex>

// What a batch's filter work reports back to the host next to the packets (pinned, one per batch).
struct FlowReport {
    unsigned long long live; // len(f.flows)
    long long floor;         // no entry's expiry lies below this
    int error;               // inserts that found no free slot, since the table was last cleared
    uint32_t used[3];        // slots of the class's region that hold a key, live or deleted
    uint32_t dead[3];        // of those, deleted ones (reclaimed by compaction)
};

// A batch's filter work between its submit and its wait (zero to start with).
struct FlowWork {
    FlowWork *next;
    long long now; // lowest clock of its submits
    bool on, notes;
};

class FlowBounds {
  public:
    explicit FlowBounds(long long floor = 0, uint64_t live = 0) : floor_(floor), live_most_(live) {}
    static constexpr long long kTtlLeast = 30ll * 1000000000ll; // the shortest lifetime, filter.go:19-21
    static constexpr uint64_t kSweepThreshold = 4096;           // filter.go:202

    // A submit is about to record up to n flows at `now` / to look flows up.  The former returns whether the table may have
    // to be swept behind its inserts.
    bool note_begins(FlowWork &w, uint32_t n, long long now) {
        std::lock_guard<std::mutex> g(mu_);
        begins(w, now);
        w.notes = true;
        live_most_ += n;
        const bool sweep = live_most_ > kSweepThreshold && now > floor_;
        floor_ = std::min(floor_, earliest(now));
        return sweep;
    }
    void check_begins(FlowWork &w, long long now) { // a lookup keeps its flow alive: it writes an expiry too
        std::lock_guard<std::mutex> g(mu_);
        begins(w, now);
        floor_ = std::min(floor_, earliest(now));
        group_floor_ = std::min(group_floor_, earliest(now));
    }
    // Lowest expiry that work in flight beside a sweep at `now` can write.
    long long beside(long long now) {
        std::lock_guard<std::mutex> g(mu_);
        for (const FlowWork *w = first_; w; w = w->next) now = std::min(now, w->now);
        return earliest(now);
    }
    // The batch has been waited for; `report` (may be null) was taken behind all of its work.
    void over(FlowWork &w, const FlowReport *report) {
        std::lock_guard<std::mutex> g(mu_);
        if (!w.on) return;
        w.on = false;
        for (FlowWork **p = &first_; *p; p = &(*p)->next)
            if (*p == &w) {
                *p = w.next;
                break;
            }
        if (report) {
            group_live_ = std::max<uint64_t>(group_live_, report->live);
            group_floor_ = std::min(group_floor_, report->floor);
            group_reported_ = true;
        } else if (w.notes) {
            group_lost_ = true;
        }
        if (first_) return;
        if (group_reported_ && !group_lost_) {
            live_most_ = group_live_;
            floor_ = group_floor_;
        }
        new_group();
    }
    // The table has been given this content; what batches still in flight report says nothing about it.
    void set(long long floor, uint64_t live) {
        std::lock_guard<std::mutex> g(mu_);
        floor_ = floor;
        live_most_ = live;
        if (first_) group_lost_ = true;
    }
    long long floor() const { return floor_; }
    uint64_t live_most() const { return live_most_; }

  private:
    static long long earliest(long long now) { return now > LLONG_MAX - kTtlLeast ? LLONG_MAX : now + kTtlLeast; }
    void new_group() {
        group_live_ = 0;
        group_floor_ = LLONG_MAX;
        group_reported_ = group_lost_ = false;
    }
    void begins(FlowWork &w, long long now) {
        if (!w.on) {
            w = FlowWork{first_, now, true, false};
            first_ = &w;
        }
        w.now = std::min(w.now, now);
    }
    std::mutex mu_;
    FlowWork *first_ = nullptr; // in flight
    long long floor_, group_floor_ = LLONG_MAX;
    uint64_t live_most_, group_live_ = 0;
    bool group_reported_ = false, group_lost_ = false;
};
