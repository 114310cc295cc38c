// Fork and join of a second stream beside the context's, within the capture
// of a step graph.  Every call's status is looked at: work is issued to the side
// stream only after the fork that makes it part of the capture, and any
// failure is returned, so that the caller drops the capture.
//
// R gives the runtime calls, each returning an error code, 0 for success:
// stream(Stream*), event(Event*), record(Event, Stream), wait(Stream, Event)
// and the destructors drop(Stream), drop(Event).
#pragma once

#include <utility>

namespace fipi {

// Fork and join events of the step's two branches.
template <class Event> struct BranchEvents {
    Event fork[2] = {}, join[2] = {};
};

template <class R, class Stream, class Event> void drop_branches(R& rt, Stream& side, BranchEvents<Event>& ev) {
    for (Event* e : {&ev.fork[0], &ev.fork[1], &ev.join[0], &ev.join[1]}) {
        if (*e) rt.drop(*e);
        *e = Event{};
    }
    if (side) rt.drop(side);
    side = Stream{};
}

// The side stream and its events: all of them, or none and the first error.
template <class R, class Stream, class Event> int make_branches(R& rt, Stream& side, BranchEvents<Event>& ev) {
    int e = rt.stream(&side);
    if (e) side = Stream{};
    for (Event* x : {&ev.fork[0], &ev.fork[1], &ev.join[0], &ev.join[1]})
        if (!e && (e = rt.event(x)) != 0) *x = Event{};
    if (e) drop_branches(rt, side, ev);
    return e;
}

// The forks and joins of one step; err: the first error, after which the rest
// of the step stays on `main`.
template <class R, class Stream, class Event> struct StepBranches {
    R& rt;
    Stream &main, &side;
    BranchEvents<Event>& ev;
    int err = 0;
    // Runs f with `main` replaced by the side stream, which waits for main's work
    // so far.
    template <class F> void fork(int k, F&& f) {
        if (!err) err = rt.record(ev.fork[k], main);
        if (!err) err = rt.wait(side, ev.fork[k]);
        if (err) {
            f();
            return;
        }
        std::swap(main, side);
        f();
        std::swap(main, side);
        err = rt.record(ev.join[k], side);
    }
    // main waits for the work of fork k.
    void join(int k) {
        if (!err) err = rt.wait(main, ev.join[k]);
    }
};

}  // namespace fipi
