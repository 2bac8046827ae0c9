// fk_branch.h -- a side branch of a context's stream: work queued between its
// construction (fork) and join() on the side stream runs beside the stream's own;
// join() makes the stream wait for it.  Host code only: the calls go through Api, so
// that a CPU test can make them fail.
#pragma once

namespace fk {

// Api: Stream, Event, Error (0: success) and record(event, stream), wait(stream, event),
// synchronize(stream), capturing(stream), clear().
template <class Api>
class Branch {
    using Stream = typename Api::Stream;
    using Error = typename Api::Error;
    Api api_;
    Stream& current_;  // the stream that launches go to
    Stream main_, side_{};
    typename Api::Event joined_;
    bool forked_ = false, recorded_ = false;
    Error error_{};

  public:
    // side: nullptr where there is none (the work then stays in line).
    Branch(Api api, Stream& current, Stream side, typename Api::Event fork, typename Api::Event joined)
        : api_(api), current_(current), main_(current), side_(side), joined_(joined) {
        if (!side) return;
        forked_ = api_.record(fork, main_) == Error{} && api_.wait(side, fork) == Error{};
        if (!forked_) api_.clear();
    }
    // Queues f's launches (which go to the current stream) on the side stream.
    template <class F>
    void run(F f) {
        if (forked_) current_ = side_;
        f();
        current_ = main_;
        if (!forked_) return;
        error_ = api_.record(joined_, side_);
        recorded_ = error_ == Error{};
    }
    // The stream waits for the branch.  Where that cannot be queued the host waits for the side
    // stream instead, except during a capture: that fails, and so does the call.
    Error join() {
        if (!forked_) return Error{};
        if (recorded_) error_ = api_.wait(main_, joined_);
        if (error_ != Error{} && !api_.capturing(main_)) {
            api_.clear();
            error_ = api_.synchronize(side_);
        }
        return error_;
    }
};

}  // namespace fk
