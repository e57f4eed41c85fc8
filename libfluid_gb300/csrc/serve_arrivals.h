// serve_arrivals.h -- whether a lone request is worth holding back for its successor (serve.cu).
#pragma once

namespace fgb {

// Requests that a client submits in a row, faster than they are served, are stepped together:
// a group made for one of them and made anew for the next costs about a third of a small
// request each time.  So where two gaps in a row were short, a request that finds the server
// idle waits for the next, 1.25 times the last gap at most.  Nobody waits otherwise: not a
// client that submits when it knows its earlier requests finished (its next request can only
// come after this one), not the first two of a stream, and not the next two after one waited
// in vain.
class Arrivals {
  public:
    static constexpr double kClose = 0.004;  // seconds: a short gap

    // A request arrives at time t; in_turn: the clients know of every earlier one that it is
    // finished.
    void arrived(double t, bool in_turn) {
        gap_ = t - last_;
        streak_ = any_ && !in_turn && gap_ < kClose ? streak_ + 1 : 0;
        last_ = t;
        any_ = true;
    }
    // Until when the last request waits for its successor if it is alone (not after its arrival:
    // it does not).
    double wait_until() const { return streak_ >= 2 ? last_ + 1.25 * gap_ : last_; }
    // It waited and none came.
    void in_vain() { streak_ = 0; }

  private:
    double last_ = 0, gap_ = 0;
    unsigned streak_ = 0;  // short gaps in a row
    bool any_ = false;
};

}  // namespace fgb
