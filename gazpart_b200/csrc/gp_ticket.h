// gp_ticket.h -- the host's record of the gather's work counter.
//
// A gather's warps take their work from a counter that has to be zero when it starts.  The
// integrate that follows takes it back to zero on its way (a clearing launch of its own costs
// each step 2 us), so a gather whose integrate was never enqueued, an error having come
// between them, leaves it used up: the next gather would find no work, and its integrate
// would advance the particles with the fluid of the call before.
#pragma once

namespace gp {

class GatherTicket {
 public:
  // A gather is about to be enqueued; true: clear the counter first.
  bool take() {
    const bool stale = used_;
    used_ = true;
    return stale;
  }
  // Its integrate has been enqueued, or the counter cleared.
  void paired() { used_ = false; }
  // Whether a gather was left without its integrate.
  bool stale() const { return used_; }

 private:
  bool used_ = false;
};

}  // namespace gp
