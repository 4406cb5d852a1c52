// query_out.h — where a query's result goes.
#pragma once

namespace cc {

// A query's result straight to the host: the launch's last block writes it
// to `host` (mapped pinned memory, complete when the stream has drained) and
// clears the accumulator and the ticket, both zero before the first query.
// host nullptr: the accumulator is the result, cleared by the caller.
struct RedOut {
  unsigned *ticket = nullptr;
  long long *host = nullptr;
};

}  // namespace cc
