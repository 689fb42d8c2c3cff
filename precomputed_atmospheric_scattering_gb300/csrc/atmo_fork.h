// atmo_fork.h -- two passes side by side on a main and a side stream.
#ifndef ATMO_FORK_H_
#define ATMO_FORK_H_

#include "../../include/atmo/atmo.h"

namespace atmo {

// Ops: Fork() makes the side stream wait for the main one, Side() and Main()
// enqueue a pass on each (several kernels, of which a failing call may have
// enqueued some), Join() makes the main stream wait for the side one: on every
// way out, as the caller frees the passes' buffers in the main stream's order.
// Returns the first failure.
template <class Ops>
atmo_status SideBySide(Ops& ops) {
  atmo_status s = ops.Fork();
  if (s != ATMO_OK) return s;
  s = ops.Side();
  if (s == ATMO_OK) s = ops.Main();
  const atmo_status joined = ops.Join();
  return s != ATMO_OK ? s : joined;
}

}  // namespace atmo

#endif  // ATMO_FORK_H_
