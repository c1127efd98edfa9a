// cg_loop.h -- the host's side of an iteration that runs ahead on the device: batches
// of launches are queued and the state is looked at one batch behind, so that the
// device never waits for the host.  Host code only (tests/cg_loop_check.cpp).
#pragma once

namespace opx {

enum CgLook { CG_GOES_ON, CG_DONE, CG_FAILED };

// queue(k): queues batch k, false where the runtime refused a launch; look(k): waits for
// batch k and says what its state is.  Ends with false where either failed, with true
// where a batch was done or `batches` of them were queued and looked at (the iteration's
// own limit): a device that never reports the end does not hold the host.
template <class Queue, class Look> inline bool cg_batches(long batches, Queue queue, Look look) {
    for (long k = 0; k <= batches; k++) {
        if (k < batches && !queue(k)) return false;
        if (k == 0) continue;
        const CgLook l = look(k - 1);
        if (l != CG_GOES_ON) return l == CG_DONE;
    }
    return true;
}

}  // namespace opx
