// Which wait record a call of the allocation-free entry point takes.  The records live in the library's built-in device array
// and a call needs one that is clear when its kernels start (a tripped one makes every wait give up).  The reader
// wants the last call's, and no call may pay for a launch that only clears.
//
//   A call of one launch takes records 0 and 1 in turn: its kernel clears all the others, once the call before has finished,
//   so the next call finds a clear one.
//   A call of two launches clears all of them in the first and uses one in the second.
//   A captured call cannot take turns: its launches are replayed as they are, any number of times, between any other calls.
//   It has record 2 to itself, cleared by a memset in front where there is only one launch.
//
// Every call clears the records it does not use, so at most one is set and the reader looks at all of them.
#pragma once

#include <stdint.h>

namespace catccos {

constexpr uint32_t kWaitRecords = 3;

struct WaitRecordTurn {
    uint32_t last = 0;  // the record of the last call that was launched directly

    uint32_t one_launch(bool captured)
    {
        if (captured) {
            return 2;
        }
        last ^= 1u;
        return last;
    }

    uint32_t two_launches(bool captured) const { return captured ? 2u : last; }
};

}  // namespace catccos
