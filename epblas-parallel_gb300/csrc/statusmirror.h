// What a host thread knows of the bounded-wait failures of a device.
//
// The device stamps a mapped word (the mirror) whenever a kernel gives up on a
// wait; nobody clears it, so that no thread can take a failure away from another
// one. A thread compares the mirror with what it read before its first launch
// since its last check: a stamp in between may be its own kernel's, and it
// reports it. (A thread may then report a failure of another thread's kernel
// that ran at the same time; none goes unreported.) Plain C++: unit-tested on
// the host.
#pragma once
#include <stdint.h>

namespace mw {

struct StatusWatch {
    uint64_t seen = 0;
    bool open = false;   // work may have been launched since the last check
    // before a launch: `now` is the mirror
    void begin(uint64_t now)
    {
        if (open) return;
        seen = now;
        open = true;
    }
    // after a synchronisation with all of the thread's work: the code of a wait
    // that gave up since begin, or 0
    int check(uint64_t now)
    {
        const int code = open && now != seen ? (int)(now & 0xFF) : 0;
        seen = now;
        open = false;
        return code;
    }
};

}  // namespace mw
