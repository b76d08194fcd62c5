// The plan of a sweeper's direction chains: the schedule positions in
// (direction, level) order and each direction's level offsets, two device
// arrays that the chain kernels and the chain records need together.
#pragma once

#include <cstdint>

#include "status.hpp"

namespace tycho {

struct ChainPlan {
    uint32_t *pos = nullptr;  // schedule positions, direction by direction, level by level
    uint32_t *off = nullptr;  // n_levels + 2 offsets into them per direction

    bool made() const { return pos && off; }

    // Makes both arrays or neither: positions(p) and offsets(o) allocate and
    // fill one each (a status; p / o may be set when they fail), release(p)
    // takes one back.  Whatever fails, the plan is as before and nothing leaks.
    template <typename Positions, typename Offsets, typename Release>
    int make(Positions positions, Offsets offsets, Release release)
    {
        if (made()) return kOk;
        uint32_t *p = nullptr, *o = nullptr;
        int st = kOk;
        try {
            st = positions(p);
            if (st == kOk) st = offsets(o);
        } catch (...) {
            release(p);
            release(o);
            throw;
        }
        if (st != kOk) {
            release(p);
            release(o);
            return st;
        }
        pos = p;
        off = o;
        return kOk;
    }

    template <typename Release>
    void drop(Release release)
    {
        release(pos);
        release(off);
        pos = off = nullptr;
    }
};

}  // namespace tycho
