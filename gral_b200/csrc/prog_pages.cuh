// prog_pages.cuh -- first touch of a call's result arrays.
#pragma once

#include <cstddef>
#include <initializer_list>

namespace gral {

struct HostRange {
    void *p;
    size_t bytes;
};

// Asks the system for the pages of result arrays that the caller has not touched yet, on a few threads, so that
// the copies from the device that follow do not take one page fault after the other (about 1 us each on
// a virtual machine: 8 of the 11 ms in which the set-up of a 200x180 quarter fills four new 7 MB arrays, in a
// process whose heap does not keep freed pages).
// Contents are not changed; arrays below 1 MB, calls with less than 4 MB and pages already there
// are left alone.
void first_touch(std::initializer_list<HostRange> ranges);

}  // namespace gral
