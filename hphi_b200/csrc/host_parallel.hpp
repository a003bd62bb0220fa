// Host loops of plan building over several threads.
#pragma once
#include <cstdint>
#include <functional>

namespace hphi {

// f(k) for every k in [0, n), the items handed out in order of k but worked on by several threads; they
// must not depend on one another.  us: estimated microseconds of all items together; a thread
// joins for 200 of them.  An exception of an item is thrown here.  A call beside another one, or
// in a forked process, does its items alone.
void host_parallel(int64_t n, double us, const std::function<void(int64_t)> &f);

}  // namespace hphi
