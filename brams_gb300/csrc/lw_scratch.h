// A device buffer that a context keeps from call to call and grows on demand.
//
// A caller may capture calls in CUDA graphs of its own, and a graph keeps the
// buffer's address.  So a buffer that a captured call has used stays allocated
// until the context is closed: a call that outgrows it takes a new one and
// sets it aside.  A new one in its place is at least twice as large (and half
// of what a call wants does where it is enough to run with), so all that are
// set aside are together smaller than the one in use.
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

struct GbAlloc {
  void* (*get)(size_t bytes);  // NULL where that much cannot be had
  void (*put)(void* p);
};

class GbScratch {
 public:
  void* p = nullptr;
  size_t bytes = 0;

  // A buffer of `want` bytes, or where that cannot be had of at least `least`
  // (a solver call then makes more passes).  Under stream capture, where
  // nothing can be allocated, `least` does.  False: there is none.
  bool ensure(size_t want, size_t least, bool capturing, const GbAlloc& a) {
    const bool does = p && bytes >= least && (bytes >= want || capturing || (captured && bytes >= want / 2));
    if (!does && !grow(captured ? std::max(want, 2 * bytes) : want, least, capturing, a)) return false;
    captured |= capturing;
    return true;
  }
  void close(const GbAlloc& a) {
    for (void* q : aside) a.put(q);
    aside.clear();
    if (p) a.put(p);
    p = nullptr;
    bytes = 0;
  }

 private:
  bool captured = false;      // a captured call has used p
  std::vector<void*> aside;   // outgrown, still held by graphs

  bool grow(size_t want, size_t least, bool capturing, const GbAlloc& a) {
    if (p) {
      if (captured || capturing)
        aside.push_back(p);
      else
        a.put(p);
    }
    p = nullptr;
    bytes = 0;
    captured = false;
    for (size_t n = want;; n = std::max(n / 2, least)) {
      if ((p = a.get(n)) != nullptr) {
        bytes = n;
        return true;
      }
      if (n <= least) return false;
    }
  }
};
