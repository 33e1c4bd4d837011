// A device buffer that a context keeps from call to call and grows on demand.
//
// A caller may capture calls in CUDA graphs of its own, and a graph keeps the
// buffer's address.  So a buffer that a captured call has used stays allocated
// until the context is closed: a call that outgrows it takes a new one and
// sets it aside.  A new one in its place is at least twice as large (and half
// of what a call wants does where it is enough to run with), so all that are
// set aside are together smaller than the one in use.
//
// Where the device has no room for what a call wants, the call runs with less,
// and that size is not asked for again: calls of its size and above keep the
// buffer they have, without an allocation (and its synchronisation) each.
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
    const bool runs = p && bytes >= least;
    const bool does = runs && (bytes >= want || capturing || want >= refused || (captured && bytes >= want / 2));
    if (!does && !grow(want, least, capturing, a)) return false;
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
  bool captured = false;       // a captured call has used p
  size_t refused = ~size_t(0);  // the least wanted that the device had no room for
  std::vector<void*> aside;    // outgrown, still held by graphs

  // the largest of want, want / 2, .. least above `over` that can be had
  static void* most(size_t want, size_t least, size_t over, const GbAlloc& a, size_t* n) {
    for (*n = want; *n > over; *n = std::max(*n / 2, least)) {
      if (void* q = a.get(*n)) return q;
      if (*n <= least) break;
    }
    return nullptr;
  }
  bool grow(size_t want, size_t least, bool capturing, const GbAlloc& a) {
    const bool runs = p && bytes >= least, held = captured || capturing;
    // the new buffer before the present one goes, which does where there is no room for a larger one
    size_t n = 2 * bytes;
    void* q = captured && n > want ? a.get(n) : nullptr;
    if (!q) q = most(want, least, runs ? bytes : 0, a, &n);
    if (!q && !runs && p && !held) {
      a.put(p);
      p = nullptr;
      bytes = 0;
      q = most(want, least, 0, a, &n);
    }
    if (!capturing && (!q || n < want)) refused = std::min(refused, want);
    if (!q) return runs;
    if (p && held)
      aside.push_back(p);
    else if (p)
      a.put(p);
    p = q;
    bytes = n;
    captured = false;
    if (n >= refused) refused = ~size_t(0);
    return true;
  }
};
