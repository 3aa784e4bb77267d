// icf_grow.cuh -- device arrays that share one capacity, and temporaries that
// return to their allocator whichever way a function ends.  Over an allocator
// `Mem` with alloc(void **, bytes) -> success and free(void *), so that it
// compiles without CUDA as well.
#pragma once
#include <cstddef>

// an array and its elements
template <class T>
struct icf_array {
  T **p;
  long long n;
};
template <class T>
icf_array<T> icf_of(T **p, long long n) {
  return {p, n};
}

// New arrays in place of the ones at a.p, whose contents are not kept, for a
// capacity of c.  It holds for all of them: it is zero from the first release
// until the last allocation has succeeded, so that after a failure the next call
// allocates all of them again, however few elements it needs.
template <class Mem, class Cap, class... T>
bool icf_grow_all(Mem &mem, Cap *cap, long long c, icf_array<T>... a) {
  *cap = 0;
  ((mem.free(*a.p), *a.p = nullptr), ...);
  bool ok = true;
  ((ok = ok && mem.alloc(reinterpret_cast<void **>(a.p), sizeof(T) * (size_t)a.n)), ...);
  if (ok) *cap = (Cap)c;
  return ok;
}
// of c elements each
template <class Mem, class Cap, class... T>
bool icf_grow_all(Mem &mem, Cap *cap, long long c, T **...p) {
  return icf_grow_all(mem, cap, c, icf_array<T>{p, c}...);
}

// Temporaries: alloc() registers what it gave, the destructor frees it.
template <class Mem, int MAX = 8>
struct icf_temps {
  Mem &mem;
  void *held[MAX] = {};
  int n = 0;
  explicit icf_temps(Mem &m) : mem(m) {}
  icf_temps(const icf_temps &) = delete;
  ~icf_temps() {
    while (n > 0) mem.free(held[--n]);
  }
  template <class T>
  bool alloc(T **p, long long count) {
    *p = nullptr;
    if (n == MAX || !mem.alloc(reinterpret_cast<void **>(p), sizeof(T) * (size_t)count)) return false;
    held[n++] = *p;
    return true;
  }
};
