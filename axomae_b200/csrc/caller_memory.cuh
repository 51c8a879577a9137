/* When a call may work in the caller's device memory itself instead of in a copy of its own: host code,
 * plain values in and out. */
#pragma once

#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <numeric>
#include <vector>

namespace nb {

/* True for memory of `device` itself.  A copy also takes another GPU's memory, without peer access, and host
 * memory; a kernel's load or store there would be an illegal address and cost the caller its context. */
inline bool on_device(const cudaPointerAttributes &a, int device) {
  return a.type == cudaMemoryTypeDevice && a.device == device;
}

struct Span {
  uintptr_t begin;
  size_t bytes;
  bool here; /* on_device of the GPU that does the work */
  uintptr_t end() const { return begin + bytes; }
};

inline bool overlap(const Span &a, const Span &b) { return a.begin < b.end() && b.begin < a.end(); }

/* Per film of a call (begin 0: none): 1 where the kernel that finishes it may store to it.  Its stores are
 * 16 bytes wide.  Films that share memory keep a buffer each until they are copied out, in the order of the
 * frames: a program that takes every frame's film to the host may pass one device buffer for all. */
inline std::vector<char> direct_films(const std::vector<Span> &films) {
  std::vector<char> direct(films.size());
  for (size_t j = 0; j < films.size(); j++) direct[j] = films[j].here && films[j].begin != 0 && (films[j].begin & 15u) == 0;
  std::vector<size_t> at(films.size()); /* by address; `last` reaches furthest of those before */
  std::iota(at.begin(), at.end(), size_t{0});
  std::sort(at.begin(), at.end(), [&](size_t a, size_t b) { return films[a].begin < films[b].begin; });
  for (size_t k = 1, last = 0; k < at.size(); k++) {
    const Span &f = films[at[k]], &l = films[at[last]];
    if (l.begin != 0 && f.begin < l.end()) direct[at[k]] = direct[at[last]] = 0;
    if (f.end() > l.end()) last = k;
  }
  return direct;
}

}  // namespace nb
