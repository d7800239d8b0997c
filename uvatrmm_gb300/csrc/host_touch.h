// Which pages of the host's memory a copy of lines touches (host code only).
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace uvt {

// The part of line l, in bytes, that a copy of `width`-byte lines of doubles
// takes.  tri: 0 all of it; 1 from element l on (the lower triangle of a
// column-major square matrix); 2 up to element l (the upper one).
struct LinePart {
  size_t lo, hi;
};
inline LinePart line_part(size_t width, size_t l, int tri) {
  const size_t at = l * sizeof(double), next = at + sizeof(double);
  return {tri == 1 ? (at < width ? at : width) : 0, tri == 2 && next < width ? next : width};
}

// Calls f(address) for one byte of every page (of `page` bytes, a power of two)
// that the lines' parts lie on, always a byte of a part, in rising order (once
// per page as long as the parts of a page follow each other).
template <class F>
void for_each_page(uintptr_t base, size_t pitch, size_t width, size_t lines, int tri, size_t page, F &&f) {
  uintptr_t seen = base;  // no page below this one is left
  for (size_t l = 0; l < lines;) {
    const LinePart p = line_part(width, l, tri);
    const uintptr_t begin = base + l * pitch + p.lo, end = base + l * pitch + p.hi;
    ++l;
    for (uintptr_t a = begin > seen ? begin : seen; a < end; a = seen) {
      f(a);
      seen = (a | (page - 1)) + 1;
      const size_t next = (seen - base) / pitch;  // the lines before it lie below `seen`
      if (next > l) l = next;
    }
  }
}

}  // namespace uvt
