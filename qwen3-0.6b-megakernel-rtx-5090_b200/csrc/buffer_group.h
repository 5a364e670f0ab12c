// Buffers that are used together: all of them, or none.  A caller that is refused memory half-way may come back; what is made by
// then must not read as the whole.  (Plain C++: the allocator is the caller's.)
#ifndef QMK_BUFFER_GROUP_H_
#define QMK_BUFFER_GROUP_H_

#include <cstddef>

namespace qmk_tc {
struct Buffer {
  void **at;            // null until the group exists
  std::size_t bytes;
};
template <std::size_t N, typename Drop>
void drop_all(const Buffer (&buffers)[N], Drop drop) {
  for (const Buffer &b : buffers)
    if (*b.at) { drop(*b.at); *b.at = nullptr; }
}
// `make(at, bytes)` returns `ok` or an error; the first error, behind which every pointer is null again, or `ok`.
template <typename Error, std::size_t N, typename Make, typename Drop>
Error make_all(const Buffer (&buffers)[N], Error ok, Make make, Drop drop) {
  for (const Buffer &b : buffers) {
    const Error e = make(b.at, b.bytes);
    if (e == ok) continue;
    *b.at = nullptr;
    drop_all(buffers, drop);
    return e;
  }
  return ok;
}
}  // namespace qmk_tc

#endif  // QMK_BUFFER_GROUP_H_
