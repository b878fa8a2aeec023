// Data of a basis that a first call builds and later calls use.
#pragma once

namespace cqf {

// slot = what make(&p) allocated and fill(p) wrote, unless it is there already.
// E is a status type, `ok` its success.  The pointer is published only after
// both have succeeded, and given to drop(p) when fill has not: a later call
// never takes memory that nothing has written.
template <class T, class E, class Make, class Fill, class Drop>
E build_once(T*& slot, E ok, Make make, Fill fill, Drop drop) {
  if (slot) return ok;
  T* p = nullptr;
  E e = make(&p);
  if (e != ok) return e;
  e = fill(p);
  if (e != ok) {
    drop(p);
    return e;
  }
  slot = p;
  return ok;
}

}  // namespace cqf
