// alloc_group.h -- buffers that are used together: all of them allocated, or none.
//
// A pointer that is set stands for its whole group, so a group that could not be made leaves
// every pointer null: a later call then tries again, and never runs on half of it.
#pragma once
#include <cstddef>
#include <initializer_list>

namespace cfd {

struct GroupItem { void** p; size_t bytes; };

// alloc(&p, bytes) -> true on success; release(p)
template <class Alloc, class Release>
bool alloc_group(std::initializer_list<GroupItem> items, Alloc alloc, Release release) {
  for (const GroupItem& it : items) *it.p = nullptr;
  for (const GroupItem& it : items) {
    if (alloc(it.p, it.bytes)) continue;
    *it.p = nullptr;
    for (const GroupItem& q : items) {
      if (*q.p) release(*q.p);
      *q.p = nullptr;
    }
    return false;
  }
  return true;
}

}  // namespace cfd
