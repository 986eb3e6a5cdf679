// sparse_heap.h -- the part of the reference's selection heap that can decide
// a pick.
//
// The reference pops a lazy std::priority_queue over every vertex's (vertex,
// count) (streaming_find_most_influential.h:546-572).  Keys only fall, so an
// item whose count at the start is below K can only come to the top once every
// key is below K.  How the items below K lie among each other never moves an
// item of K or more: pop_heap and push_heap compare them with the strict
// "less", in which all of them are equally small against any item of K or
// more, and a path that runs into them ends among them.  So the items of K or
// more keep exactly the positions they have in the full heap when every other
// position only counts as "small", and as no parent is smaller than its child a
// path ends at the first small position.  This heap keeps those items only: the
// first positions in an array a few times their number (some 16 000 items and
// 2^16 positions stay in L2; the full array of 2^24 items is 128 MB), the few
// that lie deeper in a hash table.  Or it is the full heap, in an array of its
// caller's.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <vector>

// The reference's heap holds std::pair<vertex, size_t count> ordered by count
// alone (CompareHeap, include/ripples/streaming_find_most_influential.h:410-418).
// The heap algorithms only move elements and compare them with the
// comparator, so an 8-byte item with the same comparison yields the same
// sequence of heaps (counts never exceed the number of sets, < 2^32).
struct HeapItem {
  uint32_t first;   // vertex
  uint32_t second;  // count when pushed
  bool operator==(const HeapItem &o) const { return first == o.first && second == o.second; }
};
struct CompareHeap {
  bool operator()(const HeapItem &a, const HeapItem &b) const { return a.second < b.second; }
};

class SparseHeap {
 public:
  // The heap of `len` positions that keeps R items, id 0 .. R-1, with these
  // keys (one or more) and positions.
  void build(size_t len, uint32_t R, const uint32_t *key, const uint32_t *pos) {
    all_ = nullptr;
    len_ = len;
    size_t low = 1u << 14;
    while (low < len && low < 4 * (size_t)R) low *= 2;
    low_.assign(low < len ? low : len, HeapItem{0, 0});
    deep_.assign(64, Deep{0, {0, 0}});
    used_ = 0;
    for (uint32_t i = 0; i < R; ++i) put(pos[i], HeapItem{i, key[i]});
  }
  // The full heap of `len` items, whose ids are the first halves; the array stays
  // the caller's and in use.
  void adopt(HeapItem *items, size_t len) {
    all_ = items;
    len_ = len;
  }
  bool all() const { return all_ != nullptr; }  // whether it is the full heap

  size_t size() const { return len_; }
  bool top_kept() const { return len_ && (all_ || low_[0].second); }
  uint32_t top_id() const { return all_ ? all_[0].first : low_[0].first; }
  uint32_t top_key() const { return all_ ? all_[0].second : low_[0].second; }
  // The items keyed at least T (one or more; keys never grow downwards, so subtrees
  // whose root is keyed below T are skipped), breadth first: their ids, and their
  // vertices (vertex: by id, null: the id itself).  Returns the count, or cap + 1
  // when more than cap items qualify.
  uint32_t collect(uint32_t T, uint32_t cap, const uint32_t *vertex, uint32_t *ids,
                   uint32_t *vertices, std::vector<uint32_t> &pos) const {
    pos.resize(cap);
    if (all_) return collect_in(all_, len_, T, cap, vertex, ids, vertices, pos.data());
    // the hash table is looked up only for children of the array's last items
    const size_t low = low_.size() < len_ ? low_.size() : len_;
    if (!used_) return collect_in(low_.data(), low, T, cap, vertex, ids, vertices, pos.data());
    return collect_in(*this, len_, T, cap, vertex, ids, vertices, pos.data());
  }

  // std::pop_heap and pop_back of the full heap.
  void pop() {
    if (all_) {
      pop_all();
      return;
    }
    const HeapItem last = get(len_ - 1);
    if (last.second) put(len_ - 1, HeapItem{0, 0});
    const size_t len = --len_;
    if (len == 0) return;
    // the hole sinks along the larger child (the right one unless the left is
    // strictly larger) until both are small
    HeapItem *h = low_.data();
    const size_t low = low_.size() < len ? low_.size() : len;
    size_t hole = 0;
    bool small = false;
    for (size_t r = 2; r < low; r = 2 * hole + 2) {  // both children in the array
      const size_t c = r - (h[r].second < h[r - 1].second);
      if (!h[c].second) {
        small = true;
        break;
      }
      h[hole] = h[c];
      hole = c;
    }
    while (!small) {
      size_t c = 2 * hole + 1;
      if (c >= len) break;
      HeapItem x = get(c);
      if (c + 1 < len) {
        const HeapItem r = get(c + 1);
        if (!(r.second < x.second)) {
          x = r;
          ++c;
        }
      }
      if (!x.second) break;
      put(hole, x);
      hole = c;
    }
    rise(hole, last);
  }
  // push_back and std::push_heap of the full heap (an item that is not kept is
  // small from now on).
  void push(uint32_t id, uint32_t key, bool keep) {
    const size_t at = len_++;
    if (all_) {
      rise_all(at, HeapItem{id, key});
      return;
    }
    if (!keep) return;
    // through small items to below the last kept one of its path
    size_t hole = at;
    if (hole >= low_.size()) {
      size_t p = hole;
      while (p >= low_.size()) p = (p - 1) / 2;
      if (!low_[p].second) hole = p;  // then all below it are small too
    }
    rise(hole, HeapItem{id, key});
  }

 private:
  struct Deep {
    uint32_t at;  // position + 1, 0: free
    HeapItem item;
  };
  HeapItem operator[](size_t p) const { return get(p); }
  template <class Items>
  static uint32_t collect_in(const Items &h, size_t len, uint32_t T, uint32_t cap,
                             const uint32_t *vertex, uint32_t *ids, uint32_t *vertices,
                             uint32_t *pos) {
    uint32_t cnt = 0;
    auto look = [&](size_t p) {
      const HeapItem x = h[p];
      if (x.second < T) return true;
      if (cnt == cap) return false;
      pos[cnt] = (uint32_t)p;
      ids[cnt] = x.first;
      vertices[cnt++] = vertex ? vertex[x.first] : x.first;
      return true;
    };
    if (len && !look(0)) return cap + 1;
    for (uint32_t head = 0; head < cnt; ++head) {
      const size_t l = 2 * (size_t)pos[head] + 1;
      if (l < len && !look(l)) return cap + 1;
      if (l + 1 < len && !look(l + 1)) return cap + 1;
    }
    return cnt;
  }
  // std::pop_heap and pop_back, std::push_heap on the full heap: the steps below,
  // the children's comparison without a branch (its outcome is as good as random)
  // and the lines three levels down on their way.
  void pop_all() {
    HeapItem *h = all_;
    const HeapItem last = h[len_ - 1];
    const size_t len = --len_;
    if (len == 0) return;
    size_t hole = 0;
    for (size_t r = 2; r < len; r = 2 * hole + 2) {
      const size_t c = r - (h[r].second < h[r - 1].second);
      __builtin_prefetch(h + 8 * hole + 10);
      h[hole] = h[c];
      hole = c;
    }
    if (2 * hole + 1 < len) {  // a left child alone (r == len)
      h[hole] = h[2 * hole + 1];
      hole = 2 * hole + 1;
    }
    rise_all(hole, last);
  }
  void rise_all(size_t hole, HeapItem v) {
    HeapItem *h = all_;
    while (hole > 0 && h[(hole - 1) / 2].second < v.second) {
      h[hole] = h[(hole - 1) / 2];
      hole = (hole - 1) / 2;
    }
    h[hole] = v;
  }
  HeapItem get(size_t p) const {
    if (p < low_.size()) return low_[p];
    if (!used_) return HeapItem{0, 0};
    const size_t mask = deep_.size() - 1;
    for (size_t i = slot(p, mask);; i = (i + 1) & mask) {
      if (deep_[i].at == (uint32_t)p + 1) return deep_[i].item;
      if (!deep_[i].at) return HeapItem{0, 0};
    }
  }
  void put(size_t p, HeapItem x) {
    if (p < low_.size()) {
      low_[p] = x;
      return;
    }
    const size_t mask = deep_.size() - 1;
    size_t i = slot(p, mask);
    while (deep_[i].at && deep_[i].at != (uint32_t)p + 1) i = (i + 1) & mask;
    if (!deep_[i].at) {
      if (!x.second) return;  // small already
      deep_[i].at = (uint32_t)p + 1;
      ++used_;
    }
    deep_[i].item = x;
    if (2 * used_ > deep_.size()) {  // a larger table, without what became small
      std::vector<Deep> old(4 * deep_.size(), Deep{0, {0, 0}});
      old.swap(deep_);
      used_ = 0;
      for (const Deep &d : old)
        if (d.at && d.item.second) put(d.at - 1, d.item);
    }
  }
  static size_t slot(size_t p, size_t mask) { return (p * 0x9E3779B1u >> 7) & mask; }
  void rise(size_t hole, HeapItem v) {
    while (hole > 0) {
      const size_t p = (hole - 1) / 2;
      const HeapItem x = get(p);
      if (!(x.second < v.second)) break;
      put(hole, x);
      hole = p;
    }
    put(hole, v);
  }
  HeapItem *all_ = nullptr;    // the full heap
  std::vector<HeapItem> low_;  // second: the key, 0: small
  std::vector<Deep> deep_;
  size_t used_ = 0, len_ = 0;
};
