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
// that lie deeper in a hash table.  With K = 0 every item is kept and it is the
// full heap.
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
  // keys (K or more) and positions.
  void build(size_t len, uint32_t R, uint32_t K, const uint32_t *key, const uint32_t *pos) {
    len_ = len;
    bias_ = K == 0;
    size_t low = 1u << 14;
    while (low < len && low < 4 * (size_t)R) low *= 2;
    low_.assign(low < len ? low : len, HeapItem{0, 0});
    deep_.assign(64, Deep{0, {0, 0}});
    used_ = 0;
    for (uint32_t i = 0; i < R; ++i) put(pos[i], HeapItem{i, key[i] + bias_});
  }

  size_t size() const { return len_; }
  bool top_kept() const { return len_ && low_[0].second; }
  uint32_t top_id() const { return low_[0].first; }
  uint32_t top_key() const { return low_[0].second - bias_; }
  // Whether position p holds a kept item, its id and key.
  bool kept_at(size_t p, uint32_t &id, uint32_t &key) const {
    const HeapItem x = p < len_ ? get(p) : HeapItem{0, 0};
    id = x.first;
    key = x.second - bias_;
    return x.second != 0;
  }

  // std::pop_heap and pop_back of the full heap.
  void pop() {
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
      if (!keep) return;
    // through small items to below the last kept one of its path
    size_t hole = at;
    if (hole >= low_.size()) {
      size_t p = hole;
      while (p >= low_.size()) p = (p - 1) / 2;
      if (!low_[p].second) hole = p;  // then all below it are small too
    }
    rise(hole, HeapItem{id, key + bias_});
  }

 private:
  struct Deep {
    uint32_t at;  // position + 1, 0: free
    HeapItem item;
  };
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
  std::vector<HeapItem> low_;  // second: key + bias_, 0: small
  std::vector<Deep> deep_;
  size_t used_ = 0, len_ = 0;
  uint32_t bias_ = 1;
};
