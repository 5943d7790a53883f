// Host helpers of the plan compilers: keys of input tables, label look-up and
// a flat hash map.  A call's tables (lattice, operator blocks, bases) are some
// 200 KB at m = 2000, and a plan looks up tens of thousands of labels.
#pragma once
#include <cstdint>
#include <cstring>
#include <vector>

namespace tjb {

// Key of n bytes, chained onto h: 8 bytes a step in four independent lanes (a
// byte at a time, the tables of one H*psi call took 390 us of its 1.26 ms in
// split precision on the 4x24 m = 2000 superblock, now 15).  Every step is a
// bijection of its lane for given input: an xor, degski's multiplier and a
// shift; the lanes start 2^64 / the golden ratio apart (as splitmix64 counts).
inline uint64_t key_bytes(uint64_t h, const void *p, size_t n) {
  constexpr uint64_t K = 0x9e3779b97f4a7c15ull;
  auto step = [](uint64_t a, uint64_t w) {
    a = (a ^ w) * 0xd6e8feb86659fd93ull;
    return a ^ (a >> 32);
  };
  const unsigned char *c = (const unsigned char *)p;
  auto word = [&](size_t at) {
    uint64_t w;
    std::memcpy(&w, c + at, 8);
    return w;
  };
  uint64_t a[4] = {h, h + K, h + 2 * K, h + 3 * K};
  size_t i = 0;
  for (; i + 32 <= n; i += 32)
    for (int q = 0; q < 4; ++q) a[q] = step(a[q], word(i + 8 * q));
  for (; i + 8 <= n; i += 8) a[0] = step(a[0], word(i));
  uint64_t tail = 0;
  if (i < n) std::memcpy(&tail, c + i, n - i);
  h = step(a[0], tail);
  for (int q = 1; q < 4; ++q) h = step(h, a[q]);
  return step(h, (uint64_t)n);
}

// Index of the first entry with three integer labels, label(k) = {a, b, c} of
// entry k.
class LabelIndex {
 public:
  template <class F>
  void build(int n, F label) {
    size_t cap = 16;
    while (cap < (size_t)n * 2) cap *= 2;
    mask_ = cap - 1;
    slot_.assign(cap, Entry{0, 0, 0, -1});
    for (int k = 0; k < n; ++k) {
      int l[3];
      label(k, l);
      size_t at = hash(l[0], l[1], l[2]) & mask_;
      while (slot_[at].k >= 0 && !(slot_[at].a == l[0] && slot_[at].b == l[1] && slot_[at].c == l[2])) at = (at + 1) & mask_;
      if (slot_[at].k < 0) slot_[at] = Entry{l[0], l[1], l[2], k};
    }
  }
  bool built() const { return !slot_.empty(); }
  int find(int a, int b, int c) const {
    for (size_t at = hash(a, b, c) & mask_;; at = (at + 1) & mask_) {
      const Entry &e = slot_[at];
      if (e.k < 0) return -1;
      if (e.a == a && e.b == b && e.c == c) return e.k;
    }
  }

 private:
  struct Entry {
    int a, b, c, k;
  };
  // the labels times the first three 32-bit primes of xxHash
  static size_t hash(int a, int b, int c) {
    uint64_t h = ((uint64_t)(uint32_t)a * 0x9e3779b1u) ^ ((uint64_t)(uint32_t)b * 0x85ebca77u) ^ ((uint64_t)(uint32_t)c * 0xc2b2ae3du);
    return (size_t)(h ^ (h >> 15));
  }
  std::vector<Entry> slot_;
  size_t mask_ = 0;
};

// Map from Key (with ==) to V in one open-addressed array; no erasure.
template <class Key, class V, class Hash>
class FlatMap {
 public:
  explicit FlatMap(size_t expect = 1024) {
    size_t cap = 16;
    while (cap < expect * 2) cap *= 2;
    slot_.resize(cap);
  }
  // the value of key, or null
  V *find(const Key &k) {
    Slot &s = slot_[place(k)];
    return s.used ? &s.v : nullptr;
  }
  void emplace(const Key &k, const V &v) {
    if ((n_ + 1) * 2 > slot_.size()) {
      std::vector<Slot> old;
      old.swap(slot_);
      slot_.resize(old.size() * 2);
      for (const Slot &s : old)
        if (s.used) slot_[place(s.k)] = s;
    }
    Slot &s = slot_[place(k)];
    if (s.used) return;
    s = Slot{k, v, true};
    ++n_;
  }

 private:
  struct Slot {
    Key k{};
    V v{};
    bool used = false;
  };
  size_t place(const Key &k) const {
    uint64_t h = Hash()(k);
    h = (h ^ (h >> 32)) * 0x9e3779b97f4a7c15ull;
    size_t at = (size_t)(h >> 20) & (slot_.size() - 1);
    while (slot_[at].used && !(slot_[at].k == k)) at = (at + 1) & (slot_.size() - 1);
    return at;
  }
  std::vector<Slot> slot_;
  size_t n_ = 0;
};

}  // namespace tjb
