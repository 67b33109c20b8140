// Encoded descriptors kept by what they are made of, for host code that would otherwise encode one on every call.
#pragma once

#include <stdint.h>

namespace hq {

// kPlaces entries of `Key` (hash(), operator==; a value-initialised key marks an empty place and never stands for an
// entry) and `Value`.  A key may stand in any of the kWindow places from its hash on: with one place a key, two caches
// of a model whose addresses hash alike put one another out on every token (32 layers in 128 places: some seven of
// them), although most places are free.  A full window gives up the entry that was used longest ago.
template <typename Key, typename Value, int kPlaces = 128, int kWindow = 8>
class Kept {
 public:
  // the kept value, or nullptr
  const Value* find(const Key& key) {
    const unsigned at = key.hash();
    for (int i = 0; i < kWindow; ++i) {
      Entry& e = entries_[(at + i) % kPlaces];
      if (e.key == key) { e.used = ++clock_; return &e.value; }
    }
    return nullptr;
  }
  void keep(const Key& key, const Value& value) {
    const unsigned at = key.hash();
    Entry* place = nullptr;
    for (int i = 0; i < kWindow; ++i) {
      Entry& e = entries_[(at + i) % kPlaces];
      if (place == nullptr || e.used < place->used) place = &e;        // an empty place was never used
    }
    place->key = key;
    place->value = value;
    place->used = ++clock_;
  }

 private:
  struct Entry { Key key{}; Value value{}; uint64_t used = 0; };
  Entry entries_[kPlaces];
  uint64_t clock_ = 0;
};

// what the tensor map of a cache's code planes is made of
struct PlanesKey {
  const void* base = nullptr;
  int64_t tokens = 0, planes = 0;
  int row = 0, unit = 0;
  bool operator==(const PlanesKey& o) const {
    return base == o.base && tokens == o.tokens && planes == o.planes && row == o.row && unit == o.unit;
  }
  unsigned hash() const { return (unsigned)(((uint64_t)(uintptr_t)base * 0x9E3779B97F4A7C15ull) >> 48); }
};

}  // namespace hq
