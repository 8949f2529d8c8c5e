// A small table of values computed from their arguments (encoded tensor maps). Host code, no CUDA.
#pragma once
#include <stdint.h>
#include <string.h>

namespace pb {

// Open addressing over kSlots entries, looked up by ALL bytes of the key (a plain struct without padding, or with
// its padding cleared). A key lives in one of the kProbe slots from the one its hash names; when all of those hold
// other keys, the one used longest ago makes room. Two thirds full (the 162 maps of an 80-layer model in 256 slots)
// nothing is evicted; with more keys than slots the most recently used ones stay. A value never goes stale: it is a
// pure function of its key.
template <typename Key, typename Value, int kSlots, int kProbe>
class ArgTable {
  static_assert((kSlots & (kSlots - 1)) == 0 && kProbe <= kSlots && sizeof(Key) % 8 == 0, "power of two; keys hashed in words");

 public:
  // The value stored for `key`, or NULL. `hash` is what put() wants for the same key.
  const Value* find(const Key& key, uint64_t* hash) {
    uint64_t words[sizeof(Key) / 8], h = 0;
    memcpy(words, &key, sizeof(Key));
    for (uint64_t w : words) {
      h = (h ^ w) * 0x9e3779b97f4a7c15ull;
      h ^= h >> 32;
    }
    *hash = h | 1;  // 0 marks an empty slot
    for (int i = 0; i < kProbe; ++i) {
      const int s = at(*hash, i);
      if (!hash_[s]) return nullptr;
      if (hash_[s] == *hash && memcmp(&slot_[s].key, &key, sizeof(Key)) == 0) {
        used_[s] = ++now_;
        return &slot_[s].value;
      }
    }
    return nullptr;
  }
  void put(const Key& key, uint64_t hash, const Value& value) {
    int best = at(hash, 0);
    for (int i = 0; i < kProbe; ++i) {
      const int s = at(hash, i);
      if (!hash_[s]) {
        best = s;
        break;
      }
      if (used_[s] < used_[best]) best = s;
    }
    hash_[best] = hash;
    used_[best] = ++now_;
    slot_[best].key = key;
    slot_[best].value = value;
  }

 private:
  static int at(uint64_t hash, int i) { return (int)(((hash >> 8) + i) & (kSlots - 1)); }
  struct Slot {
    Key key;
    Value value;
  };
  uint64_t hash_[kSlots] = {}, used_[kSlots] = {}, now_ = 0;
  Slot slot_[kSlots];
};

}  // namespace pb
