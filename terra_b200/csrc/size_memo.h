// Answers of a rule on sizes, kept per thread: a model of a few dozen plans takes 1 to 3 us of host time, as much as a launch, and a program
// asks for the same few sizes again and again. A table of fixed length; a slot holds the last sizes that fell on it.
#pragma once
#include <stdint.h>

#include <array>

namespace tb {

template <class Value, int KEYS, int SLOTS = 128>
class SizeMemo {
 public:
  template <class Compute>
  const Value& get(const std::array<long long, KEYS>& key, Compute compute) {
    uint64_t h = 0;
    for (const long long k : key) h = (h ^ static_cast<uint64_t>(k)) * 0x9E3779B97F4A7C15ull;
    Slot& s = slots_[(h >> 40) % SLOTS];
    if (!s.used || s.key != key) {
      s.value = compute();
      s.key = key;
      s.used = true;
    }
    return s.value;
  }

 private:
  struct Slot {
    std::array<long long, KEYS> key{};
    Value value{};
    bool used = false;
  };
  std::array<Slot, SLOTS> slots_{};
};

}  // namespace tb
