// Which calls of a backend are replayed from a captured launch sequence.  Host code without CUDA types (Exec is the executable
// graph's handle), so that its rules can be run without a GPU.
//
// A call is known by its exact arguments.  Capturing costs 0.1 to 0.3 ms and 118 KB of device memory and a replay saves 10 to
// 30 us, so a call is captured at its third occurrence and rows of ever new addresses or lengths never are.  All calls of a deep stack
// are remembered side by side (94 layers at five batch sizes are 470), whatever their arguments hash to.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <iterator>
#include <unordered_map>

struct CallKey {
  uint32_t layer;
  size_t n_tokens;
  const void *x, *out, *ids, *w;  // the buffers a caller passed, or a tag in `ids` for the entry points that have none
  bool operator==(const CallKey &o) const {
    return layer == o.layer && n_tokens == o.n_tokens && x == o.x && out == o.out && ids == o.ids && w == o.w;
  }
};
struct CallKeyHash {
  size_t operator()(const CallKey &k) const {
    uint64_t h = k.layer;
    for (const uint64_t v : {(uint64_t)k.n_tokens, (uint64_t)k.x, (uint64_t)k.out, (uint64_t)k.ids, (uint64_t)k.w})
      h = (h ^ v) * 0x9e3779b97f4a7c15ull, h ^= h >> 29;
    return (size_t)h;
  }
};

template <class Exec>
class ReplayTable {
 public:
  static constexpr size_t MAX_GRAPHS = 512, MAX_CALLS = 4096;
  // A full table gives up a graph only when it has not been replayed for this many calls: a working set larger than the table keeps
  // what it has (the rest are plain launches) instead of capturing the same calls again and again.
  static constexpr uint64_t IDLE_CALLS = 4 * MAX_GRAPHS;
  struct Call {
    Exec exec{};  // captured, if not null
    int launches = 0;
    uint32_t seen = 0;
    uint64_t last = 0;  // number of its latest occurrence
  };

  // Counts an occurrence of `key`; the call, if it is to be replayed (captured first while exec is null), else null.
  Call *occurrence(const CallKey &key, uint32_t from) {
    now_++;
    Call *c;
    try {
      c = &calls_[key];
    } catch (...) {  // no memory to remember it: a plain launch
      return nullptr;
    }
    if (c->seen != ~0u) c->seen++;
    c->last = now_;
    if (calls_.size() >= MAX_CALLS) forget();
    if (c->exec) return c;
    return c->seen >= from && (graphs_ < MAX_GRAPHS || idle()) ? c : nullptr;
  }
  // The graph of a call that occurrence() gave.  In a full table it takes the place of one that has been idle, for which
  // `destroy` is called.
  template <class Destroy>
  void captured(Call *c, Exec exec, int launches, Destroy destroy) {
    if (graphs_ >= MAX_GRAPHS)
      if (Call *old = idle()) destroy(old->exec), old->exec = Exec{}, old->seen = 0, graphs_--;
    c->exec = exec, c->launches = launches, graphs_++;
  }
  size_t graphs() const { return graphs_; }
  size_t size() const { return calls_.size(); }
  // Destroys every graph.  The calls stay known: each is captured again at its next occurrence.
  template <class Destroy>
  void drop(Destroy destroy) {
    for (auto &kv : calls_)
      if (kv.second.exec) destroy(kv.second.exec), kv.second.exec = Exec{};
    graphs_ = 0, full_until_ = 0;
  }

 private:
  // Forgets calls without a graph that did not occur among the last MAX_CALLS / 2: at most MAX_GRAPHS + MAX_CALLS / 2 stay, so
  // that the next sweep is a thousand new calls away.
  void forget() {
    for (auto it = calls_.begin(); it != calls_.end();)
      it = !it->second.exec && it->second.last + MAX_CALLS / 2 < now_ ? calls_.erase(it) : std::next(it);
  }
  // The graph replayed longest ago, if that is long enough ago.
  Call *idle() {
    if (now_ < full_until_) return nullptr;  // nothing can have become idle since the last search
    Call *oldest = nullptr;
    for (auto &kv : calls_)
      if (kv.second.exec && (!oldest || kv.second.last < oldest->last)) oldest = &kv.second;
    if (oldest && oldest->last + IDLE_CALLS < now_) return oldest;
    full_until_ = oldest ? oldest->last + IDLE_CALLS + 1 : 0;
    return nullptr;
  }

  std::unordered_map<CallKey, Call, CallKeyHash> calls_;  // its nodes do not move
  size_t graphs_ = 0;
  uint64_t now_ = 0, full_until_ = 0;
};
