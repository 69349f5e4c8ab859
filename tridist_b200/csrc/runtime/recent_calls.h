// Calls of one rank whose plan is known: the operands are compared with those of earlier calls and the plan is
// launched without a way back through Python's checks and key (a 64 x 4096 x 1376 call took 12.7 us on the host, its
// kernel 7.6). A key holds everything that those checks and the plan depend on: addresses, sizes, strides, types and
// devices of the three tensors, and the caller's tag; while the environment forces the tile, calls go to the Python key. The plans stay the Python cache's, which drops them here too.
#pragma once
#include <torch/extension.h>

#include <array>
#include <cstdint>
#include <algorithm>
#include <unordered_map>
#include <vector>

#include "../ops/fused_gemm.h"
#include "environment.h"

namespace tdb {

class RecentCalls {
 public:
  bool launch(const at::Tensor& a, const at::Tensor& b, const at::Tensor& c, int64_t tag, uint32_t round, void* stream) {
    Key k;
    if (!key_of(a, b, c, tag, k)) return false;
    auto it = calls_.find(k);
    if (it == calls_.end()) return false;
    if (tile_forced()) return false;
    it->second.used = ++clock_;
    ++hits_;
    drained_ = false;
    gemm_plan_launch(it->second.plan, round, static_cast<int>(round & 1u), 0, 0, stream);
    return true;
  }
  void remember(const at::Tensor& a, const at::Tensor& b, const at::Tensor& c, int64_t tag, int64_t plan,
                pybind11::object cache_key) {
    Key k;
    if (!tile_forced() && key_of(a, b, c, tag, k)) calls_[k] = Call{plan, 0, std::move(cache_key)};
  }
  void forget(int64_t plan) {
    for (auto it = calls_.begin(); it != calls_.end();) it = it->second.plan == plan ? calls_.erase(it) : std::next(it);
  }
  void clear() { calls_.clear(); }
  // Keys of the plans launched from here since the last time, the least recent first.
  std::vector<pybind11::object> drain() {
    std::vector<pybind11::object> out;
    if (drained_) return out;
    drained_ = true;
    std::vector<Call*> v;
    for (auto& c : calls_)
      if (c.second.used > 0) v.push_back(&c.second);
    std::sort(v.begin(), v.end(), [](const Call* x, const Call* y) { return x->used < y->used; });
    for (Call* c : v) {
      out.push_back(c->cache_key);
      c->used = 0;
    }
    return out;
  }
  int64_t hits() const { return hits_; }

 private:
  static bool tile_forced() {      // by the environment: the Python key, which such a call goes to, looks at it every time
    bool forced = false;
    each_setting([&](const char* name, size_t n, const char* value) {
      forced = forced || (*value != 0 && n == 16 && (std::memcmp(name, "TRIDIST_FORCE_BN", 16) == 0 ||
                                                     std::memcmp(name, "TRIDIST_MAX_CTAS", 16) == 0));
    });
    return forced;
  }
  static constexpr int kWords = 19;
  struct Key {
    std::array<int64_t, kWords> w;
    bool operator==(const Key& o) const { return w == o.w; }
  };
  struct Hash {
    size_t operator()(const Key& k) const {
      uint64_t h = 1469598103934665603ull;
      for (int64_t x : k.w) h = (h ^ static_cast<uint64_t>(x)) * 1099511628211ull;
      return static_cast<size_t>(h ^ (h >> 29));
    }
  };
  struct Call {
    int64_t plan;
    uint64_t used;
    pybind11::object cache_key;
  };
  static bool key_of(const at::Tensor& a, const at::Tensor& b, const at::Tensor& c, int64_t tag, Key& k) {
    int i = 0;
    for (const at::Tensor* t : {&a, &b, &c}) {
      if (t->dim() != 2 || !t->is_cuda()) return false;
      k.w[i++] = reinterpret_cast<int64_t>(t->data_ptr());
      k.w[i++] = t->size(0);
      k.w[i++] = t->size(1);
      k.w[i++] = t->stride(0);
      k.w[i++] = t->stride(1);
      k.w[i++] = static_cast<int64_t>(t->scalar_type()) * 256 + t->get_device();
    }
    k.w[i] = tag;
    return true;
  }
  std::unordered_map<Key, Call, Hash> calls_;
  uint64_t clock_ = 0;
  int64_t hits_ = 0;
  bool drained_ = true;      // nothing launched from here since the last drain
};

}  // namespace tdb
