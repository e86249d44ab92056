// launch_state.cuh -- what the library keeps per kernel between launches: the
// dynamic shared-memory limit it has raised and the cluster size it can be launched
// with.  Both are attributes of a kernel ON A DEVICE (another device starts with its
// own defaults), and the library is called from several threads, so the records are
// keyed by (device, kernel) and locked.  Host only, no CUDA calls: the caller passes
// the call to make.
#pragma once
#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace gfk {

template <typename V>
class KernelRecord {
 public:
  // update(v) under the lock, v the record of (device, kernel), V() at first
  template <class F>
  auto with(int device, const void *kernel, F update) {
    std::lock_guard<std::mutex> lock(m_);
    return update(rec_[{device, kernel}]);
  }

 private:
  std::mutex m_;
  std::map<std::pair<int, const void *>, V> rec_;
};

// The limit of (device, kernel) is at least `bytes` on return of true.  set(bytes)
// raises it; it is called only upwards, so that a thread about to launch with a
// larger amount keeps its limit, and recorded only when it succeeds.
template <class SET>
inline bool raise_smem_limit(KernelRecord<size_t> &rec, int device, const void *kernel,
                             size_t bytes, SET set) {
  return rec.with(device, kernel, [&](size_t &have) {
    if (bytes <= have) return true;
    if (!set(bytes)) return false;
    have = bytes;
    return true;
  });
}

// CTAs per cluster for (device, kernel): 16 where active(16) says that such a
// cluster fits, else the portable 8, else 0.  Asked once.
template <class ACTIVE>
inline int cluster_size_for(KernelRecord<int> &rec, int device, const void *kernel, ACTIVE active) {
  return rec.with(device, kernel, [&](int &size) {
    if (size == 0) size = active(16) ? 16 : (active(8) ? 8 : -1);
    return size > 0 ? size : 0;
  });
}

}  // namespace gfk
