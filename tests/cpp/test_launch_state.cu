// Host checks of geoflow_b200/csrc/launch_state.cuh: the records of what a kernel was
// given on a device.  Runs on the CPU; the calls that they make are counted fakes.
#include <cstdio>
#include <thread>
#include <vector>

#include "../../geoflow_b200/csrc/launch_state.cuh"

using namespace gfk;

static int failures = 0;
#define CHECK(cond, ...)                    \
  do {                                      \
    if (!(cond)) {                          \
      failures++;                           \
      std::printf("FAIL: " __VA_ARGS__);    \
      std::printf("\n");                    \
    }                                       \
  } while (0)

static void check_smem_limits() {
  KernelRecord<size_t> rec;
  const int k0 = 0, k1 = 0;
  int calls = 0;
  size_t last = 0;
  auto set = [&](size_t b) {
    calls++;
    last = b;
    return true;
  };
  CHECK(raise_smem_limit(rec, 0, &k0, 50000, set) && calls == 1 && last == 50000, "first");
  CHECK(raise_smem_limit(rec, 0, &k0, 50000, set) && calls == 1, "again");
  CHECK(raise_smem_limit(rec, 0, &k0, 20000, set) && calls == 1, "a smaller launch lowers nothing");
  CHECK(raise_smem_limit(rec, 0, &k0, 70000, set) && calls == 2 && last == 70000, "a larger one");
  CHECK(raise_smem_limit(rec, 1, &k0, 50000, set) && calls == 3 && last == 50000,
        "another device has a limit of its own");
  CHECK(raise_smem_limit(rec, 0, &k1, 10000, set) && calls == 4, "another kernel");
  auto refuse = [&](size_t) {
    calls++;
    return false;
  };
  CHECK(!raise_smem_limit(rec, 0, &k0, 900000, refuse) && calls == 5, "refused");
  CHECK(raise_smem_limit(rec, 0, &k0, 70000, refuse) && calls == 5, "the limit before stays");
  CHECK(!raise_smem_limit(rec, 0, &k0, 900000, refuse) && calls == 6, "a refusal is not recorded");
}

static void check_threads() {
  KernelRecord<size_t> rec;
  static int kernels[64];
  size_t limit[4][64] = {};  // what the fake devices hold: written under the lock
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; t++)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 4000; i++) {
        const int d = (i + t) % 4, k = (i * 7 + t) % 64;
        raise_smem_limit(rec, d, &kernels[k], 1000 + (i * 37 + t) % 9000, [&](size_t b) {
          limit[d][k] = b;
          return true;
        });
      }
    });
  for (auto &t : ts) t.join();
  for (int d = 0; d < 4; d++)
    for (int k = 0; k < 64; k++)
      rec.with(d, &kernels[k], [&](size_t &have) {
        CHECK(have == limit[d][k], "device %d kernel %d: %zu held, %zu recorded", d, k, limit[d][k], have);
        return 0;
      });
}

static void check_cluster_size() {
  const int k0 = 0, k1 = 0;
  for (int largest : {16, 8, 0}) {  // a device that holds clusters of up to so many CTAs
    KernelRecord<int> rec;
    int asked = 0;
    auto active = [&](int size) {
      asked++;
      return size <= largest;
    };
    CHECK(cluster_size_for(rec, 0, &k0, active) == largest, "largest %d", largest);
    const int once = asked;
    CHECK(cluster_size_for(rec, 0, &k0, active) == largest && asked == once, "kept, %d", largest);
    // a kernel with a need of its own, and another device, are asked for themselves
    CHECK(cluster_size_for(rec, 0, &k1, [](int size) { return size <= 8; }) == 8, "other kernel");
    CHECK(cluster_size_for(rec, 1, &k0, [](int) { return false; }) == 0, "other device");
    CHECK(cluster_size_for(rec, 0, &k0, active) == largest, "unchanged, %d", largest);
  }
}

int main() {
  check_smem_limits();
  check_threads();
  check_cluster_size();
  if (failures) return 1;
  std::printf("launch state ok\n");
  return 0;
}
