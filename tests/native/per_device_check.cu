// Host-side check of vfs::PerDevice: the settings run once on every device,
// not once per process, and a failure is returned and tried again.
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"

static int bad = 0;
static void expect(bool ok, const char* what) {
  if (ok) return;
  std::printf("wrong: %s\n", what);
  bad++;
}

int main() {
  int calls[65] = {0};
  auto set = [&](vfs::PerDevice& o, int d) { return o.on(d, [&] { calls[d]++; return cudaSuccess; }); };
  vfs::PerDevice once;
  for (int turn = 0; turn < 3; turn++)
    for (int d : {0, 1, 63}) expect(set(once, d) == cudaSuccess, "a successful setting");
  expect(calls[0] == 1 && calls[1] == 1 && calls[63] == 1, "once on each device");
  for (int turn = 0; turn < 3; turn++) set(once, 64);
  expect(calls[64] == 3, "a device beyond the table is set on every call");
  vfs::PerDevice retry;
  int n = 0;
  auto fails_first = [&] { return n++ == 0 ? cudaErrorInvalidValue : cudaSuccess; };
  expect(retry.on(2, fails_first) == cudaErrorInvalidValue, "a failure is returned");
  expect(retry.on(2, fails_first) == cudaSuccess && n == 2, "and tried again");
  expect(retry.on(2, fails_first) == cudaSuccess && n == 2, "until it held");
  vfs::PerDevice shared;
  std::atomic<int> runs{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; t++)
    ts.emplace_back([&] {
      for (int q = 0; q < 1000; q++) shared.on(5, [&] { runs++; return cudaSuccess; });
    });
  for (auto& t : ts) t.join();
  expect(runs >= 1 && runs <= 8, "threads run it at most once each");
  return bad;
}
