// Host-side check of vfs::narrow (the integer-pipe binary64 -> binary32
// rounding of the Krylov kernels) against the compiler's conversion: around
// every binary32 value of a stride the points and midpoints where rounding
// turns, pseudo-random doubles over all exponents, and the special classes;
// and of vfs::widen_normal over the same values.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "vfs_common.cuh"

static unsigned long long bad = 0, n = 0;
static void check(unsigned long long u) {
  double d;
  std::memcpy(&d, &u, 8);
  const float a = vfs::narrow(d), b = (float)d;
  n++;
  if (std::memcmp(&a, &b, 4) != 0 && !(a != a && b != b)) bad++;
}
// widen_normal agrees with the conversion unless it says special, and says so
// exactly for subnormals, infinities and NaNs.
static void check_normal(float f) {
  unsigned u;
  std::memcpy(&u, &f, 4);
  const unsigned e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
  bool special = false;
  const double a = vfs::widen_normal(f, special), b = (double)f;
  n++;
  if (special != (e == 0xffu || (e == 0u && m != 0u)) || (!special && std::memcmp(&a, &b, 8) != 0)) bad++;
}
static void around(double d) {
  unsigned long long u;
  std::memcpy(&u, &d, 8);
  for (unsigned long long q = 0; q < 3; q++) check(u - 1 + q);
}

int main(int argc, char** argv) {
  const unsigned long long stride = argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1;
  for (unsigned long long t = 0; t <= 0xffffffffull; t += stride) {
    const unsigned u = (unsigned)t;
    float f, g;
    std::memcpy(&f, &u, 4);
    check_normal(f);
    const unsigned v = u + 1;
    std::memcpy(&g, &v, 4);
    if (f != f || g != g) continue;
    around((double)f);
    around(0.5 * ((double)f + (double)g));
  }
  unsigned long long x = 88172645463325252ull;  // xorshift over all 64-bit patterns
  for (int t = 0; t < 4000000; t++) {
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    check(x);
  }
  const unsigned long long special[] = {0ull, 1ull, 0x8000000000000000ull, 0x7ff0000000000000ull, 0xfff0000000000000ull,
                                        0x7ff8000000000000ull, 0x47efffffe0000000ull, 0x47efffffefffffffull,
                                        0x47effffff0000000ull, 0x3810000000000000ull, 0x380fffffffffffffull};
  for (unsigned long long u : special) check(u);
  for (unsigned u : {0u, 0x80000000u, 1u, 0x007fffffu, 0x00800000u, 0x7f7fffffu, 0x7f800000u, 0x7fc00000u, 0xff800000u}) {
    float f;
    std::memcpy(&f, &u, 4);
    check_normal(f);
  }
  std::printf("checked %llu values, %llu mismatches\n", n, bad);
  return bad ? 1 : 0;
}
