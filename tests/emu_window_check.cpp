// Host check of the straight-line forms of the integer-pipe FP64 arithmetic
// (qss_emu.cuh: div_win, mul_win, sq_win, add_pos / add_ordered, and the
// operations built on them) on operands where the last digit is hardest to
// get right: significands with long runs of zeros or ones, quotients and
// roots next to a half-way point, sums whose shift is 0, 31, 32, 53, 54 or 55
// bits.  Usage: emu_window_check <cases> <seed>; prints "<name> <cases> <bad>".
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>

#include "qss_emu.cuh"

using namespace qss_emu;

static uint64_t g_state;
static uint64_t rnd() {  // xorshift64*
  g_state ^= g_state >> 12;
  g_state ^= g_state << 25;
  g_state ^= g_state >> 27;
  return g_state * 2685821657736338717ull;
}
static uint64_t significand() {
  uint64_t m = rnd() & kMant;
  switch (rnd() % 6) {
    case 0: return m & ~((1ull << (rnd() % 52)) - 1);
    case 1: return m | ((1ull << (rnd() % 52)) - 1);
    case 2: return rnd() % 64;
    case 3: return kMant - rnd() % 64;
    default: return m;
  }
}
static double num(int emin, int emax) {
  return from_bits(((uint64_t)(1023 + emin + (int)(rnd() % (uint64_t)(emax - emin + 1))) << 52) | significand());
}

int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : 100000;
  g_state = (argc > 2 ? strtoull(argv[2], nullptr, 10) : 1) * 0x9e3779b97f4a7c15ull | 1;
  long long bad[5] = {0, 0, 0, 0, 0};
  auto ne = [](double a, double b) { return bits(a) != bits(b) ? 1 : 0; };
  static const double numer[4] = {0.1, 0.6, 0.3, 1.0};
  static const int shifts[] = {0, 1, 2, 30, 31, 32, 33, 52, 53, 54, 55, 70};
  for (long long i = 0; i < n; i++) {
    const double x = num(-255, 256), y = num(-255, 256), q = num(0, 0);
    bad[0] += ne(qss_emu::div(x, y), x / y) + ne(qss_emu::div(-x, y), -x / y);
    const double c = numer[rnd() & 3];
    bad[0] += ne(qss_emu::div(c, y), c / y);
    const double near = (double)((long double)y * ((long double)q + 0x1p-53L));  // quotient next to half-way
    bad[0] += ne(qss_emu::div(near, y), near / y);
    bad[1] += ne(qss_emu::mul(x, y), x * y) + ne(qss_emu::mul(x, -y), x * -y);
    const double z = num(-200, 120);
    bad[2] += ne(sq_win(hi32(z), lo32(z)), z * z) + ne(sq_win(hi32(-z), lo32(z), -2), z * z * 0.25);
    // sums: exponents apart by each shift that takes another path
    const double a = num(-100, 100);
    const int d = shifts[rnd() % 12];
    const double b = from_bits((bits(a) & ~kMant) - ((uint64_t)d << 52) + significand());
    bad[3] += ne(add_pos(a, b), a + b) + ne(add_pos(b, a), a + b) + ne(add_nonneg(a, 0.0), a) +
              ne(add_pos(from_bits(rnd() & 3), a), a) + ne(add_nonneg(a * a, b * b), a * a + b * b);
    const double h = (double)(((long double)q + 0x1p-53L) * ((long double)q + 0x1p-53L));
    for (int o = -2; o <= 2; o++) {
      const double s = from_bits(bits(h) + (uint64_t)(int64_t)o);
      bad[4] += ne(qss_emu::sqrt(s), std::sqrt(s)) + ne(qss_emu::sqrt(2 * s), std::sqrt(2 * s));
    }
    bad[4] += ne(qss_emu::sqrt(x), std::sqrt(x));
  }
  for (double e : {1.0, 2.0, 4.0, 0.5})  // powers of two and their neighbours
    for (int o = -3; o <= 3; o++) {
      const double s = from_bits(bits(e) + (uint64_t)(int64_t)o);
      bad[4] += ne(qss_emu::sqrt(s), std::sqrt(s));
      bad[0] += ne(qss_emu::div(1.0, s), 1.0 / s) + ne(qss_emu::div(s, s), 1.0);
    }
  static const char* const names[5] = {"div", "mul", "sq", "add", "sqrt"};
  long long all = 0;
  for (int k = 0; k < 5; k++) {
    printf("%s %lld %lld\n", names[k], n, bad[k]);
    all += bad[k];
  }
  return all ? 1 : 0;
}
