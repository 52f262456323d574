// Host check of the lazily reduced transforms (cuda_b200/csrc/lazy_core.cuh): dif<R> and
// dit_inv<R> on any 64-bit words, and on products of such words, are congruent to the
// canonical transforms (ntt_core.cuh) of the residues, and no intermediate leaves the ranges
// that the three-word form assumes (lazy::range_error).  Extreme words sit at every position, and so
// do the ends of the stated input range, +-2^65.
#include <cstdint>
#include <cstdio>
#include <random>
#include "../../cuda_b200/csrc/lazy_core.cuh"
#include "../../cuda_b200/csrc/ntt_core.cuh"

using namespace lnt;
static int fails = 0;
static uint64_t canon(uint64_t x) { return x >= gl::P ? x - gl::P : x; }

static uint64_t pick(std::mt19937_64& rng) {
  static const uint64_t edge[] = {0ull, 1ull, 0xFFFFFFFFull, 0x100000000ull, 0x8000000000000000ull, gl::P - 1,
                                  gl::P, gl::P + 1, 0xFFFFFFFFFFFFFFFEull, 0xFFFFFFFFFFFFFFFFull};
  const uint64_t r = rng();
  return (r & 3) ? edge[(r >> 8) % 10] : rng();
}

// an end of the input range, or near it, and its residue
static lazy::W3 bound(std::mt19937_64& rng, uint64_t& residue) {
  __int128 v = lazy::kInputBound - (__int128)((rng() & 1) ? rng() % 3 : 0);
  if (rng() & 1) v = -v;
  const __int128 r = v % (__int128)gl::P;
  residue = (uint64_t)(r < 0 ? r + gl::P : r);
  return lazy::from_int(v);
}

template <int R>
void check(std::mt19937_64& rng) {
  for (int rep = 0; rep < 25000; ++rep) {
    lazy::W3 x[R];
    uint64_t want[R], got[R];
    // words of all extremes, products, one extreme value everywhere, +- halves, ends of the input range
    const int mode = rep % 5;
    const uint64_t all = pick(rng), other = pick(rng);
    for (int i = 0; i < R; ++i) {
      uint64_t a = mode == 2 ? all : (mode == 3 ? ((rng() & 1) ? all : other) : pick(rng));
      if (mode == 4) {
        x[i] = bound(rng, want[i]);
      } else if (mode == 1) {
        const uint64_t b = pick(rng);
        x[i] = lazy::mul3(a, b);
        want[i] = gl::mul(canon(a), canon(b));
        if (canon(lazy::mul(a, b)) != want[i] && fails++ < 5) std::printf("mul\n");
      } else {
        x[i] = lazy::from_word(a);
        want[i] = canon(a);
      }
    }
    lazy::W3 y[R];
    uint64_t inv[R];
    for (int i = 0; i < R; ++i) {
      y[i] = x[i];
      inv[i] = want[i];
    }
    lazy::dif<R>(x, got);
    dif<R>(want);
    for (int i = 0; i < R; ++i)
      if (canon(got[i]) != want[i] && fails++ < 5) std::printf("dif<%d> %d mode %d\n", R, i, mode);
    lazy::dit_inv<R>(y, got);
    dit_inv<R>(inv);
    for (int i = 0; i < R; ++i)
      if (canon(got[i]) != inv[i] && fails++ < 5) std::printf("dit_inv<%d> %d mode %d\n", R, i, mode);
    if (lazy::range_error()) {
      std::printf("range error, R = %d mode %d\n", R, mode);
      fails++;
      lazy::range_error() = false;
      return;
    }
  }
}

// dft5 against the definition, on words and on products
void check5(std::mt19937_64& rng) {
  const uint64_t w = gl::pow(554, (gl::P - 1) / 5);
  uint64_t c[4];
  lazy::dft5_constants(w, c);
  for (int rep = 0; rep < 30000; ++rep) {
    lazy::W3 u[5];
    uint64_t v[5], got[5];
    for (int i = 0; i < 5; ++i) {
      const uint64_t a = pick(rng), b = pick(rng);
      const int mode = rep % 3;  // words, products, ends of the input range
      u[i] = mode == 2 ? bound(rng, v[i]) : (mode ? lazy::mul3(a, b) : lazy::from_word(a));
      if (mode != 2) v[i] = mode ? gl::mul(canon(a), canon(b)) : canon(a);
    }
    lazy::dft5(u, c, got);
    for (int k = 0; k < 5; ++k) {
      uint64_t s = 0;
      for (int i = 0; i < 5; ++i) s = gl::add(s, gl::mul(v[i], gl::pow(w, (uint64_t)(i * k))));
      if (canon(got[k]) != gl::mul(4, s) && fails++ < 5) std::printf("dft5 %d\n", k);
    }
    if (lazy::range_error()) {
      std::printf("range error, dft5\n");
      fails++;
      lazy::range_error() = false;
      return;
    }
  }
}

int main() {
  std::mt19937_64 rng(11);
  check5(rng);
  check<2>(rng);
  check<4>(rng);
  check<8>(rng);
  check<16>(rng);
  if (fails) {
    std::printf("FAILED %d\n", fails);
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
