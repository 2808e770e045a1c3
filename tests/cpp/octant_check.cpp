// octant_of (xyz_b200/csrc/common.cuh) against the arc tangent it stands in
// for: random points, points on and around the octants' borders, zeros,
// infinities and NaN.  Exit code 1 on a difference; prints the share of random
// points left to the arc tangent.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../xyz_b200/csrc/common.cuh"

using namespace xyzgpu;

int main() {
  auto by_angle = [](float y, float x) {
    float phi = 0.5f * std::atan2(y, x);
    if (phi < 0.0f) phi = static_cast<float>(static_cast<double>(phi) + kPi);
    int const v = static_cast<int>(static_cast<double>(phi) * (8.0 * kInvPi));
    return v >= 8 ? 7 : v;
  };
  std::mt19937 g(3);
  std::normal_distribution<float> N;
  int wrong = 0, left = 0, n = 1000000;
  for (int i = 0; i < n; ++i) {
    float const x = N(g), y = N(g);
    int const v = octant_of(y, x);
    left += v < 0;
    wrong += v >= 0 && v != by_angle(y, x);
  }
  for (int k = 0; k < 8; ++k)
    for (int e = -60; e <= 60; ++e)
      for (float r : {1e-30f, 1e-3f, 1.0f, 1e20f}) {
        double const a = k * kPi / 4 + (e < 0 ? -1 : 1) * std::pow(10.0, -std::abs(e) / 6.0);
        float const x = r * static_cast<float>(std::cos(a)), y = r * static_cast<float>(std::sin(a));
        int const v = octant_of(y, x);
        wrong += v >= 0 && v != by_angle(y, x);
      }
  float const s[] = {0.0f, -0.0f, 1.0f, -1.0f, INFINITY, -INFINITY, NAN};
  for (float x : s)
    for (float y : s) wrong += octant_of(y, x) >= 0;  // all on a border or without an angle
  std::printf("wrong %d, left %d of %d\n", wrong, left, n);
  return wrong != 0 || left > n / 1000;
}
