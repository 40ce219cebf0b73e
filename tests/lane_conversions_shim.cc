// C entry points over the lane kernel's conversions in include/prismspf/gpu/fixed_point.cuh
// (compiled with g++ by tests/test_lane_conversions.py).
#include <prismspf/gpu/fixed_point.cuh>

namespace fx = prismspf::gpu::fx;

extern "C" {
long long lcs_to_fixed(double v, int E) { return fx::to_fixed_cut<fx::LANE_TOP_VALUES>(v, fx::high_exponent(E)); }
long long lcs_to_fixed_scaled(double v, int E, unsigned long long sig, int k) {
  return fx::to_fixed_cut_scaled<fx::LANE_TOP_INTEGRAL>(v, fx::high_exponent(E), sig, k);
}
double lcs_to_double(long long x, int lsb, unsigned long long sig, int scaled, int wide, int bad, unsigned int flip) {
  return fx::to_double_cut(x, lsb, sig, scaled != 0, wide != 0, bad != 0, flip);
}
void lcs_scale(double s, unsigned long long* sig, int* k) {
  const fx::Scale r = fx::make_scale(s);
  *sig = r.sig;
  *k = r.k;
}
int lcs_top_values() { return fx::LANE_TOP_VALUES; }
int lcs_top_integral() { return fx::LANE_TOP_INTEGRAL; }
int lcs_floor() { return fx::EXP_FLOOR; }
}
