// One transform of lh_fxfft.cuh on the host, pass by pass as the kernels run it: n complex FP64 values in, n out.
#include <algorithm>

#include "lh_fxfft.cuh"

using namespace lh;

extern "C" int fx_host(int n, int inverse, const double* in, double* out) {
  FxPlan P;
  FxTables T;
  if (!fx_build(n, &P, &T)) return 1;
  auto high = [](double x) {
    unsigned long long b;
    std::memcpy(&b, &x, 8);
    return (unsigned)(b >> 32);
  };
  int e = 0;
  for (int i = 0; i < 2 * n; ++i) e = std::max(e, fx_exp(high(in[i])));
  std::vector<fx2> b(n);
  unsigned sum = 0;
  for (int s = 0; s < n; ++s) {
    const i64 x = fx_from(in[2 * s], e), y = fx_from(in[2 * s + 1], e);
    sum += fx_mag(x) + fx_mag(y);
    b[T.pos_sample[s]] = inverse ? fx2{y, x} : fx2{x, y};
  }
  const int g = inverse ? fx_inv_shift(sum, P.shift) : P.shift;
  for (int i = 0; i < P.npass; ++i) {
    const FxPass& ps = P.ps[i];
    for (int t = 0; t < n / ps.rad; ++t) {
      const int r0 = t % ps.mI, e0 = t / ps.mI * ps.rad * ps.mI + r0;
      const int4* tw = ps.tw >= 0 ? T.tw.data() + 2 * (ps.tw + r0 / ps.inner * (ps.rad - 1)) : nullptr;
      fx2 v[9];
      for (int p = 0; p < ps.rad; ++p) v[p] = b[e0 + p * ps.mI];
      const int sh = fx_pass_shift(ps, g);
      switch (ps.rad) {
        case 2: fx_item<2>(v, tw, sh); break;
        case 3: fx_item<3>(v, tw, sh); break;
        case 4: fx_item<4>(v, tw, sh); break;
        case 8: fx_item<8>(v, tw, sh); break;
        default: fx_item<9>(v, tw, sh); break;
      }
      for (int p = 0; p < ps.rad; ++p) b[e0 + p * ps.mI] = v[p];
    }
  }
  // the last pass's frequencies lie last_step apart
  if (P.npass) {
    const FxPass& l = P.ps[P.npass - 1];
    for (int t = 0; t < n / l.rad; ++t) {
      const int e0 = t / l.mI * l.rad * l.mI + t % l.mI;
      for (int p = 0; p < l.rad; ++p)
        if (T.freq_pos[e0 + p * l.mI] != (T.freq_pos[e0] + p * P.last_step) % n) return 2;
    }
  }
  const int S = fx_scale(e) - g;
  for (int k = 0; k < n; ++k) {
    const fx2 v = b[T.pos_freq[k]];
    out[2 * k] = fx_to(inverse ? v.y : v.x, S);
    out[2 * k + 1] = fx_to(inverse ? v.x : v.y, S);
  }
  return 0;
}
