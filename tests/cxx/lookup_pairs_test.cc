// Host checks of the 4D lookup's texels as two lanes share them
// (MakePairLookup, PairRows, PairColumn of atmo_device.cuh).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

#include "../../precomputed_atmospheric_scattering_gb300/csrc/atmo_device.cuh"

using namespace atmo;

namespace {

const float kInf = std::numeric_limits<float>::infinity();
const float kNan = std::numeric_limits<float>::quiet_NaN();

Shape MakeShape(int sr, int smu, int smus, int snu) {
  Shape s;
  std::memset(&s, 0, sizeof s);
  s.sr = sr;
  s.smu = smu;
  s.smus = smus;
  s.snu = snu;
  return s;
}

// Calls f with lookups of shape s: positions on, between and past the texels
// of every axis, as far as a ray that misses the atmosphere can take them.
template <class F>
int ForLookups(const Shape& s, F f) {
  int bad = 0;
  std::vector<float> nodes{-kInf, -3e9f, -2.0f, -1.0f, float(s.snu), float(s.snu + 1), 3e9f, kInf,
                           kNan};
  for (int n = 0; n < s.snu; ++n) nodes.push_back(float(n));
  const std::vector<float> far{-0.5f, 0.25f, 1e3f, 1e6f, 2147483520.0f, 2147483648.0f, 1e12f,
                               1e30f, kInf, kNan};
  std::vector<float> zs(far), ys{-0.5f, -0.25f, kNan};
  for (int k = 0; k < s.sr; ++k) {
    zs.push_back(float(k));
    zs.push_back(float(k) + 0.5f);
  }
  for (int j = 0; j < s.smu; ++j) ys.push_back(float(j) + 0.5f * float(j & 1));
  for (float node : nodes) {
    for (int x = -1; x < s.smus; ++x) {
      for (float z : zs) {
        for (float y : ys) {
          Lookup4 L;
          L.lerp_nu = node == -1.0f ? 0.9999999f : 0.25f;
          L.b0 = ToInt(node) * s.smus;
          L.b1 = L.b0 + s.smus;
          L.xl = float(x) + 0.5f;
          L.y = y;
          L.z = z;
          if (!f(L)) ++bad;
        }
      }
    }
  }
  return bad;
}

// Every texel read lies in the LUT.
int Bounds(const Shape& s) {
  return ForLookups(s, [&](const Lookup4& L) {
    const PairLookup p = MakePairLookup(s, L);
    int rows[4];
    PairRows(s, p, rows);
    for (int q = 0; q < 4; ++q) {
      for (int node = 0; node < 2; ++node) {
        for (int upper = 0; upper < 2; ++upper) {
          const long long i = (long long)rows[q] + PairColumn(s, p, node, upper);
          if (i < 0 || i >= s.s_texels()) return false;
        }
      }
    }
    return true;
  });
}

// The texels of nonzero weight are those that a lookup by itself reads
// (Scattering4: the columns of each node clamped one by one).
int Texels(const Shape& s) {
  const int W = s.sw(), H = s.smu, D = s.sr;
  return ForLookups(s, [&](const Lookup4& L) {
    const int y = ToInt(std::floor(L.y)), z = ToInt(std::floor(L.z)), x = ToInt(std::floor(L.xl));
    const float wy = L.y - std::floor(L.y), wz = L.z - std::floor(L.z);
    const PairLookup p = MakePairLookup(s, L);
    int rows[4];
    PairRows(s, p, rows);
    for (int q = 0; q < 4; ++q) {
      if (((q & 1) && wy == 0.0f) || ((q & 2) && wz == 0.0f)) continue;
      if (L.z != L.z || std::isinf(L.z) || L.y != L.y) continue;   // weights are NaN
      // A view of no finite length: the first column has wrapped.
      if (std::abs((long long)L.b0) > 1000 * s.smus) continue;
      const int j = ClampIdx(y + (q & 1), H), k = ClampIdx(z + (q >> 1), D);
      for (int node = 0; node < 2; ++node) {
        for (int upper = 0; upper < 2; ++upper) {
          const int i = ClampIdx((node == 0 ? L.b0 : L.b1) + x + upper, W);
          if (rows[q] + PairColumn(s, p, node, upper) != (k * H + j) * W + i)
            return false;
        }
      }
    }
    return true;
  });
}

}  // namespace

int main(int argc, char** argv) {
  const Shape shapes[] = {MakeShape(2, 4, 2, 2), MakeShape(3, 6, 5, 3), MakeShape(32, 8, 8, 4),
                          MakeShape(5, 4, 32, 8)};
  int bad = 0;
  for (const Shape& s : shapes) {
    if (argc > 1 && std::strcmp(argv[1], "bounds") == 0) bad += Bounds(s);
    if (argc > 1 && std::strcmp(argv[1], "texels") == 0) bad += Texels(s);
  }
  std::printf("%d wrong\n", bad);
  return bad != 0;
}
