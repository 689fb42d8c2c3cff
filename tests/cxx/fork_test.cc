// Host checks of SideBySide (atmo_fork.h) with calls that fail on purpose.
#include <cstdio>
#include <string>

#include "../../precomputed_atmospheric_scattering_gb300/csrc/atmo_fork.h"

struct FakeOps {
  char fails;          // the call that fails: F, S, M or J
  std::string calls;   // in their order
  atmo_status Call(char c) {
    calls += c;
    return c == fails ? ATMO_CUDA_ERROR : ATMO_OK;
  }
  atmo_status Fork() { return Call('F'); }
  atmo_status Side() { return Call('S'); }
  atmo_status Main() { return Call('M'); }
  atmo_status Join() { return Call('J'); }
};

int main() {
  int bad = 0;
  for (const char fails : {'-', 'F', 'S', 'M', 'J'}) {
    FakeOps ops{fails, ""};
    const atmo_status s = atmo::SideBySide(ops);
    // What the side stream may hold is joined, last of all, on every way out.
    const bool side = ops.calls.find('S') != std::string::npos;
    const bool ok = (s == ATMO_OK) == (fails == '-') && ops.calls[0] == 'F' &&
                    (fails == 'F' || side) && (ops.calls.back() == 'J') == side;
    if (!ok) std::printf("%c: %s\n", fails, ops.calls.c_str());
    bad += !ok;
  }
  std::printf("%d wrong\n", bad);
  return bad != 0;
}
