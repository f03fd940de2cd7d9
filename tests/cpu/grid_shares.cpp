// The grid PCG's shares: for any number of CTAs every unit of the product,
// camera block and chunk of cameras has one owner, and the CTAs that stay are
// those that own something (a CTA that publishes nothing must not read what
// the others publish: nobody waits for it before the values change).
#include <algorithm>
#include <cstdio>

#include "kernels.h"

using namespace gba;

// Blocks of each camera's rows of S, the diagonal one included.
static bool check(const char *name, const std::vector<int> &m, bool idle_wanted) {
  const int n = (int)m.size(), nblk = (n + kPcgBlockCams - 1) / kPcgBlockCams, nch = (n + 31) / 32;
  long long rows = 0;
  for (int x : m) rows += x;
  bool idle_seen = false;
  for (int P = 1; P <= std::min(152, 5 * n); ++P) {
    int units = 0, blocks = 0, chunks = 0, idle = 0;
    for (int w = 0; w < P; ++w) {
      int a = 0, b = 0;
      long long before = 0;
      for (int c = 0; c < n; ++c) {
        a += units5_below(grid_bound(w, P, rows), 9 * before, m[c]);
        b += units5_below(grid_bound(w + 1, P, rows), 9 * before, m[c]);
        before += m[c];
      }
      const int k = grid_run(w + 1, P, nblk) - grid_run(w, P, nblk), h = grid_run(w + 1, P, nch) - grid_run(w, P, nch);
      if (a != units || b < a || k < 0 || h < 0) return std::printf("%s, %d CTAs: a run does not follow on\n", name, P), false;
      units = b, blocks += k, chunks += h;
      const bool stays = grid_takes_part(b - a, k, h);
      if (stays != (b > a || k > 0 || h > 0)) return std::printf("%s, %d CTAs: the wrong CTAs stay\n", name, P), false;
      if (w == 0 && b == 0) return std::printf("%s, %d CTAs: CTA 0 owns no unit\n", name, P), false;
      idle += !stays;
    }
    if (units != 5 * n || blocks != nblk || chunks != nch)
      return std::printf("%s, %d CTAs: %d units, %d blocks, %d chunks\n", name, P, units, blocks, chunks), false;
    idle_seen = idle_seen || (idle > 0 && P == std::min(152, 5 * n));
  }
  if (idle_wanted && !idle_seen) return std::printf("%s: no CTA without a share\n", name), false;
  return true;
}

int main() {
  std::vector<int> chain(200, 5), hub(200, 6);
  hub[17] = 200;
  if (!check("one camera", {1}, false) || !check("ring of 33", std::vector<int>(33, 33), true) ||
      !check("30 cameras", std::vector<int>(30, 22), false) || !check("chain", chain, false) || !check("hub", hub, true))
    return 1;
  std::printf("ok\n");
  return 0;
}
