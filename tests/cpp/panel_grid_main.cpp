// The panel grid of a surface scene: how fine it is for a given step, and
// that every point of a panel lies in a box that lists it.  Prints "ok".
#include <cmath>
#include <cstdio>
#include <random>

#include "bd_surface.h"

using namespace bd;

int main() {
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  const float boxes[3][3] = {{8, 8, 8}, {20, 3, 8}, {1, 40, 1}};
  for (const auto& hi : boxes)
    for (int n : {1, 6, 80, 1280, 5000})
      for (double step : {0.0, 0.003, 0.03, 0.3, 3.0, 100.0}) {
        const float lo[3] = {0, 0, 0};
        std::vector<bd_panel_info> panels;
        for (int k = 0; k < n; k++) {
          bd_panel q{};
          if (n == 1) {
            q.shape = BD_PANEL_SPH;
            for (int a = 0; a < 3; a++) q.p[a] = hi[a] / 2;
            q.p[3] = 0.4f * std::fmin(hi[0], std::fmin(hi[1], hi[2]));
            q.front = 1;
          } else {
            q.shape = BD_PANEL_TRI;
            float c[3];
            for (int a = 0; a < 3; a++) c[a] = (float)(u(rng) * hi[a]);
            for (int v = 0; v < 9; v++) q.p[v] = c[v % 3] + 0.1f * (float)(u(rng) - 0.5) * hi[v % 3];
          }
          bd_panel_info info;
          std::string msg;
          if (derive_panel(q, 0, &info, &msg) != BD_OK) return printf("panel: %s\n", msg.c_str()), 1;
          panels.push_back(info);
        }
        PanelGrid g;
        build_panel_grid(panels, lo, hi, step, &g);
        const double emax = std::fmax(hi[0], std::fmax(hi[1], hi[2]));
        for (int a = 0; a < 3; a++) {
          const double least =
              std::fmin(32.0, std::fmax(1.0, std::ceil(std::ceil(std::cbrt(8.0 * n)) * hi[a] / emax)));
          if (g.dims[a] < least || g.dims[a] > 64) return printf("dims %u\n", g.dims[a]), 1;
          if (g.dims[a] > least && hi[a] / g.dims[a] < 3.999 * step)
            return printf("box %g of step %g\n", hi[a] / g.dims[a], step), 1;
        }
        for (int k = 0; k < 20000; k++) {
          const size_t id = (size_t)(u(rng) * panels.size());
          const bd_panel_info& P = panels[id];
          double x[3];
          if (P.shape == BD_PANEL_SPH) {
            std::normal_distribution<double> normal;
            double d[3], r = 0;
            for (double& v : d) v = normal(rng), r += v * v;
            for (int a = 0; a < 3; a++) x[a] = P.a[a] + P.r * d[a] / std::sqrt(r);
          } else {
            double s = u(rng), t = u(rng);
            if (s + t > 1) s = 1 - s, t = 1 - t;
            for (int a = 0; a < 3; a++) x[a] = P.a[a] + s * (P.v1[a] - P.a[a]) + t * (P.v2[a] - P.a[a]);
          }
          uint32_t c[3];
          for (int a = 0; a < 3; a++) {
            const int v = (int)std::floor(((float)x[a] - g.lo[a]) * g.inv[a]);
            c[a] = (uint32_t)std::min(std::max(v, 0), (int)g.dims[a] - 1);
          }
          const uint32_t box = (c[2] * g.dims[1] + c[1]) * g.dims[0] + c[0];
          bool listed = false;
          for (uint32_t e = g.start[box]; e < g.start[box + 1]; e++) listed |= g.list[e] == id;
          if (!listed) return printf("panel %zu not listed at %g %g %g\n", id, x[0], x[1], x[2]), 1;
        }
      }
  puts("ok");
  return 0;
}
