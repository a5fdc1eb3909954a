// Host check of the candidate masks (tomo_span.cuh) over the pixel sizes a
// caller may pass, up to the largest float: the pixels to look at lie within the
// triangle's pixel box (the walk over the cells ends), and every pixel of the
// box that the reference's barycentric test accepts is a candidate.  Compiled
// with -fwrapv: a count that wraps is a violation here, as on the device.
// Prints one line: "cases N accepted A violations V".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../tomo_shell2026_b200/csrc/tomo_span.cuh"

static float pix_center(int x, float half) { return ((float)x + 0.001f) + half; }
static float dot2(float ax, float ay, float bx, float by) { return ((ax * bx) + (ay * by)) + 0.0f; }

int main(int argc, char** argv)
{
  const int per = argc > 1 ? std::atoi(argv[1]) : 1000;
  std::mt19937_64 rng(argc > 2 ? (unsigned)std::atoi(argv[2]) : 1u);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  const float mags[] = {0.5f, 7.0f, 60.0f, 4.0e3f, 1.0e6f, 3.0e6f, 1.0e9f, 2.1e9f, 2.2e9f, 5.0e9f, 1.0e12f, 1.0e30f, 1.7e38f};
  float vmax = (float)(1.0 + (double)0.001f);
  while ((double)vmax > 1.0 + (double)0.001f) vmax = std::nextafter(vmax, 0.0f);
  long long cases = 0, accepted = 0, bad = 0;
  for (float mag : mags)
    for (float sign : {1.0f, -1.0f})
      for (int i = 0; i < per; i++) {
        const float half = sign * mag, s = (i % 16 == 0) ? 300.0f : ((i & 1) ? 40.0f : 5.0f);
        const float ox = (float)(U(rng) * 3700.0), oy = (float)(U(rng) * 3700.0);
        float v[6];
        for (int k = 0; k < 6; k++) v[k] = (k & 1 ? oy : ox) + (float)(U(rng) * s);
        const float minx = std::fmin(std::fmin(v[0], v[2]), v[4]), maxx = std::fmax(std::fmax(v[0], v[2]), v[4]);
        const float miny = std::fmin(std::fmin(v[1], v[3]), v[5]), maxy = std::fmax(std::fmax(v[1], v[3]), v[5]);
        const float e0x = v[2] - v[0], e0y = v[3] - v[1], e1x = v[4] - v[0], e1y = v[5] - v[1];
        const float d00 = dot2(e0x, e0y, e0x, e0y), d01 = dot2(e0x, e0y, e1x, e1y), d11 = dot2(e1x, e1y, e1x, e1y);
        const float denom = (d00 * d11) - (d01 * d01);
        if (!(std::fabs(denom) > 0.001f)) continue;
        const int x0 = (int)minx, x1 = (int)maxx, y0 = (int)miny, y1 = (int)maxy;
        const tomo::MaskTri T = tomo::mask_setup(v[0], v[1], e0x, e0y, e1x, e1y, d00, d01, d11, denom, minx, maxx, miny,
                                                 maxy, x0, x1, y0, y1, half);
        cases++;
        const bool none = T.nx <= 0 || T.ny <= 0;
        if (!none && !(T.x0 >= x0 && T.y0 >= y0 && T.nx <= x1 - x0 + 1 && T.ny <= y1 - y0 + 1)) {
          if (bad++ < 5)
            std::printf("violation: half %g box %d..%d %d..%d grid %d+%d %d+%d\n", half, x0, x1, y0, y1, T.x0, T.nx, T.y0, T.ny);
          continue;
        }
        for (int x = x0; x <= x1; x++)
          for (int y = y0; y <= y1; y++) {
            const float e2x = pix_center(x, half) - v[0], e2y = pix_center(y, half) - v[1];
            const float d20 = dot2(e2x, e2y, e0x, e0y), d21 = dot2(e2x, e2y, e1x, e1y);
            const float b = ((d11 * d20) - (d01 * d21)) / denom, c = ((d00 * d21) - (d01 * d20)) / denom;
            const float a = (float)(1.0 - (double)b - (double)c);
            if (!((a >= -0.001f) && (b >= -0.001f) && (b <= vmax) && ((a + b) <= vmax))) continue;
            accepted++;
            const int i8 = x - T.x0, j4 = y - T.y0;
            const bool in = !none && i8 >= 0 && j4 >= 0 && i8 < T.nx && j4 < T.ny &&
                            ((tomo::mask_cell(T, i8 / tomo::kCellX, j4 / tomo::kCellY) >>
                              (31 - (4 * (i8 % tomo::kCellX) + j4 % tomo::kCellY))) & 1u);
            if (!in && bad++ < 5) std::printf("violation: half %g pixel %d %d accepted, no candidate\n", half, x, y);
          }
      }
  std::printf("cases %lld accepted %lld violations %lld\n", cases, accepted, bad);
  return bad == 0 ? 0 : 1;
}
