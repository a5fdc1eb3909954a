// Host check of the candidate masks (tomo_span.cuh): for random triangles of
// several shapes, every pixel of the bounding box that the reference's
// barycentric test accepts must have its bit set in its cell's mask.  The
// test is restated here with the kernels' float operations in their order
// (IEEE single precision, no contraction).  Prints one line:
// "triangles T pixels P accepted A candidates C violations V".
#include <cstdio>
#include <cstdlib>
#include <cstdint>
#include <cmath>
#include <random>
#include <vector>

#include "../tomo_shell2026_b200/csrc/tomo_span.cuh"

using tomo::MaskTri;

static float pix_center(int x, float half) { return ((float)x + 0.001f) + half; }
static float dot2(float ax, float ay, float bx, float by) { return ((ax * bx) + (ay * by)) + 0.0f; }

struct Counts { long long tris = 0, pixels = 0, accepted = 0, candidates = 0, violations = 0; };

static void check(float ax, float ay, float bx, float by, float cx, float cy, float half, Counts& n)
{
  const float minx = std::fmin(std::fmin(ax, bx), cx), maxx = std::fmax(std::fmax(ax, bx), cx);
  const float miny = std::fmin(std::fmin(ay, by), cy), maxy = std::fmax(std::fmax(ay, by), cy);
  const int x0 = (int)std::trunc(minx), y0 = (int)std::trunc(miny);
  const int x1 = (int)std::trunc(maxx), y1 = (int)std::trunc(maxy);
  const float e0x = bx - ax, e0y = by - ay, e1x = cx - ax, e1y = cy - ay;
  const float d00 = dot2(e0x, e0y, e0x, e0y), d01 = dot2(e0x, e0y, e1x, e1y), d11 = dot2(e1x, e1y, e1x, e1y);
  const float denom = (d00 * d11) - (d01 * d01);
  if (!(std::fabs(denom) > 0.001f)) return;   // no pixel of such a triangle is tested
  float vmax = (float)(1.0 + (double)0.001f);
  while ((double)vmax > 1.0 + (double)0.001f) vmax = std::nextafter(vmax, 0.0f);
  const MaskTri T = tomo::mask_setup(ax, ay, e0x, e0y, e1x, e1y, d00, d01, d11, denom, minx, maxx, miny, maxy, x0, x1,
                                     y0, y1, half);
  n.tris++;
  const int w = x1 - x0 + 1, h = y1 - y0 + 1;
  std::vector<char> cand((size_t)w * h, 0);
  for (int ci = 0; ci * tomo::kCellX < T.nx; ci++)
    for (int cj = 0; cj * tomo::kCellY < T.ny; cj++) {
      unsigned m = tomo::mask_cell(T, ci, cj);
      for (int b = 0; b < 32; b++) {
        if (!((m >> (31 - b)) & 1u)) continue;
        const int x = T.x0 + ci * tomo::kCellX + (b >> 2), y = T.y0 + cj * tomo::kCellY + (b & 3);
        n.candidates++;
        if (x < x0 || x > x1 || y < y0 || y > y1) { n.violations++; std::printf("violation: outside the box\n"); continue; }
        cand[(size_t)(x - x0) * h + (y - y0)] = 1;
      }
    }
  for (int x = x0; x <= x1; x++)
    for (int y = y0; y <= y1; y++) {
      const float e2x = pix_center(x, half) - ax, e2y = pix_center(y, half) - ay;
      const float d20 = dot2(e2x, e2y, e0x, e0y), d21 = dot2(e2x, e2y, e1x, e1y);
      const float v = ((d11 * d20) - (d01 * d21)) / denom, ww = ((d00 * d21) - (d01 * d20)) / denom;
      const float u = (float)(1.0 - (double)v - (double)ww);
      n.pixels++;
      if (!((u >= -0.001f) && (v >= -0.001f) && (v <= vmax) && ((u + v) <= vmax))) continue;
      n.accepted++;
      if (!cand[(size_t)(x - x0) * h + (y - y0)]) {
        if (n.violations < 10)
          std::printf("violation: tri (%.9g %.9g) (%.9g %.9g) (%.9g %.9g) half %g column %d row %d\n", ax, ay, bx, by,
                      cx, cy, half, x, y);
        n.violations++;
      }
    }
}

int main(int argc, char** argv)
{
  const long long per_kind = argc > 1 ? std::atoll(argv[1]) : 100000;
  const unsigned seed = argc > 2 ? (unsigned)std::atoi(argv[2]) : 1u;
  std::mt19937_64 rng(seed);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  auto uf = [&](double a, double b) { return (float)(a + (b - a) * U(rng)); };
  const float halves[] = {0.5f, 0.25f, 1.0f, 0.125f};
  Counts n;
  for (long long i = 0; i < per_kind; i++) {
    const float half = halves[i & 3];
    const float ox = uf(0.0, 4000.0), oy = uf(0.0, 4000.0);
    // small triangles, a few pixels across
    check(ox + uf(0, 4), oy + uf(0, 4), ox + uf(0, 4), oy + uf(0, 4), ox + uf(0, 4), oy + uf(0, 4), half, n);
    // medium and large (up to the 63-row span limit and beyond)
    const double s = (i % 7 == 0) ? 200.0 : 40.0;
    check(ox + uf(0, s), oy + uf(0, s), ox + uf(0, s), oy + uf(0, s), ox + uf(0, s), oy + uf(0, s), half, n);
    // slivers: a long edge and a third vertex very near it
    {
      const float ax = ox, ay = oy, bx = ox + uf(-30, 30), by = oy + uf(-30, 30);
      const float t = uf(0, 1), d = (float)std::ldexp(U(rng), -(int)(U(rng) * 20));
      const float cx = ax + t * (bx - ax) - d * (by - ay) * 0.01f, cy = ay + t * (by - ay) + d * (bx - ax) * 0.01f;
      check(ax, ay, bx, by, cx, cy, half, n);
    }
    // axis-aligned edges and vertices on pixel centres and pixel edges
    {
      const float bx0 = std::floor(ox), by0 = std::floor(oy);
      const float fx = (i % 3 == 0) ? 0.0f : (i % 3 == 1 ? 0.001f + half : 0.5f);
      const float w = (float)(1 + (int)(U(rng) * 6)), h = (float)(1 + (int)(U(rng) * 6));
      if (i & 4) check(bx0 + fx, by0 + fx, bx0 + fx + w, by0 + fx, bx0 + fx, by0 + fx + h, half, n);
      else check(bx0 + fx + w, by0 + fx + h, bx0 + fx, by0 + fx + h, bx0 + fx + w, by0 + fx, half, n);
    }
    // near-degenerate (almost collinear) small triangles
    {
      const float ax = ox + uf(0, 3), ay = oy + uf(0, 3), bx = ax + uf(-3, 3), by = ay + uf(-3, 3);
      const float e = (float)std::ldexp(1.0, -(int)(8 + U(rng) * 14));
      check(ax, ay, bx, by, ax + 2.0f * (bx - ax) + e, ay + 2.0f * (by - ay) - e, half, n);
    }
  }
  std::printf("triangles %lld pixels %lld accepted %lld candidates %lld violations %lld\n", n.tris, n.pixels,
              n.accepted, n.candidates, n.violations);
  return n.violations == 0 ? 0 : 1;
}
