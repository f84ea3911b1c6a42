// Copy-block plans of random rigs (hmp_copyplan.h): the lists replanned for another down-tile edge equal
// those of a plan made for it, and the RGB8 canvas plane holds, pixel by pixel, the copied slot's entry
// in copy blocks and what it held before elsewhere.
//
//   copyplan_test <iterations> <seed>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>
#include <vector>
#include "hmp_copyplan.h"

using namespace hmp;

static bool same(const CopyPlan& a, const CopyPlan& b, int n) {
  for (int k = 0; k < n; ++k)
    if (a.need_w[k] != b.need_w[k] || a.need_h[k] != b.need_h[k]) return false;
  return a.usable == b.usable && a.fx0 == b.fx0 && a.fy0 == b.fy0 && a.nfx == b.nfx && a.nfy == b.nfy &&
         a.pyramid_block == b.pyramid_block && a.block_class == b.block_class && a.fine_list == b.fine_list &&
         a.coarse_list == b.coarse_list && a.down_list == b.down_list && a.support_mark == b.support_mark &&
         a.support_pitch == b.support_pitch && a.support_shift == b.support_shift && a.copy_blocks == b.copy_blocks &&
         a.empty_blocks == b.empty_blocks && a.pyramid_blocks == b.pyramid_blocks &&
         a.pyramid_pixels == b.pyramid_pixels && a.dense_down == b.dense_down && a.dense_coarse == b.dense_coarse;
}

// The canvas plane's entries, plain.
static void expected(const Plan& p, const CopyPlan& c, bool had, const GatherPlane& before, std::vector<uint32_t>& map,
                     std::vector<uint8_t>& owner) {
  const size_t px = size_t(p.canvas_w) * p.canvas_h;
  map = had ? before.map : std::vector<uint32_t>(px, kNoEntry);
  owner = had ? before.owner : std::vector<uint8_t>(px, kNoOwner);
  const int wx0 = p.write.x - p.blend.x, wy0 = p.write.y - p.blend.y;
  for (int y = wy0; y < wy0 + p.write.h; ++y)
    for (int x = wx0; x < wx0 + p.write.w; ++x) {
      const int i = (x - c.fx0) / 64, j = (y - c.fy0) / 16;
      if (c.block_class[size_t(j) * c.nfx + i] != kBlockCopy) continue;
      const int label = p.mask0[size_t(y) * p.lw[0] + x];
      const GatherPlane& s = p.slots[p.rule == kRuleTwo ? (label == 1 ? 0 : 1) : label];
      const size_t d = size_t(y + p.blend.y) * p.canvas_w + (x + p.blend.x);
      map[d] = kNoEntry;
      owner[d] = kNoOwner;
      if (!s.rect.contains(x, y)) continue;
      const size_t q = size_t(y - s.rect.y) * s.rect.w + (x - s.rect.x);
      map[d] = s.map[q];
      if (s.map[q] != kNoEntry) owner[d] = s.owner.empty() ? uint8_t(s.default_owner) : s.owner[q];
    }
}

int main(int argc, char** argv) {
  const int iters = atoi(argv[1]);
  std::mt19937 rng(atoi(argv[2]));
  long planned = 0, planes = 0;
  for (int it = 0; it < iters; ++it) {
    const int kinds[3] = {HMP_KIND_PANON, HMP_KIND_PANO2, HMP_KIND_PANO3};
    const int kind = kinds[rng() % 3];
    const int n = kind == HMP_KIND_PANO2 ? 2 : kind == HMP_KIND_PANO3 ? 3 : 2 + int(rng() % 5);
    const int h = 40 + int(rng() % 150), fw = 140 + int(rng() % 160), step = fw - 30 - int(rng() % 60);
    const int W = step * (n - 1) + fw, first = rng() % 4 == 0 ? int(rng() % 9) : 0;
    std::vector<std::vector<uint16_t>> mx(n), my(n);
    std::vector<hmp_remap> rm(n);
    for (int i = 0; i < n; ++i) {
      const int top = int(rng() % 5), rows = h - top - int(rng() % 5);
      mx[i].resize(size_t(fw) * rows);
      my[i].resize(mx[i].size());
      for (size_t q = 0; q < mx[i].size(); ++q) {
        mx[i][q] = uint16_t(q % fw);
        my[i][q] = uint16_t(q / fw);
        if (rng() % 4000 == 0) mx[i][q] = my[i][q] = 65535;
      }
      rm[i] = hmp_remap{mx[i].data(), my[i].data(), fw, rows, i * step + (i == 0 ? first : 0), top};
    }
    std::vector<uint8_t> seam(size_t(W) * h);
    int at[8] = {};
    for (int y = 0; y < h; ++y)
      for (int i = 0, x = 0; i < n; ++i) {
        at[i] += int(rng() % 3) - 1;
        const int end = i == n - 1 ? W : step * (i + 1) + (fw - step) / 2 + std::max(-10, std::min(10, at[i]));
        for (; x < end && x < W; ++x) seam[size_t(y) * W + x] = uint8_t(kind == HMP_KIND_PANO2 ? 1 - i : i);
      }
    if (rng() % 5 == 0) seam[rng() % seam.size()] = 9;
    hmp_config c{};
    c.kind = kind;
    c.n_images = n;
    c.num_levels = 2 + int(rng() % 6);
    c.batch_size = 1;
    c.channels = rng() % 3 ? 3 : 4;
    c.minimize_blend = rng() % 2;
    c.fused = 1;
    c.remaps = rm.data();
    c.seam = seam.data();
    c.seam_width = W;
    c.seam_height = h;
    Plan p;
    std::string m;
    if (build_plan(c, p, m) != HMP_OK) continue;
    const int align = 1 << (p.levels - 1), t1 = std::max(32, align / 2);
    CopyPlan a, b, d;
    plan_copy_blocks(p, 64, t1, a);
    if (32 % align == 0) {
      replan_tiles(p, 32, t1, a, b);
      plan_copy_blocks(p, 32, t1, d);
      if (!same(b, d, n)) return printf("iteration %d: replanned lists differ\n", it), 1;
    }
    replan_tiles(p, 64, t1, a, b);
    if (!same(a, b, n)) return printf("iteration %d: the plan of the same edge differs\n", it), 1;
    planned += a.usable;
    if (!p.rgb8() || !a.usable) continue;
    const bool had = p.canvas_plane_used;
    std::vector<uint32_t> map;
    std::vector<uint8_t> owner;
    expected(p, a, had, p.canvas, map, owner);
    rgb_canvas_plane(p, a);
    if (!p.canvas_plane_used || p.canvas.map != map || p.canvas.owner != owner)
      return printf("iteration %d: canvas plane differs\n", it), 1;
    ++planes;
  }
  printf("planned %ld planes %ld\n", planned, planes);
  return 0;
}
