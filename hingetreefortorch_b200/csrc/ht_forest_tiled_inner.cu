// Trees on inputs with inner positions, and the plan for both kinds.
#include "ht_forest_tiled_inner.cuh"

namespace ht {
namespace tile {

// Inputs with inner positions (x [B, C, K], K > 1): a sample is a (row, position)
// pair and its features are K elements apart, so consecutive samples of a tile are consecutive
// positions — contiguous in x and, for a fixed tree, in the output.  No staging of results is needed.
bool make_inner_plan(const ht_forest_problem *p, TilePlan &plan) {
  if (p->K <= 1 || p->M < 1 || p->M > 64) return false;
  if (p->C > 65536 || p->depth > 12 || p->K > 0x3fffffff) return false;
  if (p->B * p->K * p->T < 32 * 1024) return false;
  plan.ord_bytes = p->C <= 256 ? 1 : 2;
  const bool paired = paired_ordinals(p->kind, p->depth, (uint32_t)plan.ord_bytes);
  auto fits = [&](int S, bool weights) {
    plan.weights = weights;
    plan.rec = record_layout(p->kind, p->depth, (uint32_t)plan.ord_bytes, weights, paired);
    if (weights) plan.rec.bytes = round16(plan.rec.w + 4u * (uint32_t)p->M * (1u << p->depth));
    plan.S = S;
    for (plan.per_warp = 4; plan.per_warp >= 1; plan.per_warp >>= 1) {
      plan.G = (kWarps / (S / 32)) * plan.per_warp;
      plan.smem = (size_t)p->C * S * 4 + 2 * (size_t)plan.G * plan.rec.bytes + 64;
      if (plan.smem <= kSmemBudget) return true;
    }
    return false;
  };
  // One output per leaf: its weights in the records wherever those of four trees per warp fit.
  if (p->M == 1)
    for (int S = 256; S >= 32; S >>= 1)
      if (fits(S, true) && plan.per_warp == 4) return true;
  // Several outputs per leaf: the weights join the records where a warp's walk pays for bringing them (a record is shared by the S / 32
  // warps that walk its tree) and two trees at a time still fit.
  for (int S = 256; S >= 32; S >>= 1) {
    if (p->M > 1 && (((int64_t)p->M << p->depth) + 512) * 4 * 32 / S <= 4096 && fits(S, true) && plan.per_warp > 1) return true;
    if (fits(S, false)) return true;
  }
  return false;
}

}  // namespace tile

// Rounds of CTAs, each staging its tile and walking its share of the tree groups, like forward_tiled_cost(); the outputs of a group
// cost what their form does.
double inner_tiled_cost(const ht_forest_problem *p, bool keep) {
  tile::TilePlan plan;
  if (!tile::make_inner_plan(p, plan)) return -1.0;
  const int64_t tiles = (p->B * p->K + plan.S - 1) / plan.S, groups = (p->T + plan.G - 1) / plan.G;
  const int splits = tile::choose_splits(tiles, groups);
  const double waves = (double)((tiles * splits + 147) / 148), per_cta = (double)((groups + splits - 1) / splits);
  const double level = plan.per_warp == 1 ? 0.0241 : plan.per_warp == 2 ? 0.0832 : 0.150;
  const double evals = 1e-3 * plan.G * plan.S, pieces = evals * (double)p->M / vector_width(p->M, sizeof(float), {});
  const double output = pieces * ((p->M > 4 ? 0.182 : p->M > 1 ? 0.0225 : 0.0) + (plan.weights ? 0.0 : 0.107)) +
                        evals * (0.0110 * (double)p->M + (keep && p->M > 1 ? 0.217 : 0.0));
  return 0.3 + waves * (1.87 + 0.226e-3 * plan.S * (double)p->C + per_cta * (0.968 + level * p->depth + output));
}

namespace tile {

int launch_inner(int kind, int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  return kind == TREE ? launch_inner_kind<TREE>(depth, plan, a, grid, stream) : launch_inner_ferns(depth, plan, a, grid, stream);
}

}  // namespace tile
}  // namespace ht
