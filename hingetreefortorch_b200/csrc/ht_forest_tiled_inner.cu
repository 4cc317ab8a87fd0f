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

// Rounds of CTAs, each staging its tile and walking its share of the tree groups, like forward_tiled_cost().  A group costs the walks
// of a warp's trees and, for several outputs per leaf, what their form does: dealing out (five and more) pays for the 32 / K rows that a
// warp's samples are on.  Tiles read all of x and write all outputs, in bursts that the walks hide in part: 0.15 and 0.06 us per MB, and
// as much again for x where it does not stay in L2.  Scalar loads (K no multiple of four) stage a tile in 0.29 us per 1000 numbers.
double inner_tiled_cost(const ht_forest_problem *p, bool keep) {
  tile::TilePlan plan;
  if (!tile::make_inner_plan(p, plan)) return -1.0;
  const int64_t tiles = (p->B * p->K + plan.S - 1) / plan.S, groups = (p->T + plan.G - 1) / plan.G;
  const int splits = tile::choose_splits(tiles, groups);
  const double waves = (double)((tiles * splits + 147) / 148), per_cta = (double)((groups + splits - 1) / splits);
  const double walk = plan.per_warp == 4 ? 0.553 + 0.161 * p->depth : plan.per_warp == 2 ? 0.675 + 0.0986 * p->depth : 0.952 + 0.0326 * p->depth;
  const double evals = 1e-3 * plan.G * plan.S, pieces = evals * (double)p->M / vector_width(p->M, sizeof(float), {});
  const double output = pieces * ((p->M > 4 ? 0.136 + 0.0166 * 32.0 / (double)p->K : p->M > 1 ? 0.0260 : 0.0) + (plan.weights ? 0.0 : 0.0855)) +
                        (keep && p->M > 1 ? 0.223 * evals : 0.0);
  const double staging = (double)p->C * (0.0899e-3 + ((p->K & 3) != 0 ? 0.292e-3 * plan.S : 0.0));
  const double read = 4e-6 * (double)p->B * (double)p->C * (double)p->K, written = 4e-6 * (double)p->B * (double)p->K * (double)p->T * (double)p->M;
  return 3.60 + waves * (2.42 + staging + per_cta * (walk + output)) + 0.154 * read + 0.158 * std::max(0.0, read - 100.0) + 0.0645 * written;
}

namespace tile {

int launch_inner(int kind, int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  return kind == TREE ? launch_inner_kind<TREE>(depth, plan, a, grid, stream) : launch_inner_ferns(depth, plan, a, grid, stream);
}

}  // namespace tile
}  // namespace ht
