// group.hpp -- work lists of the cell-group kernels: a block of W warps solves
// G grid cells in lockstep with their LU factors and vectors in shared memory,
// element e of cell g at e * G + g.
//
// A warp is 32 / G item lanes of G cells each.  The items of a phase (LU
// entries, solution components, gathered sums) are cut into chunks of 32 / G
// items, one per item lane, padded to the chunk's longest sum with products of
// the zero element, which leave every sum bit-identical.  Chunks are packed into
// units of 16 terms per lane -- four chunks of up to four terms, two of up to
// eight, or a stretch of one long chunk -- so that a warp works on independent
// sums side by side and decides what to do once per unit.  Every warp walks its
// own list of units; the lists of a phase agree on where the block synchronises.
#pragma once

#include "mechanism.hpp"

#include <cstdint>
#include <vector>

namespace micmb
{
  // element index space of one cell in shared memory
  struct GroupLayout
  {
    int32_t zero, one;  // constants 0.0 and 1.0
    int32_t v0;         // S: the state a rate reads, then the stage vector being solved
    int32_t trash;      // what idle lanes write
    int32_t w0;         // Jacobian rates (n_info), later inv and the rates
    int32_t inv;        // S: 1 / u_ii, and 1.0 as the trash element's
    int32_t rate;       // max(R, S): reaction rates, then the scaled squared errors
    int32_t g2;         // backward sweep, in place of the rates: S, what reactions project on
    int32_t slot;       // and their contributions, one per (reaction, reactant) ...
    int32_t elements;
  };
  // sweep_stages: 0, or the stages of the adjoint's backward sweep.  The
  // contributions of a whole step, of which there are more, begin in the factor,
  // which is no longer needed then: contribution i is element i below nnz, and
  // slot + i - nnz from there on.
  GroupLayout MakeGroupLayout(const CompiledMechanism& m, int32_t sweep_stages = 0);

  // What becomes of a unit's sums v.  Level phases: kGroupPlain stores v * [aux] in
  // the LU and v in the solves; kGroupPivot stores v and [aux] = 1 / v in the LU, and
  // v / [aux] in the solves (the reciprocal of [aux] is at target - v0 + inv).
  // kGroupNone: a stretch of a long sum that goes on in the next unit.
  constexpr int32_t kGroupPlain = 0, kGroupPivot = 1, kGroupNone = 2;
  // what follows a unit
  constexpr int32_t kGroupNoSync = 0, kGroupWarpSync = 1, kGroupBlockSync = 2;

  // Unit shapes: chunks and terms per chunk.  A unit has room for 16 terms; those
  // past a chunk's longest sum are not run.
  struct GroupShape
  {
    int32_t chunks, terms;
  };
  constexpr GroupShape kGroupShapes[7] = { { 1, 4 }, { 1, 8 }, { 1, 16 }, { 2, 4 }, { 2, 8 }, { 4, 2 }, { 4, 4 } };
  constexpr int32_t kGroupTerms = 16;

  // Unit u, item lane p (chunk k starts at term k * 16 / chunks):
  //   ctrl[u]: shape * 3 + what becomes of the sums | sync << 8 | (first unit of a
  //            sum) << 10
  //   item[(u * ipw + p) * 4 + k]: chunk k's target | aux << 16 (gathers: aux 1 adds
  //            alpha); idle lanes work on the trash element
  //   the unit's terms t = 0..15 of the lane:
  //     level phases: row[((u * 4 + t / 4) * ipw + p) * 4 + t % 4], a | b << 16
  //     gathers: row[((u * 2 + t / 8) * ipw + p) * 4 + t % 8 / 2], the values, two per
  //              word; coef[((u * 8 + t / 2) * ipw + p) * 2 + t % 2]
  struct GroupPhase
  {
    std::vector<int32_t> warp_start;  // [W + 1] first unit of each warp
    std::vector<uint32_t> ctrl;
    std::vector<uint32_t> item;
    std::vector<uint32_t> row;
    std::vector<double> coef;
  };

  struct GroupProgram
  {
    int32_t G = 0, W = 0;
    GroupLayout layout{};
    GroupPhase forcing;  // sweep: one evaluation's contributions to each species, into V
    GroupPhase jacobian, lu;
    GroupPhase solve;  // forward, then backward substitution (sweep: with the transposed factors)
    GroupPhase step;   // sweep: a step's contributions to each species, added to V
    std::vector<int32_t> step_start;  // sweep: [R] a reaction's first contribution
    std::vector<uint32_t> rate;   // [2R]: reactant elements a | b << 16, c (one where there are fewer)
    std::vector<uint32_t> drate;  // [2 n_info]: rate column | a << 16, b | c << 16
  };

  // Whether the mechanism has group work lists at all (16-bit elements, at most
  // three reactants, no algebraic constraints).
  bool GroupApplies(const CompiledMechanism& m);
  GroupProgram BuildGroupProgram(const CompiledMechanism& m, int32_t G, int32_t W, int32_t sweep_stages = 0);
}  // namespace micmb
