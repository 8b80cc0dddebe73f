// group.hpp -- work lists of the cell-group kernels: a block of W warps solves
// G grid cells in lockstep with their LU factors and vectors in shared memory,
// element e of cell g at e * G + g.
//
// A warp is 32 / G item lanes of G cells each.  The items of a phase (LU
// entries, solution components, gathered sums) are cut into chunks of 32 / G
// items, one per item lane; a chunk's terms are stored lane-interleaved and
// padded to its longest item with products of the zero element, which leave
// every sum bit-identical.  Every warp walks its own chunk list; the lists of
// a phase agree on where the block synchronises.
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
    int32_t inv;        // S: 1 / u_ii
    int32_t rate;       // max(R, S): reaction rates, then the scaled squared errors
    int32_t elements;
  };
  GroupLayout MakeGroupLayout(const CompiledMechanism& m);

  constexpr uint32_t kGroupNoItem = 0xFFFFFFFFu;
  // how a chunk's sums become values
  constexpr int32_t kGroupScale = 0;  // v * [aux]
  constexpr int32_t kGroupRecip = 1;  // v, and [aux] = 1 / v
  constexpr int32_t kGroupDiv = 2;    // v / [aux], with the reciprocal of [aux] at target - v0 + inv
  constexpr int32_t kGroupStore = 3;  // v
  // what follows a chunk
  constexpr int32_t kGroupNoSync = 0, kGroupWarpSync = 1, kGroupBlockSync = 2;

  // A warp's chunks become a straight run of records of up to four terms, read in
  // units of four records so that a whole unit is fetched while the one before
  // it is worked on.  Elements appear as byte offsets (element * G * 8), so that
  // an operand's address is one addition.  Record r = 4 u + j, item lane p:
  //   ctrl[r]: T | first << 3 | last << 4 | kind << 5 | sync << 7 (T: the record's
  //            terms, 0..4; first/last record of a chunk)
  //   level phases: item[((u * ipw + p) * 4 + j) * 2 ..], target and aux;
  //                 row[((r * 2 + h) * ipw + p) * 4 ..], terms 2 h and 2 h + 1, two
  //                 operands each; idle lanes work on the trash element
  //   gathers: item[(u * ipw + p) * 4 + j], target index | flag << 16 (flag: adds
  //            alpha) or kGroupNoItem; row[(r * ipw + p) * 4 ..], the four values;
  //            coef[((r * 2 + h) * ipw + p) * 2 ..], their coefficients
  constexpr int32_t kGroupUnit = 4;
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
    GroupPhase forcing, jacobian, lu;
    GroupPhase solve;  // forward, then backward substitution
    std::vector<uint32_t> rate;   // [2R]: reactant elements a | b << 16, c (one where there are fewer)
    std::vector<uint32_t> drate;  // [2 n_info]: rate column | a << 16, b | c << 16
  };

  // Whether the mechanism has group work lists at all (16-bit elements, at most
  // three reactants, no algebraic constraints).
  bool GroupApplies(const CompiledMechanism& m);
  GroupProgram BuildGroupProgram(const CompiledMechanism& m, int32_t G, int32_t W);
}  // namespace micmb
