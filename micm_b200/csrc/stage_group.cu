// stage_group.cu -- the single-stage entry points on the cell-group engine
// (group.cuh): a block brings G cells' arrays into shared memory, runs one stage
// on them and writes its result back, so a factor is read and written once
// instead of once per term.  The sums and their order are those of the
// thread-per-cell kernels.
#include "runtime.hpp"
#include "group.cuh"

#include <algorithm>

namespace micmb
{
  namespace
  {
    __device__ __forceinline__ size_t cell_base(int64_t c, int32_t L, int32_t ncol)
    {
      return (size_t)(c / L) * (size_t)L * (size_t)ncol + (size_t)(c % L);
    }

    struct StageArgs
    {
      int64_t n;
      int32_t L;
      const double* y;
      const double* k;
      double* f;    // S columns: forcing, or the solve's vector
      double* jac;  // nnz columns
    };

    // elements [e0, e0 + n) of this thread's cell from / to global memory, eight
    // loads under way at a time
    template<int G>
    __device__ __forceinline__ void bring(const GroupThread<G>& X, int32_t e0, int32_t n, const double* from, int32_t L)
    {
      constexpr int B = 8;
      for (int32_t i0 = X.lane; i0 < n; i0 += B * X.lanes)
      {
        double v[B];
#pragma unroll
        for (int b = 0; b < B; ++b)
          v[b] = from[(int64_t)min(i0 + b * X.lanes, n - 1) * L];
#pragma unroll
        for (int b = 0; b < B; ++b)
          if (i0 + b * X.lanes < n)
            X[e0 + i0 + b * X.lanes] = v[b];
      }
    }
    template<int G>
    __device__ __forceinline__ void put(const GroupThread<G>& X, int32_t e0, int32_t n, double* to, int32_t L)
    {
#pragma unroll 4
      for (int32_t i = X.lane; i < n; i += X.lanes)
        to[(int64_t)i * L] = X[e0 + i];
    }

    template<int G, GroupStage STAGE>
    __global__ void __launch_bounds__(256, 1) k_group_stage(DevGroup P, const int32_t* diag_pos, StageArgs a)
    {
      extern __shared__ __align__(16) double shared[];
      const GroupThread<G> X(shared);
      const int32_t S = P.S, L = a.L;
      if (X.lane == 0)
      {
        X[P.zero] = 0.0;
        X[P.one] = 1.0;
        X[P.trash] = 1.0;
      }
      for (int64_t first = (int64_t)blockIdx.x * G; first < a.n; first += (int64_t)gridDim.x * G)
      {
        const int64_t c = first + (threadIdx.x & (G - 1));
        const bool live = c < a.n;
        const int64_t cc = live ? c : a.n - 1;  // spare lanes repeat the last cell and write nothing
        double* f = a.f + cell_base(cc, L, S);
        double* jac = a.jac + cell_base(cc, L, P.nnz);
        if (STAGE == GroupStage::kForcing || STAGE == GroupStage::kJacobian)
        {
          bring(X, P.v0, S, a.y + cell_base(cc, L, S), L);
          if (STAGE == GroupStage::kJacobian)
            bring(X, 0, P.nnz, jac, L);
          __syncthreads();
          const double* k = a.k + cell_base(cc, L, P.R);
          if (STAGE == GroupStage::kForcing)
            group_rates<G>(P, X, k, L);
          else
            group_drates<G>(P, X, k, L);
          __syncthreads();
          if (STAGE == GroupStage::kForcing)
            run_gather<G>(P.forcing, X, 0.0);
          else
            run_gather<G, true>(P.jacobian, X, 0.0);
          __syncthreads();
          if (live && STAGE == GroupStage::kForcing)
            for (int32_t i = X.lane; i < S; i += X.lanes)
              f[(int64_t)i * L] = f[(int64_t)i * L] + X[P.v0 + i];
          if (live && STAGE == GroupStage::kJacobian)
            put(X, 0, P.nnz, jac, L);
        }
        else
        {
          bring(X, 0, P.nnz, jac, L);
          if (STAGE == GroupStage::kSolve)
            bring(X, P.v0, S, f, L);
          if (X.lane == 0)
            X[P.inv + S] = 1.0;
          __syncthreads();
          if (STAGE == GroupStage::kLu)
            run_levels<G, true>(P.lu, X, P);
          else
          {
            for (int32_t i = X.lane; i < S; i += X.lanes)
              X[P.inv + i] = 1.0 / X[__ldg(diag_pos + i)];
            __syncthreads();
            run_levels<G, false>(P.solve, X, P);
          }
          __syncthreads();
          if (live && STAGE == GroupStage::kLu)
            put(X, 0, P.nnz, jac, L);
          if (live && STAGE == GroupStage::kSolve)
            put(X, P.v0, S, f, L);
        }
        __syncthreads();
      }
    }

    using StageKernel = void (*)(DevGroup, const int32_t*, StageArgs);

    template<GroupStage STAGE>
    StageKernel StageKernelFor(int32_t G)
    {
      switch (G)
      {
        case 1: return k_group_stage<1, STAGE>;
        case 2: return k_group_stage<2, STAGE>;
        case 4: return k_group_stage<4, STAGE>;
        case 8: return k_group_stage<8, STAGE>;
        case 16: return k_group_stage<16, STAGE>;
        default: return k_group_stage<32, STAGE>;
      }
    }
  }  // namespace

  namespace
  {
    // The cells that a cell-group launch of one stage does in the time of one set of
    // threads.  The groups bring all of a cell's arrays into shared memory and back, the
    // threads read what a stage needs: the solve, which reads the factor once either
    // way, has the lowest line, the LU, which reads it once per term, the highest.
    // Measured, thousands of cells (thread kernels' time of one set: 60 species 0.29,
    // 0.64, 0.62, 0.25 ms; TS1 1.4, 3.2, 4.1, 1.1; 600 species 3.1, 9.3, 29, 4.2):
    //                                forcing  Jacobian   LU   solve
    //   Chapman                         40        90      45    45
    //   60 species (32 cells per SM)   115       125     140    62
    //   TS1 (8)                        100       115     130    40
    //   210 species (8)                 74        98     132    42
    //   600 species (1)                 21        36      63    13
    int64_t EqualCells(const micmb_solver& s, GroupStage stage)
    {
      static constexpr int64_t many[4] = { 770, 840, 940, 420 }, some[4] = { 500, 660, 880, 270 },
                               one[4] = { 145, 240, 430, 88 };  // cells per SM of the GPU
      const int i = (int)stage;
      if (s.mech->nnz < kTinyNonZeros)
        return 300 * (int64_t)s.sm_count;
      const int64_t cells = GroupCellsPerSm(s);
      return s.sm_count * (cells >= 16 ? many[i] : (cells >= 4 ? some[i] : std::min(cells * one[i], some[i])));
    }
  }  // namespace

  bool LaunchGroupStage(micmb_solver& s, micmb_state& st, GroupStage stage, const void* thread_kernel, int block)
  {
    const int64_t n = st.n_cells;
    if (n < 1 || !GroupFaster(s, n) || !GroupBeatsThreads(s, n, EqualCells(s, stage), thread_kernel, block))
      return false;
    const GroupChoice choice = ChooseGroup(s, n);
    const StageKernel kernel = stage == GroupStage::kForcing    ? StageKernelFor<GroupStage::kForcing>(choice.G)
                               : stage == GroupStage::kJacobian ? StageKernelFor<GroupStage::kJacobian>(choice.G)
                               : stage == GroupStage::kLu       ? StageKernelFor<GroupStage::kLu>(choice.G)
                                                                : StageKernelFor<GroupStage::kSolve>(choice.G);
    const int per_sm = GroupBlocksPerSm(s, reinterpret_cast<const void*>(kernel), choice);
    if (per_sm < 1)
      return false;
    StageArgs a{};
    a.n = n;
    a.L = st.L;
    a.y = st.variables.as<double>();
    a.k = st.rate_constants.as<double>();
    a.f = st.forcing0.as<double>();
    a.jac = st.jacobian.as<double>();
    const int64_t grid = std::min<int64_t>((int64_t)per_sm * s.sm_count, (n + choice.G - 1) / choice.G);
    kernel<<<(unsigned)grid, 32 * choice.W, GroupSharedBytes(s, choice), st.stream>>>(GroupTablesFor(s, choice).dev,
                                                                                     s.dev.diag_pos, a);
    MICMB_CUDA(cudaGetLastError());
    return true;
  }
}  // namespace micmb
