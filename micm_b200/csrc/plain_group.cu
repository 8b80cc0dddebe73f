// plain_group.cu -- the plain method with one step size for all cells (micm's
// own semantics) on the cell-group kernels: one launch runs a whole step attempt
// of every cell (group.cuh), so the factor and the stage vectors of a cell never
// make a round trip through memory between the stages; a second, small launch
// reduces the cells' error sums in the fixed order of the per-stage kernels and
// takes the step-size decision.
#include "runtime.hpp"
#include "group.cuh"

#include <algorithm>

namespace micmb
{
  namespace
  {
    constexpr int kBlock = 256;

    __device__ __forceinline__ size_t cell_base(int64_t c, int32_t L, int32_t ncol)
    {
      return (size_t)(c / L) * (size_t)L * (size_t)ncol + (size_t)(c % L);
    }

    struct GlobalCtl
    {
      CellCtl c;
      int32_t status;    // MICMB_SOLVER_*
      int32_t accepted;  // the last attempt's Ynew is the state
      uint32_t ticket;   // blocks of the running reduction that are done
    };

    struct GlobalArgs
    {
      int64_t n;
      int32_t L;
      double* y;
      double* ynew;
      const double* k;
      const double* atol;
      double rtol;
      GlobalCtl* ctl;
      double* cell_err;  // [n] sums of scaled squared errors
      double* blk_err;   // per 256 cells
    };

    // top of micm's outer loop
    __device__ __forceinline__ void begin_step(CellCtl& c, int32_t& status, const DevParams& D, const StepBounds& B)
    {
      if (ctl_begin_step(c, D, B))
      {
        c.function_calls += 1;    // initial forcing
        c.jacobian_updates += 1;  // Jacobian at the start of the step
      }
      else
      {
        status = c.state;
        c.new_step = 0;
      }
    }

    __global__ void k_global_begin(GlobalCtl* ctl, DevParams D, StepBounds B)
    {
      GlobalCtl g;
      ctl_init(g.c, B);
      g.status = MICMB_SOLVER_RUNNING;
      g.accepted = 0;
      g.ticket = 0;
      begin_step(g.c, g.status, D, B);
      *ctl = g;
    }

    // One attempt of every cell; a block takes the cells group by group.  Ynew
    // goes to its own array; where the last attempt was accepted, this one reads
    // the state from there and completes it in y.
    template<int G>
    __global__ void __launch_bounds__(256, 1) k_global_attempt(DevGroup P, DevParams D, GlobalArgs a, double* ws, int64_t slot_doubles)
    {
      extern __shared__ __align__(16) double shared[];
      if (a.ctl->status != MICMB_SOLVER_RUNNING)
        return;
      const GroupThread<G> X(shared);
      const int32_t S = P.S, L = a.L;
      GroupVectors v = group_vectors<G>(ws + (int64_t)blockIdx.x * slot_doubles, P);
      v.ks = L;
      const bool accepted = a.ctl->accepted != 0;
      const double H = a.ctl->c.H;
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
        const int64_t cc = live ? c : a.n - 1;
        const size_t by = cell_base(cc, L, S);
        const double* y = (accepted ? a.ynew : a.y) + by;
        v.kk = a.k + cell_base(cc, L, P.R);
        for (int32_t i = X.lane; i < S; i += X.lanes)
        {
          const double yi = live ? y[(int64_t)i * L] : 0.0;
          X[P.v0 + i] = yi;
          v.Y[(int64_t)i * G] = yi;
          if (live && accepted)
            a.y[by + (size_t)i * L] = yi;
        }
        __syncthreads();
        group_attempt<G>(P, D, X, v, H, a.atol, a.rtol);
        if (live)
          for (int32_t i = X.lane; i < S; i += X.lanes)
            a.ynew[by + (size_t)i * L] = X[P.v0 + i];
        __syncthreads();
        if (threadIdx.x < G && live)
        {
          double sum = 0.0;
#pragma unroll 8
          for (int32_t i = 0; i < S; ++i)
            sum += X[P.rate + i];
          a.cell_err[c] = sum;
        }
        __syncthreads();
      }
    }

    // Fixed-shape tree over the kBlock values of a block (every thread returns the total).
    __device__ __forceinline__ double block_tree_sum(double v, double* red)
    {
      red[threadIdx.x] = v;
      __syncthreads();
      for (int w = kBlock / 2; w > 0; w >>= 1)
      {
        if ((int)threadIdx.x < w)
          red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
      }
      return red[0];
    }

    // The cells' sums to one total in the per-stage kernels' order: a tree per
    // 256 cells, then the block totals by one block (each thread a strided
    // sequential sum, then a tree).  The block that finishes last does the
    // second part; it returns true there, with the total.
    __device__ __forceinline__ bool reduce_cells(const GlobalArgs& a, double* red, double& total)
    {
      __shared__ bool last;
      const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
      const double t = block_tree_sum(c < a.n ? a.cell_err[c] : 0.0, red);
      if (threadIdx.x == 0)
      {
        a.blk_err[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(&a.ctl->ticket, 1u) + 1 == gridDim.x;
        __threadfence();
      }
      __syncthreads();
      if (!last)
        return false;
      double acc = 0.0;
      for (int64_t i = threadIdx.x; i < (int64_t)gridDim.x; i += kBlock)
        acc += __ldcg(a.blk_err + i);
      total = block_tree_sum(acc, red);
      return true;
    }

    // micm's step control from the job's sum of squared scaled errors
    __device__ __forceinline__ void decide(const GlobalArgs& a, const DevParams& D, const StepBounds& B, double total,
                                           double n_values)
    {
      const double error = error_from_sum(total, n_values > 0.0 ? n_values : 1.0);
      GlobalCtl g = *a.ctl;
      g.c.decompositions += 1;
      g.c.solves += D.stages;
      for (int32_t s = 1; s < D.stages; ++s)
        g.c.function_calls += D.new_f[s] ? 1 : 0;
      const int res = ctl_after_error(g.c, D, B, error);
      g.accepted = res == 1;
      g.status = g.c.state;
      g.ticket = 0;
      if (res == 1)
        begin_step(g.c, g.status, D, B);
      *a.ctl = g;
    }

    __global__ void k_global_step(GlobalArgs a, DevParams D, StepBounds B, int32_t S)
    {
      __shared__ double red[kBlock];
      if (a.ctl->status != MICMB_SOLVER_RUNNING)
        return;
      double total;
      if (reduce_cells(a, red, total) && threadIdx.x == 0)
        decide(a, D, B, total, (double)(a.n * (int64_t)S));
    }

    // Several ranks, first half: this shard's sum for the exchange.
    __global__ void k_global_shard(GlobalArgs a, double* shard_sum)
    {
      __shared__ double red[kBlock];
      if (a.ctl->status != MICMB_SOLVER_RUNNING)
        return;
      double total;
      if (reduce_cells(a, red, total) && threadIdx.x == 0)
      {
        *shard_sum = total;
        a.ctl->ticket = 0;
      }
    }

    // Several ranks, second half: the gathered shard sums added in rank order.
    __global__ void k_global_step_gathered(GlobalArgs a, DevParams D, StepBounds B, const double* gathered,
                                           int32_t world, double n_values)
    {
      if (a.ctl->status != MICMB_SOLVER_RUNNING)
        return;
      double total = 0.0;
      for (int32_t r = 0; r < world; ++r)
        total += gathered[r];
      decide(a, D, B, total, n_values);
    }

    // the final state, clamped at zero (Solver::PostSolveClamp, solver.hpp:275-297)
    __global__ void k_global_finish(GlobalArgs a, int32_t S)
    {
      const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
      const int64_t per_group = (int64_t)S * a.L;
      const int64_t g = idx / per_group;
      if (g * a.L + idx % a.L >= a.n)
        return;
      const double y = a.ctl->accepted ? a.ynew[idx] : a.y[idx];
      a.y[idx] = (y < 0.0) ? 0.0 : y;
    }

    using AttemptKernel = void (*)(DevGroup, DevParams, GlobalArgs, double*, int64_t);

    AttemptKernel AttemptKernelFor(int32_t G)
    {
      switch (G)
      {
        case 1: return k_global_attempt<1>;
        case 2: return k_global_attempt<2>;
        case 4: return k_global_attempt<4>;
        case 8: return k_global_attempt<8>;
        case 16: return k_global_attempt<16>;
        default: return k_global_attempt<32>;
      }
    }

    inline unsigned Blocks(int64_t n)
    {
      return (unsigned)std::max<int64_t>(1, (n + kBlock - 1) / kBlock);
    }
  }  // namespace

  bool SolveGlobalGroup(micmb_solver& s, micmb_state& st, double dt, micmb_solver_stats* stats,
                        int32_t* per_cell_status, int32_t* per_cell_accepted)
  {
    const auto& m = *s.mech;
    const int64_t n = st.n_cells;
    // With one step size every cell takes every attempt, and the per-stage kernels
    // have no lanes that wait for others': they are the faster form at large counts
    // (210 species, 1,048,576 cells, ms per attempt: 95 against 129), the cell groups
    // below the count that fills the GPU with threads.  Measured, ms, cell groups /
    // per-stage kernels: Chapman 151,000 cells 2.3 / 3.1; 60 species (32 cells per SM)
    // 151,000 469 / 621; TS1 (8) 10,000 70 / 641, 130,000 884 / 926; 210 species (8) 98,000
    // 1,137 / 1,373, 120,000 1,456 / 1,474, 131,000 1,520 / 1,413; 600 species (1) 16,000
    // 3,569 / 7,599.
    if (n < 1 || !GroupVariantApplies(s, n))
      return false;
    const int64_t cells = GroupCellsPerSm(s);
    if (n > std::min<int64_t>((int64_t)s.sm_count * (cells >= 16 ? 1024 : 820), 16384 * cells))
      return false;
    if (n == 1 && !st.gx_fn)
    {
      // one cell: the single step size is the cell's own, and the whole solve is
      // one launch (Chapman: 0.52 ms with two launches per attempt)
      if (!st.group_ctl.p)
        st.group_ctl = DeviceMemory(sizeof(GlobalCtl));
      double* t = reinterpret_cast<double*>(st.group_ctl.p);
      if (!SolvePlainPerCellGroup(s, st, dt, stats, per_cell_status, per_cell_accepted, t))
        return false;
      if (stats)
        MICMB_CUDA(cudaMemcpy(&stats->final_time, t, sizeof(double), cudaMemcpyDeviceToHost));
      return true;
    }
    const GroupChoice choice = ChooseGroup(s, n);
    const size_t smem = GroupSharedBytes(s, choice);
    const AttemptKernel kernel = AttemptKernelFor(choice.G);
    const int per_sm = GroupBlocksPerSm(s, reinterpret_cast<const void*>(kernel), choice);
    if (per_sm < 1)
      return false;
    const GroupTables& t = GroupTablesFor(s, choice);
    const int64_t grid = std::min<int64_t>((int64_t)per_sm * s.sm_count, (n + choice.G - 1) / choice.G);
    const int64_t slot = GroupVectorDoubles(m.S, s.params.stages) * choice.G;
    EnsureWorkspace(st, st.group_ws, grid * slot);
    const unsigned n_blk = Blocks(n);
    if (!st.group_ynew.p)
      st.group_ynew = DeviceMemory(st.dense_bytes(m.S));
    if (!st.group_err.p)
      st.group_err = DeviceMemory(sizeof(double) * ((size_t)n + n_blk));
    if (!st.group_ctl.p)
      st.group_ctl = DeviceMemory(sizeof(GlobalCtl));
    const DevParams D = s.params;
    const StepBounds B = step_bounds(D, dt);
    GlobalArgs a{};
    a.n = n;
    a.L = st.L;
    a.y = st.variables.as<double>();
    a.ynew = st.group_ynew.as<double>();
    a.k = st.rate_constants.as<double>();
    a.atol = st.atol.as<double>();
    a.rtol = st.rtol;
    a.ctl = st.group_ctl.as<GlobalCtl>();
    a.cell_err = st.group_err.as<double>();
    a.blk_err = a.cell_err + n;
    cudaStream_t stream = st.stream;
    const int threads = 32 * choice.W;

    k_global_begin<<<1, 1, 0, stream>>>(a.ctl, D, B);
    MICMB_CUDA(cudaGetLastError());
    int64_t attempts = 0, batch = 8;
    const int64_t max_attempts = (int64_t)(D.max_steps + 2) * 2000;
    for (;;)
    {
      for (int64_t it = 0; it < batch; ++it)
      {
        kernel<<<(unsigned)grid, threads, smem, stream>>>(t.dev, D, a, st.group_ws.as<double>(), slot);
        if (st.gx_fn)
        {
          double* gx = st.gx_buf.as<double>();
          k_global_shard<<<n_blk, kBlock, 0, stream>>>(a, gx);
          MICMB_CUDA(cudaGetLastError());
          if (st.gx_fn(gx, gx + 1, st.gx_world, stream, st.gx_user) != 0)
            throw Error(MICMB_ERR_INTERNAL, "global step control: the all-gather of the error sums failed");
          k_global_step_gathered<<<1, 1, 0, stream>>>(a, D, B, gx + 1, st.gx_world,
                                                      (double)st.gx_total_cells * (double)m.S);
        }
        else
          k_global_step<<<n_blk, kBlock, 0, stream>>>(a, D, B, m.S);
        MICMB_CUDA(cudaGetLastError());
      }
      attempts += batch;
      // one host round trip per batch
      MICMB_CUDA(cudaMemcpyAsync(st.host_counters, &a.ctl->status, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
      MICMB_CUDA(cudaStreamSynchronize(stream));
      if (st.host_counters[0] != MICMB_SOLVER_RUNNING)
        break;
      if (attempts > max_attempts)
        throw Error(MICMB_ERR_INTERNAL, "plain solve did not terminate");
      batch = std::min<int64_t>(batch * 2, 64);
    }
    k_global_finish<<<Blocks(st.n_pad * m.S), kBlock, 0, stream>>>(a, m.S);
    MICMB_CUDA(cudaGetLastError());
    GlobalCtl h;
    MICMB_CUDA(cudaMemcpyAsync(&h, a.ctl, sizeof(h), cudaMemcpyDeviceToHost, stream));
    MICMB_CUDA(cudaStreamSynchronize(stream));
    for (int64_t c = 0; c < n; ++c)
    {
      if (per_cell_status)
        per_cell_status[c] = h.status;
      if (per_cell_accepted)
        per_cell_accepted[c] = h.c.accepted;
    }
    if (stats)
    {
      *stats = micmb_solver_stats{};
      stats->function_calls = h.c.function_calls;
      stats->jacobian_updates = h.c.jacobian_updates;
      stats->number_of_steps = h.c.number_of_steps;
      stats->accepted = h.c.accepted;
      stats->rejected = h.c.rejected;
      stats->decompositions = h.c.decompositions;
      stats->solves = h.c.solves;
      stats->cells_not_converged = h.status == MICMB_SOLVER_CONVERGED ? 0 : (int32_t)n;
      stats->final_time = h.c.t;
      stats->state = h.c.state;
    }
    return true;
  }
}  // namespace micmb
