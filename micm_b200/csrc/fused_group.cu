// fused_group.cu -- the persistent fused solve with the cells' working sets in
// shared memory: a block advances G cells in lockstep (group.cuh), each with its
// own step size; a cell that finishes is replaced by the next unsolved one from
// a global atomic counter between two attempts.  Per-cell results are
// bit-identical to the other fused kernels and to the plain ones.
#include "runtime.hpp"
#include "group.cuh"

#include <algorithm>
#include <cstring>

namespace micmb
{
  namespace
  {
    __device__ __forceinline__ size_t cell_base(int64_t c, int32_t L, int32_t ncol)
    {
      return (size_t)(c / L) * (size_t)L * (size_t)ncol + (size_t)(c % L);
    }

    __device__ __forceinline__ void count_attempt(CellCtl& cc, const DevParams& P)
    {
      cc.decompositions += 1;
      cc.solves += P.stages;
      for (int32_t s = 1; s < P.stages; ++s)
        cc.function_calls += P.new_f[s] ? 1 : 0;
    }

    // what the block does with a slot's cell between two attempts
    constexpr int32_t kSlotIdle = 0;      // no cell
    constexpr int32_t kSlotRejected = 1;  // attempt again from Y
    constexpr int32_t kSlotAccepted = 2;  // Ynew becomes Y, next step
    constexpr int32_t kSlotLast = 3;      // Ynew becomes Y, the cell is done
    constexpr int32_t kSlotStopped = 4;   // the cell is done, Y as it is
    constexpr int32_t kSlotFresh = 5;     // a new cell to load
    constexpr int32_t kSlotNothing = 6;   // a new cell that needs no step

    template<int G>
    __global__ void __launch_bounds__(256, 1) k_group_solve(DevGroup P, DevParams D, StepBounds B, FusedArgs A, double* ws, int64_t slot_doubles)
    {
      extern __shared__ __align__(16) double shared[];
      __shared__ CellCtl ctl[G];
      __shared__ int64_t cell_of[G];
      __shared__ int32_t what[G], n_ckpt[G];
      __shared__ double h_used[G];
      __shared__ unsigned long long block_stats[8];
      const GroupThread<G> X(shared);
      const int32_t g = threadIdx.x & (G - 1), S = P.S, L = A.L;
      double* slot = ws + (int64_t)blockIdx.x * slot_doubles;
      GroupVectors v = group_vectors<G>(slot, P);
      double* kk = slot + GroupVectorDoubles(S, D.stages) * G + g;
      v.kk = kk;
      v.ks = G;
      if (threadIdx.x < 8)
        block_stats[threadIdx.x] = 0;
      if (X.lane == 0)
      {
        X[P.zero] = 0.0;
        X[P.one] = 1.0;
        X[P.trash] = 1.0;
        ctl_init(ctl[g], B);
        cell_of[g] = -1;
      }
      for (int32_t i = X.lane; i < S; i += X.lanes)
      {
        X[P.v0 + i] = 0.0;
        v.Y[(int64_t)i * G] = 0.0;
      }
      for (int32_t r = X.lane; r < P.R; r += X.lanes)
        kk[(int64_t)r * G] = 0.0;

      // thread g < G: the next unsolved cell for slot g
      auto claim = [&]() {
        const int64_t c = atomicAdd(A.next_cell, 1);
        if (c >= A.n_cells)
        {
          cell_of[g] = -1;
          what[g] = kSlotIdle;
          return;
        }
        cell_of[g] = c;
        n_ckpt[g] = 0;
        CellCtl cc;
        ctl_init(cc, B);
        if (ctl_begin_step(cc, D, B))
        {
          cc.function_calls += 1;
          cc.jacobian_updates += 1;
          what[g] = kSlotFresh;
        }
        else
          what[g] = kSlotNothing;
        ctl[g] = cc;
      };
      // thread g < G: the finished cell's status and counters
      auto retire = [&]() {
        const CellCtl& c = ctl[g];
        if (A.cell_status)
          A.cell_status[cell_of[g]] = c.state;
        if (A.cell_accepted)
          A.cell_accepted[cell_of[g]] = A.ckpt_y ? n_ckpt[g] : c.accepted;
        if (A.cell_time)
          A.cell_time[cell_of[g]] = c.t;
        atomicAdd(block_stats + 0, (unsigned long long)c.function_calls);
        atomicAdd(block_stats + 1, (unsigned long long)c.jacobian_updates);
        atomicAdd(block_stats + 2, (unsigned long long)c.number_of_steps);
        atomicAdd(block_stats + 3, (unsigned long long)c.accepted);
        atomicAdd(block_stats + 4, (unsigned long long)c.rejected);
        atomicAdd(block_stats + 5, (unsigned long long)c.decompositions);
        atomicAdd(block_stats + 6, (unsigned long long)c.solves);
        if (c.state != MICMB_SOLVER_CONVERGED)
          atomicAdd(block_stats + 7, 1ull);
      };
      auto write_out = [&]() {
        double* out = A.variables_out + cell_base(cell_of[g], L, S);
        for (int32_t i = X.lane; i < S; i += X.lanes)
        {
          const double y = v.Y[(int64_t)i * G];
          out[(int64_t)i * L] = (y < 0.0) ? 0.0 : y;
        }
      };

      if (threadIdx.x < G)
        claim();
      for (;;)
      {
        // cells taken since the last attempt
        __syncthreads();
        int32_t w = what[g];
        while (__syncthreads_or(w >= kSlotFresh))
        {
          if (w >= kSlotFresh)
          {
            const double* y = A.variables_in + cell_base(cell_of[g], L, S);
            const double* k = A.rate_constants + cell_base(cell_of[g], L, P.R);
            for (int32_t i = X.lane; i < S; i += X.lanes)
            {
              const double yi = y[(int64_t)i * L];
              X[P.v0 + i] = yi;
              v.Y[(int64_t)i * G] = yi;
            }
            for (int32_t r = X.lane; r < P.R; r += X.lanes)
              kk[(int64_t)r * G] = k[(int64_t)r * L];
            if (w == kSlotNothing)
              write_out();
          }
          __syncthreads();
          if (threadIdx.x < G)
          {
            if (w == kSlotFresh)
              what[g] = kSlotAccepted;
            else if (w == kSlotNothing)
            {
              retire();
              claim();
            }
          }
          __syncthreads();
          w = what[g];
        }
        const bool live = w != kSlotIdle;
        if (!__syncthreads_or(live))
          break;
        group_attempt<G>(P, D, X, v, ctl[g].H, A.atol, A.rtol);
        __syncthreads();
        if (threadIdx.x < G && live)
        {
          double sum = 0.0;
#pragma unroll 8
          for (int32_t i = 0; i < S; ++i)
            sum += X[P.rate + i];
          const double error = error_from_sum(sum, (double)S);
          CellCtl c = ctl[g];
          count_attempt(c, D);
          h_used[g] = c.H;
          const int res = ctl_after_error(c, D, B, error);
          int32_t next = res == 0 ? kSlotRejected : kSlotStopped;
          if (res == 1)
          {
            if (A.ckpt_y)
              n_ckpt[g] += 1;
            bool more = ctl_begin_step(c, D, B);
            if (more && A.ckpt_y && n_ckpt[g] >= A.max_ckpt)
            {
              c.state = MICMB_SOLVER_CONVERGENCE_EXCEEDED_MAX_STEPS;
              more = false;
            }
            if (more)
            {
              c.function_calls += 1;
              c.jacobian_updates += 1;
            }
            next = more ? kSlotAccepted : kSlotLast;
          }
          ctl[g] = c;
          what[g] = next;
        }
        __syncthreads();
        w = what[g];
        if (w == kSlotAccepted || w == kSlotLast)
        {
          if (A.ckpt_y)
          {
            const size_t at = (size_t)cell_of[g] * A.max_ckpt + (n_ckpt[g] - 1);
            double* dst = A.ckpt_y + at * S;
            for (int32_t i = X.lane; i < S; i += X.lanes)
              dst[i] = v.Y[(int64_t)i * G];
            if (A.ckpt_k)
            {
              double* kd = A.ckpt_k + at * (size_t)D.stages * S;
              for (int32_t st = 0; st < D.stages; ++st)
                for (int32_t i = X.lane; i < S; i += X.lanes)
                  kd[(size_t)st * S + i] = v.K[((int64_t)st * S + i) * G];
            }
            if (X.lane == 0)
              A.ckpt_h[at] = h_used[g];
          }
          for (int32_t i = X.lane; i < S; i += X.lanes)
            v.Y[(int64_t)i * G] = X[P.v0 + i];
        }
        else if (w == kSlotRejected)
          for (int32_t i = X.lane; i < S; i += X.lanes)
            X[P.v0 + i] = v.Y[(int64_t)i * G];
        if (w == kSlotLast || w == kSlotStopped)
          write_out();
        __syncthreads();
        if (threadIdx.x < G && (w == kSlotLast || w == kSlotStopped))
        {
          retire();
          claim();
        }
      }
      if (threadIdx.x < 8 && block_stats[threadIdx.x])
        atomicAdd(A.stats + threadIdx.x, block_stats[threadIdx.x]);
    }

    using SolveKernel = void (*)(DevGroup, DevParams, StepBounds, FusedArgs, double*, int64_t);

    SolveKernel SolveKernelFor(int32_t G)
    {
      switch (G)
      {
        case 1: return k_group_solve<1>;
        case 2: return k_group_solve<2>;
        case 4: return k_group_solve<4>;
        case 8: return k_group_solve<8>;
        case 16: return k_group_solve<16>;
        default: return k_group_solve<32>;
      }
    }
  }  // namespace

  // Cells per block: as many as leave two blocks for every SM (four from eight cells
  // on: a block's last cells wait for one another), as long as one block's cells fit
  // in shared memory.  Warps per block: registers allow eight per SM, shared by the
  // blocks that share the SM; one where a cell is so small that there is nothing to
  // split.  Measured, ms: 210 species, 4,096 cells: (cells, warps) = (2, 2) 43.8, (4,
  // 4) 41.4, (8, 8) 41.3; 60 species, 1,013 cells: (4, 4) 8.1, (4, 2) 9.8, (8, 4) 10.1;
  // 3,000: (4, 4) 11.6, (8, 4) 10.5, (16, 4) 12.7; 30,000: (8, 4) 53.1, (16, 4) 42.5,
  // (32, 4) 50.3, (32, 8) 41.6; Chapman, 3,000: (1, 1) 1.08, (4, 1) 0.44, (16, 1) 0.50;
  // 100,000: (16, 1) 3.6, (32, 1) 2.0, (32, 2) 2.8.
  GroupChoice ChooseGroup(const micmb_solver& s, int64_t n_cells, int32_t sweep_stages)
  {
    const CompiledMechanism& m = *s.mech;
    const size_t per_cell = GroupSharedBytes(s, GroupChoice{ 1, 1, sweep_stages }) + 96;  // static shared memory included
    GroupChoice c{ 1, 1, sweep_stages };
    while (c.G < 32 && n_cells >= (c.G < 8 ? 2 : 4) * (int64_t)c.G * s.sm_count &&
           2 * c.G * per_cell + 1024 <= s.smem_optin)
      c.G *= 2;
    if (m.nnz < kTinyNonZeros)
      return c;
    const int64_t fit = std::max<int64_t>(1, (int64_t)((s.smem_optin + 1024) / (c.G * per_cell + 2048)));
    const int64_t wanted = (n_cells + (int64_t)c.G * s.sm_count - 1) / ((int64_t)c.G * s.sm_count);
    const int64_t blocks = std::min(fit, std::max<int64_t>(1, wanted));
    while (c.W * blocks < 8)
      c.W *= 2;
    return c;
  }

  const GroupTables& GroupTablesFor(micmb_solver& s, const GroupChoice& choice)
  {
    std::lock_guard<std::mutex> lock(s.group_mutex);
    for (const auto& t : s.group)
      if (t->choice.G == choice.G && t->choice.W == choice.W && t->choice.sweep_stages == choice.sweep_stages)
        return *t;
    const GroupProgram p = BuildGroupProgram(*s.mech, choice.G, choice.W, choice.sweep_stages);
    auto t = std::make_unique<GroupTables>();
    t->choice = choice;
    std::vector<char> bytes;
    auto add = [&](const auto& vec) {
      const size_t off = (bytes.size() + 255) & ~size_t(255), n = vec.size() * sizeof(vec[0]);
      bytes.resize(off + std::max<size_t>(n, 16), 0);
      if (n)
        std::memcpy(bytes.data() + off, vec.data(), n);
      return off;
    };
    struct Offsets
    {
      size_t ws, ctrl, item, row, coef;
    };
    auto add_phase = [&](const GroupPhase& ph) {
      Offsets o;
      o.ws = add(ph.warp_start);
      o.ctrl = add(ph.ctrl);
      o.item = add(ph.item);
      o.row = add(ph.row);
      o.coef = add(ph.coef);
      return o;
    };
    const Offsets of = add_phase(p.forcing), oj = add_phase(p.jacobian), ol = add_phase(p.lu), os = add_phase(p.solve);
    const Offsets ostep = add_phase(p.step);
    const size_t ostart = add(p.step_start);
    const size_t orate = add(p.rate), odrate = add(p.drate);
    t->memory = DeviceMemory(bytes.size());
    MICMB_CUDA(cudaMemcpy(t->memory.p, bytes.data(), bytes.size(), cudaMemcpyHostToDevice));
    // a copy from pageable memory may return before it has arrived, and the
    // states' streams do not wait for the default stream
    MICMB_CUDA(cudaStreamSynchronize(nullptr));
    const char* b = t->memory.as<const char>();
    auto phase = [&](const Offsets& o) {
      DevGroupPhase d;
      d.warp_start = reinterpret_cast<const int32_t*>(b + o.ws);
      d.ctrl = reinterpret_cast<const uint32_t*>(b + o.ctrl);
      d.item = reinterpret_cast<const uint4*>(b + o.item);
      d.row = reinterpret_cast<const uint4*>(b + o.row);
      d.coef = reinterpret_cast<const double2*>(b + o.coef);
      return d;
    };
    DevGroup& g = t->dev;
    g.S = s.mech->S;
    g.R = s.mech->R;
    g.nnz = s.mech->nnz;
    g.n_info = (int32_t)s.mech->info_rxn.size();
    g.zero = p.layout.zero;
    g.one = p.layout.one;
    g.v0 = p.layout.v0;
    g.trash = p.layout.trash;
    g.w0 = p.layout.w0;
    g.inv = p.layout.inv;
    g.rate = p.layout.rate;
    g.g2 = p.layout.g2;
    g.slot = p.layout.slot;
    g.elements = p.layout.elements;
    g.forcing = phase(of);
    g.jacobian = phase(oj);
    g.lu = phase(ol);
    g.solve = phase(os);
    g.step = phase(ostep);
    g.step_start = reinterpret_cast<const int32_t*>(b + ostart);
    g.rate_tab = reinterpret_cast<const uint2*>(b + orate);
    g.drate_tab = reinterpret_cast<const uint2*>(b + odrate);
    s.group.push_back(std::move(t));
    return *s.group.back();
  }

  size_t GroupSharedBytes(const micmb_solver& s, const GroupChoice& choice)
  {
    return sizeof(double) * (size_t)MakeGroupLayout(*s.mech, choice.sweep_stages).elements * choice.G;
  }

  int GroupBlocksPerSm(const micmb_solver& s, const void* kernel, const GroupChoice& choice)
  {
    const size_t smem = GroupSharedBytes(s, choice);
    // the kernels' static shared memory: at most 96 bytes per cell and a few words
    if (smem + 96 * (size_t)choice.G + 1024 > s.smem_optin)
      return 0;
    AllowSharedMemory(s, kernel);
    int per_sm = 0;
    MICMB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * choice.W, smem));
    return per_sm;
  }

  bool GroupVariantApplies(const micmb_solver& s, int64_t n_cells)
  {
    // the register-blocked schedules, asked for by the environment, are the
    // thread-per-cell kernels'
    if (!GroupApplies(*s.mech) || s.dev.has_blocked)
      return false;
    const GroupChoice choice = ChooseGroup(s, n_cells);
    return GroupBlocksPerSm(s, reinterpret_cast<const void*>(SolveKernelFor(choice.G)), choice) > 0;
  }

  // The thread-per-cell kernels need about 300,000 cells to fill the GPU and take
  // nearly the same time for fewer; the cell-group kernel's time is proportional
  // to the cells from a few thousand on, and inversely to the cells an SM holds.
  // Measured, cell-group against one-cell-per-thread fused kernel, ms: Chapman
  // 150,000 cells 2.6 / 2.9, 225,000 3.9 / 3.8, 300,000 5.2 / 4.5; 60 species (32 cells
  // per SM) 300,000 294 / 570, 1,000,000 1,550 / 1,218; TS1 (8 per SM) 260,000 1,388 /
  // 1,613, 1,000,000 5,806 / 4,531; 210 species (8 per SM) 260,000 1,747 / 1,915,
  // 524,288 3,710 / 3,340; 600 species (1 per SM) 32,000 4,013 / 6,332, 100,000 12,593 /
  // 7,442.
  bool GroupFaster(const micmb_solver& s, int64_t n_cells)
  {
    if (!GroupVariantApplies(s, n_cells))
      return false;
    const int64_t per_sm = s.mech->nnz < kTinyNonZeros ? 1500 : 2048;
    return n_cells <= std::min<int64_t>(s.sm_count * per_sm, 32768 * (int64_t)GroupCellsPerSm(s));
  }

  // The per-stage kernels take 1.3-1.6 times the thread kernel's time, so with
  // eight cells per SM the cell-group kernel is faster at any count (210 species,
  // 1,048,576 cells: 7.4 s against 8.7 s; TS1, 600,000 3.2 against 4.4; Chapman,
  // 1,000,000 17 ms against 20); with one (600 species) it is up to the thread
  // kernel's limit.
  bool GroupFasterThanStages(const micmb_solver& s, int64_t n_cells)
  {
    return GroupVariantApplies(s, n_cells) && (GroupCellsPerSm(s) >= 8 || GroupFaster(s, n_cells));
  }

  bool GroupBeatsThreads(const micmb_solver& s, int64_t n_cells, int64_t equal, const void* kernel, int block)
  {
    if (n_cells <= equal)
      return true;
    int per_sm = 0;
    MICMB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0));
    const int64_t set = std::max<int64_t>(1, (int64_t)per_sm * block * s.sm_count);
    return n_cells <= (n_cells + set - 1) / set * equal;
  }

  int32_t GroupCellsPerSm(const micmb_solver& s)
  {
    const GroupChoice most = ChooseGroup(s, (int64_t)1 << 40);
    return most.G * GroupBlocksPerSm(s, reinterpret_cast<const void*>(SolveKernelFor(most.G)), most);
  }

  void SolveFusedGroup(micmb_solver& s, micmb_state& st, const FusedArgs& A, double dt)
  {
    const GroupChoice choice = ChooseGroup(s, A.n_cells);
    const SolveKernel kernel = SolveKernelFor(choice.G);
    const int per_sm = GroupBlocksPerSm(s, reinterpret_cast<const void*>(kernel), choice);
    const GroupTables& t = GroupTablesFor(s, choice);
    const int64_t grid =
        std::max<int64_t>(1, std::min<int64_t>((int64_t)per_sm * s.sm_count, (A.n_cells + choice.G - 1) / choice.G));
    const int64_t slot = (GroupVectorDoubles(s.mech->S, s.params.stages) + s.mech->R) * choice.G;
    EnsureWorkspace(st, st.group_ws, grid * slot);
    kernel<<<(unsigned)grid, 32 * choice.W, GroupSharedBytes(s, choice), st.stream>>>(
        t.dev, s.params, step_bounds(s.params, dt), A, st.group_ws.as<double>(), slot);
    MICMB_CUDA(cudaGetLastError());
  }
}  // namespace micmb
