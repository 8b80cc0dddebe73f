// adjoint.cu -- discrete adjoint of the accepted Rosenbrock steps of a
// per-cell fused solve (no counterpart in micm).
//
// The forward solve (SolveFused with checkpointing) stores, for every accepted
// step n of every cell, the starting state y_n, the step size H_n and (where
// memory allows) the stage vectors K_s.  The backward sweep, on cell groups in
// shared memory or one cell per thread, then walks each cell's steps backwards.  For step n it rebuilds
// alpha I - J(y_n) and its LU factor, takes the stored stages or recomputes
// them exactly as the forward pass did (same routines, so the same bits), and
// applies the transposed step with the step size held fixed:
//
//   y_{n+1} = y_n + sum_s m_s K_s,   M K_s = F(Y_s) + sum_{j<s} (c_sj / H) K_j,
//   M = 1/(H gamma_0) I - J(y_n),    Y_s = y_n + sum_{j<s} a_sj K_j
//
//   Kbar_s = m_s ybar;  for s = S-1..0: Rbar_s = M^-T Kbar_s, Gbar_s += Rbar_s,
//   Kbar_j += (c_sj / H) Rbar_s, and the chain rule through Y_s (new function
//   evaluation: ybar += J(Y_s)^T Gbar_s, Kbar_j += a_sj J(Y_s)^T Gbar_s) or
//   through the reused evaluation (Gbar_{s-1} += Gbar_s);
//   finally ybar += J(y_n)^T Gbar_0 + sum_s H_r-terms of M's dependence on y_n.
//
// Rate-parameter gradients are taken with respect to log k_r (w_r = k_r prod y,
// so d w_r / d log k_r = w_r).  The same recurrences, in the same order, are
// restated on the CPU by the test oracle (om_adjoint_per_cell).
#include "runtime.hpp"
#include "group.cuh"

#include <algorithm>
#include <vector>

namespace micmb
{
  namespace
  {
    constexpr int kMaxAdjStages = 6;

    __device__ __forceinline__ size_t cell_base(int64_t c, int32_t L, int32_t ncol)
    {
      return (size_t)(c / L) * (size_t)L * (size_t)ncol + (size_t)(c % L);
    }

    struct AdjArgs
    {
      int64_t n_cells;
      int32_t L;
      int32_t max_ckpt;
      const double* rate_constants;  // vector layout [R]
      const double* y0;              // vector layout [S]: initial state (clamp derivative when no step)
      const double* ybar_final;      // vector layout [S]
      const double* ckpt_y;          // [cell][max_ckpt][S]
      const double* ckpt_h;          // [cell][max_ckpt]
      const double* ckpt_k;          // [cell][max_ckpt][stages][S] stored stage vectors, or null
      const int32_t* n_ckpt;         // [cell]
      double* ybar0;                 // vector layout [S]
      double* kbar;                  // [cell][R]
      int32_t* next_cell;
      const int32_t* order;          // cells in decreasing step count, or null
    };

    // ---- one cell per thread, private working sets in global memory ----

    // entry offsets of a thread's working set (each entry is 32 doubles, one per lane)
    struct AdjThreadLayout
    {
      int32_t oy, oF0, oFc, oInv, oYb, oTmp, oYs, oK, oKb, oGb, oRb, oKk, oKbar, oScr, oLU, per_slot;
    };

    AdjThreadLayout MakeAdjThreadLayout(int32_t S, int32_t R, int32_t ns, int32_t n_info, int32_t nnz)
    {
      AdjThreadLayout t;
      int32_t o = 0;
      auto take = [&](int32_t n) {
        const int32_t at = o;
        o += n;
        return at;
      };
      t.oy = take(S);
      t.oF0 = take(S);
      t.oFc = take(S);
      t.oInv = take(S);
      t.oYb = take(S);
      t.oTmp = take(S);
      t.oYs = take(ns * S);
      t.oK = take(ns * S);
      t.oKb = take(ns * S);
      t.oGb = take(ns * S);
      t.oRb = take(ns * S);
      t.oKk = take(R);
      t.oKbar = take(R);
      t.oScr = take(R > n_info ? R : n_info);
      t.oLU = take(nnz);
      t.per_slot = o;
      return t;
    }

    template<class V>
    __device__ __forceinline__ double nu_dot_t(const DevMech& M, int32_t r, V v)
    {
      double s = 0.0;
      for (int32_t i = M.prod_start[r]; i < M.prod_start[r + 1]; ++i)
        s += M.prod_yield[i] * v[M.prod_ids[i]];
      for (int32_t i = M.react_start[r]; i < M.react_start[r + 1]; ++i)
        s -= v[M.react_ids[i]];
      return s;
    }

    template<class V>
    __device__ __forceinline__ double prod_except_t(const DevMech& M, int32_t r, V y, int32_t a, int32_t b)
    {
      double v = 1.0;
      for (int32_t i = M.react_start[r]; i < M.react_start[r + 1]; ++i)
        if (i != a && i != b)
          v *= y[M.react_ids[i]];
      return v;
    }

    // yb += J(y)^T g ; kb[r] += (nu_r . g) w_r(y)  (reactions in order, as the oracle)
    template<class V>
    __device__ void vjp_f_t(const DevMech& M, V kk, V y, V g, V yb, V kb)
    {
      for (int32_t r = 0; r < M.R; ++r)
      {
        const double c = nu_dot_t(M, r, g);
        if (c == 0.0)
          continue;
        kb[r] += c * (kk[r] * prod_except_t(M, r, y, -1, -1));
        for (int32_t i = M.react_start[r]; i < M.react_start[r + 1]; ++i)
          yb[M.react_ids[i]] += c * kk[r] * prod_except_t(M, r, y, i, -1);
      }
    }

    template<class V>
    __device__ void jacobian_term_t(const DevMech& M, V kk, V y, V Rb, V Kv, V yb, V kb)
    {
      for (int32_t r = 0; r < M.R; ++r)
      {
        const double rho = nu_dot_t(M, r, Rb);
        if (rho == 0.0)
          continue;
        const int32_t r0 = M.react_start[r], r1 = M.react_start[r + 1];
        double gk = 0.0;
        for (int32_t i = r0; i < r1; ++i)
          gk += kk[r] * prod_except_t(M, r, y, i, -1) * Kv[M.react_ids[i]];
        kb[r] += rho * gk;
        for (int32_t i = r0; i < r1; ++i)
          for (int32_t j = r0; j < r1; ++j)
            if (i != j)
              yb[M.react_ids[j]] += rho * kk[r] * prod_except_t(M, r, y, i, j) * Kv[M.react_ids[i]];
      }
    }

    // vjp_f_t over fixed-width reactant lists (rate_desc)
    template<class V>
    __device__ void vjp_narrow(const DevMech& M, V kk, V y, V g, V yb, V kb)
    {
      const int32_t S = M.S;
      for (int32_t r = 0; r < M.R; ++r)
      {
        const double c = nu_dot_t(M, r, g);
        if (c == 0.0)
          continue;
        const int4 d = M.rate_desc[r];
        const int32_t id[3] = { d.x, d.y, d.z };
        double yv[3];
        int32_t nr = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
          yv[q] = id[q] < S ? y[id[q]] : 1.0;
          nr += id[q] < S ? 1 : 0;
        }
        const double k = kk[r];
        kb[r] += c * (k * (((1.0 * yv[0]) * yv[1]) * yv[2]));
        for (int q = 0; q < nr; ++q)
        {
          double v = 1.0;
          for (int o = 0; o < nr; ++o)
            if (o != q)
              v *= yv[o];
          yb[id[q]] += c * k * v;
        }
      }
    }

    // Reactions with at most three reactants (rate_desc): one pass over the
    // reactions at the step's starting state applies J(y)^T Gbar_0 and the
    // second-order terms of every stage, with w_r's partial derivatives formed
    // once per reaction instead of once per use.
    template<class V>
    __device__ void step_terms_narrow(const DevMech& M, int32_t ns, V kk, V y, V Gb0, const V* Rb, const V* K, V yb,
                                      V kb)
    {
      const int32_t S = M.S;
      for (int32_t r = 0; r < M.R; ++r)
      {
        const int4 d = M.rate_desc[r];
        const int32_t id[3] = { d.x, d.y, d.z };
        int32_t nr = 0;
        double yv[3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
          yv[q] = id[q] < S ? y[id[q]] : 1.0;
          nr += id[q] < S ? 1 : 0;
        }
        const double k = kk[r];
        // first derivatives k * prod of the other reactants (in reactant order)
        double P1[3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
          double v = 1.0;
#pragma unroll
          for (int o = 0; o < 3; ++o)
            if (o != q && o < nr)
              v *= yv[o];
          P1[q] = v;
        }
        // J(y)^T Gbar_0
        const double c = nu_dot_t(M, r, Gb0);
        if (c != 0.0)
        {
          kb[r] += c * (k * (((1.0 * (nr > 0 ? yv[0] : 1.0)) * (nr > 1 ? yv[1] : 1.0)) * (nr > 2 ? yv[2] : 1.0)));
          for (int q = 0; q < nr; ++q)
            yb[id[q]] += c * k * P1[q];
        }
        // second-order terms of every stage
        for (int32_t st = 0; st < ns; ++st)
        {
          const double rho = nu_dot_t(M, r, Rb[st]);
          if (rho == 0.0)
            continue;
          double kv[3];
          for (int q = 0; q < nr; ++q)
            kv[q] = K[st][id[q]];
          double gk = 0.0;
          for (int q = 0; q < nr; ++q)
            gk += k * P1[q] * kv[q];
          kb[r] += rho * gk;
          for (int q = 0; q < nr; ++q)
            for (int o = 0; o < nr; ++o)
              if (q != o)
              {
                double v = 1.0;  // product of the reactants other than q and o
                for (int z = 0; z < nr; ++z)
                  if (z != q && z != o)
                    v *= yv[z];
                yb[id[o]] += rho * k * v * kv[q];
              }
        }
      }
    }

    __device__ __forceinline__ void adjoint_thread_body(const DevMech& M, const DevParams& P, const AdjArgs& A,
                                                        const AdjThreadLayout& T, double* ws)
    {
      const int lane = threadIdx.x & 31;
      const int64_t wslot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
      double* w = ws + (size_t)wslot * (size_t)T.per_slot * 32 + lane;
      const int32_t S = M.S, R = M.R, L = A.L, ns = P.stages;
      auto at = [&](int32_t entry) { return Strided{ w + (size_t)entry * 32, 32 }; };
      Strided y = at(T.oy), F0 = at(T.oF0), Fc = at(T.oFc), inv = at(T.oInv), yb = at(T.oYb), tmp = at(T.oTmp);
      Strided kk = at(T.oKk), kb = at(T.oKbar), scr = at(T.oScr), LU = at(T.oLU);
      auto Ys = [&](int32_t s) { return at(T.oYs + s * S); };
      auto K = [&](int32_t s) { return at(T.oK + s * S); };
      auto Kb = [&](int32_t s) { return at(T.oKb + s * S); };
      auto Gb = [&](int32_t s) { return at(T.oGb + s * S); };
      auto Rb = [&](int32_t s) { return at(T.oRb + s * S); };

      int64_t cell = 0;
      int32_t n = -1;  // checkpoint being processed; -1: no cell
      auto finish = [&]() {
        const size_t by = cell_base(cell, L, S);
        for (int32_t i = 0; i < S; ++i)
          A.ybar0[by + (size_t)i * L] = yb[i];
        for (int32_t r = 0; r < R; ++r)
          A.kbar[(size_t)cell * R + r] = kb[r];
      };
      auto claim = [&]() {
        for (;;)
        {
          const int64_t k = atomicAdd(A.next_cell, 1);
          if (k >= A.n_cells)
          {
            n = -1;
            return;
          }
          cell = A.order ? A.order[k] : k;
          const size_t by = cell_base(cell, L, S);
          const size_t bk = cell_base(cell, L, R);
          for (int32_t r = 0; r < R; ++r)
          {
            kk[r] = A.rate_constants[bk + (size_t)r * L];
            kb[r] = 0.0;
          }
          const int32_t n_ck = A.n_ckpt[cell];
          if (n_ck > 0)
          {
            n = n_ck - 1;
            return;
          }
          for (int32_t i = 0; i < S; ++i)
            yb[i] = (A.y0[by + (size_t)i * L] < 0.0) ? 0.0 : A.ybar_final[by + (size_t)i * L];
          finish();
        }
      };

      claim();
      while (__any_sync(0xffffffffu, n >= 0))
      {
        if (n < 0)
          continue;
        const size_t by = cell_base(cell, L, S);
        const double* yc = A.ckpt_y + ((size_t)cell * A.max_ckpt + n) * S;
        const double H = A.ckpt_h[(size_t)cell * A.max_ckpt + n];
        for (int32_t i = 0; i < S; ++i)
          y[i] = yc[i];
        // ---- the accepted step's factor, stages and stage inputs ----
        const double alpha = 1.0 / (H * P.gamma0);
        jacobian_rates<1>(M, kk, y, scr, 0);
        thread_lu_gathered(M, scr, alpha, LU, inv);  // -J + alpha I, then LU
        if (A.ckpt_k)
        {
          // stages stored by the forward pass; stage inputs rebuilt from them
          const double* kc = A.ckpt_k + ((size_t)cell * A.max_ckpt + n) * (size_t)ns * S;
          for (int32_t st = 0; st < ns; ++st)
          {
            Strided Ks = K(st);
            for (int32_t i = 0; i < S; ++i)
              Ks[i] = kc[(size_t)st * S + i];
          }
          for (int32_t st = 0; st < ns; ++st)
          {
            const int32_t sc = st * (st - 1) / 2;
            Strided Yst = Ys(st);
            if (st > 0 && P.new_f[st])
              for (int32_t i = 0; i < S; ++i)
              {
                double v = y[i];
                for (int32_t j = 0; j < st; ++j)
                  v += P.a[sc + j] * K(j)[i];
                Yst[i] = v;
              }
            else
              for (int32_t i = 0; i < S; ++i)
                Yst[i] = y[i];
          }
        }
        else
        {
          reaction_rates<1>(M, kk, y, scr, 0);
          forcing_gather<1>(M, scr, F0, 0);
          bool fc_is_src = false;
          for (int32_t st = 0; st < ns; ++st)
          {
            const int32_t sc = st * (st - 1) / 2;
            Strided Yst = Ys(st);
            if (st > 0 && P.new_f[st])
            {
              for (int32_t i = 0; i < S; ++i)
              {
                double v = y[i];
                for (int32_t j = 0; j < st; ++j)
                  v += P.a[sc + j] * K(j)[i];
                Yst[i] = v;
              }
              reaction_rates<1>(M, kk, Yst, scr, 0);
              forcing_gather<1>(M, scr, Fc, 0);
              fc_is_src = true;
            }
            else
              for (int32_t i = 0; i < S; ++i)
                Yst[i] = y[i];
            double coh[kMaxAdjStages];
            for (int32_t j = 0; j < st; ++j)
              coh[j] = P.c[sc + j] / H;
            Strided Ks = K(st);
            for (int32_t i = 0; i < S; ++i)
            {
              double v = fc_is_src ? Fc[i] : F0[i];
              for (int32_t j = 0; j < st; ++j)
                v += coh[j] * K(j)[i];
              Ks[i] = v;
            }
            thread_solve(M, LU, Ks);
          }
        }
        if (n == A.n_ckpt[cell] - 1)
          for (int32_t i = 0; i < S; ++i)
          {
            double v = y[i];
            for (int32_t st = 0; st < ns; ++st)
              v += P.m[st] * K(st)[i];
            yb[i] = (v < 0.0) ? 0.0 : A.ybar_final[by + (size_t)i * L];
          }
        // ---- reverse sweep ----
        for (int32_t i = 0; i < S; ++i)
        {
          const double g = yb[i];
          for (int32_t st = 0; st < ns; ++st)
          {
            Kb(st)[i] = P.m[st] * g;
            Gb(st)[i] = 0.0;
          }
        }
        for (int32_t st = ns - 1; st >= 0; --st)
        {
          const int32_t sc = st * (st - 1) / 2;
          Strided rb = Rb(st);
          for (int32_t i = 0; i < S; ++i)
            rb[i] = Kb(st)[i];
          solve_upper<1>(M.fwd_t_s, LU, rb, 0);  // U^T w = Kbar (divides by u_ii)
          solve_lower<1>(M.bwd_t_s, LU, rb, 0);  // L^T z = w
          double coh[kMaxAdjStages];
          for (int32_t j = 0; j < st; ++j)
            coh[j] = P.c[sc + j] / H;
          for (int32_t i = 0; i < S; ++i)
          {
            const double v = rb[i];
            Gb(st)[i] += v;
            for (int32_t j = 0; j < st; ++j)
              Kb(j)[i] += coh[j] * v;
          }
          if (st == 0)
            continue;
          if (P.new_f[st])
          {
            for (int32_t i = 0; i < S; ++i)
              tmp[i] = 0.0;
            if (M.rate_desc)
              vjp_narrow(M, kk, Ys(st), Gb(st), tmp, kb);
            else
              vjp_f_t(M, kk, Ys(st), Gb(st), tmp, kb);
            for (int32_t i = 0; i < S; ++i)
            {
              const double t = tmp[i];
              yb[i] += t;
              for (int32_t j = 0; j < st; ++j)
                Kb(j)[i] += P.a[sc + j] * t;
            }
          }
          else
            for (int32_t i = 0; i < S; ++i)
              Gb(st - 1)[i] += Gb(st)[i];
        }
        if (M.rate_desc)
        {
          Strided rbs[kMaxAdjStages], ks[kMaxAdjStages];
          for (int32_t st = 0; st < ns; ++st)
          {
            rbs[st] = Rb(st);
            ks[st] = K(st);
          }
          step_terms_narrow(M, ns, kk, y, Gb(0), rbs, ks, yb, kb);
        }
        else
        {
          vjp_f_t(M, kk, y, Gb(0), yb, kb);
          for (int32_t st = 0; st < ns; ++st)
            jacobian_term_t(M, kk, y, Rb(st), K(st), yb, kb);
        }
        if (--n < 0)
        {
          finish();
          claim();
        }
      }
    }

    // ---- cell groups: a block sweeps G cells in lockstep, their factors in shared memory ----

    // nu_r . v for elements v0 + column
    template<int G>
    __device__ __forceinline__ double nu_dot_g(const DevMech& M, int32_t r, const GroupThread<G>& X, int32_t v0)
    {
      double s = 0.0;
      for (int32_t i = M.prod_start[r]; i < M.prod_start[r + 1]; ++i)
        s += M.prod_yield[i] * X[v0 + M.prod_ids[i]];
      for (int32_t i = M.react_start[r]; i < M.react_start[r + 1]; ++i)
        s -= X[v0 + M.react_ids[i]];
      return s;
    }

    // a reaction's reactants (rate_desc), their values in V and the products of the others
    struct Reactants
    {
      int32_t id[3], n;
      double y[3], others[3];
    };
    template<int G>
    __device__ __forceinline__ Reactants reactants_of(const DevMech& M, const DevGroup& P, const GroupThread<G>& X,
                                                      int32_t r)
    {
      Reactants a;
      const int4 d = M.rate_desc[r];
      a.id[0] = d.x;
      a.id[1] = d.y;
      a.id[2] = d.z;
      a.n = 0;
#pragma unroll
      for (int q = 0; q < 3; ++q)
      {
        a.y[q] = a.id[q] < M.S ? X[P.v0 + a.id[q]] : 1.0;
        a.n += a.id[q] < M.S ? 1 : 0;
      }
#pragma unroll
      for (int q = 0; q < 3; ++q)
      {
        double v = 1.0;
#pragma unroll
        for (int o = 0; o < 3; ++o)
          if (o != q && o < a.n)
            v *= a.y[o];
        a.others[q] = v;
      }
      return a;
    }

    // kb[r] += (nu_r . g) w_r, and the reaction's terms of J^T g to element first + q
    // for reactant q (state in V, g in G2).  What the thread kernel skips is -0,
    // which leaves every sum as it is.
    template<int G>
    __device__ __forceinline__ void project(const Reactants& a, double k, double c, const GroupThread<G>& X,
                                            const int32_t (&to)[3], double& kb)
    {
      if (c != 0.0)
        kb += c * (k * (((1.0 * a.y[0]) * a.y[1]) * a.y[2]));
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (q < a.n)
          X[to[q]] = c != 0.0 ? c * k * a.others[q] : -0.0;
    }

    template<int G>
    __device__ __forceinline__ void group_vjp(const DevMech& M, const DevGroup& P, const GroupThread<G>& X,
                                              const double* kk, double* kb)
    {
      for (int32_t r = X.lane; r < P.R; r += X.lanes)
      {
        const int32_t first = P.slot + M.react_start[r];
        const int32_t to[3] = { first, first + 1, first + 2 };
        project<G>(reactants_of(M, P, X, r), kk[(int64_t)r * G], nu_dot_g(M, r, X, P.g2), X, to, kb[(int64_t)r * G]);
      }
    }

    // Contributions of a whole step at its start: stage < 0, J^T Gbar_0; else the
    // second-order terms of that stage (Rbar in G2, K in the inv elements, which no
    // solve needs any more).
    template<int G>
    __device__ __forceinline__ void group_step_terms(const DevMech& M, const DevGroup& P, const GroupThread<G>& X,
                                                     int32_t stage, const double* kk, double* kb)
    {
      for (int32_t r = X.lane; r < P.R; r += X.lanes)
      {
        const double k = kk[(int64_t)r * G], c = nu_dot_g(M, r, X, P.g2);
        const Reactants a = reactants_of(M, P, X, r);
        int32_t i = P.step_start[r];
        auto element = [&](int32_t e) { return e < P.nnz ? e : P.slot + e - P.nnz; };
        if (stage < 0)
        {
          const int32_t to[3] = { element(i), element(i + 1), element(i + 2) };
          project<G>(a, k, c, X, to, kb[(int64_t)r * G]);
          continue;
        }
        i += a.n + stage * a.n * (a.n - 1);
        double kv[3], gk = 0.0;
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
          kv[q] = q < a.n ? X[P.inv + a.id[q]] : 0.0;
          if (q < a.n)
            gk += k * a.others[q] * kv[q];
        }
        if (c != 0.0)
          kb[(int64_t)r * G] += c * gk;
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
          for (int o = 0; o < 3; ++o)
            if (q != o && q < a.n && o < a.n)
            {
              const double v = a.n == 3 ? 1.0 * a.y[3 - q - o] : 1.0;
              X[element(i++)] = c != 0.0 ? c * k * v * kv[q] : -0.0;
            }
      }
    }

    // The backward sweep with stored stages: the thread kernel's sums, in the same
    // order, so the same bits.  Per step one factorisation and a transposed solve per
    // stage as in the forward kernel, and per evaluation a pass over the reactions
    // whose contributions go to shared memory and are gathered per species, as the
    // sums of a species have to keep the reactions' order.  Bound by the solves'
    // dependency levels, as the forward kernel; the stages' vectors (Kbar, Gbar,
    // Rbar) stay in L2.  The thread kernel, with a working set per thread in HBM, is
    // bound by latency below some 100,000 cells.  Measured, forward and sweep of
    // 8,192 cells of 60 species: 347 -> 54 ms; 16,384 of 210: 1,608 -> 500; 2,048 of
    // 600: 5,706 -> 611.
    template<int G>
    __global__ void __launch_bounds__(256, 1)
        k_adjoint_group(DevMech M, DevGroup P, DevParams D, AdjArgs A, double* ws, int64_t slot_doubles)
    {
      extern __shared__ __align__(16) double shared[];
      __shared__ int64_t cell_of[G];
      __shared__ int32_t step[G];  // checkpoint being swept; -1: none
      const GroupThread<G> X(shared);
      const int32_t g = threadIdx.x & (G - 1), S = P.S, L = A.L, ns = D.stages;
      double* w = ws + (int64_t)blockIdx.x * slot_doubles + g;
      auto take = [&](int64_t n) {
        double* at = w;
        w += n * G;
        return at;
      };
      double *yv = take(S), *yb = take(S), *Kb = take((int64_t)ns * S), *Gb = take((int64_t)ns * S),
             *Rb = take((int64_t)ns * S), *kk = take(P.R), *kb = take(P.R);
      auto at = [&](double* v, int32_t st, int32_t i) -> double& { return v[((int64_t)st * S + i) * G]; };
      if (X.lane == 0)
      {
        X[P.zero] = 0.0;
        X[P.one] = 1.0;
        X[P.trash] = 1.0;
      }
      for (int32_t i = X.lane; i < S; i += X.lanes)
      {
        yv[(int64_t)i * G] = yb[(int64_t)i * G] = 0.0;
        for (int32_t st = 0; st < ns; ++st)
          at(Kb, st, i) = at(Gb, st, i) = at(Rb, st, i) = 0.0;
      }
      for (int32_t r = X.lane; r < P.R; r += X.lanes)
        kk[(int64_t)r * G] = kb[(int64_t)r * G] = 0.0;
      constexpr int32_t kWants = -2, kNone = -1;
      if (threadIdx.x < G)
        step[g] = kWants;
      auto finish = [&]() {
        double* out = A.ybar0 + cell_base(cell_of[g], L, S);
        for (int32_t i = X.lane; i < S; i += X.lanes)
          out[(int64_t)i * L] = yb[(int64_t)i * G];
        for (int32_t r = X.lane; r < P.R; r += X.lanes)
          A.kbar[(size_t)cell_of[g] * P.R + r] = kb[(int64_t)r * G];
      };
      for (;;)
      {
        // new cells; those without a step are done at once
        __syncthreads();
        while (__syncthreads_or(step[g] == kWants))
        {
          const bool wants = step[g] == kWants;
          __syncthreads();
          if (threadIdx.x < G && wants)
          {
            const int64_t k = atomicAdd(A.next_cell, 1);
            cell_of[g] = k < A.n_cells ? (A.order ? A.order[k] : k) : -1;
          }
          __syncthreads();
          const int64_t c = cell_of[g];
          const int32_t n_ck = wants && c >= 0 ? A.n_ckpt[c] : 0;
          if (wants && c >= 0)
          {
            const double* k = A.rate_constants + cell_base(c, L, P.R);
            for (int32_t r = X.lane; r < P.R; r += X.lanes)
            {
              kk[(int64_t)r * G] = k[(int64_t)r * L];
              kb[(int64_t)r * G] = 0.0;
            }
            if (n_ck == 0)
            {
              const size_t by = cell_base(c, L, S);
              for (int32_t i = X.lane; i < S; i += X.lanes)
                yb[(int64_t)i * G] = (A.y0[by + (size_t)i * L] < 0.0) ? 0.0 : A.ybar_final[by + (size_t)i * L];
              finish();
            }
          }
          __syncthreads();
          if (threadIdx.x < G && wants)
            step[g] = c < 0 ? kNone : (n_ck > 0 ? n_ck - 1 : kWants);
          __syncthreads();
        }
        const int32_t n = step[g];
        const bool live = n >= 0;
        if (!__syncthreads_or(live))
          break;
        const int64_t c = live ? cell_of[g] : 0;
        const size_t row = (size_t)c * A.max_ckpt + (live ? n : 0);
        const double* yc = A.ckpt_y + row * S;
        const double* kc = A.ckpt_k + row * (size_t)ns * S;
        const double H = live ? A.ckpt_h[row] : 1.0;
        // the step's factor
        for (int32_t i = X.lane; i < S; i += X.lanes)
          X[P.v0 + i] = yv[(int64_t)i * G] = live ? yc[i] : 0.0;
        __syncthreads();
        group_drates<G>(P, X, kk, G);
        __syncthreads();
        run_gather<G>(P.jacobian, X, 1.0 / (H * D.gamma0));
        __syncthreads();
        if (X.lane == 0)
          X[P.inv + S] = 1.0;  // the Jacobian rates were there
        run_levels<G, true>(P.lu, X, P);
        __syncthreads();
        if (X.lane == 0)
          X[P.trash] = 1.0;  // idle lanes left what is slow to divide
        const bool last_step = live && n == A.n_ckpt[c] - 1;
        for (int32_t i = X.lane; i < S; i += X.lanes)
        {
          if (last_step)
          {
            double v = yv[(int64_t)i * G];
            for (int32_t st = 0; st < ns; ++st)
              v += D.m[st] * kc[(int64_t)st * S + i];
            yb[(int64_t)i * G] = (v < 0.0) ? 0.0 : A.ybar_final[cell_base(c, L, S) + (size_t)i * L];
          }
          const double b = live ? yb[(int64_t)i * G] : 0.0;
          for (int32_t st = 0; st < ns; ++st)
          {
            at(Kb, st, i) = D.m[st] * b;
            at(Gb, st, i) = 0.0;
          }
        }
        for (int32_t st = ns - 1; st >= 0; --st)
        {
          const int32_t sc = st * (st - 1) / 2;
          for (int32_t i = X.lane; i < S; i += X.lanes)
            X[P.v0 + i] = at(Kb, st, i);
          __syncthreads();
          run_levels<G, false>(P.solve, X, P);
          __syncthreads();
          double coh[kMaxAdjStages];
          for (int32_t j = 0; j < st; ++j)
            coh[j] = D.c[sc + j] / H;
          const bool fresh = st > 0 && D.new_f[st];
          for (int32_t i = X.lane; i < S; i += X.lanes)
          {
            const double v = X[P.v0 + i];
            at(Rb, st, i) = v;
            const double gb = at(Gb, st, i) + v;
            at(Gb, st, i) = gb;
            for (int32_t j = 0; j < st; ++j)
              at(Kb, j, i) += coh[j] * v;
            if (fresh)
            {
              double y = yv[(int64_t)i * G];
              for (int32_t j = 0; j < st; ++j)
                y += D.a[sc + j] * (live ? kc[(int64_t)j * S + i] : 0.0);
              X[P.v0 + i] = y;
              X[P.g2 + i] = gb;
            }
            else if (st > 0)
              at(Gb, st - 1, i) += gb;
          }
          if (!fresh)
            continue;
          __syncthreads();
          group_vjp<G>(M, P, X, kk, kb);
          __syncthreads();
          run_gather<G>(P.forcing, X, 0.0);
          __syncthreads();
          for (int32_t i = X.lane; i < S; i += X.lanes)
          {
            const double t = X[P.v0 + i];
            yb[(int64_t)i * G] += t;
            for (int32_t j = 0; j < st; ++j)
              at(Kb, j, i) += D.a[sc + j] * t;
          }
        }
        // the terms at the step's start
        for (int32_t i = X.lane; i < S; i += X.lanes)
        {
          X[P.v0 + i] = yv[(int64_t)i * G];
          X[P.g2 + i] = at(Gb, 0, i);
        }
        __syncthreads();
        group_step_terms<G>(M, P, X, -1, kk, kb);
        for (int32_t st = 0; st < ns; ++st)
        {
          __syncthreads();
          for (int32_t i = X.lane; i < S; i += X.lanes)
          {
            X[P.g2 + i] = at(Rb, st, i);
            X[P.inv + i] = live ? kc[(int64_t)st * S + i] : 0.0;
          }
          __syncthreads();
          group_step_terms<G>(M, P, X, st, kk, kb);
        }
        __syncthreads();  // the state in V has been read
        for (int32_t i = X.lane; i < S; i += X.lanes)
          X[P.v0 + i] = yb[(int64_t)i * G];
        __syncthreads();
        run_gather<G, true>(P.step, X, 0.0);
        __syncthreads();
        for (int32_t i = X.lane; i < S; i += X.lanes)
          yb[(int64_t)i * G] = X[P.v0 + i];
        __syncthreads();
        if (live && n == 0)
          finish();
        if (threadIdx.x < G && live)
          step[g] = n > 0 ? n - 1 : kWants;
      }
    }

    using AdjGroupKernel = void (*)(DevMech, DevGroup, DevParams, AdjArgs, double*, int64_t);

    // Where the cell-group sweep is the faster one.  Measured, with the forward solve,
    // ms, cell groups / one cell per thread: Chapman 16,384 cells 3.9 / 4.0, 50,000
    // 9.4 / 9.1; 60 species 65,536 345 / 596, 131,072 691 / 799, 262,144 1,381 / 1,316;
    // 210 species (8 cells per SM) 49,152 1,504 / 2,177, and from the slopes equal at
    // about 97,000.  For small
    // mechanisms, whose blocks are single warps, the line lies lower.
    bool SweepGroupFaster(const micmb_solver& s, int64_t n)
    {
      if (!GroupFaster(s, n))
        return false;
      if (s.mech->nnz < kTinyNonZeros)
        return n <= (int64_t)s.sm_count * 128;
      return n <= std::min<int64_t>((int64_t)s.sm_count * 1024, 12288 * (int64_t)GroupCellsPerSm(s));
    }

    AdjGroupKernel AdjointGroupFor(int32_t G)
    {
      switch (G)
      {
        case 1: return k_adjoint_group<1>;
        case 2: return k_adjoint_group<2>;
        case 4: return k_adjoint_group<4>;
        case 8: return k_adjoint_group<8>;
        case 16: return k_adjoint_group<16>;
        default: return k_adjoint_group<32>;
      }
    }

    // 96 registers, 5 blocks of 128 per SM, no spills.  A full-occupancy build
    // (32 registers, as the forward kernel's fastest) measured slower here:
    // 1.38 s against 1.16 s on 131,072 cells of the 60-species mechanism, and
    // 67.6 s against 52.5 s on 262,144 cells of the 600-species one, where its
    // larger working-set footprint also leaves less memory for checkpoints.
    __global__ void __launch_bounds__(128, 5)
        k_adjoint_thread(DevMech M, DevParams P, AdjArgs A, AdjThreadLayout T, double* ws)
    {
      adjoint_thread_body(M, P, A, T, ws);
    }

    using AdjThreadKernel = void (*)(DevMech, DevParams, AdjArgs, AdjThreadLayout, double*);

    AdjThreadKernel AdjointThreadKernelFor(const micmb_solver&)
    {
      return k_adjoint_thread;
    }

    // Cells in decreasing order of accepted steps (counting sort on the step
    // count): the backward sweep takes the longest cells first, so the last
    // cells finish together, and the 32 cells of a warp have similar counts.
    __global__ void k_step_histogram(const int32_t* n_ckpt, int64_t n, int32_t max_ckpt, int32_t* bins)
    {
      const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
      if (c < n)
        atomicAdd(bins + (max_ckpt - min(max(n_ckpt[c], 0), max_ckpt)), 1);
    }

    __global__ void k_step_offsets(int32_t* bins, int32_t n_bins)
    {
      int32_t run = 0;
      for (int32_t b = 0; b < n_bins; ++b)
      {
        const int32_t v = bins[b];
        bins[b] = run;
        run += v;
      }
    }

    __global__ void k_step_scatter(const int32_t* n_ckpt, int64_t n, int32_t max_ckpt, int32_t* cursor,
                                   int32_t* order)
    {
      const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
      if (c < n)
        order[atomicAdd(cursor + (max_ckpt - min(max(n_ckpt[c], 0), max_ckpt)), 1)] = (int32_t)c;
    }

    // out[r] = sum over cells of kbar[cell][r], in a fixed order (deterministic)
    __global__ void k_sum_cells(const double* kbar, int64_t n_cells, int32_t R, double* out)
    {
      __shared__ double part[256];
      const int32_t r = blockIdx.x;
      double s = 0.0;
      for (int64_t c = threadIdx.x; c < n_cells; c += blockDim.x)
        s += kbar[(size_t)c * R + r];
      part[threadIdx.x] = s;
      __syncthreads();
      for (int w = blockDim.x / 2; w > 0; w >>= 1)
      {
        if ((int)threadIdx.x < w)
          part[threadIdx.x] += part[threadIdx.x + w];
        __syncthreads();
      }
      if (threadIdx.x == 0)
        out[r] = part[0];
    }
  }  // namespace

  namespace
  {
    // arguments for cells [begin, begin + count) of the state; begin is a
    // multiple of L, so every vector-layout array of the chunk starts at
    // begin * columns and is laid out like a state of `count` cells.  The
    // checkpoints hold the chunk's cells only.
    AdjArgs ChunkArgs(micmb_solver& s, micmb_state& st, int32_t max_ckpt, int64_t begin, int64_t count)
    {
      const auto& m = *s.mech;
      AdjArgs A{};
      A.n_cells = count;
      A.L = st.L;
      A.max_ckpt = max_ckpt;
      A.rate_constants = st.rate_constants.as<double>() + (size_t)begin * m.R;
      A.y0 = st.adj_y0.as<double>() + (size_t)begin * m.S;
      A.ybar_final = st.adj_ybar.as<double>() + (size_t)begin * m.S;
      A.ckpt_y = st.adj_ckpt_y.as<double>();
      A.ckpt_h = st.adj_ckpt_h.as<double>();
      A.ckpt_k = st.adj_ckpt_k.p ? st.adj_ckpt_k.as<double>() : nullptr;
      A.n_ckpt = st.accepted.as<int32_t>() + begin;
      A.ybar0 = st.adj_ybar.as<double>() + (size_t)begin * m.S;  // overwritten cell by cell after its last read
      A.kbar = st.adj_kbar_cells.as<double>() + (size_t)begin * m.R;
      char* cbase = st.counters.as<char>();
      A.next_cell = reinterpret_cast<int32_t*>(cbase + 8);
      return A;
    }
  }  // namespace

  // cell groups, or one cell per thread with working sets in global memory; no atomics
  void LaunchAdjointThread(micmb_solver& s, micmb_state& st, int32_t max_ckpt, int64_t begin, int64_t count)
  {
    const auto& m = *s.mech;
    if (s.params.stages > kMaxAdjStages)
      throw Error(MICMB_ERR_UNSUPPORTED, "too many stages for the adjoint kernel");
    const AdjThreadLayout T = MakeAdjThreadLayout(m.S, m.R, s.params.stages, (int32_t)m.info_rxn.size(), m.nnz);
    const AdjThreadKernel kernel = AdjointThreadKernelFor(s);
    int per_sm = 0;
    MICMB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 128, 0));
    if (per_sm < 1)
      throw Error(MICMB_ERR_UNSUPPORTED, "adjoint kernel cannot be resident");
    const int64_t n = count;
    int64_t grid = (int64_t)per_sm * s.sm_count;
    grid = std::max<int64_t>(1, std::min<int64_t>(grid, (n + 127) / 128));
    AdjArgs A = ChunkArgs(s, st, max_ckpt, begin, count);
    MICMB_CUDA(cudaMemsetAsync(A.next_cell, 0, 8, st.stream));
    if (n > 0)
    {
      const int32_t n_bins = max_ckpt + 1;
      const size_t need = sizeof(int32_t) * ((size_t)n + (size_t)n_bins);
      if (!st.adj_order.p || st.adj_order.bytes < need)
        st.adj_order = DeviceMemory(need);
      int32_t* order = st.adj_order.as<int32_t>();
      int32_t* bins = order + n;
      const unsigned blocks = (unsigned)((n + 255) / 256);
      MICMB_CUDA(cudaMemsetAsync(bins, 0, sizeof(int32_t) * n_bins, st.stream));
      k_step_histogram<<<blocks, 256, 0, st.stream>>>(A.n_ckpt, n, max_ckpt, bins);
      k_step_offsets<<<1, 1, 0, st.stream>>>(bins, n_bins);
      k_step_scatter<<<blocks, 256, 0, st.stream>>>(A.n_ckpt, n, max_ckpt, bins, order);
      MICMB_CUDA(cudaGetLastError());
      A.order = order;
      const GroupChoice choice = ChooseGroup(s, n, s.params.stages);
      const AdjGroupKernel group = AdjointGroupFor(choice.G);
      const int group_blocks = A.ckpt_k && SweepGroupFaster(s, n)
                                   ? GroupBlocksPerSm(s, reinterpret_cast<const void*>(group), choice)
                                   : 0;
      if (group_blocks > 0)
      {
        const int64_t blocks = std::min<int64_t>((int64_t)group_blocks * s.sm_count, (n + choice.G - 1) / choice.G);
        const int64_t slot = ((int64_t)m.S * (2 + 3 * s.params.stages) + 2 * (int64_t)m.R) * choice.G;
        EnsureWorkspace(st, st.group_ws, blocks * slot);
        group<<<(unsigned)blocks, 32 * choice.W, GroupSharedBytes(s, choice), st.stream>>>(
            s.dev, GroupTablesFor(s, choice).dev, s.params, A, st.group_ws.as<double>(), slot);
        MICMB_CUDA(cudaGetLastError());
        return;
      }
      const int64_t doubles = grid * 128 * (int64_t)T.per_slot;
      EnsureWorkspace(st, st.thread_ws, doubles);
      kernel<<<(unsigned)grid, 128, 0, st.stream>>>(s.dev, s.params, A, T, st.thread_ws.as<double>());
      MICMB_CUDA(cudaGetLastError());
    }
  }

  int64_t AdjointThreadWorkspaceDoubles(const micmb_solver& s, int64_t n_cells)
  {
    const auto& m = *s.mech;
    const AdjThreadLayout T = MakeAdjThreadLayout(m.S, m.R, s.params.stages, (int32_t)m.info_rxn.size(), m.nnz);
    int per_sm = 0;
    MICMB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, AdjointThreadKernelFor(s), 128, 0));
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)per_sm * s.sm_count, (n_cells + 127) / 128));
    return grid * 128 * (int64_t)T.per_slot;
  }

  void ReduceAdjointParameters(micmb_solver& s, micmb_state& st)
  {
    const auto& m = *s.mech;
    if (m.R > 0)
    {
      k_sum_cells<<<(unsigned)m.R, 256, 0, st.stream>>>(st.adj_kbar_cells.as<double>(), st.n_cells, m.R,
                                                         st.adj_kbar.as<double>());
      MICMB_CUDA(cudaGetLastError());
    }
  }

  void LaunchAdjoint(micmb_solver& s, micmb_state& st, int32_t max_ckpt, int64_t begin, int64_t count)
  {
    LaunchAdjointThread(s, st, max_ckpt, begin, count);
  }
}  // namespace micmb
