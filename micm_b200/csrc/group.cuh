// group.cuh -- device side of the cell-group kernels (work lists: group.hpp).
//
// A block of W warps advances G grid cells in lockstep; thread t works on cell
// t % G, item lane t / G.  The cells' factors and vectors are interleaved in
// shared memory (element e of cell g at e * G + g), so the G threads of an item
// read G consecutive doubles and share every table word.
#pragma once

#include "device.cuh"
#include "group.hpp"

namespace micmb
{
  struct DevGroupPhase
  {
    const int32_t* warp_start;
    const uint32_t* ctrl;  // per unit
    const uint4* item;     // per unit and lane
    const uint4* row;      // per unit and lane: four (level phases) or two (gathers)
    const double2* coef;   // gathers: eight per unit and lane
  };

  struct DevGroup
  {
    int32_t S, R, n_info, nnz;
    int32_t zero, one, v0, trash, w0, inv, rate, g2, slot, elements;
    DevGroupPhase forcing, jacobian, lu, solve, step;
    const int32_t* step_start;
    const uint2* rate_tab;
    const uint2* drate_tab;
  };

  // One thread's view of its cell.  The table-driven loops address shared memory
  // by 32-bit addresses formed in one instruction from a 16-bit element index
  // (dp2a: base + index * 8 G).
  template<int G>
  struct GroupThread
  {
    double* s;      // element e at s[e * G]
    uint32_t base;  // its shared-memory address
    int32_t lane;   // item lane in the block
    int32_t lanes;  // item lanes of the block
    int32_t warp;   // warp in the block
    int32_t sub;    // item lane in the warp

    __device__ __forceinline__ explicit GroupThread(double* shared)
        : s(shared + (threadIdx.x & (G - 1))),
          base((uint32_t)__cvta_generic_to_shared(s)),
          lane((int32_t)(threadIdx.x / G)),
          lanes((int32_t)(blockDim.x / G)),
          warp(__shfl_sync(0xffffffffu, (int32_t)(threadIdx.x >> 5), 0)),  // known to be the warp's
          sub((int32_t)((threadIdx.x & 31) / G))
    {
    }
    __device__ __forceinline__ double& operator[](uint32_t e) const
    {
      return s[e * G];
    }
    // addresses of the elements in a table word's halves
    __device__ __forceinline__ uint32_t lo(uint32_t w) const
    {
      if constexpr (G * 8 < 256)
        return __dp2a_lo(w, (uint32_t)(G * 8), base);
      else
        return base + (w & 0xFFFFu) * (G * 8);
    }
    __device__ __forceinline__ uint32_t hi(uint32_t w) const
    {
      if constexpr (G * 8 < 256)
        return __dp2a_lo(w, (uint32_t)(G * 8) << 8, base);
      else
        return base + (w >> 16) * (G * 8);
    }
    static __device__ __forceinline__ double load(uint32_t address)
    {
      double v;
      asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(address) : "memory");
      return v;
    }
    static __device__ __forceinline__ void store(uint32_t address, double v)
    {
      asm volatile("st.shared.f64 [%0], %1;" ::"r"(address), "d"(v) : "memory");
    }
  };

  // v / d given r = 1 / d rounded to nearest, by Markstein's method (IBM J. Res.
  // Dev. 34(1), 1990): a quotient q within an ulp of v / d has an exact remainder
  // v - q d (one fma), and q + r (v - q d) in one fma is v / d rounded to nearest.
  // v r itself can be one and a half ulps off, so a first correction brings it
  // within the ulp.  Five dependent operations where the divide takes about 110
  // cycles; operands whose exponents could leave the normal range anywhere on
  // the way (zeros, infinities and NaN among them) take the divide.
  static __device__ __noinline__ double divide_slowly(double v, double d)
  {
    return v / d;
  }

  __device__ __forceinline__ double divide_by(double v, double d, double r)
  {
    double q = v * r;
    q = fma(fma(-q, d, v), r, q);
    q = fma(fma(-q, d, v), r, q);
    const int32_t ev = (__double2hiint(v) >> 20) & 0x7FF, ed = (__double2hiint(d) >> 20) & 0x7FF;
    // exponents within 2^-500 .. 2^500
    if ((uint32_t)(ev - 523) > 1000u || (uint32_t)(ed - 523) > 1000u)
      q = (v == 0.0 && (uint32_t)(ed - 523) <= 1000u) ? v * r  // a zero with the quotient's sign
                                                      : divide_slowly(v, d);
    return q;
  }

  // A unit's table words.
  template<int G, bool LU>
  struct LevelUnit
  {
    uint32_t ctrl;
    uint4 item, row[4];

    __device__ __forceinline__ void fetch(const uint32_t*& cp, const uint4*& ip, const uint4*& rp)
    {
      constexpr int ipw = 32 / G;
      ctrl = __ldg(cp);
      item = __ldg(ip);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        row[j] = __ldg(rp + j * ipw);
      cp += 1;
      ip += ipw;
      rp += 4 * ipw;
    }

    __device__ __forceinline__ uint32_t item_word(int k) const
    {
      return k == 0 ? item.x : (k == 1 ? item.y : (k == 2 ? item.z : item.w));
    }
    __device__ __forceinline__ uint32_t term_word(int t) const
    {
      const uint4 q = row[t / 4];
      return t % 4 == 0 ? q.x : (t % 4 == 1 ? q.y : (t % 4 == 2 ? q.z : q.w));
    }

    // The unit with C chunks of T terms; the chunks' sums run side by side.
    template<int C, int T, int FIN>
    __device__ __forceinline__ void run(const GroupThread<G>& X, uint32_t inv_offset, double& carry) const
    {
      double v[C], d[C], r[C];
#pragma unroll
      for (int k = 0; k < C; ++k)
      {
        v[k] = X.load(X.lo(item_word(k)));
        if (FIN == (LU ? kGroupPlain : kGroupPivot))
          d[k] = X.load(X.hi(item_word(k)));
        if (!LU && FIN == kGroupPivot)
          r[k] = X.load(X.lo(item_word(k)) + inv_offset);
      }
      if (C == 1 && T == 16 && !(ctrl & 1024u))
        v[0] = carry;
#pragma unroll
      for (int t = 0; t < T; ++t)
      {
        double p[C];
#pragma unroll
        for (int k = 0; k < C; ++k)
        {
          const uint32_t w = term_word(k * (16 / C) + t);
          const double a = X.load(X.lo(w)), b = X.load(X.hi(w));
          p[k] = a * b;
        }
#pragma unroll
        for (int k = 0; k < C; ++k)
          v[k] -= p[k];
      }
      if (C == 1 && FIN == kGroupNone)
        carry = v[0];
      else
#pragma unroll
        for (int k = 0; k < C; ++k)
        {
          const uint32_t target = X.lo(item_word(k));
          if (FIN == kGroupPlain)
            X.store(target, LU ? v[k] * d[k] : v[k]);
          else if (!LU)
            X.store(target, divide_by(v[k], d[k], r[k]));
          else
          {
            X.store(target, v[k]);
            X.store(X.hi(item_word(k)), 1.0 / v[k]);
          }
        }
    }

    // one jump per unit: a taken branch costs a lone warp about 25 cycles
    __device__ __forceinline__ void run(const GroupThread<G>& X, uint32_t inv_offset, double& carry) const
    {
#define MICMB_GROUP_CASES(shape, C, T)                        \
  case shape * 3 + kGroupPlain: run<C, T, kGroupPlain>(X, inv_offset, carry); break; \
  case shape * 3 + kGroupPivot: run<C, T, kGroupPivot>(X, inv_offset, carry); break;
      switch (ctrl & 255u)
      {
        MICMB_GROUP_CASES(0, 1, 4)
        MICMB_GROUP_CASES(1, 1, 8)
        MICMB_GROUP_CASES(2, 1, 16)
        MICMB_GROUP_CASES(3, 2, 4)
        MICMB_GROUP_CASES(4, 2, 8)
        MICMB_GROUP_CASES(5, 4, 2)
        MICMB_GROUP_CASES(6, 4, 4)
        case 2 * 3 + kGroupNone: run<1, 16, kGroupNone>(X, inv_offset, carry); break;
      }
#undef MICMB_GROUP_CASES
      if (ctrl & (kGroupBlockSync << 8))
        __syncthreads();
      else
        __syncwarp();
    }
  };

  // The units of this warp in one level phase.  The next unit's table words are
  // fetched while this one is worked on, across barriers, since nothing in them
  // depends on the cells.  The copy waits for all of a unit's words before the
  // next ones are asked for.
  template<int G, bool LU>
  __device__ __forceinline__ void run_levels(const DevGroupPhase& ph, const GroupThread<G>& X, const DevGroup& P)
  {
    constexpr int ipw = 32 / G;
    const uint32_t inv_offset = (uint32_t)(P.inv - P.v0) * (G * 8);
    int32_t u = ph.warp_start[X.warp];
    const int32_t u1 = ph.warp_start[X.warp + 1];
    const uint32_t* cp = ph.ctrl + u;
    const uint4* ip = ph.item + ((int64_t)u * ipw + X.sub);
    const uint4* rp = ph.row + ((int64_t)u * (4 * ipw) + X.sub);
    LevelUnit<G, LU> next;
    double carry = 0.0;
    if (u < u1)
      next.fetch(cp, ip, rp);
#pragma unroll 1
    for (; u < u1; ++u)
    {
      const LevelUnit<G, LU> unit = next;
      next.fetch(cp, ip, rp);
      unit.run(X, inv_offset, carry);
    }
  }

  // One unit of a gather: sums of coef * element, in term order.
  template<int G>
  struct GatherUnit
  {
    uint32_t ctrl;
    uint4 item, row[2];
    double2 f[8];

    __device__ __forceinline__ void fetch(const uint32_t*& cp, const uint4*& ip, const uint4*& rp, const double2*& fp)
    {
      constexpr int ipw = 32 / G;
      ctrl = __ldg(cp);
      item = __ldg(ip);
      row[0] = __ldg(rp);
      row[1] = __ldg(rp + ipw);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        f[j] = __ldg(fp + j * ipw);
      cp += 1;
      ip += ipw;
      rp += 2 * ipw;
      fp += 8 * ipw;
    }

    // ADD: the sums start from their elements' values, and nothing gains alpha
    template<bool ADD, int C, int T, bool LAST>
    __device__ __forceinline__ void run(const GroupThread<G>& X, double alpha, double& carry) const
    {
      double acc[C];
#pragma unroll
      for (int k = 0; k < C; ++k)
        acc[k] = ADD ? X.load(X.lo(k == 0 ? item.x : (k == 1 ? item.y : (k == 2 ? item.z : item.w)))) : 0.0;
      if (C == 1 && T == 16 && !(ctrl & 1024u))
        acc[0] = carry;
#pragma unroll
      for (int t = 0; t < T; ++t)
      {
        double p[C];
#pragma unroll
        for (int k = 0; k < C; ++k)
        {
          const int i = k * (16 / C) + t;
          const uint4 q = row[i / 8];
          const uint32_t w = (i / 2) % 4 == 0 ? q.x : ((i / 2) % 4 == 1 ? q.y : ((i / 2) % 4 == 2 ? q.z : q.w));
          p[k] = (i % 2 ? f[i / 2].y : f[i / 2].x) * X.load(i % 2 ? X.hi(w) : X.lo(w));
        }
#pragma unroll
        for (int k = 0; k < C; ++k)
          acc[k] += p[k];
      }
      if (C == 1 && !LAST)
        carry = acc[0];
      else
#pragma unroll
        for (int k = 0; k < C; ++k)
        {
          const uint32_t it = k == 0 ? item.x : (k == 1 ? item.y : (k == 2 ? item.z : item.w));
          // a sum that starts at +0 is never -0, so adding 0 changes none
          X.store(X.lo(it), ADD ? acc[k] : acc[k] + (it >> 16 ? alpha : 0.0));
        }
    }

    template<bool ADD>
    __device__ __forceinline__ void run(const GroupThread<G>& X, double alpha, double& carry) const
    {
      switch (ctrl & 255u)
      {
        case 0 * 3: run<ADD, 1, 4, true>(X, alpha, carry); break;
        case 1 * 3: run<ADD, 1, 8, true>(X, alpha, carry); break;
        case 2 * 3: run<ADD, 1, 16, true>(X, alpha, carry); break;
        case 3 * 3: run<ADD, 2, 4, true>(X, alpha, carry); break;
        case 4 * 3: run<ADD, 2, 8, true>(X, alpha, carry); break;
        case 5 * 3: run<ADD, 4, 2, true>(X, alpha, carry); break;
        case 6 * 3: run<ADD, 4, 4, true>(X, alpha, carry); break;
        case 2 * 3 + kGroupNone: run<ADD, 1, 16, false>(X, alpha, carry); break;
      }
    }
  };

  // Gathered sums of this warp's items into their elements (ADD: added to them);
  // flagged ones gain alpha.
  template<int G, bool ADD = false>
  __device__ __forceinline__ void run_gather(const DevGroupPhase& ph, const GroupThread<G>& X, double alpha)
  {
    constexpr int ipw = 32 / G;
    int32_t u = ph.warp_start[X.warp];
    const int32_t u1 = ph.warp_start[X.warp + 1];
    const uint32_t* cp = ph.ctrl + u;
    const uint4* ip = ph.item + ((int64_t)u * ipw + X.sub);
    const uint4* rp = ph.row + ((int64_t)u * (2 * ipw) + X.sub);
    const double2* fp = ph.coef + ((int64_t)u * (8 * ipw) + X.sub);
    GatherUnit<G> next;
    double carry = 0.0;
    if (u < u1)
      next.fetch(cp, ip, rp, fp);
#pragma unroll 1
    for (; u < u1; ++u)
    {
      const GatherUnit<G> unit = next;
      next.fetch(cp, ip, rp, fp);
      unit.template run<ADD>(X, alpha, carry);
    }
  }

  // rate[r] = k_r * products of the state in V (kk: this thread's cell, rate r at
  // r * ks in global memory).  Rate constants are fetched a batch at a time: a
  // store to shared memory may alias them as far as the compiler knows.
  template<int G>
  __device__ __forceinline__ void group_rates(const DevGroup& P, const GroupThread<G>& X, const double* kk, int32_t ks)
  {
    constexpr int B = 8;
    for (int32_t r0 = X.lane; r0 < P.R; r0 += B * X.lanes)
    {
      uint2 d[B];
      double k[B];
#pragma unroll
      for (int b = 0; b < B; ++b)
      {
        const int32_t r = min(r0 + b * X.lanes, P.R - 1);
        d[b] = __ldg(P.rate_tab + r);
        k[b] = kk[(int64_t)r * ks];
      }
#pragma unroll
      for (int b = 0; b < B; ++b)
      {
        const int32_t r = r0 + b * X.lanes;
        if (r < P.R)
        {
          double v = k[b];
          v *= X[d[b].x & 0xFFFFu];
          v *= X[d[b].x >> 16];
          v *= X[d[b].y];
          X[P.rate + r] = v;
        }
      }
    }
  }

  // Jacobian rates into W
  template<int G>
  __device__ __forceinline__ void group_drates(const DevGroup& P, const GroupThread<G>& X, const double* kk,
                                               int32_t ks)
  {
    constexpr int B = 8;
    for (int32_t i0 = X.lane; i0 < P.n_info; i0 += B * X.lanes)
    {
      uint2 d[B];
      double k[B];
#pragma unroll
      for (int b = 0; b < B; ++b)
        d[b] = __ldg(P.drate_tab + min(i0 + b * X.lanes, P.n_info - 1));
#pragma unroll
      for (int b = 0; b < B; ++b)
        k[b] = kk[(int64_t)(d[b].x & 0xFFFFu) * ks];
#pragma unroll
      for (int b = 0; b < B; ++b)
      {
        const int32_t i = i0 + b * X.lanes;
        if (i < P.n_info)
        {
          double v = k[b];
          v *= X[d[b].x >> 16];
          v *= X[d[b].y & 0xFFFFu];
          v *= X[d[b].y >> 16];
          X[P.w0 + i] = v;
        }
      }
    }
  }

  // The cells' vectors that stay in global memory (L2), element i at i * G
  struct GroupVectors
  {
    double *Y, *Fc, *K;
    const double* kk;  // rate constants, stride ks
    int32_t ks;
  };

  // doubles of Y, Fc and K per cell
  __host__ __device__ inline int64_t GroupVectorDoubles(int32_t S, int32_t stages)
  {
    return (int64_t)S * (2 + stages);
  }

  template<int G>
  __device__ __forceinline__ GroupVectors group_vectors(double* slot, const DevGroup& P)
  {
    double* p = slot + (threadIdx.x & (G - 1));
    GroupVectors v;
    v.Y = p;
    v.Fc = v.Y + (int64_t)P.S * G;
    v.K = v.Fc + (int64_t)P.S * G;
    v.kk = nullptr;
    v.ks = 0;
    return v;
  }

  // f(i) for this thread's species, in batches of B whose loads can all be under
  // way together: load(b, i) fetches (i clamped to the last species), use(b, i)
  // computes and stores.
  template<int B, int G, class Load, class Use>
  __device__ __forceinline__ void for_species_by(const GroupThread<G>& X, int32_t S, Load load, Use use)
  {
    for (int32_t i0 = X.lane; i0 < S; i0 += B * X.lanes)
    {
#pragma unroll
      for (int b = 0; b < B; ++b)
        load(b, min(i0 + b * X.lanes, S - 1));
#pragma unroll
      for (int b = 0; b < B; ++b)
        if (i0 + b * X.lanes < S)
          use(b, i0 + b * X.lanes);
    }
  }

  template<int B, int G, class Load, class Use>
  __device__ __forceinline__ void for_species(const GroupThread<G>& X, int32_t S, Load load, Use use)
  {
    if (S <= 2 * X.lanes)
      for_species_by<2, G>(X, S, load, use);
    else
      for_species_by<B, G>(X, S, load, use);
  }

  // One step attempt of the block's cells from the state in V (and v.Y), step
  // size H of this thread's cell: alpha I - J, LU, then per stage the forcing
  // (where it is new) and the solve.  On return V holds Ynew, v.K the stage
  // vectors, and the elements P.rate + i the scaled squared errors; the caller
  // synchronises.  The sums and their order are those of the thread-per-cell
  // routines.
  template<int G>
  __device__ __forceinline__ void group_attempt(const DevGroup& P, const DevParams& D, const GroupThread<G>& X,
                                                const GroupVectors& v, double H, const double* __restrict__ atol,
                                                double rtol)
  {
    const int32_t S = P.S;
    group_drates<G>(P, X, v.kk, v.ks);
    __syncthreads();
    run_gather<G>(P.jacobian, X, 1.0 / (H * D.gamma0));
    __syncthreads();
    if (X.lane == 0)
      X[P.inv + S] = 1.0;  // the Jacobian rates were there
    run_levels<G, true>(P.lu, X, P);
    for (int32_t st = 0; st < D.stages; ++st)
    {
      const int32_t sc = st * (st - 1) / 2;
      const bool fresh = st == 0 || D.new_f[st];
      if (fresh)
      {
        // V holds Y in the first stage
        if (st > 0)
        {
          double y[8];
          for_species<8, G>(
              X, S,
              [&](int b, int32_t i) {
                y[b] = v.Y[(int64_t)i * G];
#pragma unroll
                for (int32_t j = 0; j < 5; ++j)
                  if (j < st)
                    y[b] += D.a[sc + j] * v.K[((int64_t)j * S + i) * G];
              },
              [&](int b, int32_t i) { X[P.v0 + i] = y[b]; });
          __syncthreads();
        }
        group_rates<G>(P, X, v.kk, v.ks);
        __syncthreads();
        run_gather<G>(P.forcing, X, 0.0);
        __syncthreads();
      }
      // the stage's right-hand side into V
      const bool keep = fresh && st + 1 < D.stages && !D.new_f[st + 1];
      if (st > 0 || keep)
      {
        double coh[5];
#pragma unroll
        for (int32_t j = 0; j < 5; ++j)
          coh[j] = j < st ? D.c[sc + j] / H : 0.0;
        double f[8], f0[8];
        for_species<8, G>(
            X, S,
            [&](int b, int32_t i) {
              f0[b] = f[b] = fresh ? X[P.v0 + i] : v.Fc[(int64_t)i * G];
#pragma unroll
              for (int32_t j = 0; j < 5; ++j)
                if (j < st)
                  f[b] += coh[j] * v.K[((int64_t)j * S + i) * G];
            },
            [&](int b, int32_t i) {
              if (keep)
                v.Fc[(int64_t)i * G] = f0[b];
              X[P.v0 + i] = f[b];
            });
        __syncthreads();
      }
      run_levels<G, false>(P.solve, X, P);
      __syncthreads();
      for (int32_t i = X.lane; i < S; i += X.lanes)
        v.K[((int64_t)st * S + i) * G] = X[P.v0 + i];
    }
    double y[4], yn[4], e[4], at[4];
    for_species<4, G>(
        X, S,
        [&](int b, int32_t i) {
          y[b] = yn[b] = v.Y[(int64_t)i * G];
          at[b] = atol[i];
          e[b] = 0.0;
#pragma unroll
          for (int32_t st = 0; st < 6; ++st)
            if (st < D.stages)
            {
              const double kv = v.K[((int64_t)st * S + i) * G];
              yn[b] += D.m[st] * kv;
              e[b] += D.e[st] * kv;
            }
        },
        [&](int b, int32_t i) {
          X[P.v0 + i] = yn[b];
          X[P.rate + i] = scaled_sq(y[b], yn[b], e[b], at[b], rtol);
        });
  }

  // One Newton iteration of Backward Euler on the block's cells (backward_euler.cu:
  // newton_iteration) from the state in V and v.Y, with the step's start in v.Fc:
  // Y <- max(0, Y + (LU)^-1 (f(Y) - (Y - Yn) / H)), into V and v.Y.  test(i, d, y)
  // sees every correction and new value.
  template<int G, class Test>
  __device__ __forceinline__ void group_newton(const DevGroup& P, const GroupThread<G>& X, const GroupVectors& v,
                                               double H, Test test)
  {
    const int32_t S = P.S;
    group_drates<G>(P, X, v.kk, v.ks);
    __syncthreads();
    run_gather<G>(P.jacobian, X, 1.0 / H);
    __syncthreads();
    if (X.lane == 0)
      X[P.inv + S] = 1.0;  // the Jacobian rates were there
    run_levels<G, true>(P.lu, X, P);
    group_rates<G>(P, X, v.kk, v.ks);
    __syncthreads();
    run_gather<G>(P.forcing, X, 0.0);
    __syncthreads();
    double y[4], yn[4];
    for_species<4, G>(
        X, S,
        [&](int b, int32_t i) {
          y[b] = v.Y[(int64_t)i * G];
          yn[b] = v.Fc[(int64_t)i * G];
        },
        [&](int b, int32_t i) { X[P.v0 + i] = X[P.v0 + i] - (y[b] - yn[b]) / H; });
    __syncthreads();
    run_levels<G, false>(P.solve, X, P);
    __syncthreads();
    for_species<4, G>(
        X, S, [&](int b, int32_t i) { y[b] = v.Y[(int64_t)i * G]; },
        [&](int b, int32_t i) {
          const double d = X[P.v0 + i], sum = y[b] + d, yi = (0.0 > sum) ? 0.0 : sum;
          v.Y[(int64_t)i * G] = yi;
          X[P.v0 + i] = yi;
          test(i, d, yi);
        });
  }
}  // namespace micmb
