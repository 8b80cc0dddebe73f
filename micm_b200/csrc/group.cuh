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
    const uint4* ctrl;    // per unit
    const uint4* item;    // per unit and lane: two (level phases) or one (gathers)
    const uint4* row;     // per record and lane: two (level phases) or one (gathers)
    const double2* coef;  // gathers: two per record and lane
  };

  struct DevGroup
  {
    int32_t S, R, n_info, nnz;
    int32_t zero, one, v0, trash, w0, inv, rate, elements;
    DevGroupPhase forcing, jacobian, lu, solve;
    const uint2* rate_tab;
    const uint2* drate_tab;
  };

  // one thread's view of its cell
  template<int G>
  struct GroupThread
  {
    double* s;      // element e at s[e * G]
    int32_t lane;   // item lane in the block
    int32_t lanes;  // item lanes of the block
    int32_t warp;   // warp in the block
    int32_t sub;    // item lane in the warp

    __device__ __forceinline__ explicit GroupThread(double* shared)
        : s(shared + (threadIdx.x & (G - 1))),
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
    // element at a byte offset of the tables
    __device__ __forceinline__ double& at(uint32_t offset) const
    {
      return *reinterpret_cast<double*>(reinterpret_cast<char*>(s) + offset);
    }
  };

  // v / d given r = 1 / d rounded to nearest, by Markstein's method (IBM J. Res.
  // Dev. 34(1), 1990): a quotient q within an ulp of v / d has an exact remainder
  // v - q d (one fma), and q + r (v - q d) in one fma is v / d rounded to nearest.
  // v r itself can be one and a half ulps off, so a first correction brings it
  // within the ulp.  Five dependent operations where the divide takes about 110
  // cycles; operands whose exponents could leave the normal range anywhere on
  // the way (zeros, infinities and NaN among them) take the divide.
  __device__ __forceinline__ double divide_by(double v, double d, double r)
  {
    const int32_t ev = (__double2hiint(v) >> 20) & 0x7FF, ed = (__double2hiint(d) >> 20) & 0x7FF;
    if (v == 0.0 && (uint32_t)(ed - 523) <= 1000u)
      return v * r;  // a zero with the quotient's sign
    // exponents within 2^-500 .. 2^500
    if ((uint32_t)(ev - 523) <= 1000u && (uint32_t)(ed - 523) <= 1000u)
    {
      double q = v * r;
      q = fma(fma(-q, d, v), r, q);
      return fma(fma(-q, d, v), r, q);
    }
    return v / d;
  }

  // The records of this warp in one level phase, a unit of four at a time: the
  // next unit's table words are fetched (all together, so that they share one
  // wait) while this one is worked on, across barriers, since nothing in them
  // depends on the cells.  A unit takes a few hundred cycles, about what a
  // fetch from L2 takes.
  template<int G>
  __device__ __forceinline__ void run_levels(const DevGroupPhase& ph, const GroupThread<G>& X, const DevGroup& P)
  {
    constexpr int ipw = 32 / G, U = kGroupUnit;
    const uint32_t inv_offset = (uint32_t)(P.inv - P.v0) * (G * 8);
    int32_t u = ph.warp_start[X.warp];
    const int32_t u1 = ph.warp_start[X.warp + 1];
    if (u == u1)
      return;
    const uint4* cp = ph.ctrl + u;
    const uint4* ip = ph.item + ((int64_t)u * ipw + X.sub) * 2;
    const uint4* rp = ph.row + (int64_t)u * (U * 2 * ipw) + X.sub;
    uint4 nctrl = __ldg(cp), nitem[2] = { __ldg(ip), __ldg(ip + 1) }, nrow[2 * U];
#pragma unroll
    for (int j = 0; j < 2 * U; ++j)
      nrow[j] = __ldg(rp + j * ipw);
    double v = 0.0;
    for (; u < u1; ++u)
    {
      const uint32_t ctrl[U] = { nctrl.x, nctrl.y, nctrl.z, nctrl.w };
      const uint32_t target[U] = { nitem[0].x, nitem[0].z, nitem[1].x, nitem[1].z };
      const uint32_t aux[U] = { nitem[0].y, nitem[0].w, nitem[1].y, nitem[1].w };
      uint4 row[2 * U];
#pragma unroll
      for (int j = 0; j < 2 * U; ++j)
        row[j] = nrow[j];
      cp += 1;
      ip += 2 * ipw;
      rp += U * 2 * ipw;
      nctrl = __ldg(cp);
      nitem[0] = __ldg(ip);
      nitem[1] = __ldg(ip + 1);
#pragma unroll
      for (int j = 0; j < 2 * U; ++j)
        nrow[j] = __ldg(rp + j * ipw);
#pragma unroll
      for (int j = 0; j < U; ++j)
      {
        const uint32_t c = ctrl[j], T = c & 7u;
        const uint4 a = row[2 * j], b = row[2 * j + 1];
        if (c & 8u)
          v = X.at(target[j]);
        if (T > 2)
        {
          const double p0 = X.at(a.x) * X.at(a.y), p1 = X.at(a.z) * X.at(a.w);
          const double p2 = X.at(b.x) * X.at(b.y), p3 = X.at(b.z) * X.at(b.w);
          v -= p0;
          v -= p1;
          v -= p2;
          v -= p3;
        }
        else if (T > 0)
        {
          const double p0 = X.at(a.x) * X.at(a.y), p1 = X.at(a.z) * X.at(a.w);
          v -= p0;
          v -= p1;
        }
        if (c & 16u)
        {
          const uint32_t kind = (c >> 5) & 3u;
          if (kind == kGroupStore)
            X.at(target[j]) = v;
          else if (kind == kGroupScale)
            X.at(target[j]) = v * X.at(aux[j]);
          else if (kind == kGroupDiv)
            X.at(target[j]) = divide_by(v, X.at(aux[j]), X.at(target[j] + inv_offset));
          else
          {
            X.at(target[j]) = v;
            X.at(aux[j]) = 1.0 / v;
          }
        }
        const uint32_t sync = c >> 7;
        if (sync == 2)
          __syncthreads();
        else if (sync == 1)
          __syncwarp();
      }
    }
  }

  // Gathered sums of this warp's items: acc = sum coef * element, in term
  // order; out(target, flag, acc) takes each sum.  Units as in run_levels.
  template<int G, class Out>
  __device__ __forceinline__ void run_gather(const DevGroupPhase& ph, const GroupThread<G>& X, Out out)
  {
    constexpr int ipw = 32 / G, U = kGroupUnit;
    int32_t u = ph.warp_start[X.warp];
    const int32_t u1 = ph.warp_start[X.warp + 1];
    if (u == u1)
      return;
    const uint4* cp = ph.ctrl + u;
    const uint4* ip = ph.item + (int64_t)u * ipw + X.sub;
    const uint4* rp = ph.row + (int64_t)u * (U * ipw) + X.sub;
    const double2* fp = ph.coef + (int64_t)u * (U * 2 * ipw) + X.sub;
    uint4 nctrl = __ldg(cp), nitem = __ldg(ip), nrow[U];
    double2 nf[2 * U];
#pragma unroll
    for (int j = 0; j < U; ++j)
    {
      nrow[j] = __ldg(rp + j * ipw);
      nf[2 * j] = __ldg(fp + 2 * j * ipw);
      nf[2 * j + 1] = __ldg(fp + (2 * j + 1) * ipw);
    }
    double acc = 0.0;
    for (; u < u1; ++u)
    {
      const uint32_t ctrl[U] = { nctrl.x, nctrl.y, nctrl.z, nctrl.w };
      const uint32_t item[U] = { nitem.x, nitem.y, nitem.z, nitem.w };
      uint4 row[U];
      double2 f[2 * U];
#pragma unroll
      for (int j = 0; j < U; ++j)
      {
        row[j] = nrow[j];
        f[2 * j] = nf[2 * j];
        f[2 * j + 1] = nf[2 * j + 1];
      }
      cp += 1;
      ip += ipw;
      rp += U * ipw;
      fp += U * 2 * ipw;
      nctrl = __ldg(cp);
      nitem = __ldg(ip);
#pragma unroll
      for (int j = 0; j < U; ++j)
      {
        nrow[j] = __ldg(rp + j * ipw);
        nf[2 * j] = __ldg(fp + 2 * j * ipw);
        nf[2 * j + 1] = __ldg(fp + (2 * j + 1) * ipw);
      }
#pragma unroll
      for (int j = 0; j < U; ++j)
      {
        const uint32_t c = ctrl[j];
        if (c & 8u)
          acc = 0.0;
        if (c & 7u)
        {
          const double p0 = f[2 * j].x * X.at(row[j].x), p1 = f[2 * j].y * X.at(row[j].y);
          const double p2 = f[2 * j + 1].x * X.at(row[j].z), p3 = f[2 * j + 1].y * X.at(row[j].w);
          acc += p0;
          acc += p1;
          acc += p2;
          acc += p3;
        }
        if ((c & 16u) && item[j] != kGroupNoItem)
          out(item[j] & 0xFFFFu, item[j] >> 16, acc);
      }
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
    double *Y, *F0, *Fc, *K;
    const double* kk;  // rate constants, stride ks
    int32_t ks;
  };

  // doubles of Y, F0, Fc and K per cell
  __host__ __device__ inline int64_t GroupVectorDoubles(int32_t S, int32_t stages)
  {
    return (int64_t)S * (3 + stages);
  }

  template<int G>
  __device__ __forceinline__ GroupVectors group_vectors(double* slot, const DevGroup& P)
  {
    double* p = slot + (threadIdx.x & (G - 1));
    GroupVectors v;
    v.Y = p;
    v.F0 = v.Y + (int64_t)P.S * G;
    v.Fc = v.F0 + (int64_t)P.S * G;
    v.K = v.Fc + (int64_t)P.S * G;
    v.kk = nullptr;
    v.ks = 0;
    return v;
  }

  // One step attempt of the block's cells from the state in V (and v.Y), step
  // size H of this thread's cell: forcing (where new_f0), alpha I - J, LU, the
  // stages.  On return V holds Ynew, v.K the stage vectors, and the elements
  // P.rate + i the scaled squared errors; the caller synchronises.  The sums
  // and their order are those of the thread-per-cell routines.
  template<int G>
  __device__ __forceinline__ void group_attempt(const DevGroup& P, const DevParams& D, const GroupThread<G>& X,
                                                const GroupVectors& v, double H, bool new_f0,
                                                const double* __restrict__ atol, double rtol)
  {
    const int32_t S = P.S;
    if (new_f0)
    {
      group_rates<G>(P, X, v.kk, v.ks);
      __syncthreads();
      run_gather<G>(P.forcing, X, [&](uint32_t i, uint32_t, double acc) { v.F0[i * G] = acc; });
      __syncthreads();
    }
    group_drates<G>(P, X, v.kk, v.ks);
    __syncthreads();
    {
      const double alpha = 1.0 / (H * D.gamma0);
      run_gather<G>(P.jacobian, X,
                    [&](uint32_t e, uint32_t diag, double acc) { X[e] = diag ? acc + alpha : acc; });
    }
    __syncthreads();
    run_levels<G>(P.lu, X, P);
    const double* F = v.F0;
    for (int32_t st = 0; st < D.stages; ++st)
    {
      const int32_t sc = st * (st - 1) / 2;
      double coh[5];
#pragma unroll
      for (int32_t j = 0; j < 5; ++j)
        coh[j] = j < st ? D.c[sc + j] / H : 0.0;
      // the stage's right-hand side into V
      auto rhs = [&](uint32_t i, double f) {
#pragma unroll
        for (int32_t j = 0; j < 5; ++j)
          if (j < st)
            f += coh[j] * v.K[((int64_t)j * S + i) * G];
        X[P.v0 + i] = f;
      };
      if (st > 0 && D.new_f[st])
      {
#pragma unroll 4
        for (int32_t i = X.lane; i < S; i += X.lanes)
        {
          double y = v.Y[(int64_t)i * G];
#pragma unroll
          for (int32_t j = 0; j < 5; ++j)
            if (j < st)
              y += D.a[sc + j] * v.K[((int64_t)j * S + i) * G];
          X[P.v0 + i] = y;
        }
        __syncthreads();
        group_rates<G>(P, X, v.kk, v.ks);
        __syncthreads();
        const bool keep = st + 1 < D.stages && !D.new_f[st + 1];
        run_gather<G>(P.forcing, X, [&](uint32_t i, uint32_t, double acc) {
          if (keep)
            v.Fc[i * G] = acc;
          rhs(i, acc);
        });
        F = v.Fc;
      }
      else
        for (int32_t i = X.lane; i < S; i += X.lanes)
          rhs((uint32_t)i, F[(int64_t)i * G]);
      __syncthreads();
      run_levels<G>(P.solve, X, P);
      __syncthreads();
      for (int32_t i = X.lane; i < S; i += X.lanes)
        v.K[((int64_t)st * S + i) * G] = X[P.v0 + i];
    }
#pragma unroll 2
    for (int32_t i = X.lane; i < S; i += X.lanes)
    {
      const double y = v.Y[(int64_t)i * G];
      double yn = y, e = 0.0;
#pragma unroll
      for (int32_t st = 0; st < 6; ++st)
        if (st < D.stages)
        {
          const double kv = v.K[((int64_t)st * S + i) * G];
          yn += D.m[st] * kv;
          e += D.e[st] * kv;
        }
      X[P.v0 + i] = yn;
      X[P.rate + i] = scaled_sq(y, yn, e, atol[i], rtol);
    }
  }
}  // namespace micmb
