// Runs the cell-group work lists (micm_b200/csrc/group.hpp) of a mechanism on one
// cell on the host, unit by unit as a block's warps do, and compares every LU
// entry, solution component and gather list with the serial schedules bit for bit.
// Also counted: elements out of range, and elements that one item lane writes while
// another one reads or writes them without a synchronisation in between.
#include "../../micm_b200/csrc/group.hpp"

#include <cstring>
#include <functional>
#include <random>
#include <set>

using namespace micmb;

namespace
{
  struct Checker
  {
    const CompiledMechanism& m;
    const GroupProgram p;
    const GroupLayout& L;
    const int ipw, W;
    std::vector<double> E;  // the cell's elements
    int64_t bad = 0;

    Checker(const CompiledMechanism& mech, int G, int warps, int sweep_stages)
        : m(mech),
          p(BuildGroupProgram(mech, G, warps, sweep_stages)),
          L(p.layout),
          ipw(32 / G),
          W(warps),
          E(L.elements, 0.0)
    {
      E[L.one] = 1.0;
    }

    bool InRange(int e)
    {
      bad += e < 0 || e >= L.elements;
      return e >= 0 && e < L.elements;
    }

    void RunLevels(const GroupPhase& ph, bool lu)
    {
      std::vector<int> at(ph.warp_start.begin(), ph.warp_start.begin() + W);
      std::vector<double> carry(W * 32, 0.0);
      for (bool done = false; !done;)
      {
        // one stretch between two block synchronisations
        done = true;
        std::vector<std::set<int>> read(W), written(W);
        for (int w = 0; w < W; ++w)
        {
          std::vector<std::set<int>> r(ipw), wr(ipw);
          auto lanes_apart = [&] {
            for (int a = 0; a < ipw; ++a)
              for (int b = 0; b < ipw; ++b)
                if (a != b)
                  for (int e : wr[a])
                    bad += r[b].count(e) + wr[b].count(e);
            r.assign(ipw, {});
            wr.assign(ipw, {});
          };
          while (at[w] < ph.warp_start[w + 1])
          {
            const int u = at[w]++;
            const uint32_t c = ph.ctrl.at(u);
            const GroupShape shape = kGroupShapes[(c & 255) / 3];
            const int fin = (c & 255) % 3, sync = (c >> 8) & 3, room = kGroupTerms / shape.chunks;
            const bool first = c & 1024;
            bad += (fin == kGroupNone || !first) && shape.terms != kGroupTerms;
            std::vector<std::pair<int, double>> stores;
            for (int q = 0; q < ipw; ++q)
              for (int k = 0; k < shape.chunks; ++k)
              {
                const uint32_t item = ph.item.at(((size_t)u * ipw + q) * 4 + k);
                const int target = item & 0xFFFF, aux = item >> 16;
                if (!InRange(target) || !InRange(aux) || !InRange(target - L.v0 + L.inv))
                  continue;
                const bool idle = target == L.trash;
                bad += idle && aux != (lu && fin == kGroupPivot ? L.trash : L.one);
                double v = first ? (idle ? 1.0 : E[target]) : carry[w * 32 + q];
                if (!idle)
                  r[q].insert(target);
                for (int t = k * room; t < k * room + room; ++t)
                {
                  const uint32_t word = ph.row.at((((size_t)u * 4 + t / 4) * ipw + q) * 4 + t % 4);
                  const int a = word & 0xFFFF, b = word >> 16;
                  if (!InRange(a) || !InRange(b))
                    continue;
                  if (t - k * room >= shape.terms)  // not run
                  {
                    bad += a != L.zero || b != L.zero;
                    continue;
                  }
                  r[q].insert({ a, b });
                  const double product = E[a] * E[b];
                  v = v - product;
                }
                if (fin == kGroupNone)
                  carry[w * 32 + q] = v;
                if (fin == kGroupNone || idle)
                  continue;
                wr[q].insert(target);
                if (lu || fin == kGroupPivot)
                  r[q].insert(aux);
                if (fin == kGroupPlain)
                  stores.push_back({ target, lu ? v * E[aux] : v });
                else if (!lu)
                {
                  r[q].insert(target - L.v0 + L.inv);
                  stores.push_back({ target, v / E[aux] });
                }
                else
                {
                  wr[q].insert(aux);
                  r[q].erase(aux);
                  stores.push_back({ target, v });
                  stores.push_back({ aux, 1.0 / v });
                }
              }
            for (const auto& s : stores)
              E[s.first] = s.second;
            for (int q = 0; q < ipw; ++q)
            {
              read[w].insert(r[q].begin(), r[q].end());
              written[w].insert(wr[q].begin(), wr[q].end());
            }
            if (sync != kGroupNoSync)
              lanes_apart();
            if (sync == kGroupBlockSync)
              break;
          }
          lanes_apart();
          done = done && at[w] == ph.warp_start[w + 1];
        }
        for (int a = 0; a < W; ++a)
          for (int b = 0; b < W; ++b)
            if (a != b)
              for (int e : written[a])
                bad += read[b].count(e) + written[b].count(e);
      }
    }

    void CheckGather(const GroupPhase& ph, const std::vector<int32_t>& start, const std::vector<int32_t>& src,
                     const std::vector<double>& coef, int src0, int target0, const std::function<int(int)>& flag)
    {
      std::vector<int> seen(start.size() - 1, 0);
      for (int w = 0; w < W; ++w)
      {
        std::vector<int> from(ipw, 0);
        for (int u = ph.warp_start[w]; u < ph.warp_start[w + 1]; ++u)
        {
          const uint32_t c = ph.ctrl.at(u);
          const GroupShape shape = kGroupShapes[(c & 255) / 3];
          const bool first = c & 1024, last = (c & 255) % 3 != kGroupNone;
          const int room = kGroupTerms / shape.chunks;
          for (int q = 0; q < ipw; ++q)
            for (int k = 0; k < shape.chunks; ++k)
            {
              const uint32_t item = ph.item.at(((size_t)u * ipw + q) * 4 + k);
              if ((int)(item & 0xFFFF) == L.trash)
                continue;
              const int i = (int)(item & 0xFFFF) - target0, n = start[i + 1] - start[i];
              bad += (int)(item >> 16) != flag(i);
              const int t0 = first ? 0 : from[q];
              from[q] = t0 + shape.terms;
              seen.at(i) += last;
              bad += last && t0 + shape.terms < n;
              for (int t = 0; t < shape.terms; ++t)
              {
                const int x = k * room + t;
                const uint32_t word = ph.row.at((((size_t)u * 2 + x / 8) * ipw + q) * 4 + x % 8 / 2);
                const int e = (word >> (16 * (x % 2))) & 0xFFFF;
                const double f = ph.coef.at((((size_t)u * 8 + x / 2) * ipw + q) * 2 + x % 2);
                bad += t0 + t < n ? (e != src0 + src[start[i] + t0 + t] || f != coef[start[i] + t0 + t])
                                  : (e != L.zero || f != 0.0);
              }
            }
        }
      }
      for (int s : seen)
        bad += s != 1;
    }
  };
}  // namespace

// number of faults; -1: the mechanism has no group work lists
extern "C" int64_t check_group_lists(const micmb_mechanism_desc* desc, int32_t G, int32_t W,
                                     int32_t sweep_stages)
{
  const CompiledMechanism m = Compile(*desc);
  if (!GroupApplies(m))
    return -1;
  Checker c(m, G, W, sweep_stages);
  const GroupLayout& L = c.L;
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> uniform(0.5, 1.5);
  std::vector<double> A(m.nnz), inv(m.S), x(m.S);
  for (double& a : A)
    a = uniform(rng);
  for (int32_t i = 0; i < m.S; ++i)
  {
    A[m.diag_pos[i]] += 50.0;
    c.E[L.v0 + i] = x[i] = uniform(rng);
  }
  std::copy(A.begin(), A.end(), c.E.begin());

  c.RunLevels(c.p.lu, true);
  std::vector<int32_t> row_of(m.nnz, -1);
  for (int32_t i = 0; i < m.S; ++i)
    row_of[m.diag_pos[i]] = i;
  for (int32_t it = 0; it < m.lu_serial.n_items(); ++it)
  {
    const LevelSchedule& s = m.lu_serial;
    double v = A[s.item_target[it]];
    for (int32_t t = s.term_start[it]; t < s.term_start[it + 1]; ++t)
    {
      const double product = A[s.term_a[t]] * A[s.term_b[t]];
      v = v - product;
    }
    if (s.item_aux[it] >= 0)
      v = v * inv[row_of[s.item_aux[it]]];
    A[s.item_target[it]] = v;
    if (row_of[s.item_target[it]] >= 0)
      inv[row_of[s.item_target[it]]] = 1.0 / v;
  }
  auto same = [&](const double* got, const std::vector<double>& want) {
    for (size_t i = 0; i < want.size(); ++i)
      c.bad += std::memcmp(got + i, &want[i], sizeof(double)) != 0;
  };
  same(c.E.data(), A);
  same(c.E.data() + L.inv, inv);

  c.RunLevels(c.p.solve, false);
  const LevelSchedule* const order[2] = { sweep_stages ? &m.fwd_t_serial : &m.fwd_serial,
                                          sweep_stages ? &m.bwd_t_serial : &m.bwd_serial };
  for (const LevelSchedule* s : order)
    for (int32_t it = 0; it < s->n_items(); ++it)
    {
      double v = x[s->item_target[it]];
      for (int32_t t = s->term_start[it]; t < s->term_start[it + 1]; ++t)
      {
        const double product = A[s->term_a[t]] * x[s->term_b[t]];
        v = v - product;
      }
      x[s->item_target[it]] = s->item_aux[it] >= 0 ? v / A[s->item_aux[it]] : v;
    }
  same(c.E.data() + L.v0, x);

  const auto plain = [](int) { return 0; };
  if (sweep_stages == 0)
    c.CheckGather(c.p.forcing, m.f_start, m.f_rxn, m.f_coef, L.rate, L.v0, plain);
  else
  {
    // contributions are numbered reaction by reaction: reactants, then (stage, q, o)
    std::vector<int32_t> owner;
    for (int32_t r = 0; r < m.R; ++r)
    {
      const int32_t r0 = m.react_start[r], r1 = m.react_start[r + 1];
      c.bad += c.p.step_start.at(r) != (int32_t)owner.size();
      owner.insert(owner.end(), m.react_ids.begin() + r0, m.react_ids.begin() + r1);
      for (int32_t st = 0; st < sweep_stages; ++st)
        for (int32_t q = r0; q < r1; ++q)
          for (int32_t o = r0; o < r1; ++o)
            if (q != o)
              owner.push_back(m.react_ids[o]);
    }
    auto check = [&](const GroupPhase& ph, const std::vector<int32_t>& species, const std::function<int(int)>& element) {
      std::vector<int32_t> start{ 0 }, src;
      for (int32_t i = 0; i < m.S; ++i)
      {
        for (int32_t x = 0; x < (int32_t)species.size(); ++x)
          if (species[x] == i)
          {
            src.push_back(element(x));
            c.InRange(src.back());
            c.bad += src.back() >= m.nnz && src.back() < L.slot;  // neither vectors nor constants
          }
        start.push_back((int32_t)src.size());
      }
      c.CheckGather(ph, start, src, std::vector<double>(src.size(), 1.0), 0, L.v0, plain);
    };
    check(c.p.forcing, m.react_ids, [&](int x) { return L.slot + x; });
    check(c.p.step, owner, [&](int x) { return x < m.nnz ? x : L.slot + x - m.nnz; });
  }
  c.CheckGather(c.p.jacobian, m.j_start, m.j_info, m.j_coef, L.w0, 0, [&](int e) { return row_of[e] >= 0; });
  for (const GroupPhase* ph : { &c.p.forcing, &c.p.jacobian, &c.p.lu, &c.p.solve, &c.p.step })
  {
    if (ph == &c.p.step && sweep_stages == 0)
      continue;
    // one unit past the last warp's is fetched
    const bool gather = ph != &c.p.lu && ph != &c.p.solve;
    const size_t units = ph->warp_start.back() + 1, lanes = units * (32 / G);
    c.bad += ph->ctrl.size() != units || ph->item.size() != 4 * lanes || ph->row.size() != (gather ? 8 : 16) * lanes ||
             ph->coef.size() != (gather ? 16 * lanes : 0);
  }
  return c.bad;
}
