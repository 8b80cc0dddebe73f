// group.cpp -- builds the cell-group kernels' work lists (see group.hpp).
#include "group.hpp"

#include <algorithm>
#include <stdexcept>

namespace micmb
{
  namespace
  {
    struct Unit
    {
      int32_t target, aux, kind;
      std::vector<uint32_t> term;  // elements: pairs of operands, or gathered values
      std::vector<double> coef;
      int32_t n_terms(bool gather) const
      {
        return (int32_t)term.size() / (gather ? 1 : 2);
      }
    };

    struct Chunk
    {
      std::vector<const Unit*> units;
      int32_t T = 0, kind = 0;
    };

    // the units of one level in chunks of ipw, longest first within each kind
    std::vector<Chunk> Cut(const std::vector<Unit>& units, int32_t ipw, bool gather)
    {
      std::vector<const Unit*> order;
      for (const Unit& u : units)
        order.push_back(&u);
      std::stable_sort(order.begin(), order.end(), [](const Unit* a, const Unit* b) {
        return a->kind != b->kind ? a->kind < b->kind : a->term.size() > b->term.size();
      });
      std::vector<Chunk> chunks;
      for (const Unit* u : order)
      {
        if (chunks.empty() || (int32_t)chunks.back().units.size() == ipw || chunks.back().kind != u->kind)
        {
          chunks.emplace_back();
          chunks.back().kind = u->kind;
        }
        chunks.back().units.push_back(u);
        chunks.back().T = std::max<int32_t>(chunks.back().T, u->n_terms(gather));
      }
      return chunks;
    }

    // Chunk lists of all warps while a phase is being built.
    struct Lists
    {
      struct Entry
      {
        Chunk chunk;
        int32_t sync;
      };
      std::vector<std::vector<Entry>> warp;

      explicit Lists(int32_t W)
          : warp(W)
      {
      }

      void BlockSync()
      {
        for (auto& list : warp)
        {
          if (list.empty() || list.back().sync == kGroupBlockSync)
            list.push_back({ Chunk{}, kGroupNoSync });
          list.back().sync = kGroupBlockSync;
        }
      }
    };

    // Longest chunk first onto the least loaded warp.  The cost of a chunk is
    // about its fixed part (descriptor, item, first load, store) plus its terms.
    void Deal(Lists& lists, std::vector<Chunk> chunks)
    {
      std::stable_sort(chunks.begin(), chunks.end(), [](const Chunk& a, const Chunk& b) { return a.T > b.T; });
      std::vector<int64_t> load(lists.warp.size(), 0);
      for (Chunk& c : chunks)
      {
        const size_t w = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
        load[w] += 4 + c.T;
        lists.warp[w].push_back({ std::move(c), kGroupNoSync });
      }
    }

    void Emit(GroupPhase& ph, const Lists& lists, const GroupLayout& L, int32_t G, bool gather)
    {
      const int32_t ipw = 32 / G;
      auto offset = [&](int32_t e) { return (uint32_t)e * (uint32_t)G * 8u; };
      std::vector<std::vector<uint32_t>> items;  // per record, [lane][words]
      const int32_t item_words = gather ? 1 : 2;
      auto record = [&](const Chunk& c, int32_t t0, uint32_t ctrl) {
        ph.ctrl.push_back(ctrl);
        items.emplace_back();
        auto unit = [&](int32_t p) { return p < (int32_t)c.units.size() ? c.units[p] : nullptr; };
        for (int32_t p = 0; p < ipw; ++p)
        {
          const Unit* u = unit(p);
          if (gather)
            items.back().push_back(u ? (uint32_t)u->target | ((uint32_t)u->aux << 16) : kGroupNoItem);
          else
          {
            items.back().push_back(offset(u ? u->target : L.trash));
            items.back().push_back(offset(u ? u->aux : (c.kind == kGroupRecip ? L.trash : L.one)));
          }
        }
        auto term = [&](int32_t p, int32_t t, int32_t k) {
          const Unit* u = unit(p);
          return offset(u && t < u->n_terms(gather) ? (int32_t)u->term[gather ? t : 2 * t + k] : L.zero);
        };
        if (gather)
        {
          for (int32_t p = 0; p < ipw; ++p)
            for (int32_t q = 0; q < 4; ++q)
              ph.row.push_back(term(p, t0 + q, 0));
          for (int32_t h = 0; h < 2; ++h)
            for (int32_t p = 0; p < ipw; ++p)
              for (int32_t q = 2 * h; q < 2 * h + 2; ++q)
              {
                const Unit* u = unit(p);
                ph.coef.push_back(u && t0 + q < u->n_terms(true) ? u->coef[t0 + q] : 0.0);
              }
        }
        else
          for (int32_t h = 0; h < 2; ++h)
            for (int32_t p = 0; p < ipw; ++p)
              for (int32_t q = 2 * h; q < 2 * h + 2; ++q)
                for (int32_t k = 0; k < 2; ++k)
                  ph.row.push_back(term(p, t0 + q, k));
      };
      ph.warp_start.push_back(0);
      for (const auto& list : lists.warp)
      {
        for (const auto& e : list)
        {
          const Chunk& c = e.chunk;
          const int32_t n = std::max<int32_t>(1, (c.T + 3) / 4);
          for (int32_t j = 0; j < n; ++j)
          {
            uint32_t ctrl = (uint32_t)std::min<int32_t>(4, c.T - 4 * j);
            if (!c.units.empty())
              ctrl |= (j == 0 ? 1u << 3 : 0u) | (j == n - 1 ? 1u << 4 : 0u) | ((uint32_t)c.kind << 5);
            if (j == n - 1)
              ctrl |= (uint32_t)e.sync << 7;
            record(c, 4 * j, ctrl);
          }
        }
        while (ph.ctrl.size() % kGroupUnit)
          record(Chunk{}, 0, 0);
        ph.warp_start.push_back((int32_t)(ph.ctrl.size() / kGroupUnit));
      }
      // fetched ahead, never run
      for (int32_t j = 0; j < kGroupUnit; ++j)
        record(Chunk{}, 0, 0);
      for (size_t u = 0; u < ph.ctrl.size() / kGroupUnit; ++u)
        for (int32_t p = 0; p < ipw; ++p)
          for (int32_t j = 0; j < kGroupUnit; ++j)
            for (int32_t k = 0; k < item_words; ++k)
              ph.item.push_back(items[u * kGroupUnit + j][(size_t)p * item_words + k]);
    }

    // A level with at most this many chunks runs on the first warp alone, with
    // warp synchronisation: a block barrier costs more than a second chunk.
    constexpr int32_t kNarrowChunks = 2;

    // Chunk lists of one or more level schedules run one after the other.
    struct LevelLists
    {
      Lists lists;
      std::vector<std::vector<Unit>> kept;  // the chunks point into them
      bool narrow_run = false;

      explicit LevelLists(int32_t W)
          : lists(W)
      {
      }

      template<class MakeUnit>
      void Add(const LevelSchedule& s, int32_t ipw, MakeUnit make)
      {
        for (int32_t l = 0; l < s.n_levels(); ++l)
        {
          std::vector<Unit> units;
          for (int32_t i = s.level_start[l]; i < s.level_start[l + 1]; ++i)
          {
            Unit u = make(i);
            // an item without terms that keeps its value has nothing to do
            if (u.term.empty() && u.kind == kGroupStore)
              continue;
            units.push_back(std::move(u));
          }
          kept.push_back(std::move(units));
          std::vector<Chunk> chunks = Cut(kept.back(), ipw, false);
          if (chunks.empty())
            continue;
          const bool narrow = lists.warp.size() == 1 || (int32_t)chunks.size() <= kNarrowChunks;
          if (!lists.warp[0].empty())
          {
            if (narrow && narrow_run)
              lists.warp[0].back().sync = std::max(lists.warp[0].back().sync, kGroupWarpSync);
            else
              lists.BlockSync();
          }
          if (narrow)
            for (Chunk& c : chunks)
              lists.warp[0].push_back({ std::move(c), kGroupNoSync });
          else
            Deal(lists, std::move(chunks));
          narrow_run = narrow;
        }
      }
    };

    GroupPhase GatherPhase(const std::vector<int32_t>& start, const std::vector<int32_t>& src,
                           const std::vector<double>& coef, int32_t src0, const GroupLayout& L, int32_t G, int32_t W,
                           const std::vector<char>& flag)
    {
      std::vector<Unit> units;
      for (int32_t i = 0; i + 1 < (int32_t)start.size(); ++i)
      {
        Unit u;
        u.target = i;
        u.aux = flag.empty() ? 0 : flag[i];
        u.kind = kGroupScale;
        for (int32_t t = start[i]; t < start[i + 1]; ++t)
        {
          u.term.push_back((uint32_t)(src0 + src[t]));
          u.coef.push_back(coef[t]);
        }
        units.push_back(std::move(u));
      }
      Lists lists(W);
      Deal(lists, Cut(units, 32 / G, true));
      GroupPhase ph;
      Emit(ph, lists, L, G, true);
      return ph;
    }
  }  // namespace

  GroupLayout MakeGroupLayout(const CompiledMechanism& m)
  {
    GroupLayout L;
    const int32_t n_info = (int32_t)m.info_rxn.size();
    L.zero = m.nnz;
    L.one = m.nnz + 1;
    L.v0 = m.nnz + 2;
    L.trash = L.v0 + m.S;
    L.w0 = L.trash + 1;
    L.inv = L.w0;
    L.rate = L.w0 + m.S;
    L.elements = L.w0 + std::max(n_info, m.S + std::max(m.R, m.S));
    return L;
  }

  bool GroupApplies(const CompiledMechanism& m)
  {
    return m.constraints.empty() && m.R > 0 && m.R <= 0xFFFF && MakeGroupLayout(m).elements <= 0x7FFF &&
           !m.rate_desc.empty();
  }

  GroupProgram BuildGroupProgram(const CompiledMechanism& m, int32_t G, int32_t W)
  {
    if (!GroupApplies(m))
      throw std::runtime_error("group program: the mechanism has none");
    GroupProgram P;
    P.G = G;
    P.W = W;
    const GroupLayout L = P.layout = MakeGroupLayout(m);
    const int32_t ipw = 32 / G;

    // products: rate_desc / drate_desc pad with column S + 1
    auto vec = [&](int32_t col) { return (uint32_t)(col < m.S ? L.v0 + col : L.one); };
    for (int32_t r = 0; r < m.R; ++r)
    {
      const int32_t* d = &m.rate_desc[4 * (size_t)r];
      P.rate.push_back(vec(d[0]) | (vec(d[1]) << 16));
      P.rate.push_back(vec(d[2]));
    }
    for (size_t i = 0; i < m.info_rxn.size(); ++i)
    {
      const int32_t* d = &m.drate_desc[4 * i];
      P.drate.push_back((uint32_t)d[0] | (vec(d[1]) << 16));
      P.drate.push_back(vec(d[2]) | (vec(d[3]) << 16));
    }

    P.forcing = GatherPhase(m.f_start, m.f_rxn, m.f_coef, L.rate, L, G, W, {});
    std::vector<char> diag(m.nnz, 0);
    for (int32_t i = 0; i < m.S; ++i)
      diag[m.diag_pos[i]] = 1;
    P.jacobian = GatherPhase(m.j_start, m.j_info, m.j_coef, L.w0, L, G, W, diag);

    LevelLists lu(W);
    lu.Add(m.lu, ipw, [&](int32_t i) {
      Unit u;
      u.target = m.lu.item_target[i];
      const bool partial = m.lu.item_aux[i] == -2;
      const int32_t row = m.nz_row[u.target], col = m.nz_col[u.target];
      // scaling by one keeps partial sums and U entries in the chunks of the L entries
      u.kind = partial || row < col ? (m.lu.term_start[i] == m.lu.term_start[i + 1] ? kGroupStore : kGroupScale)
                                    : (row == col ? kGroupRecip : kGroupScale);
      u.aux = partial || row < col ? L.one : L.inv + (row == col ? row : col);
      for (int32_t t = m.lu.term_start[i]; t < m.lu.term_start[i + 1]; ++t)
        u.term.insert(u.term.end(), { (uint32_t)m.lu.term_a[t], (uint32_t)m.lu.term_b[t] });
      return u;
    });
    Emit(P.lu, lu.lists, L, G, false);

    LevelLists solve(W);
    for (const LevelSchedule* s : { &m.fwd, &m.bwd })
      solve.Add(*s, ipw, [&](int32_t i) {
        Unit u;
        u.target = L.v0 + s->item_target[i];
        u.kind = s->item_aux[i] >= 0 ? kGroupDiv : kGroupStore;
        u.aux = s->item_aux[i] >= 0 ? s->item_aux[i] : L.one;
        for (int32_t t = s->term_start[i]; t < s->term_start[i + 1]; ++t)
          u.term.insert(u.term.end(), { (uint32_t)s->term_a[t], (uint32_t)(L.v0 + s->term_b[t]) });
        return u;
      });
    Emit(P.solve, solve.lists, L, G, false);
    return P;
  }
}  // namespace micmb
