// group.cpp -- builds the cell-group kernels' work lists (see group.hpp).
#include "group.hpp"

#include <algorithm>
#include <map>
#include <stdexcept>

namespace micmb
{
  namespace
  {
    struct Sum
    {
      int32_t target, aux, kind;
      std::vector<uint32_t> term;  // operands a | b << 16, or a gathered value's element
      std::vector<double> coef;
    };

    struct Chunk
    {
      std::vector<const Sum*> units;
      int32_t T = 0, kind = 0;
    };

    // the units of one level in chunks of ipw, longest first within each kind
    std::vector<Chunk> Cut(const std::vector<Sum>& units, int32_t ipw)
    {
      std::vector<const Sum*> order;
      for (const Sum& u : units)
        order.push_back(&u);
      std::stable_sort(order.begin(), order.end(), [](const Sum* a, const Sum* b) {
        return a->kind != b->kind ? a->kind < b->kind : a->term.size() > b->term.size();
      });
      std::vector<Chunk> chunks;
      for (const Sum* u : order)
      {
        if (chunks.empty() || (int32_t)chunks.back().units.size() == ipw || chunks.back().kind != u->kind)
        {
          chunks.emplace_back();
          chunks.back().kind = u->kind;
        }
        chunks.back().units.push_back(u);
        chunks.back().T = std::max<int32_t>(chunks.back().T, (int32_t)u->term.size());
      }
      return chunks;
    }

    // One unit: up to four chunks, or terms [t0, t0 + 16) of one.
    struct Step
    {
      std::vector<Chunk> chunks;
      int32_t t0 = 0;
      bool first = true, last = true;
      int32_t sync = kGroupNoSync;
    };

    // The chunks of one level, longest first within each kind, as units of at most
    // `limit` chunks; a long chunk's units stay together.
    std::vector<std::vector<Step>> Pack(const std::vector<Chunk>& chunks, size_t limit = 4)
    {
      std::vector<std::vector<Step>> out;
      for (size_t i = 0; i < chunks.size();)
      {
        const int32_t T = chunks[i].T, kind = chunks[i].kind;
        out.emplace_back();
        if (T > kGroupTerms / 2)
        {
          for (int32_t t0 = 0; t0 < T; t0 += kGroupTerms)
          {
            Step st;
            st.chunks = { chunks[i] };
            st.t0 = t0;
            st.first = t0 == 0;
            st.last = t0 + kGroupTerms >= T;
            out.back().push_back(std::move(st));
          }
          ++i;
          continue;
        }
        Step st;
        const size_t most = std::min<size_t>(limit, T > kGroupTerms / 4 ? 2 : 4);
        for (; i < chunks.size() && st.chunks.size() < most && chunks[i].kind == kind; ++i)
          st.chunks.push_back(chunks[i]);
        out.back().push_back(std::move(st));
      }
      return out;
    }

    // Unit lists of all warps while a phase is being built.
    struct Lists
    {
      std::vector<std::vector<Step>> warp;

      explicit Lists(int32_t W)
          : warp(W)
      {
      }

      void BlockSync()
      {
        for (auto& list : warp)
        {
          if (list.empty() || list.back().sync == kGroupBlockSync)
            list.emplace_back();  // nothing but the barrier
          list.back().sync = kGroupBlockSync;
        }
      }

      void Append(size_t w, std::vector<Step> steps)
      {
        for (Step& st : steps)
          warp[w].push_back(std::move(st));
      }
    };

    // longest first onto the least loaded warp
    void Deal(Lists& lists, std::vector<std::vector<Step>> packed)
    {
      std::stable_sort(packed.begin(), packed.end(), [](const auto& a, const auto& b) { return a.size() > b.size(); });
      std::vector<size_t> load(lists.warp.size(), 0);
      for (auto& steps : packed)
      {
        const size_t w = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
        load[w] += steps.size();
        lists.Append(w, std::move(steps));
      }
    }

    // pivot_is_aux: kGroupPivot writes aux (the LU)
    void Emit(GroupPhase& ph, const Lists& lists, const GroupLayout& L, int32_t G, bool gather,
              bool pivot_is_aux = false)
    {
      const int32_t ipw = 32 / G;
      auto emit = [&](const Step& st) {
        int32_t T = 0;
        for (const Chunk& c : st.chunks)
          T = std::max(T, std::min(kGroupTerms, c.T - st.t0));
        uint32_t shape = 0;
        while (kGroupShapes[shape].chunks < (int32_t)st.chunks.size() || kGroupShapes[shape].terms < T)
          ++shape;
        if (!st.first || !st.last)
          shape = 2;  // stretches of a long sum
        const int32_t per_chunk = kGroupTerms / kGroupShapes[shape].chunks;
        const int32_t kind = st.chunks.empty() ? kGroupPlain : st.chunks[0].kind;
        ph.ctrl.push_back((shape * 3 + (uint32_t)(st.last ? kind : kGroupNone)) | (uint32_t)st.sync << 8 |
                          (st.first ? 1u << 10 : 0u));
        auto unit = [&](int32_t k, int32_t p) -> const Sum* {
          return k < (int32_t)st.chunks.size() && p < (int32_t)st.chunks[k].units.size() ? st.chunks[k].units[p]
                                                                                         : nullptr;
        };
        for (int32_t p = 0; p < ipw; ++p)
          for (int32_t k = 0; k < 4; ++k)
          {
            const Sum* u = unit(k, p);
            const uint32_t idle = (uint32_t)L.trash |
                                  (gather ? 0u : (uint32_t)(pivot_is_aux && kind == kGroupPivot ? L.trash : L.one) << 16);
            ph.item.push_back(u ? (uint32_t)u->target | (uint32_t)u->aux << 16 : idle);
          }
        auto term = [&](int32_t p, int32_t t, double* coef) {
          const Sum* u = unit(t / per_chunk, p);
          const int32_t i = st.t0 + t % per_chunk;
          const bool real = u && i < (int32_t)u->term.size();
          if (coef)
            *coef = real ? u->coef[i] : -0.0;  // -0 times the zero element changes no sum, -0 among them
          const uint32_t zero = (uint32_t)L.zero;
          return real ? u->term[i] : (gather ? zero : zero | zero << 16);
        };
        if (gather)
        {
          for (int32_t r = 0; r < 2; ++r)
            for (int32_t p = 0; p < ipw; ++p)
              for (int32_t t = 8 * r; t < 8 * r + 8; t += 2)
                ph.row.push_back(term(p, t, nullptr) | term(p, t + 1, nullptr) << 16);
          for (int32_t r = 0; r < 8; ++r)
            for (int32_t p = 0; p < ipw; ++p)
              for (int32_t t = 2 * r; t < 2 * r + 2; ++t)
              {
                double c;
                term(p, t, &c);
                ph.coef.push_back(c);
              }
        }
        else
          for (int32_t r = 0; r < 4; ++r)
            for (int32_t p = 0; p < ipw; ++p)
              for (int32_t t = 4 * r; t < 4 * r + 4; ++t)
                ph.row.push_back(term(p, t, nullptr));
      };
      ph.warp_start.push_back(0);
      for (const auto& list : lists.warp)
      {
        for (const Step& st : list)
          emit(st);
        ph.warp_start.push_back((int32_t)ph.ctrl.size());
      }
      emit(Step{});  // fetched ahead, never run
    }

    // One stretch of an item's terms, in the level where it runs.
    struct Piece
    {
      int32_t level, item, t0, t1;
      bool last;  // the item's value is final after it
    };

    // Dependency levels of a serial schedule.  Term t of an item can run one level
    // after its operands are final (and after the item's earlier terms); an item
    // is finished in the first level that has all of its terms.  Terms that are
    // ready earlier run in batches of kBatch as they come (a stretch loads and
    // stores the item's sum, so short stretches cost more than they do), the rest
    // with the last ones.  Exact: the sum is only stored and reloaded in between.
    constexpr int32_t kBatch = 4;
    std::vector<std::vector<Piece>> Levels(const LevelSchedule& s, bool factor)
    {
      const int32_t n = s.n_items();
      std::map<int32_t, int32_t> item_of;
      for (int32_t i = 0; i < n; ++i)
        item_of[s.item_target[i]] = i;
      std::vector<int32_t> final_level(n, 0);
      std::vector<std::vector<Piece>> levels;
      auto put = [&](const Piece& p) {
        if ((int32_t)levels.size() <= p.level)
          levels.resize(p.level + 1);
        levels[p.level].push_back(p);
      };
      for (int32_t i = 0; i < n; ++i)
      {
        const int32_t t0 = s.term_start[i], t1 = s.term_start[i + 1];
        std::vector<int32_t> ready;
        int32_t level = 0;
        for (int32_t t = t0; t < t1; ++t)
        {
          if (factor)
            level = std::max(level, final_level[item_of.at(s.term_a[t])] + 1);
          level = std::max(level, final_level[item_of.at(s.term_b[t])] + 1);
          ready.push_back(level);
        }
        // an L entry's scaling needs its pivot
        if (factor && s.item_aux[i] >= 0)
          level = std::max(level, final_level[item_of.at(s.item_aux[i])] + 1);
        final_level[i] = level;
        int32_t start = 0;
        for (int32_t t = 0; t < t1 - t0; ++t)
          if (ready[t] < level && t + 1 - start >= kBatch && (t + 1 == t1 - t0 || ready[t + 1] > ready[t]))
          {
            put({ ready[t], i, t0 + start, t0 + t + 1, false });
            start = t + 1;
          }
        put({ level, i, t0 + start, t1, true });
      }
      return levels;
    }

    // A level with at most this many units runs on the first warp alone, with warp
    // synchronisation.  A second unit costs about as much as a block barrier:
    // measured with 1 / 2 / 3 / 4 units, ms: TS1 10,000 cells 62.0 / 64.1 / 67.7 /
    // 69.2, 210 species 65,536 cells 453 / 460 / 486 / 513, 600 species 700 cells
    // 100.5 / 99.3 / - / 101.9; with none, 64.2, 477, 104.8.
    constexpr size_t kNarrowUnits = 1;

    // Unit lists of one or more level schedules run one after the other.
    struct LevelLists
    {
      Lists lists;
      std::vector<std::vector<Sum>> kept;  // the chunks point into them
      bool narrow_run = false;

      explicit LevelLists(int32_t W)
          : lists(W)
      {
      }

      template<class MakeSum>
      void Add(const LevelSchedule& s, bool factor, int32_t ipw, int32_t one, MakeSum make)
      {
        for (const std::vector<Piece>& pieces : Levels(s, factor))
        {
          std::vector<Sum> units;
          for (const Piece& piece : pieces)
          {
            Sum u = make(piece);
            // an item without terms that keeps its value has nothing to do
            if (u.term.empty() && u.kind == kGroupPlain && u.aux == one)
              continue;
            units.push_back(std::move(u));
          }
          if (units.empty())
            continue;
          kept.push_back(std::move(units));
          // as few chunks per unit as give every warp one unit: a warp's time goes with
          // its unit's terms (TS1, 10,000 cells: 62.0 -> 59.9 ms)
          const std::vector<Chunk> chunks = Cut(kept.back(), ipw);
          std::vector<std::vector<Step>> packed;
          for (size_t limit = 1; limit <= 4; limit *= 2)
          {
            packed = Pack(chunks, limit);
            if (packed.size() <= lists.warp.size())
              break;
          }
          size_t n_units = 0;
          for (const auto& steps : packed)
            n_units += steps.size();
          const bool narrow = lists.warp.size() == 1 || n_units <= kNarrowUnits;
          if (!lists.warp[0].empty())
          {
            if (narrow && narrow_run)
              lists.warp[0].back().sync = std::max(lists.warp[0].back().sync, kGroupWarpSync);
            else
              lists.BlockSync();
          }
          if (narrow)
            for (auto& steps : packed)
              lists.Append(0, std::move(steps));
          else
            Deal(lists, std::move(packed));
          narrow_run = narrow;
        }
      }
    };

    // sums of coef * (element src0 + src) into elements target0 + i; flag: adds alpha
    GroupPhase GatherPhase(const std::vector<int32_t>& start, const std::vector<int32_t>& src,
                           const std::vector<double>& coef, int32_t src0, int32_t target0, const GroupLayout& L,
                           int32_t G, int32_t W, const std::vector<char>& flag)
    {
      std::vector<Sum> sums;
      for (int32_t i = 0; i + 1 < (int32_t)start.size(); ++i)
      {
        Sum u;
        u.target = target0 + i;
        u.aux = flag.empty() ? 0 : flag[i];
        u.kind = kGroupPlain;
        for (int32_t t = start[i]; t < start[i + 1]; ++t)
        {
          u.term.push_back((uint32_t)(src0 + src[t]));
          u.coef.push_back(coef[t]);
        }
        sums.push_back(std::move(u));
      }
      Lists lists(W);
      Deal(lists, Pack(Cut(sums, 32 / G)));
      GroupPhase ph;
      Emit(ph, lists, L, G, true);
      return ph;
    }
  }  // namespace

  namespace
  {
    // contributions of reaction r in a step: first derivatives per reactant, then
    // per stage the pairs of different reactants
    int32_t Contributions(const CompiledMechanism& m, int32_t r, int32_t stages)
    {
      const int32_t n = m.react_start[r + 1] - m.react_start[r];
      return n + stages * n * (n - 1);
    }
  }  // namespace

  GroupLayout MakeGroupLayout(const CompiledMechanism& m, int32_t sweep_stages)
  {
    GroupLayout L;
    const int32_t n_info = (int32_t)m.info_rxn.size();
    L.zero = m.nnz;
    L.one = m.nnz + 1;
    L.v0 = m.nnz + 2;
    L.trash = L.v0 + m.S;
    L.w0 = L.trash + 1;
    L.inv = L.w0;
    L.rate = L.inv + m.S + 1;
    L.g2 = L.rate;
    L.slot = L.g2 + m.S;
    int32_t vectors = m.S + 1 + std::max(m.R, m.S);
    if (sweep_stages > 0)
    {
      int32_t total = 0;
      for (int32_t r = 0; r < m.R; ++r)
        total += Contributions(m, r, sweep_stages);
      vectors = 2 * m.S + 1 + std::max((int32_t)m.react_ids.size(), total - m.nnz);
    }
    L.elements = L.w0 + std::max(n_info, vectors);
    return L;
  }

  bool GroupApplies(const CompiledMechanism& m)
  {
    return m.constraints.empty() && m.R > 0 && m.R <= 0xFFFF && MakeGroupLayout(m).elements <= 0x7FFF &&
           !m.rate_desc.empty();
  }

  GroupProgram BuildGroupProgram(const CompiledMechanism& m, int32_t G, int32_t W, int32_t sweep_stages)
  {
    if (!GroupApplies(m))
      throw std::runtime_error("group program: the mechanism has none");
    GroupProgram P;
    P.G = G;
    P.W = W;
    const GroupLayout L = P.layout = MakeGroupLayout(m, sweep_stages);
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

    if (sweep_stages == 0)
      P.forcing = GatherPhase(m.f_start, m.f_rxn, m.f_coef, L.rate, L.v0, L, G, W, {});
    else
    {
      // every species' contributions in the order of the one-cell-per-thread sweep:
      // by reaction, first derivatives by reactant, then by stage the pairs (q, o)
      // of different reactants, which go to reactant o
      std::vector<std::vector<int32_t>> first(m.S), all(m.S);
      int32_t at = 0;
      for (int32_t r = 0; r < m.R; ++r)
      {
        const int32_t r0 = m.react_start[r], n = m.react_start[r + 1] - r0;
        P.step_start.push_back(at);
        auto add = [&](int32_t reactant) {
          all[m.react_ids[r0 + reactant]].push_back(at < m.nnz ? at : L.slot + at - m.nnz);
          ++at;
        };
        for (int32_t q = 0; q < n; ++q)
        {
          first[m.react_ids[r0 + q]].push_back(L.slot + r0 + q);
          add(q);
        }
        for (int32_t st = 0; st < sweep_stages; ++st)
          for (int32_t q = 0; q < n; ++q)
            for (int32_t o = 0; o < n; ++o)
              if (o != q)
                add(o);
      }
      auto phase = [&](const std::vector<std::vector<int32_t>>& of) {
        std::vector<int32_t> start{ 0 }, element;
        for (const auto& list : of)
        {
          element.insert(element.end(), list.begin(), list.end());
          start.push_back((int32_t)element.size());
        }
        return GatherPhase(start, element, std::vector<double>(element.size(), 1.0), 0, L.v0, L, G, W, {});
      };
      P.forcing = phase(first);
      P.step = phase(all);
    }
    std::vector<char> diag(m.nnz, 0);
    for (int32_t i = 0; i < m.S; ++i)
      diag[m.diag_pos[i]] = 1;
    P.jacobian = GatherPhase(m.j_start, m.j_info, m.j_coef, L.w0, 0, L, G, W, diag);

    LevelLists lu(W);
    lu.Add(m.lu_serial, true, ipw, L.one, [&](const Piece& p) {
      Sum u;
      u.target = m.lu_serial.item_target[p.item];
      const int32_t row = m.nz_row[u.target], col = m.nz_col[u.target];
      const bool scaled = p.last && row > col;
      // partial sums and U entries share the units of the L entries: scaled by one
      u.kind = p.last && row == col ? kGroupPivot : kGroupPlain;
      u.aux = scaled ? L.inv + col : (u.kind == kGroupPivot ? L.inv + row : L.one);
      for (int32_t t = p.t0; t < p.t1; ++t)
        u.term.push_back((uint32_t)m.lu_serial.term_a[t] | (uint32_t)m.lu_serial.term_b[t] << 16);
      return u;
    });
    Emit(P.lu, lu.lists, L, G, false, true);

    LevelLists solve(W);
    const LevelSchedule* const order[2] = { sweep_stages ? &m.fwd_t_serial : &m.fwd_serial,
                                            sweep_stages ? &m.bwd_t_serial : &m.bwd_serial };
    for (const LevelSchedule* s : order)
      solve.Add(*s, false, ipw, L.one, [&](const Piece& p) {
        Sum u;
        u.target = L.v0 + s->item_target[p.item];
        const bool divided = p.last && s->item_aux[p.item] >= 0;
        u.kind = divided ? kGroupPivot : kGroupPlain;
        u.aux = divided ? s->item_aux[p.item] : L.one;
        for (int32_t t = p.t0; t < p.t1; ++t)
          u.term.push_back((uint32_t)s->term_a[t] | (uint32_t)(L.v0 + s->term_b[t]) << 16);
        return u;
      });
    Emit(P.solve, solve.lists, L, G, false);
    return P;
  }
}  // namespace micmb
