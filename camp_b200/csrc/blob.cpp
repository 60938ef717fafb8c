// Builds the compact shared-memory tables of the solve kernel (blob.hpp).
#include "blob.hpp"

#include <algorithm>
#include <cstring>
#include <map>
#include <numeric>

#include "bdf_consts.hpp"
#include "model.hpp"

namespace campb {

namespace {

constexpr int kLanes = 32;
constexpr uint16_t kNoSlot = 0xFFFF;

struct Writer {
  std::vector<uint8_t> buf;
  template <typename T>
  int put(const std::vector<T>& v) {
    size_t off = (buf.size() + 15) & ~size_t(15);
    buf.resize(off + std::max<size_t>(v.size(), 1) * sizeof(T), 0);
    if (!v.empty()) memcpy(buf.data() + off, v.data(), v.size() * sizeof(T));
    return (int)off;
  }
};

// where a Writer would be after the same puts
struct Sizer {
  size_t at;
  template <typename T>
  int put(const std::vector<T>& v) {
    at = ((at + 15) & ~size_t(15)) + std::max<size_t>(v.size(), 1) * sizeof(T);
    return 0;
  }
};

// Longest-processing-time assignment of weighted items to the 32 lanes.
std::vector<std::vector<int>> lpt(const std::vector<long>& weight) {
  std::vector<int> idx(weight.size());
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return weight[a] > weight[b]; });
  std::vector<long> load(kLanes, 0);
  std::vector<std::vector<int>> lanes(kLanes);
  for (int i : idx) {
    int best = 0;
    for (int l = 1; l < kLanes; ++l)
      if (load[l] < load[best]) best = l;
    lanes[best].push_back(i);
    load[best] += weight[i];
  }
  return lanes;
}

// One item of the f or J gather: index | coef<<16 entries of its sums (a loss
// or an unguarded product carries the coefficient 1), which lie one after the
// other in a vector shared by all items: a vector per list made up half of the
// time that packing takes
struct GatherList {
  const uint32_t* p = nullptr;
  size_t n = 0;
  size_t size() const { return n; }
  bool empty() const { return n == 0; }
  uint32_t operator[](size_t k) const { return p[k]; }
};

struct GatherItem {
  int id = 0, tag = 0xFFFF;
  GatherList lead, loss, prod;
  GatherList neg;  // f: guarded losses, after the others into L1
  // the four chains: losses alternate between L0 and L1, products between P0,
  // which starts with the unguarded ones, and P1
  std::vector<uint32_t> chain(int c) const {
    std::vector<uint32_t> o;
    const GatherList& v = c < 2 ? loss : prod;
    if (c == 2) o.assign(lead.p, lead.p + lead.n);
    for (size_t k = c & 1; k < v.size(); k += 2) o.push_back(v[k]);
    if (c == 1) o.insert(o.end(), neg.p, neg.p + neg.n);
    return o;
  }
  int longest = 0, padded = 0;  // longest chain; entries in multiples of four
  void measure() {
    const int len[4] = {(int)(loss.size() + 1) / 2, (int)(loss.size() / 2 + neg.size()),
                        (int)(lead.size() + (prod.size() + 1) / 2), (int)prod.size() / 2};
    for (int v : len) {
      longest = std::max(longest, v);
      padded += (v + 3) / 4 * 4;
    }
  }
};

struct GatherTables {
  std::vector<uint32_t> a_rec, a_ent, b_hdr, b_id, b_ent, neg;
};

// Splits the items into rounds of eight with a lane per chain and rounds of 32
// with a lane per item (blob.hpp).  A chain round costs its longest chain (11
// instructions an entry, 45 for the reduction), an item round its longest
// lists (9 a word, 30 besides) and their padded words; with the longest chains
// first, the number of chain rounds and the order of the rest with the least
// sum are taken, `bytes_per_inst` table bytes counting as one instruction.
void pack_gather(std::vector<GatherItem>& items, uint32_t zero, int bytes_per_inst,
                 GatherTables* o) {
  auto half = [](size_t n) { return (int)(n + 1) / 2; };
  auto up = [](int n, int m) { return (n + m - 1) / m * m; };
  for (GatherItem& x : items) x.measure();
  const int n = (int)items.size();
  // sorts indices by decreasing value, equal ones in order (by counting: the
  // values are list lengths)
  auto sort_by = [&](std::vector<int>* order, auto value) {
    int most = 0;
    for (int k : *order) most = std::max(most, value(k));
    std::vector<int> at(most + 2, 0), to(n);
    for (int k : *order) at[most - value(k) + 1]++;
    for (int v = 0; v <= most; ++v) at[v + 1] += at[v];
    for (int k : *order) to[at[most - value(k)]++] = k;
    order->swap(to);
  };
  std::vector<int> in_order(n);
  std::iota(in_order.begin(), in_order.end(), 0);
  {
    std::vector<int> by = in_order;
    sort_by(&by, [&](int k) { return items[k].longest; });
    sort_by(&by, [&](int k) { return (int)!items[k].neg.empty(); });
    std::vector<GatherItem> v;
    v.reserve(n);
    for (int k : by) v.push_back(items[k]);
    items.swap(v);
  }
  struct Steps {
    int u = 0, l = 0, p = 0;
  };
  std::vector<Steps> sh(n);
  for (int k = 0; k < n; ++k)
    sh[k] = {(int)items[k].lead.size(), half(items[k].loss.size()), (int)items[k].prod.size()};
  // orders that put similar lists together: by words, products, losses
  std::vector<int> orders[3];
  for (int w = 0; w < 3; ++w) {
    orders[w] = in_order;
    sort_by(&orders[w], [&](int k) { return sh[k].u + sh[k].l + sh[k].p; });
    if (w == 1) sort_by(&orders[w], [&](int k) { return sh[k].p; });
    if (w == 2) sort_by(&orders[w], [&](int k) { return sh[k].l; });
  }
  // the items from `first` on, in order w, as rounds of 32
  auto rounds = [&](int first, int w) {
    std::vector<std::vector<int>> r;
    for (int k : orders[w]) {
      if (k < first) continue;
      if (r.empty() || r.back().size() == kLanes) r.emplace_back();
      r.back().push_back(k);
    }
    return r;
  };
  auto steps = [&](const std::vector<int>& r) {
    Steps s;
    for (int k : r) {
      s.u = std::max(s.u, sh[k].u);
      s.l = std::max(s.l, sh[k].l);
      s.p = std::max(s.p, sh[k].p);
    }
    s.l = s.l > 1 ? up(s.l, 2) : s.l;
    s.p = s.p > 1 ? up(s.p, 2) : s.p;
    return s;
  };
  // the same orders with the lengths beside the items, for the search
  struct Shape {
    int item, u, l, p;
  };
  std::vector<Shape> shapes[3];
  for (int w = 0; w < 3; ++w) {
    shapes[w].reserve(n);
    for (int k : orders[w]) shapes[w].push_back({k, sh[k].u, sh[k].l, sh[k].p});
  }
  int n_neg = 0;
  while (n_neg < n && !items[n_neg].neg.empty()) ++n_neg;
  const int r_min = (n_neg + 7) / 8;
  int best_r = r_min, best_w = 0;
  long best = -1, chains = 0;
  // past the long lists the cost only rises: a few rounds beyond the best end
  // the search
  for (int ra = 0; 8 * ra < n + 8 && (best < 0 || ra < best_r + 6); ++ra) {
    if (ra > 0) {
      long len = 0, bytes = 32 * 8;
      for (int k = 8 * (ra - 1); k < std::min(n, 8 * ra); ++k) {
        len = std::max(len, (long)up(items[k].longest, 4));
        bytes += 4 * items[k].padded;
      }
      chains += 45 + 11 * len + bytes / bytes_per_inst;
    }
    if (ra < r_min) continue;
    for (int w = 0; w < 3; ++w) {
      long cost = chains;
      Steps s;
      int in_round = 0;
      auto close = [&]() {
        s.l = s.l > 1 ? up(s.l, 2) : s.l;
        s.p = s.p > 1 ? up(s.p, 2) : s.p;
        cost += 30 + 9 * (s.u + s.l + s.p) + 128L * (1 + s.u + s.l + s.p) / bytes_per_inst;
        s = Steps{};
        in_round = 0;
      };
      for (const Shape& x : shapes[w]) {
        if (x.item < 8 * ra) continue;
        s.u = std::max(s.u, x.u);
        s.l = std::max(s.l, x.l);
        s.p = std::max(s.p, x.p);
        if (++in_round < kLanes) continue;
        close();
        if (best >= 0 && cost >= best) break;
      }
      if (in_round) close();
      if (best < 0 || cost < best) {
        best = cost;
        best_r = ra;
        best_w = w;
      }
    }
  }
  for (int k = 0; k < 8 * best_r; ++k) {
    for (int c = 0; c < 4; ++c) {
      std::vector<uint32_t> e;
      if (k < n) e = items[k].chain(c);
      e.resize(up((int)e.size(), 4), zero);
      o->a_rec.push_back((uint32_t)o->a_ent.size() | ((uint32_t)e.size() << 16));
      o->a_rec.push_back(
          k < n ? (uint32_t)items[k].id | ((uint32_t)items[k].tag << 16) : 0xFFFFu);
      o->a_ent.insert(o->a_ent.end(), e.begin(), e.end());
    }
  }
  for (const auto& r : rounds(8 * best_r, best_w)) {
    const Steps s = steps(r);
    o->b_hdr.push_back((uint32_t)s.l | ((uint32_t)s.p << 16));
    o->b_hdr.push_back((uint32_t)s.u);
    auto at = [&](const GatherList GatherItem::*list, int k, size_t j) {
      return k < (int)r.size() && j < (items[r[k]].*list).size() ? (items[r[k]].*list)[j] : zero;
    };
    for (int k = 0; k < kLanes; ++k)
      o->b_id.push_back(k < (int)r.size() ? (uint32_t)items[r[k]].id |
                                                ((uint32_t)items[r[k]].tag << 16)
                                          : 0xFFFFu);
    for (int j = 0; j < s.u; ++j)
      for (int k = 0; k < kLanes; ++k) o->b_ent.push_back(at(&GatherItem::lead, k, j));
    for (int j = 0; j < s.l; ++j)
      for (int k = 0; k < kLanes; ++k)
        o->b_ent.push_back((at(&GatherItem::loss, k, 2 * j) & 0xFFFFu) |
                           (at(&GatherItem::loss, k, 2 * j + 1) << 16));
    for (int j = 0; j < s.p; ++j)
      for (int k = 0; k < kLanes; ++k) o->b_ent.push_back(at(&GatherItem::prod, k, j));
  }
  o->a_ent.resize(o->a_ent.size() + 4, zero);  // read ahead, never used
  o->b_ent.resize(o->b_ent.size() + 2 * kLanes, zero);
}

}  // namespace

Layout make_layout(const BlobOff& o, int lt_size, bool with_hist, bool with_tempv) {
  Layout L{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t r = off;
    off = (off + bytes + 15) & ~size_t(15);
    return (int)r;
  };
  const size_t vec = sizeof(double) * o.n;
  L.zn = with_hist ? take(vec * bdf::LMAX) : -1;
  L.ewt = take(vec);
  L.acor = take(vec);
  L.y = take(vec + sizeof(double));  // y[n]: see set_unit
  L.ftemp = take(vec);
  L.tempv = with_tempv ? take(vec) : -1;
  // the f scratch (pseudo-rates, then the computed species, a zero and the
  // guarded terms) and the J scratch (partials, computed species, parameter
  // partials, virtual slots, a zero and the guarded terms), with the
  // sub-models' scratch over or behind them; the solves' vector lies over all
  const int n_scr = std::max(o.scr_end[0], o.scr_end[1]);
  L.rates = L.z = take(std::max(sizeof(double) * n_scr, (size_t)lt_size * (o.n + 1)));
  L.keff = take(sizeof(double) * o.n_keff);
  // the split species' parts lie behind f's terms, over J's where those leave room
  const int f_end = o.scr_end[0], n_fscr = 2 * std::max(1, o.n_fscratch);
  L.fscr = f_end + n_fscr <= n_scr ? L.rates + (int)sizeof(double) * f_end
                                   : take(sizeof(double) * n_fscr);
  // a spare slot: see clear_spare
  L.lu = take((size_t)lt_size * (o.n_lu + 1));
  L.dinv = take((size_t)lt_size * o.n);
  // control block: tau[LMAX + 2], tq[8], l[LMAX + 1], quot[8]
  L.ctl = take(sizeof(double) * (2 * bdf::LMAX + 19));
  L.bytes = (int)off;
  return L;
}

bool build_blob(const Tables& t, const std::vector<double>& atol_dep, int max_smem,
                std::vector<uint8_t>* blob, BlobOff* off, std::string* err) {
  const int n = t.n;
  if (n > 1023) {
    *err = "more than 1023 dependent variables";
    return false;
  }
  if (t.n_rates + t.n_cv > 65535 || t.n_keff > 65535 ||
      t.n_part_all + t.n_cv + t.n_pj + t.n_virt > 65535 || t.n_lu > 65535 ||
      t.n_jac > 65535 ||
      (int)t.fg_rxn.size() > 65535 || (int)t.jg_part.size() > 65535 ||
      (int)t.fa_pos.size() > 65535) {
    *err = "mechanism exceeds the 16-bit table encodings";
    return false;
  }
  // coefficient table
  std::map<uint64_t, int> cid;
  std::vector<double> coef;
  auto coef_id = [&](double v) {
    uint64_t b;
    memcpy(&b, &v, 8);
    auto it = cid.find(b);
    if (it != cid.end()) return it->second;
    int id = (int)coef.size();
    coef.push_back(v);
    cid[b] = id;
    return id;
  };
  // reactions
  std::vector<uint32_t> rx_word(t.n_rxn);
  std::vector<uint16_t> rx_vptr(t.n_rxn + 1);
  for (int r = 0; r < t.n_rxn; ++r) {
    int v0 = t.rx_vptr[r], v1 = t.rx_vptr[r + 1];
    if (v1 - v0 > 3) {
      *err = "reaction " + std::to_string(r) + " has more than 3 variable reactants";
      return false;
    }
    uint32_t w = (uint32_t)(v1 - v0) << 30;
    for (int k = 0; k < v1 - v0; ++k) w |= (uint32_t)t.rx_vdep[v0 + k] << (10 * k);
    for (int k = v1 - v0; k < 2; ++k) w |= (uint32_t)n << (10 * k);
    rx_word[r] = w;
    rx_vptr[r] = (uint16_t)v0;
  }
  rx_vptr[t.n_rxn] = (uint16_t)t.n_part;
  // f gather entries.  Each species list is regrouped, keeping reaction
  // order within a group: reactant occurrences (loss, coefficient -1), then
  // products with a non-negative yield, then products with a negative yield,
  // so that the device's common path adds each group without classifying
  // every term.  grp_end[2 * i + g] is the end of group g of species i.
  std::vector<uint32_t> fg_ent;
  fg_ent.reserve(t.fg_rxn.size());
  std::vector<int> grp_end(2 * n);
  for (int i = 0; i < n; ++i) {
    for (int g = 0; g < 3; ++g) {
      for (int e = t.fg_ptr[i]; e < t.fg_ptr[i + 1]; ++e) {
        const int eg = t.fg_prod[e] == FG_LOSS ? 0 : (t.fg_coef[e] >= 0.0 ? 1 : 2);
        if (eg != g) continue;
        int c = coef_id(t.fg_coef[e]);
        // bit 31: the term is guarded (a product; not a loss or a source)
        fg_ent.push_back((uint32_t)t.fg_rxn[e] | ((uint32_t)c << 16) |
                         ((uint32_t)(t.fg_prod[e] == FG_PRODUCT ? 1 : 0) << 31));
      }
      if (g < 2) grp_end[2 * i + g] = (int)fg_ent.size();
    }
  }
  // balanced f units: species lists longer than the per-lane share are split
  // into slots that a combine pass adds up
  const int total = t.fg_ptr[n];
  const int share = std::max(1, (total + kLanes - 1) / kLanes);
  struct Unit {
    int sp, b, e, slot;
  };
  auto clampi = [](int v, int lo, int hi) { return std::max(lo, std::min(hi, v)); };
  std::vector<Unit> units;
  std::vector<uint16_t> split;
  int n_slots = 0;
  for (int i = 0; i < n; ++i) {
    int b = t.fg_ptr[i], e = t.fg_ptr[i + 1], c = e - b;
    if (c <= share) {
      units.push_back({i, b, e, kNoSlot});
      continue;
    }
    int k = (c + share - 1) / share;
    split.push_back((uint16_t)i);
    split.push_back((uint16_t)n_slots);
    split.push_back((uint16_t)k);
    for (int j = 0; j < k; ++j) {
      int ub = b + (int)((long)c * j / k), ue = b + (int)((long)c * (j + 1) / k);
      units.push_back({i, ub, ue, n_slots++});
    }
  }
  std::vector<long> uw(units.size());
  for (size_t u = 0; u < units.size(); ++u) uw[u] = 2 + (units[u].e - units[u].b);
  auto ulanes = lpt(uw);
  // unit record (8 x uint16, one 16-byte load): species, first entry, end
  // of its loss entries, end of its non-negative-yield products, end, slot
  std::vector<uint16_t> fg_unit, fg_lane(kLanes + 1, 0);
  for (int l = 0; l < kLanes; ++l) {
    fg_lane[l] = (uint16_t)(fg_unit.size() / 8);
    for (int u : ulanes[l]) {
      const Unit& x = units[u];
      fg_unit.push_back((uint16_t)x.sp);
      fg_unit.push_back((uint16_t)x.b);
      fg_unit.push_back((uint16_t)clampi(grp_end[2 * x.sp], x.b, x.e));
      fg_unit.push_back((uint16_t)clampi(grp_end[2 * x.sp + 1], x.b, x.e));
      fg_unit.push_back((uint16_t)x.e);
      fg_unit.push_back((uint16_t)x.slot);
      fg_unit.push_back(0);
      fg_unit.push_back(0);
    }
  }
  fg_lane[kLanes] = (uint16_t)(fg_unit.size() / 8);
  // the same units as chains and rounds (blob.hpp)
  const uint32_t one = (uint32_t)coef_id(1.0) << 16;
  const int f_zero = t.n_rates + t.n_cv;
  GatherTables fgt;
  {
    std::vector<uint32_t> ent;  // the items' lists: never more than reserved
    ent.reserve(fg_ent.size());
    auto list = [&](size_t from) { return GatherList{ent.data() + from, ent.size() - from}; };
    std::vector<GatherItem> items;
    items.reserve(units.size());
    for (const Unit& x : units) {
      const int m1 = clampi(grp_end[2 * x.sp], x.b, x.e);
      const int m2 = clampi(grp_end[2 * x.sp + 1], x.b, x.e);
      GatherItem it;
      it.id = x.sp;
      it.tag = x.slot;
      size_t at = ent.size();
      for (int k = x.b; k < m1; ++k) ent.push_back((fg_ent[k] & 0xFFFFu) | one);
      it.loss = list(at);
      at = ent.size();
      for (int k = m1; k < m2; ++k) ent.push_back(fg_ent[k] & 0x7FFFFFFFu);
      it.prod = list(at);
      at = ent.size();
      for (int k = m2; k < x.e; ++k) {
        fgt.neg.push_back(fg_ent[k] & 0x7FFFFFFFu);
        fgt.neg.push_back((uint32_t)x.sp);
        ent.push_back((uint32_t)(f_zero + (int)fgt.neg.size() / 2) | one);
      }
      it.neg = list(at);
      items.push_back(it);
    }
    pack_gather(items, (uint32_t)f_zero, 16, &fgt);
  }
  // J gather: each slot's partials regrouped: unguarded products (SIMPOL,
  // into the production part), losses (into the loss part) and guarded
  // products (into the production part); jg_umid[e] / jg_mid[e] are the
  // first loss / guarded product entry of slot e
  std::vector<uint32_t> jg_w0;
  std::vector<uint16_t> jg_w1, jg_mid(t.n_jac), jg_umid(t.n_jac);
  jg_w0.reserve(t.jg_part.size());
  jg_w1.reserve(t.jg_part.size());
  bool has_ug = false;
  for (int e = 0; e < t.n_jac; ++e) {
    for (int pass = 0; pass < 3; ++pass) {
      if (pass == 1) jg_umid[e] = (uint16_t)jg_w0.size();
      if (pass == 2) jg_mid[e] = (uint16_t)jg_w0.size();
      for (int g = t.jg_ptr[e]; g < t.jg_ptr[e + 1]; ++g) {
        const int kind = t.jg_ind[g] == -2 ? 0 : (t.jg_ind[g] == -1 ? 1 : 2);
        if (kind != pass) continue;
        has_ug |= kind == 0;
        int c = coef_id(t.jg_coef[g]);
        jg_w0.push_back((uint32_t)t.jg_part[g] | ((uint32_t)c << 16));
        jg_w1.push_back((uint16_t)(t.jg_ind[g] >= 0 ? t.jg_ind[g] + 1 : 0));
      }
    }
  }
  if (coef.size() > 32767) {
    *err = "too many distinct yields for the table encoding";
    return false;
  }
  std::vector<uint16_t> jg_ptr(t.n_jac + 1), jg_lupos(t.n_jac), jg_row(t.n_jac);
  for (int e = 0; e <= t.n_jac; ++e) jg_ptr[e] = (uint16_t)t.jg_ptr[e];
  // SIMPOL instance tables (dependent elements only: the constant ones are
  // folded into the per-cell constants)
  std::vector<uint16_t> si_rec, si_elem;
  std::vector<double> si_ef;
  for (int k = 0; k < t.n_simpol; ++k) {
    const SimpolInst& si = t.simpol[k];
    const int first = (int)si_elem.size();
    int nd = 0;
    // HL instances have no element partials (see SimpolInst)
    const size_t ne = si.type == RXN_SIMPOL_PHASE_TRANSFER ? si.elem.size() : 0;
    for (size_t j = 0; j < ne; ++j) {
      const int d = std::lower_bound(t.dep_state.begin(), t.dep_state.end(), si.elem[j]) -
                    t.dep_state.begin();
      if (d >= n || t.dep_state[d] != si.elem[j]) continue;  // not a dependent variable
      si_elem.push_back((uint16_t)d);
      si_ef.push_back(si.inv_rho[j]);
      si_ef.push_back(si.inv_mw[j]);
      si_ef.push_back(si.in_phase[j] ? 1.0 : 0.0);
      ++nd;
    }
    const auto dep_of = [&](int st) {
      return (int)(std::lower_bound(t.dep_state.begin(), t.dep_state.end(), st) -
                   t.dep_state.begin());
    };
    // rec[5]: HL's computed water + 1 (0: a constant water, folded per cell)
    const uint16_t rec[8] = {(uint16_t)dep_of(si.gas), (uint16_t)dep_of(si.aero),
                             (uint16_t)nd,                (uint16_t)first,
                             (uint16_t)t.si_part0[k],     (uint16_t)(si.water_cv + 1), 0, 0};
    si_rec.insert(si_rec.end(), rec, rec + 8);
  }
  for (int e = 0; e < t.n_jac; ++e) {
    jg_lupos[e] = (uint16_t)t.jg_lupos[e];
    jg_row[e] = (uint16_t)t.jg_row[e];
  }
  // per 32 LU positions: those that a solver-J slot fills, the diagonals, and
  // the slots before them (M = I - gamma*J in one pass)
  if (t.n_jac >= 32767) {
    *err = "too many Jacobian elements for the table encoding";
    return false;
  }
  std::vector<int> jslot(t.n_jac);  // J slot of each CSC entry: by LU position
  {
    std::vector<int> at(t.n_lu, 0);
    for (int e = 0; e < t.n_jac; ++e) at[t.jg_lupos[e]] = e + 1;
    for (int q = 0, k = 0; q < t.n_lu; ++q)
      if (at[q]) jslot[at[q] - 1] = k++;
  }
  std::vector<uint32_t> lu_src(3 * ((t.n_lu + 127) / 128 * 4), 0);
  for (int e = 0; e < t.n_jac; ++e) lu_src[3 * (t.jg_lupos[e] / 32)] |= 1u << (t.jg_lupos[e] % 32);
  for (int i = 0; i < n; ++i) lu_src[3 * (t.lu_diag[i] / 32) + 1] |= 1u << (t.lu_diag[i] % 32);
  for (size_t c = 1; c < lu_src.size() / 3; ++c)
    lu_src[3 * c + 2] = lu_src[3 * c - 1] + (uint32_t)__builtin_popcount(lu_src[3 * c - 3]);
  std::vector<int> jcsc(t.n_jac);
  for (int e = 0; e < t.n_jac; ++e) jcsc[jslot[e]] = e;
  std::vector<long> jw(t.n_jac);
  for (int e = 0; e < t.n_jac; ++e) jw[e] = 2 + (t.jg_ptr[e + 1] - t.jg_ptr[e]);
  auto jlanes = lpt(jw);
  std::vector<uint16_t> jg_lane(kLanes + 1, 0), jg_slots;
  for (int l = 0; l < kLanes; ++l) {
    jg_lane[l] = (uint16_t)jg_slots.size();
    // longest slots first on every lane: the lanes of a warp step through
    // their k-th slots together, so slots of similar length line up and the
    // warp runs sum_k max_lane(len) ~ the per-lane total instead of far more
    std::vector<int> s = jlanes[l];
    std::stable_sort(s.begin(), s.end(), [&](int a, int b) {
      return t.jg_ptr[a + 1] - t.jg_ptr[a] > t.jg_ptr[b + 1] - t.jg_ptr[b];
    });
    for (int e : s) jg_slots.push_back((uint16_t)e);
  }
  jg_lane[kLanes] = (uint16_t)jg_slots.size();
  // the same slots as chains and rounds (blob.hpp); a Jacobian is evaluated a
  // few times less often than f, so its table bytes weigh more
  const int j_zero = t.n_part_all + t.n_cv + t.n_pj + t.n_virt;
  GatherTables jgt;
  {
    std::vector<uint32_t> ent;
    ent.reserve(jg_w0.size());
    auto list = [&](size_t from) { return GatherList{ent.data() + from, ent.size() - from}; };
    std::vector<GatherItem> items;
    items.reserve(t.n_jac);
    for (int e = 0; e < t.n_jac; ++e) {
      GatherItem it;
      it.id = jslot[e];
      size_t at = ent.size();
      for (int g = t.jg_ptr[e]; g < jg_umid[e]; ++g) ent.push_back((jg_w0[g] & 0xFFFFu) | one);
      it.lead = list(at);
      at = ent.size();
      for (int g = jg_umid[e]; g < jg_mid[e]; ++g) ent.push_back((jg_w0[g] & 0xFFFFu) | one);
      it.loss = list(at);
      at = ent.size();
      for (int g = jg_mid[e]; g < t.jg_ptr[e + 1]; ++g) {
        if (coef[jg_w0[g] >> 16] >= 0.0) {
          ent.push_back(jg_w0[g]);
          continue;
        }
        jgt.neg.push_back(jg_w0[g]);
        jgt.neg.push_back((uint32_t)(jg_w1[g] - 1) | ((uint32_t)t.jg_row[e] << 16));
        ent.push_back((uint32_t)(j_zero + (int)jgt.neg.size() / 2) | one);
      }
      it.prod = list(at);
      items.push_back(it);
    }
    pack_gather(items, (uint32_t)j_zero, 8, &jgt);
  }
  // LU
  auto u16 = [](const std::vector<int>& v) {
    std::vector<uint16_t> o(v.size());
    for (size_t i = 0; i < v.size(); ++i) o[i] = (uint16_t)v[i];
    return o;
  };
  // Grouped phases as rounds of 32 targets, longest first within a level, so
  // that a round's targets have similar lengths and its padding stays small.
  // Targets of four pairs or more take two lanes, one for each of their
  // alternating sums, 16 to a round.  Per round its pair count per lane (two
  // lanes: | lanes in use<<9 | 1<<15), 32 records (first pair,
  // target, pivot or finish mark) and its further pairs, with two lanes only
  // those of the lanes in use: a hub species' target has hundreds, and 32 words
  // for each pair of lanes filled 75 KB for 400 species around one.
  struct Rounds {
    std::vector<uint32_t> pair0, target, recip, ext;
    std::vector<int> cnt, level;
  };
  auto rounds_of = [&](const Tables::Grouped& g, Rounds* o, uint32_t no_pair, int spare,
                       bool with_empty) {
    for (int l = 0; l < g.n_levels; ++l) {
      std::vector<int> us;
      for (int u = g.lane_ptr[33 * l]; u < g.lane_ptr[33 * l + kLanes]; ++u)
        if (with_empty || g.unit_count[u] > 0) us.push_back(u);
      std::stable_sort(us.begin(), us.end(), [&](int a, int b) {
        return g.unit_count[a] > g.unit_count[b];
      });
      for (size_t k0 = 0; k0 < us.size();) {
        const int most = std::max(1, g.unit_count[us[k0]]);
        const bool two = most >= 4;
        // a round of very long targets leaves those of less than half their
        // length to the next, which would be padding otherwise
        size_t m = std::min(us.size() - k0, (size_t)(two ? kLanes / 2 : kLanes));
        if (most >= 64)
          while (2 * g.unit_count[us[k0 + m - 1]] < most) --m;
        int row = two ? 2 : kLanes;  // lanes with a table word of their own
        while (two && row < 2 * (int)m) row *= 2;
        auto pair = [&](size_t lane, int j) {
          const size_t k = two ? lane / 2 : lane;
          const int at = two ? 2 * j + (int)(lane & 1) : j;
          if (k >= m || at >= g.unit_count[us[k0 + k]]) return no_pair;
          const int p = g.unit_begin[us[k0 + k]] + at;
          return (uint32_t)g.pair_a[p] | ((uint32_t)g.pair_b[p] << 16);
        };
        const int cnt = two ? (most + 1) / 2 : most;
        o->cnt.push_back(two ? 0x8000 | (row << 9) | cnt : cnt);
        o->level.push_back(l);
        const size_t at0 = o->pair0.size(), ext0 = o->ext.size();
        o->pair0.resize(at0 + kLanes);
        o->target.resize(at0 + kLanes, (uint32_t)spare);
        o->recip.resize(at0 + kLanes, 0u);
        for (size_t lane = 0; lane < kLanes; ++lane) o->pair0[at0 + lane] = pair(lane, 0);
        for (size_t k = 0; k < m; ++k) {
          const size_t lane = at0 + (two ? 2 * k : k);
          o->target[lane] = (uint32_t)g.unit_target[us[k0 + k]];
          o->recip[lane] = (uint32_t)g.unit_recip[us[k0 + k]];
        }
        o->ext.resize(ext0 + (size_t)row * (cnt - 1));
        for (int j = 1; j < cnt; ++j)
          for (int lane = 0; lane < row; ++lane)
            o->ext[ext0 + (size_t)row * (j - 1) + lane] = pair(lane, j);
        k0 += m;
      }
    }
  };
  for (const Tables::Grouped* g : {&t.fb, &t.fwd, &t.bwd})
    if (g->unit_target.size() > 65535 || g->pair_a.size() > 65535) {
      *err = "LU schedule exceeds the 16-bit table encodings";
      return false;
    }
  Rounds fbr, svr;
  for (Rounds* r : {&fbr, &svr})
    for (auto* v : {&r->pair0, &r->target, &r->recip, &r->ext}) v->reserve(128 * kLanes);
  const uint32_t lu_none = (uint32_t)t.n_lu | ((uint32_t)t.n_lu << 16);
  const uint32_t sv_none = (uint32_t)t.n_lu | ((uint32_t)n << 16);
  // the factorization takes reciprocal pivots with the scaling, so its units
  // without pairs drop out (the schedule's phase g holds level g - 1's updates)
  rounds_of(t.fb, &fbr, lu_none, t.n_lu, false);
  rounds_of(t.fwd, &svr, sv_none, n, true);
  if (svr.cnt.empty()) {
    // L has no entries: an empty round, as the solve starts with a forward one
    svr.cnt.push_back(1);
    svr.pair0.resize(kLanes, sv_none);
    svr.target.resize(kLanes, (uint32_t)n);
    svr.recip.resize(kLanes, 0u);
  }
  const int n_fwd = (int)svr.cnt.size();
  rounds_of(t.bwd, &svr, sv_none, n, true);
  std::vector<uint32_t> fb_rec, sv_rec, fs_rec;
  std::vector<uint16_t> fl_hdr(2 * t.n_plev, 0);
  for (size_t r = 0; r < fbr.cnt.size(); ++r)
    fl_hdr[2 * (fbr.level[r] - 1) + 1]++;
  for (size_t k = 0; k < fbr.pair0.size(); ++k) {
    fb_rec.push_back(fbr.pair0[k]);
    fb_rec.push_back(fbr.target[k] | ((uint32_t)fbr.cnt[k / kLanes] << 16));
  }
  for (int k = 0; k < 2 * kLanes; ++k) {
    fb_rec.push_back(lu_none);
    fb_rec.push_back((uint32_t)t.n_lu | (1u << 16));
  }
  for (int l = 0; l < t.n_plev; ++l) {
    std::vector<std::pair<int, int>> e;  // L position (n_lu: none), pivot
    std::vector<char> has(n, 0);
    for (int i = t.fa_ptr[l]; i < t.fa_ptr[l + 1]; ++i) {
      e.push_back({t.fa_pos[i], t.fa_piv[i]});
      has[t.fa_piv[i]] = 1;
    }
    // the pivots of a level are those whose reciprocal its phase takes
    for (int u = t.fb.lane_ptr[33 * l]; u < t.fb.lane_ptr[33 * l + kLanes]; ++u)
      if (t.fb.unit_recip[u] && !has[t.fb.unit_recip[u] - 1])
        e.push_back({t.n_lu, t.fb.unit_recip[u] - 1});
    std::vector<char> stored(n, 0);
    for (const auto& x : e) {
      fs_rec.push_back((uint32_t)x.first | ((uint32_t)t.lu_diag[x.second] << 16));
      fs_rec.push_back((uint32_t)x.second | (stored[x.second] ? 0u : 0x8000u));
      stored[x.second] = 1;
    }
    fl_hdr[2 * l] = (uint16_t)(fs_rec.size() / 2);
  }
  svr.ext.resize(svr.ext.size() + kLanes, sv_none);  // read ahead, never used
  fbr.ext.resize(fbr.ext.size() + kLanes, lu_none);
  for (size_t k = 0; k < svr.pair0.size(); ++k) {
    sv_rec.push_back(svr.pair0[k]);
    sv_rec.push_back(svr.target[k] | (svr.recip[k] ? 0x8000u : 0u) |
                     ((uint32_t)svr.cnt[k / kLanes] << 16));
  }
  for (int k = 0; k < 2 * kLanes; ++k) {
    sv_rec.push_back(sv_none);
    sv_rec.push_back((uint32_t)n | (1u << 16));
  }

  Writer w;
  // the offsets themselves lead the blob, so device code can rebuild its
  // table pointers from shared memory alone
  w.buf.resize(kBlobHeader, 0);
  static_assert(sizeof(BlobOff) <= kBlobHeader, "BlobOff must fit the blob header");
  BlobOff o{};
  o.n = n;
  o.n_rxn = t.n_rxn;
  o.n_part = t.n_part;
  o.n_jac = t.n_jac;
  o.n_lu = t.n_lu;
  o.n_coef = (int)coef.size();
  o.n_fsplit = (int)split.size() / 3;
  o.n_fscratch = n_slots;
  o.rx_word = w.put(rx_word);
  o.coef = w.put(coef);
  o.fg_split = w.put(split);
  o.rx_vptr = w.put(rx_vptr);
  o.has_ug = has_ug ? 1 : 0;
  o.n_simpol = t.n_simpol;
  o.n_keff = t.n_keff;
  o.n_rates = t.n_rates;
  o.n_part_all = t.n_part_all;
  o.si_rec = w.put(si_rec);
  o.si_elem = w.put(si_elem);
  o.si_ef = w.put(si_ef);
  // aqueous equilibrium instance records
  std::vector<uint16_t> aq_rec, aq_sp, aq_cp;
  std::vector<double> aq_sm, aq_cpm;
  for (int k = 0; k < t.n_aq; ++k) {
    const AqInst& q = t.aq[k];
    const int first = (int)aq_sp.size();
    int S = 0, R = 0;
    const auto dep_of = [&](int st) {
      const int d = (int)(std::lower_bound(t.dep_state.begin(), t.dep_state.end(), st) -
                          t.dep_state.begin());
      return d < n && t.dep_state[d] == st ? d : -1;
    };
    for (int pass = 0; pass < 2; ++pass) {
      const std::vector<int>& list = pass == 0 ? q.react : q.prod;
      for (size_t i = 0; i < list.size(); ++i) {
        const int d = dep_of(list[i]);
        if (d < 0) continue;
        aq_sp.push_back((uint16_t)d);
        aq_sm.push_back(q.m2m[(pass == 0 ? 0 : q.react.size()) + i]);
        ++S;
        R += pass == 0;
      }
    }
    // rec[6]: computed water + 1 (0: constant, folded per cell) | reactant
    // count << 8 | product count << 12 (constant species included: the
    // powers of the water); rec[7]: computed activity coefficient + 1
    const uint16_t wrec = (uint16_t)((q.water_cv + 1) | (q.react.size() << 8) |
                                     (q.prod.size() << 12));
    const int cp0 = (int)aq_cp.size();
    for (size_t j = 0; j < q.cp_cv.size(); ++j) {
      aq_cp.push_back((uint16_t)(q.cp_cv[j] | (q.cp_r[j] ? 0x8000 : 0)));
      aq_cpm.push_back(q.cp_m[j]);
    }
    const uint16_t rec[12] = {(uint16_t)S, (uint16_t)R, (uint16_t)first,
                              (uint16_t)t.aq_rate0[k], (uint16_t)t.aq_part0[k],
                              (uint16_t)t.aq_keff0[k], wrec, (uint16_t)(q.act_cv + 1),
                              (uint16_t)cp0, (uint16_t)q.cp_cv.size(), 0, 0};
    aq_rec.insert(aq_rec.end(), rec, rec + 12);
  }
  o.n_aq = t.n_aq;
  o.aq_rec = w.put(aq_rec);
  o.aq_sp = w.put(aq_sp);
  o.aq_sm = w.put(aq_sm);
  {
    std::vector<double> sim(aq_sm.size());
    for (size_t k = 0; k < sim.size(); ++k) sim[k] = 1.0 / aq_sm[k];
    o.aq_sim = w.put(sim);
  }
  o.aq_cp = w.put(aq_cp);
  o.aq_cpm = w.put(aq_cpm);
  // sub-model programs, virtual slots and the chain
  std::vector<uint32_t> sm_item, sm_scr, sm_pel;
  std::vector<uint16_t> sm_pq;
  int sm_slots = 0;
  {
    std::vector<uint32_t> rec;
    std::vector<int32_t> ints;
    std::vector<double> flts;
    for (const SubProgram& g : t.cv) {
      rec.push_back((uint32_t)ints.size());
      rec.push_back((uint32_t)flts.size());
      ints.insert(ints.end(), g.ints.begin(), g.ints.end());
      flts.insert(flts.end(), g.flts.begin(), g.flts.end());
    }
    o.n_cv = t.n_cv;
    o.n_pj = t.n_pj;
    o.sm_keff = t.sm_keff;
    o.sm_rec = w.put(rec);
    std::vector<int> cv_state;
    for (const SubProgram& g : t.cv) cv_state.push_back(g.state);
    o.sm_state = w.put(u16(cv_state));
    // parallel parts of the programs (blob.hpp)
    std::vector<uint32_t> item[5];  // by kind
    uint32_t slots = 0;
    // slots of the pairs' moles, by their ions and factors
    std::map<std::vector<double>, uint32_t> moles;
    for (size_t c = 0; c < t.cv.size(); ++c) {
      const std::vector<int>& I = t.cv[c].ints;
      const uint32_t i0 = rec[2 * c], f0 = rec[2 * c + 1], cc = (uint32_t)c << 8;
      auto add = [&](uint32_t kind, uint32_t i, uint32_t f, int n) {
        for (uint32_t v : {kind | cc, i0 + i, f0 + f, slots}) item[kind].push_back(v);
        slots += n;
      };
      const uint32_t s0 = slots;
      if (I[0] == 1) {
        int ii = 3, fi = 0;
        for (int x = 0; x < I[2]; ++x) {
          const int type = I[ii++];
          if (type == 1) {
            add(1, ii, fi, 7);
            fi += 3 + I[ii + 2];
            ii += 6;
          } else if (type == 2) {
            fi += 2 + I[ii];
            ii += 2 + 2 * I[ii];
          }
        }
        for (uint32_t v : {s0, 0u, 0u, 0u}) sm_scr.push_back(v);
        continue;
      }
      const int npair = I[2], x = I[3], ninter = I[4];
      const int* pr = I.data() + 6;
      const int* it = pr + 5 * npair;
      int fi = 2 * npair;
      for (int k = 0; k < ninter; ++k) {
        add(3, 6 + 5 * npair + 2 * k, fi, 3);
        fi += 2 + it[2 * k + 1];
      }
      std::vector<double> key;
      for (int j = 0; j < npair; ++j)
        for (double v : {(double)pr[5 * j], (double)pr[5 * j + 1], t.cv[c].flts[2 * j],
                         t.cv[c].flts[2 * j + 1]})
          key.push_back(v);
      const auto at = moles.insert({key, slots});
      if (at.second)
        for (int j = 0; j < npair; ++j) add(4, 6 + 5 * j, 2 * j, 2);
      for (uint32_t v : {s0, (uint32_t)ninter, at.first->second, slots}) sm_scr.push_back(v);
      slots += 2;
      // every partial of this coefficient, with the other pairs whose cation or
      // anion it is against
      std::vector<int> ids{I[5]};
      for (int j = 0; j < npair; ++j)
        for (int a : {pr[5 * j + 3], pr[5 * j + 4]})
          if (std::find(ids.begin(), ids.end(), a) == ids.end()) ids.push_back(a);
      for (int id : ids) {
        const size_t q0 = sm_pq.size();
        for (int q = 0; q < npair; ++q) {
          if (q == x) continue;
          if (id == pr[5 * q + 3]) sm_pq.push_back((uint16_t)q);
          if (id == pr[5 * q + 4]) sm_pq.push_back((uint16_t)(q | 0x8000));
        }
        sm_pel.push_back((uint32_t)id | ((uint32_t)c << 16));
        sm_pel.push_back((uint32_t)q0 | ((uint32_t)(sm_pq.size() - q0) << 16));
      }
    }
    for (int kind : {1, 3, 4}) sm_item.insert(sm_item.end(), item[kind].begin(), item[kind].end());
    sm_slots = (int)slots;
    o.sm_int = w.put(ints);
    o.sm_flt = w.put(flts);
    o.n_virt = t.n_virt;
    o.jv_ptr = w.put(u16(t.jv_ptr));
    o.jv_part = w.put(u16(t.jv_part));
    o.n_chain = (int)t.ch_tgt.size();
    std::vector<int> tgt;
    for (int e : t.ch_tgt) tgt.push_back(jslot[e]);
    o.ch_tgt = w.put(u16(tgt));
    o.ch_ptr = w.put(u16(t.ch_ptr));
    std::vector<uint32_t> ent(t.ch_v.size());
    for (size_t i = 0; i < ent.size(); ++i)
      ent[i] = (uint32_t)t.ch_v[i] | ((uint32_t)t.ch_p[i] << 16);
    o.ch_ent = w.put(ent);
    if (t.n_cv > 254 || t.n_pj > 65535 || t.n_virt > 65535 || t.jv_part.size() > 65535 ||
        t.ch_v.size() > 65535) {
      *err = "sub-model tables exceed the 16-bit encodings";
      return false;
    }
  }
  o.n_plev = t.n_plev;
  o.lu_iperm = w.put(u16(t.lu_iperm));
  o.lu_src = w.put(lu_src);
  o.fl_hdr = w.put(fl_hdr);
  o.fs_rec = w.put(fs_rec);
  o.fb_rec = w.put(fb_rec);
  o.fb_ext = w.put(fbr.ext);
  o.n_fwd = n_fwd;
  o.n_bwd = (int)svr.cnt.size() - n_fwd;
  o.sv_rec = w.put(sv_rec);
  o.sv_ext = w.put(svr.ext);
  o.dep_state = w.put(u16(t.dep_state));
  o.atol = w.put(atol_dep);
  auto put_known = [&](auto& v, BlobOff* q) {
    for (int k = 0; k < 2; ++k) {
      GatherTables& x = k == 0 ? fgt : jgt;
      BlobOff::Gather& g = q->g[k];
      g.n_a = (int)x.a_rec.size() / (2 * kLanes);
      g.n_b = (int)x.b_hdr.size() / 2;
      g.n_neg = (int)x.neg.size() / 2;
      g.a_rec = v.put(x.a_rec);
      g.a_ent = v.put(x.a_ent);
      g.b_hdr = v.put(x.b_hdr);
      g.b_id = k == 0 ? v.put(x.b_id)
                      : v.put(std::vector<uint16_t>(x.b_id.begin(), x.b_id.end()));
      g.b_ent = v.put(x.b_ent);
      g.neg = v.put(x.neg);
    }
  };
  auto put_any = [&](auto& v, BlobOff* q) {
    q->fg_ent = v.put(fg_ent);
    q->fg_unit = v.put(fg_unit);
    q->fg_lane = v.put(fg_lane);
    q->j_csc = v.put(u16(jcsc));
    q->jg_slot = v.put(u16(jslot));
    q->jg_w0 = v.put(jg_w0);
    q->jg_w1 = v.put(jg_w1);
    q->jg_ptr = v.put(jg_ptr);
    q->jg_mid = v.put(jg_mid);
    q->jg_row = v.put(jg_row);
    q->jg_lane = v.put(jg_lane);
    q->jg_slots = v.put(jg_slots);
    q->jg_umid = v.put(jg_umid);
  };
  auto put_parts = [&](auto& v, BlobOff* q) {
    q->n_smi = (int)sm_item.size() / 4;
    q->n_smp = (int)sm_pel.size() / 2;
    q->n_sms = sm_slots;
    q->sm_item = v.put(sm_item);
    q->sm_scr = v.put(sm_scr);
    q->sm_pel = v.put(sm_pel);
    q->sm_pq = v.put(sm_pq);
  };
  for (int k = 0; k < 2; ++k) o.g[k].zero = k == 0 ? f_zero : j_zero;
  // The sub-models' scratch lies over the pseudo-rates (f) and partials (J),
  // which are computed after them, or, where it does not fit there, behind the
  // rest.
  auto place_scratch = [&](BlobOff* q) {
    const bool over = q->n_sms <= std::min(t.n_rates, t.n_part_all);
    for (int k = 0; k < 2; ++k) {
      const int end = q->g[k].zero + 1 + q->g[k].n_neg;
      q->scr0[k] = over ? 0 : end;
      q->scr_end[k] = over ? end : end + q->n_sms;
    }
  };
  // cells per block (FP64, all in shared memory) with the given tables staged
  const int most_cells =
      t.n_simpol > 0 || t.n_aq > 0 || t.n_cv > 0 ? kMaxCellsAero : kMaxCellsPerBlock;
  auto cells = [&](bool any, bool parts) {
    BlobOff q = o;
    Sizer v{w.buf.size()};
    if (parts) put_parts(v, &q);
    any ? put_any(v, &q) : put_known(v, &q);
    place_scratch(&q);
    const int room = max_smem - (int)((v.at + 127) & ~size_t(127));
    return std::min(std::max(0, room / make_layout(q, 8, true, false).bytes), most_cells);
  };
  // The parts of the sub-models' programs over the lanes, unless their tables and
  // scratch cost a quarter of the cells (4 000 cells of one phase in
  // several modes, FP64, cells and ms of the parts / a lane per program: 4 ion
  // pairs x 16 modes 3 / 4, 7.6 / 6.0; 9 x 4 5 / 8, 3.9 / 3.5; 9 x 8 1 / 2,
  // 26.8 / 12.8; 20 x 1 6 / 14, 2.52 / 2.59; 9 x 2 12 / 20, 2.00 / 2.20; the
  // shipped mod37 configuration 5 / 5, 214 / 241).
  if (sm_pq.size() <= 65535 && !t.cv.empty()) {
    const int parts = cells(false, true);
    if (parts == most_cells || 4 * parts > 3 * cells(false, false)) put_parts(w, &o);
  }
  // A guarded term takes eight bytes of every cell's slab beside its table
  // entry, so a mechanism with many of them holds fewer cells, or none at all,
  // with the known-sign gathers staged; it keeps the gathers for any signs
  // where those hold a fifth more cells (1 500 cells of random mechanisms,
  // FP64, cells and ms of known / any signs: 20 species x 300 reactions, all
  // yields negative, 3 / 12 cells 111 / 37 ms; 15 x 600 1 / 7, 372 / 72;
  // 40 x 100, half negative, 3 / 4, 131 / 110; 15 x 300 6 / 12, 51 / 47; 20 x
  // 100 10 / 12, 42 / 27; with as many cells known signs are 0.99 to 1.8 times as
  // fast, cb05 1.11, mod37 gas 1.18).
  const bool fits = fgt.a_ent.size() <= 65535 && jgt.a_ent.size() <= 65535 &&
                    f_zero + fgt.neg.size() / 2 <= 65535 && j_zero + jgt.neg.size() / 2 <= 65535;
  const bool guards = !fgt.neg.empty() || !jgt.neg.empty();
  if (!fits) {
    o.any_sign = 1;
  } else if (guards) {
    const int known = cells(false, false);
    const int any = known < most_cells ? cells(true, false) : 0;
    o.any_sign = any > 0 && 6 * known <= 5 * any;
  }
  o.any_sign ? put_any(w, &o) : put_known(w, &o);
  place_scratch(&o);
  // the level-scheduled mode stages only the bytes up to here into shared
  // memory, the one-lane LU mode its LU tables too; the gathers for any signs,
  // where they are the exception, come last and stay in global memory
  w.buf.resize((w.buf.size() + 15) & ~size_t(15), 0);
  o.stage_bytes = (int)w.buf.size();
  {
    std::vector<uint32_t> up(t.upd_ptr.begin(), t.upd_ptr.end()), ud(t.upd_src.size());
    for (size_t p = 0; p < ud.size(); ++p)
      ud[p] = (uint32_t)t.upd_src[p] | ((uint32_t)t.upd_dst[p] << 16);
    o.jg_lupos = w.put(jg_lupos);
    o.lu_diag = w.put(u16(t.lu_diag));
    o.lu_rowptr = w.put(u16(t.lu_rowptr));
    o.lu_col = w.put(u16(t.lu_col));
    o.upd_ptr = w.put(up);
    o.upd = w.put(ud);
  }
  w.buf.resize((w.buf.size() + 15) & ~size_t(15), 0);
  o.seq_bytes = (int)w.buf.size();
  if (!o.any_sign) put_any(w, &o);
  w.buf.resize((w.buf.size() + 15) & ~size_t(15), 0);
  o.bytes = (int)w.buf.size();
  memcpy(w.buf.data(), &o, sizeof(o));
  blob->swap(w.buf);
  *off = o;
  return true;
}

}  // namespace campb

namespace campb {

bool build_lane_blob(const Tables& t, const std::vector<double>& atol_dep,
                     std::vector<uint8_t>* blob, LaneOff* off, std::string* err) {
  if (t.n_simpol > 0 || t.n_aq > 0 || t.n_cv > 0) {
    *err = "the lane-per-cell kernel does not evaluate SIMPOL, HL or aqueous equilibrium "
           "reactions or sub-models";
    return false;
  }
  const int n = t.n;
  if (n > 1023 || t.n_rxn > 65535 || t.n_lu > 65535) {
    *err = "mechanism exceeds the lane-kernel table encodings";
    return false;
  }
  std::map<uint64_t, int> cid;
  std::vector<double> coef;
  auto coef_id = [&](double v) {
    uint64_t b;
    memcpy(&b, &v, 8);
    auto it = cid.find(b);
    if (it != cid.end()) return it->second;
    int id = (int)coef.size();
    coef.push_back(v);
    cid[b] = id;
    return id;
  };
  // LU positions by (pivot row, pivot column)
  std::vector<std::vector<int>> pos(n, std::vector<int>(n, -1));
  for (int i = 0; i < n; ++i)
    for (int q = t.lu_rowptr[i]; q < t.lu_rowptr[i + 1]; ++q) pos[i][t.lu_col[q]] = q;
  // participants in term order: the variable reactant occurrences
  // (rx_vdep), then the variable products and sources (recovered from the f
  // gather lists, which hold every product of a term with its yield)
  struct Gain {
    int d;
    double c;
    bool guarded;
  };
  std::vector<std::vector<Gain>> prods(t.n_rxn);
  for (int d = 0; d < n; ++d)
    for (int e = t.fg_ptr[d]; e < t.fg_ptr[d + 1]; ++e)
      if (t.fg_prod[e] != FG_LOSS)
        prods[t.fg_rxn[e]].push_back({d, t.fg_coef[e], t.fg_prod[e] == FG_PRODUCT});
  std::vector<uint32_t> rx_word(t.n_rxn), rx_part;
  std::vector<uint16_t> rx_pptr(t.n_rxn + 1), rx_jptr(t.n_rxn + 1), jpos;
  for (int r = 0; r < t.n_rxn; ++r) {
    int v0 = t.rx_vptr[r], v1 = t.rx_vptr[r + 1];
    if (v1 - v0 > 3) {
      *err = "reaction " + std::to_string(r) + " has more than 3 variable reactants";
      return false;
    }
    uint32_t w = (uint32_t)(v1 - v0) << 30;
    for (int k = 0; k < v1 - v0; ++k) w |= (uint32_t)t.rx_vdep[v0 + k] << (10 * k);
    rx_word[r] = w;
    rx_pptr[r] = (uint16_t)rx_part.size();
    std::vector<int> sp;
    for (int k = v0; k < v1; ++k) {
      rx_part.push_back((uint32_t)t.rx_vdep[k] | ((uint32_t)coef_id(-1.0) << 10));
      sp.push_back(t.rx_vdep[k]);
    }
    for (const Gain& pr : prods[r]) {
      rx_part.push_back((uint32_t)pr.d | ((uint32_t)coef_id(pr.c) << 10) |
                        ((pr.guarded ? 1u : 0u) << 31));
      sp.push_back(pr.d);
    }
    rx_jptr[r] = (uint16_t)jpos.size();
    for (int k = v0; k < v1; ++k) {
      int col = t.lu_iperm[t.rx_vdep[k]];
      for (int s : sp) {
        int q = pos[t.lu_iperm[s]][col];
        if (q < 0) {
          *err = "internal: Jacobian entry outside the LU pattern";
          return false;
        }
        jpos.push_back((uint16_t)q);
      }
    }
  }
  rx_pptr[t.n_rxn] = (uint16_t)rx_part.size();
  rx_jptr[t.n_rxn] = (uint16_t)jpos.size();
  if (rx_part.size() > 65535 || jpos.size() > 65535 || coef.size() > 32767) {
    *err = "mechanism exceeds the lane-kernel table encodings";
    return false;
  }
  auto u16 = [](const std::vector<int>& v) {
    std::vector<uint16_t> o(v.size());
    for (size_t i = 0; i < v.size(); ++i) o[i] = (uint16_t)v[i];
    return o;
  };
  std::vector<uint32_t> up(t.upd_ptr.begin(), t.upd_ptr.end()), ud(t.upd_src.size());
  for (size_t p = 0; p < ud.size(); ++p)
    ud[p] = (uint32_t)t.upd_src[p] | ((uint32_t)t.upd_dst[p] << 16);
  Writer w;
  w.buf.resize(256, 0);
  static_assert(sizeof(LaneOff) <= 256, "LaneOff must fit the blob header");
  LaneOff o{};
  o.n = n;
  o.n_rxn = t.n_rxn;
  o.n_lu = t.n_lu;
  o.n_coef = (int)coef.size();
  o.n_part = (int)rx_part.size();
  o.n_jpos = (int)jpos.size();
  o.n_upd = (int)ud.size();
  o.rx_word = w.put(rx_word);
  o.rx_pptr = w.put(rx_pptr);
  o.rx_part = w.put(rx_part);
  o.rx_jptr = w.put(rx_jptr);
  o.jpos = w.put(jpos);
  o.coef = w.put(coef);
  o.lu_perm = w.put(u16(t.lu_perm));
  o.lu_rowptr = w.put(u16(t.lu_rowptr));
  o.lu_col = w.put(u16(t.lu_col));
  o.lu_diag = w.put(u16(t.lu_diag));
  o.upd_ptr = w.put(up);
  o.upd = w.put(ud);
  o.dep_state = w.put(u16(t.dep_state));
  o.atol = w.put(atol_dep);
  w.buf.resize((w.buf.size() + 15) & ~size_t(15), 0);
  o.bytes = (int)w.buf.size();
  memcpy(w.buf.data(), &o, sizeof(o));
  blob->swap(w.buf);
  *off = o;
  return true;
}

}  // namespace campb

namespace campb {

bool build_block_blob(const Tables& t, const std::vector<double>& atol_dep,
                      std::vector<uint8_t>* blob, BlockOff* off, std::string* err) {
  if (t.n_simpol > 0 || t.n_aq > 0 || t.n_cv > 0) {
    *err = "the CTA-per-cell kernel does not evaluate SIMPOL, HL or aqueous equilibrium "
           "reactions or sub-models";
    return false;
  }
  const int n = t.n;
  if (n < 1 || n > 1023 || t.n_rxn > 65535 || t.n_lu > 65535 || t.n_part > 65535 ||
      t.n_jac > 32767) {
    *err = "mechanism exceeds the CTA-kernel table encodings";
    return false;
  }
  std::map<uint64_t, int> cid;
  std::vector<double> coef;
  auto coef_id = [&](double v) {
    uint64_t b;
    memcpy(&b, &v, 8);
    auto it = cid.find(b);
    if (it != cid.end()) return it->second;
    int id = (int)coef.size();
    coef.push_back(v);
    cid[b] = id;
    return id;
  };
  // reactions
  std::vector<uint32_t> rx_word(t.n_rxn), rx_vptr(t.n_rxn + 1);
  for (int r = 0; r < t.n_rxn; ++r) {
    const int v0 = t.rx_vptr[r], v1 = t.rx_vptr[r + 1];
    if (v1 - v0 > 3) {
      *err = "reaction " + std::to_string(r) + " has more than 3 variable reactants";
      return false;
    }
    uint32_t w = (uint32_t)(v1 - v0) << 30;
    for (int k = 0; k < v1 - v0; ++k) w |= (uint32_t)t.rx_vdep[v0 + k] << (10 * k);
    rx_word[r] = w;
    rx_vptr[r] = (uint32_t)v0;
  }
  rx_vptr[t.n_rxn] = (uint32_t)t.rx_vptr[t.n_rxn];
  // f gather in the species lists' own order
  std::vector<uint32_t> fg_ptr(n + 1), fg_ent(t.fg_rxn.size());
  for (int i = 0; i <= n; ++i) fg_ptr[i] = (uint32_t)t.fg_ptr[i];
  for (size_t e = 0; e < fg_ent.size(); ++e)
    fg_ent[e] = (uint32_t)t.fg_rxn[e] | ((uint32_t)coef_id(t.fg_coef[e]) << 16) |
                ((uint32_t)(t.fg_prod[e] == FG_PRODUCT ? 1 : 0) << 31);
  // J gather: losses, then guarded products, per slot
  std::vector<uint32_t> jg_ptr(t.n_jac + 1), jg_mid(t.n_jac), jg_w0;
  std::vector<uint16_t> jg_w1, jg_row(t.n_jac);
  for (int e = 0; e < t.n_jac; ++e) {
    jg_ptr[e] = (uint32_t)jg_w0.size();
    for (int pass = 0; pass < 2; ++pass) {
      if (pass == 1) jg_mid[e] = (uint32_t)jg_w0.size();
      for (int g = t.jg_ptr[e]; g < t.jg_ptr[e + 1]; ++g) {
        if (t.jg_ind[g] == -2) {
          *err = "the CTA-per-cell kernel has no unguarded Jacobian products";
          return false;
        }
        if ((t.jg_ind[g] == -1) != (pass == 0)) continue;
        jg_w0.push_back((uint32_t)t.jg_part[g] | ((uint32_t)coef_id(t.jg_coef[g]) << 16));
        jg_w1.push_back((uint16_t)(t.jg_ind[g] >= 0 ? t.jg_ind[g] + 1 : 0));
      }
    }
    jg_row[e] = (uint16_t)t.jg_row[e];
  }
  jg_ptr[t.n_jac] = (uint32_t)jg_w0.size();
  if (coef.size() > 32767) {
    *err = "too many distinct yields for the table encoding";
    return false;
  }
  // LU: sorted rows, the diagonal in every row
  for (int i = 0; i < n; ++i) {
    for (int q = t.lu_rowptr[i] + 1; q < t.lu_rowptr[i + 1]; ++q)
      if (t.lu_col[q] <= t.lu_col[q - 1]) {
        *err = "internal: LU row columns not sorted";
        return false;
      }
    if (t.lu_col[t.lu_diag[i]] != i) {
      *err = "internal: LU diagonal position";
      return false;
    }
  }
  std::vector<uint16_t> lu_src(t.n_lu, 0);
  for (int e = 0; e < t.n_jac; ++e) lu_src[t.jg_lupos[e]] = (uint16_t)(e + 1);
  for (int i = 0; i < n; ++i) lu_src[t.lu_diag[i]] |= 0x8000u;
  // position lookup and the trailing dense block: the smallest r0 with every
  // (i, j), i, j >= r0, present
  std::vector<int> pos((size_t)n * n, -1);
  for (int i = 0; i < n; ++i)
    for (int q = t.lu_rowptr[i]; q < t.lu_rowptr[i + 1]; ++q)
      pos[(size_t)i * n + t.lu_col[q]] = q;
  int r0 = n - 1;
  for (int c = n - 2; c >= 0; --c) {
    bool full = true;
    for (int i = c; i < n && full; ++i)
      full = pos[(size_t)i * n + c] >= 0 && pos[(size_t)c * n + i] >= 0;
    if (!full) break;
    r0 = c;
  }
  if (n - r0 > kBlockMaxDense) {
    *err = "the LU's trailing dense block (" + std::to_string(n - r0) +
           " rows) exceeds the CTA kernel's " + std::to_string(kBlockMaxDense);
    return false;
  }
  std::vector<uint16_t> dpos(n - r0), ub(r0);
  for (int i = r0; i < n; ++i) dpos[i - r0] = (uint16_t)pos[(size_t)i * n + r0];
  for (int i = 0; i < r0; ++i) {
    int q = t.lu_rowptr[i + 1];
    while (q > t.lu_diag[i] + 1 && t.lu_col[q - 1] >= r0) --q;
    ub[i] = (uint16_t)q;
  }
  // head pivots: L entries of each column (row order), and the tabulated
  // update targets: head rows against every U entry of row k, dense rows
  // against the U entries in head columns
  std::vector<uint32_t> lk_ptr(r0 + 1, 0), lk_mid(std::max(r0, 1), 0), tg_ptr(r0 + 1, 0);
  std::vector<uint16_t> lk_pos, lk_row;
  std::vector<uint64_t> hrec;
  for (int k = 0; k < r0; ++k) {
    lk_ptr[k] = (uint32_t)lk_pos.size();
    tg_ptr[k] = (uint32_t)hrec.size();
    std::vector<int> rows;
    for (int i = k + 1; i < n; ++i) {
      const int q = pos[(size_t)i * n + k];
      if (q < 0) continue;
      rows.push_back(i);
      lk_pos.push_back((uint16_t)q);
      lk_row.push_back((uint16_t)i);
    }
    lk_mid[k] = (uint32_t)lk_ptr[k];
    for (int i : rows)
      if (i < r0) ++lk_mid[k];
    for (int pass = 0; pass < 2; ++pass)
      for (int i : rows) {
        if ((i >= r0) != (pass == 1)) continue;
        const int p1 = pass == 0 ? t.lu_rowptr[k + 1] : ub[k];
        const int lpos = pos[(size_t)i * n + k];
        for (int p = t.lu_diag[k] + 1; p < p1; ++p) {
          const int d = pos[(size_t)i * n + t.lu_col[p]];
          if (d < 0) {
            *err = "internal: LU fill pattern not closed";
            return false;
          }
          hrec.push_back((uint64_t)d | ((uint64_t)lpos << 16) | ((uint64_t)p << 32));
        }
      }
  }
  lk_ptr[r0] = (uint32_t)lk_pos.size();
  tg_ptr[r0] = (uint32_t)hrec.size();
  std::vector<uint32_t> lk(lk_pos.size());
  for (size_t e = 0; e < lk.size(); ++e) lk[e] = (uint32_t)lk_pos[e] | ((uint32_t)lk_row[e] << 16);
  // head row levels: forward over the L entries, backward over the U entries
  // with columns < r0 (the dense block's values reach head rows in one pass)
  std::vector<int> flev(r0, 0), blev(r0, 0);
  int n_hf = 0, n_hb = 0;
  for (int i = 0; i < r0; ++i) {
    int l = 0;
    for (int q = t.lu_rowptr[i]; q < t.lu_diag[i]; ++q) l = std::max(l, flev[t.lu_col[q]] + 1);
    flev[i] = l;
    n_hf = std::max(n_hf, l + 1);
  }
  for (int i = r0 - 1; i >= 0; --i) {
    int l = 0;
    for (int q = t.lu_diag[i] + 1; q < ub[i]; ++q) l = std::max(l, blev[t.lu_col[q]] + 1);
    blev[i] = l;
    n_hb = std::max(n_hb, l + 1);
  }
  auto levels = [&](const std::vector<int>& lev, int nl, std::vector<uint16_t>* ptr,
                    std::vector<uint16_t>* rows) {
    ptr->assign(nl + 1, 0);
    rows->clear();
    for (int l = 0; l < nl; ++l) {
      (*ptr)[l] = (uint16_t)rows->size();
      for (int i = 0; i < (int)lev.size(); ++i)
        if (lev[i] == l) rows->push_back((uint16_t)i);
    }
    (*ptr)[nl] = (uint16_t)rows->size();
  };
  std::vector<uint16_t> hf_ptr, hf_rows, hb_ptr, hb_rows;
  levels(flev, n_hf, &hf_ptr, &hf_rows);
  levels(blev, n_hb, &hb_ptr, &hb_rows);
  // the solve's staged section
  std::vector<uint16_t> stage;
  auto sec = [&](const std::vector<uint16_t>& v) {
    const int off = (int)stage.size();
    stage.insert(stage.end(), v.begin(), v.end());
    return off;
  };
  std::vector<uint16_t> ndoff(n + 1, 0), ndcol, dbase(n - r0);
  for (int i = 0; i < n; ++i) {
    ndoff[i] = (uint16_t)ndcol.size();
    const int q1 = i < r0 ? t.lu_rowptr[i + 1] : dpos[i - r0];
    for (int q = t.lu_rowptr[i]; q < q1; ++q) ndcol.push_back((uint16_t)t.lu_col[q]);
  }
  ndoff[n] = (uint16_t)ndcol.size();
  for (int i = r0; i < n; ++i) dbase[i - r0] = (uint16_t)(dpos[i - r0] - r0);
  if (ndcol.size() > 65535) {
    *err = "mechanism exceeds the CTA-kernel table encodings";
    return false;
  }
  auto u16 = [](const std::vector<int>& v) {
    std::vector<uint16_t> o(v.size());
    for (size_t i = 0; i < v.size(); ++i) o[i] = (uint16_t)v[i];
    return o;
  };
  Writer w;
  w.buf.resize(256, 0);
  static_assert(sizeof(BlockOff) <= 256, "BlockOff must fit the blob header");
  BlockOff o{};
  o.n = n;
  o.n_rxn = t.n_rxn;
  o.n_part = t.n_part;
  o.n_jac = t.n_jac;
  o.n_lu = t.n_lu;
  o.n_coef = (int)coef.size();
  o.r0 = r0;
  o.n_hf = n_hf;
  o.n_hb = n_hb;
  o.rx_word = w.put(rx_word);
  o.rx_vptr = w.put(rx_vptr);
  o.coef = w.put(coef);
  o.fg_ptr = w.put(fg_ptr);
  o.fg_ent = w.put(fg_ent);
  o.jg_ptr = w.put(jg_ptr);
  o.jg_mid = w.put(jg_mid);
  o.jg_w0 = w.put(jg_w0);
  o.jg_w1 = w.put(jg_w1);
  o.jg_row = w.put(jg_row);
  o.lu_src = w.put(lu_src);
  o.lu_perm = w.put(u16(t.lu_perm));
  o.lu_rowptr = w.put(u16(t.lu_rowptr));
  o.lu_col = w.put(u16(t.lu_col));
  o.lu_diag = w.put(u16(t.lu_diag));
  o.dpos = w.put(dpos);
  o.ub = w.put(ub);
  o.lk_ptr = w.put(lk_ptr);
  o.lk = w.put(lk);
  o.lk_mid = w.put(lk_mid);
  o.tg_ptr = w.put(tg_ptr);
  o.hrec = w.put(hrec);
  o.hf_ptr = w.put(hf_ptr);
  o.hf_rows = w.put(hf_rows);
  o.hb_ptr = w.put(hb_ptr);
  o.hb_rows = w.put(hb_rows);
  o.dep_state = w.put(u16(t.dep_state));
  o.atol = w.put(atol_dep);
  o.sg_rowptr = sec(u16(t.lu_rowptr));
  o.sg_diag = sec(u16(t.lu_diag));
  o.sg_ub = sec(ub);
  o.sg_perm = sec(u16(t.lu_perm));
  o.sg_hf_ptr = sec(hf_ptr);
  o.sg_hf_rows = sec(hf_rows);
  o.sg_hb_ptr = sec(hb_ptr);
  o.sg_hb_rows = sec(hb_rows);
  o.sg_ndoff = sec(ndoff);
  o.sg_ndcol = sec(ndcol);
  o.sg_dbase = sec(dbase);
  if (lk_ptr[r0] > 65535 || tg_ptr[r0] > 65535) {
    *err = "mechanism exceeds the CTA-kernel table encodings";
    return false;
  }
  std::vector<uint16_t> hlk(lk_ptr.begin(), lk_ptr.end()), hmid(r0), htg(tg_ptr.begin(), tg_ptr.end());
  for (int k = 0; k < r0; ++k) hmid[k] = (uint16_t)lk_mid[k];
  o.sg_hlk = sec(hlk);
  o.sg_hmid = sec(hmid);
  o.sg_htg = sec(htg);
  stage.resize((stage.size() + 7) & ~size_t(7), 0);  // whole 16-byte units
  o.sg_len = (int)stage.size();
  o.stage = w.put(stage);
  w.buf.resize((w.buf.size() + 15) & ~size_t(15), 0);
  o.bytes = (int)w.buf.size();
  memcpy(w.buf.data(), &o, sizeof(o));
  blob->swap(w.buf);
  *off = o;
  return true;
}

}  // namespace campb
