// Compact mechanism tables for the solve kernel.  The host packs them into one
// 16-byte aligned blob; every block copies the blob into the front of its
// shared memory with one bulk (TMA) copy, and all warps of the block read it
// from there.  Offsets are in bytes from the start of the blob, whose first
// kBlobHeader bytes hold the BlobOff itself.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace campb {

struct BlobOff {
  int bytes;        // whole blob
  int stage_bytes;  // prefix the level-scheduled mode stages
  int seq_bytes;    // prefix the one-lane LU mode stages (its LU tables too)
  // counts
  int n, n_rxn, n_part, n_jac, n_lu, n_coef, n_fsplit, n_fscratch, n_plev;
  int any_sign;  // the gathers for any signs are staged and used throughout
  // reactions: variable reactants packed (nv<<30 | d2<<20 | d1<<10 | d0; d0
  // and d1 default to n, where y holds 1), partial base
  int rx_word, rx_vptr;
  // coefficient table (double)
  int coef;
  // f gather for any signs: entries (rxn | coef<<16 | prod<<31), units
  // (species, begin, end of losses, end of non-negative-yield products, end,
  // slot) as 8 x uint16, lane pointers (33 x uint16); read from the blob in
  // global memory (self) where they are the exception.  Split species (species,
  // first slot, count) as 3 x uint16
  int fg_ent, fg_unit, fg_lane, fg_split;
  // f (g[0]) and J (g[1]) gathers where no rate (partial), concentration or
  // step is negative (empty with any_sign); every item is a unit of the f gather
  // or a slot of the solver Jacobian, its sums L0, L1, P0 and P1 four chains of
  // entries (uint32 index | coef<<16).  Long items come first, as n_a rounds of eight items
  // with one lane per chain: per lane a_rec (uint32 first entry | entries<<16,
  // id | tag<<16) into a_ent (lists of a multiple of four).  The rest follows
  // as n_b rounds of 32 items, one lane each: per round b_hdr (uint32 x 2:
  // words of loss pairs | products<<16, leading unguarded products), per lane
  // b_id (f: uint32 id | tag<<16, J: uint16 id), and in b_ent, 32 lanes at a
  // time, the unguarded products, the loss pairs (uint32 index | index<<16) and
  // the products, both one or a multiple of two.  Padding uses an index that
  // the gather keeps at zero; four entries and two rows are read ahead of the
  // ends.
  // Terms with a negative yield are evaluated before the gather, n_neg records
  // (uint32 index | coef<<16; f: species, J: guard species | row<<16), into
  // the slots after that zero.
  // f: id species, tag split slot (0xFFFF none); J: id slot; idle lanes have
  // id 0xFFFF.
  struct Gather {
    int n_a, n_b, n_neg, zero, a_rec, a_ent, b_hdr, b_id, b_ent, neg;
  } g[2];
  unsigned long long self;  // the blob's own address in global memory
  // J gather for any signs: w0 = part | coef<<16, w1 = independent species + 1
  // (0 = loss entry); per slot: entry pointer, LU position, row; lane slot
  // lists.  Read as those of f.
  int jg_w0, jg_w1, jg_ptr, jg_mid, jg_lupos, jg_row, jg_lane, jg_slots;
  // device J slots are numbered by LU position; CSC entry of each slot and
  // slot of each CSC entry (uint16; self)
  int j_csc, jg_slot;
  // LU: dependent index -> pivot row (iperm), diag (uint16); per 32 LU positions
  // lu_src (uint32 x 3): those that a J slot fills (slots are numbered by LU
  // position), the diagonals, and the number of slots before them.
  int lu_iperm, lu_diag, lu_src;
  // factorization by pivot level (n_plev): fl_hdr (uint16 x 2 per level): end
  // of the level's scaling records, rounds of updates.  A scaling record fs_rec
  // is an L entry (uint32 L position | diagonal position<<16, uint32 pivot |
  // store its reciprocal<<15; L position n_lu: nothing to scale).  An update
  // round gives every lane one target LU[tgt] -= sum LU[a] LU[b]: record uint32
  // a | b<<16, uint32 tgt | cnt<<16 (fb_rec), the first pair in the record,
  // cnt - 1 more per lane in fb_ext (uint32 a | b<<16, 32 per step).  cnt is the
  // round's largest, the same in every lane: shorter targets and idle lanes are
  // padded with the spare slot LU[n_lu] = 0.  Bit 15 of cnt: a round of targets
  // of four pairs or more on two neighbouring lanes each, one of the two
  // alternating sums per lane; bits 10 to 14 are then half of the lanes in use (a
  // power of two), which are the words of a step in fb_ext.
  int fl_hdr, fs_rec, fb_rec, fb_ext;
  // triangular solves: n_fwd rounds forward, then n_bwd backward.  A round
  // gives every lane one target z[tgt] -= sum LU[a] z[x] (backward: then times
  // its reciprocal pivot when bit 15 of the second word is set): record
  // uint32 a | x<<16, uint32 tgt | finish<<15 | cnt<<16 (sv_rec), further pairs
  // in sv_ext (uint32 a | x<<16) as for the updates, padded with LU[n_lu] and
  // z[n] = 0.  Two rounds of records are read ahead of the ends.
  int n_fwd, n_bwd, sv_rec, sv_ext;
  // row-wise LU for the sequential (one-lane) mode: J slot -> LU position
  // (jg_lupos), diagonal positions, rowptr, col (uint16), update pointer per
  // L entry (uint32) and updates (src | dst<<16); staged only in that mode
  int lu_rowptr, lu_col, upd_ptr, upd;
  // dependent index -> state index (uint16); absolute tolerances (double)
  int dep_state, atol;
  // SIMPOL phase transfer: per instance a record of 8 x uint16 (gas and
  // aerosol dependent indices, dependent element count, first element, first
  // Jacobian partial), per dependent element its index (uint16) and factors
  // (1/density, 1/MW when in the instance's phase else 0, in-phase flag;
  // 3 x double).  Its 4 pseudo-rates per instance follow the terms' rates,
  // its 8 per-cell constants the terms' rate constants.
  int n_simpol, n_keff, n_rates, n_part_all;
  int si_rec, si_elem, si_ef;
  // aqueous equilibrium instances: record (uint16 x 12: dependent slots,
  // dependent reactant slots, first slot, first pseudo-rate, first partial,
  // keff slot, computed water | reactant and product counts, computed
  // activity coefficient, first and count of the computed participants),
  // per slot its dependent index (uint16) and 1e3 / MW (double); per
  // computed participant its computed index | reactant << 15 (uint16) and
  // 1e3 / MW (double)
  int n_aq, aq_rec, aq_sp, aq_sm, aq_cp, aq_cpm;
  int aq_sim;  // per slot MW / 1e3 (1 / aq_sm), double
  // J gather with unguarded products (SIMPOL): they lead each slot, and
  // jg_umid (uint16 per slot) is the slot's first loss entry
  int has_ug, jg_umid;
  // sub-models: computed species, parameter-Jacobian elements, keff slot of
  // PPM_TO_RH_; per computed species its program's first int and first
  // float (2 x uint32), the program ints (int32) and floats (double).  The
  // values sit after the pseudo-rates (f) or the partials (J), the
  // parameter partials and the virtual slots after the values.
  int n_cv, n_pj, sm_keff, sm_rec, sm_int, sm_flt;
  int sm_state;  // state index of each computed species (uint16)
  // their parallel parts (n_smi 0: none, a lane per computed species): n_smi
  // items (sm_item, uint32 x 4: kind | computed species<<8, first int, first
  // float, scratch slot), kind 1 a Jacobson pair of ZSR (7 slots: the water's
  // factor, then factor and multiplier of its three partials), kind 3 a PD-FiTE
  // interaction (slots li, dli, in range), kind 4 a PD-FiTE pair (slots its
  // cation's and anion's moles; shared by the coefficients of a phase); per
  // computed species sm_scr (uint32 x 4: first slot; PD-FiTE: interactions, slot
  // of the first pair, slot of gamma and 1 / omega).  PD-FiTE's partials: n_smp
  // elements, sm_pel (uint32 x 2: parameter id | computed species<<16, first |
  // count<<16 of the other pairs, in order, whose cation or anion it is
  // against), sm_pq (uint16: pair | anion<<15).  The scratch of n_sms slots lies
  // at scr0[0] (f) or scr0[1] (J) of the f / J scratch, which end at scr_end.
  int n_smi, sm_item, sm_scr, n_smp, sm_pel, sm_pq, n_sms, scr0[2], scr_end[2];
  // virtual Jacobian slots: partial lists (uint16 pointers, n_virt + 1, and
  // uint16 partial indices); the chain by target slot: target (uint16),
  // entry pointers (uint16, n_chain + 1), entries (uint32: virtual slot |
  // parameter id << 16)
  int n_virt, jv_ptr, jv_part, n_chain, ch_tgt, ch_ptr, ch_ent;
};

constexpr int kBlobHeader = 512;
// Cells (warps) per block of the solve kernel: its launch bound leaves 168
// registers per thread, enough to keep the BDF state without spilling.
constexpr int kMaxCellsPerBlock = 12;
constexpr int kMaxCellsAero = 8;  // cells per block of the aerosol form
constexpr int kBlockSmem = 232448;  // the most shared memory of a block on sm_100a

struct Tables;

// Builds the blob; false (with a message) if the mechanism exceeds the
// encodings (more than 3 variable reactants in a reaction, more than 1023
// dependent variables, or index spaces beyond 16 bits).
// max_smem: the most shared memory of a block, for the choice of the gathers.
bool build_blob(const Tables& t, const std::vector<double>& atol_dep, int max_smem,
                std::vector<uint8_t>* blob, BlobOff* off, std::string* err);

// A cell's shared-memory slice (byte offsets; -1 = not in it).  Without the
// Nordsieck history it leaves room for more resident cells; tempv is for the
// evaluation hooks.
struct Layout {
  int zn, ewt, acor, y, ftemp, tempv, rates, keff, fscr, lu, z, dinv, ctl, bytes;
};
Layout make_layout(const BlobOff& o, int lt_size, bool with_hist, bool with_tempv);

}  // namespace campb

namespace campb {

// Tables of the lane-per-cell kernel (one cell per lane, all lanes of a warp
// read the same table entry at the same time).  Header first, then sections;
// offsets in bytes from the start of the blob.
struct LaneOff {
  int bytes;
  int n, n_rxn, n_lu, n_coef, n_part, n_jpos, n_upd;
  // reactions: variable reactants (nv<<30 | d2<<20 | d1<<10 | d0, uint32);
  // participants (variable reactant occurrences, then variable products) per
  // reaction: pointer (uint16) and entries (species | coef<<10 | product<<31)
  int rx_word, rx_pptr, rx_part;
  // Jacobian scatter: per reaction, for each variable reactant occurrence k
  // and each participant p, the LU position of d(p)/d(k) (uint16)
  int rx_jptr, jpos;
  int coef;  // double
  // row-wise LU in pivot order (uint16) and update lists (uint32)
  int lu_perm, lu_rowptr, lu_col, lu_diag, upd_ptr, upd;
  int dep_state;  // uint16
  int atol;       // double
};

bool build_lane_blob(const Tables& t, const std::vector<double>& atol_dep,
                     std::vector<uint8_t>* blob, LaneOff* off, std::string* err);

}  // namespace campb

namespace campb {

// Tables of the CTA-per-cell kernel (one thread block per cell), for
// mechanisms whose LU is too large for the warp-per-cell tables.  The block
// reads them from global memory through L1.  The LU is row-wise in pivot
// order with sorted columns; its trailing rows r0..n-1 form a dense block
// (every column r0..n-1 present), addressed without tables: entry (i, j) of
// that block sits at dpos[i - r0] + (j - r0).  The sparse head (pivots and
// rows before r0) is factored pivot by pivot from tabulated update targets
// and solved by row levels.  Offsets in bytes from the start of the blob.
struct BlockOff {
  int bytes;
  int n, n_rxn, n_part, n_jac, n_lu, n_coef;
  int r0;          // first row (pivot) of the trailing dense block
  int n_hf, n_hb;  // forward / backward row levels of the head rows
  // reactions: variable reactants (nv<<30 | d2<<20 | d1<<10 | d0, uint32)
  // and the first rate partial of each (uint32, n_rxn + 1)
  int rx_word, rx_vptr;
  int coef;  // double
  // f gather by species: pointers (uint32, n + 1), entries (uint32: term |
  // coef<<16 | guarded product<<31)
  int fg_ptr, fg_ent;
  // J gather by solver slot: pointers (uint32, n_jac + 1), first guarded
  // product (uint32), entries (uint32: partial | coef<<16), guard species + 1
  // (uint16), row species (uint16)
  int jg_ptr, jg_mid, jg_w0, jg_w1, jg_row;
  // per LU position: J slot + 1 (0 = none) | diagonal<<15 (uint16)
  int lu_src;
  // LU structure (uint16): pivot -> dependent index, row pointers, columns,
  // diagonal positions
  int lu_perm, lu_rowptr, lu_col, lu_diag;
  int dpos;  // per dense row: position of its column r0 (uint16)
  int ub;    // per head row: first position with a column >= r0 (uint16)
  // head pivots k < r0: L entries of column k in row order (pointers
  // uint32, r0 + 1; entries uint32: position | row << 16), the first of
  // them in a dense row (uint32 per pivot), and the tabulated updates
  // (pointers uint32, r0 + 1; records uint64: target | L position << 16 |
  // U position << 32): the head rows' L entries against every U entry of
  // row k, then the dense rows' against the U entries of row k in head
  // columns, row-major.  The dense rows' updates in dense columns are
  // addressed through the dense block.
  int lk_ptr, lk, lk_mid, tg_ptr, hrec;
  // head row levels (pointers uint16, levels + 1; rows uint16)
  int hf_ptr, hf_rows, hb_ptr, hb_rows;
  int dep_state;  // uint16
  int atol;       // double
  // the solve's tables, one uint16 section the block copies into shared
  // memory (stage: byte offset, sg_len: elements); element offsets inside:
  // row pointers (n + 1), diagonals (n), head rows' ub (r0), permutation
  // (n), head levels (forward pointers and rows, backward pointers and
  // rows), per row the first of its non-dense entries in ndcol (n + 1; the
  // head rows' entries, the dense rows' head-column entries) and their
  // columns, and the dense rows' bases (dpos - r0, m)
  int stage, sg_len;
  int sg_rowptr, sg_diag, sg_ub, sg_perm, sg_hf_ptr, sg_hf_rows, sg_hb_ptr, sg_hb_rows;
  int sg_ndoff, sg_ndcol, sg_dbase;
  // and the head pivots' pointers: lk_ptr (r0 + 1), lk_mid (r0), tg_ptr
  // (r0 + 1), as uint16
  int sg_hlk, sg_hmid, sg_htg;
};

// the largest trailing dense block the CTA kernel holds in registers
// (a 16 x 16 thread grid, 7 x 7 entries per thread)
constexpr int kBlockMaxDense = 112;

bool build_block_blob(const Tables& t, const std::vector<double>& atol_dep,
                      std::vector<uint8_t>* blob, BlockOff* off, std::string* err);

}  // namespace campb
