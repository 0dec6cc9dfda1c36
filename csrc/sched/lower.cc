// Lowering of a global plan to the work list of one GPU.
//
// The reference lowers to per-GPU parameter blocks and splits every peer transfer evenly over the
// CTAs (alltoall_global_scheduler.cc:1109-1150) and into <=16 chunks of >=32 MiB with cumulative
// ready thresholds (:1152-1178). Here one chunk IS one CTA work item, chunks of concurrent ops are
// interleaved so that every peer of a slot is in flight at once, and ordering between phases is
// carried by byte counters (balance / per-stage rail / output) instead of per-block flags.
#include <algorithm>
#include <cstdint>

#include "plan.h"

namespace fastb {

namespace {

// Arrival counters of the rail staging. Without segments there is one per stage (slot = stage).
// With segments a rank's rail staging is cut into pieces of `seg` bytes by absolute offset and a
// piece of stage k gets the counter `offset / seg + k`, so that a forwarder waits only for the
// pieces it reads (the reference's cumulative chunk_ready_threshold,
// alltoall_global_scheduler.cc:1152-1178, without its assumption that chunks arrive in order).
// Adding the stage index keeps the counters of neighbouring stages apart even where their regions
// share a `seg`-sized window: a forward of stage k must never wait for bytes of a later stage,
// whose pushes come after it in the work lists (that would be a cycle between ranks). This relies
// on the regions lying in stage order, which holds up to Plan::rail_tail_start; what is staged
// behind it (remainders of aligned cuts, a few units per pair) gets one counter per stage instead.
// The numbering needs nothing but per-rank sizes, so a one-rank view of the plan lowers exactly
// like the full plan.
struct RailSlots {
  int64_t seg = 0, ub = 1;    // segment bytes (0 = one slot per stage); unit bytes
  int K = 0;
  const Plan* plan = nullptr;
  std::vector<int> count;     // [rank] counters of the rank

  bool in_tail(int owner, int64_t byte_off) const { return seg > 0 && byte_off >= plan->rail_tail_start[owner] * ub; }
  int ordered_slots(int owner) const { return static_cast<int>((plan->buffers[owner].rail_units * ub + seg - 1) / seg) + K; }
  int slot(int owner, int stage, int64_t byte_off) const {
    if (seg <= 0) return stage;
    return in_tail(owner, byte_off) ? ordered_slots(owner) + stage : static_cast<int>(byte_off / seg) + stage;
  }
  // End (bytes, exclusive) of the piece that contains byte_off; tail pieces are not cut.
  int64_t piece_end(int owner, int64_t byte_off) const {
    if (seg <= 0 || in_tail(owner, byte_off)) return INT64_MAX;
    return std::min((byte_off / seg + 1) * seg, plan->rail_tail_start[owner] * ub);
  }
};

RailSlots make_slots(const Plan& p, const LowerOptions& lo_opt) {
  RailSlots rs;
  const int n = p.matrix.n, K = p.num_stages;
  rs.plan = &p; rs.K = K; rs.ub = lo_opt.unit_bytes;
  rs.count.assign(n, K);
  if (lo_opt.rail_segment_bytes <= 0 || K == 0) return rs;
  int64_t widest = 0;
  for (int r = 0; r < n; ++r) widest = std::max(widest, p.buffers[r].rail_units * lo_opt.unit_bytes);
  if (widest == 0) return rs;  // nothing is staged (flat plans): nothing to segment
  rs.seg = (std::max<int64_t>(lo_opt.rail_segment_bytes, 16) + 15) / 16 * 16;
  // Every rank must fit the signal block: coarsen until the largest staging area does (never
  // below one counter per stage, plus one per stage for the tail).
  const int64_t room = std::max<int64_t>(lo_opt.max_rail_slots - 2 * K, 1);
  while ((widest + rs.seg - 1) / rs.seg > room && rs.seg < widest) rs.seg *= 2;
  for (int r = 0; r < n; ++r) rs.count[r] = rs.ordered_slots(r) + K;
  return rs;
}

}  // namespace

RankProgram lower_for_rank(const Plan& p, int rank, const LowerOptions& lo) {
  const int n = p.matrix.n;
  if (rank < 0 || rank >= n) throw std::invalid_argument("lower_for_rank: rank out of range");
  if (lo.unit_bytes < 1 || lo.chunk_bytes < 1) throw std::invalid_argument("lower_for_rank: bad options");
  RankProgram prog;
  prog.rank = rank;
  const int K = p.num_stages;
  const int64_t ub = lo.unit_bytes;
  const RailSlots slots = make_slots(p, lo);
  prog.expect_rail_bytes.assign(slots.count[rank], 0);
  const RankBuffers& b = p.buffers[rank];
  prog.buffers_bytes = RankBuffers{b.input_units * ub, b.output_units * ub, b.balance_units * ub, b.rail_units * ub};

  // A piece is the part of an op that signals (rail push) or waits for (forward) one rail slot.
  struct Piece { const Op* op; int64_t begin, bytes; int signal_slot, wait_slot; };
  auto pieces_of = [&](const Op& o, std::vector<Piece>& out) {
    const int64_t total = o.len * ub;
    const bool to_rail = o.dst_buf == Buf::kRail, from_rail = o.src_buf == Buf::kRail;
    if (slots.seg <= 0 || (!to_rail && !from_rail)) {
      out.push_back(Piece{&o, 0, total, o.stage, from_rail ? o.stage : -1});
      return;
    }
    // Cut where the rail-side offset crosses a piece boundary (a forward reads rail, a push writes it).
    const int owner = to_rail ? o.dst_rank : o.src_rank;
    const int64_t rail0 = (to_rail ? o.dst_off : o.src_off) * ub;
    int64_t done = 0;
    while (done < total) {
      const int64_t at = rail0 + done;
      const int64_t take = std::min(total - done, slots.piece_end(owner, at) - at);
      const int s = slots.slot(owner, o.stage, at);
      out.push_back(Piece{&o, done, take, to_rail ? s : o.stage, from_rail ? s : -1});
      done += take;
    }
  };

  // slot 0: balance | slot 1: rail 0, intrinsic, un-staged direct ops | slot k+1: rail k (+ staged
  // direct ops of round k) and redistribution of stage k-1 | last slot: final redistribution.
  // One list for all pieces, filed by (slot, push before forward) afterwards: a vector per slot allocates 2 (K + 3) times, mostly for one piece.
  std::vector<Piece> pieces, tmp;
  std::vector<int> cell_of;
  pieces.reserve(p.ops.size() / static_cast<size_t>(n) + static_cast<size_t>(K) + 16);
  cell_of.reserve(pieces.capacity());
  const int cells = 2 * (K + 3);
  for (const Op& o : p.ops) {
    if (o.dst_rank == rank) {
      const int64_t bytes = o.len * ub;
      if (o.dst_buf == Buf::kOutput) prog.expect_output_bytes += bytes;
      else if (o.dst_buf == Buf::kBalance) prog.expect_balance_bytes += bytes;
      else {
        tmp.clear();
        pieces_of(o, tmp);
        for (const Piece& pc : tmp) prog.expect_rail_bytes[pc.signal_slot] += pc.bytes;
      }
    }
    if (o.src_rank != rank) continue;
    int cell = 0;
    switch (o.phase) {
      case Phase::kBalance: cell = 0; break;
      case Phase::kIntrinsic: cell = 2 * (o.stage < 0 ? 1 : 1 + o.stage); break;
      case Phase::kRail: cell = 2 * (1 + o.stage); break;
      case Phase::kRedistribute: cell = 2 * (2 + o.stage) + 1; break;
    }
    pieces_of(o, pieces);
    cell_of.resize(pieces.size(), cell);
  }
  std::vector<size_t> cell_start(static_cast<size_t>(cells) + 1, 0);
  for (int c : cell_of) ++cell_start[static_cast<size_t>(c) + 1];
  for (int c = 0; c < cells; ++c) cell_start[static_cast<size_t>(c) + 1] += cell_start[static_cast<size_t>(c)];
  if (!std::is_sorted(cell_of.begin(), cell_of.end())) {
    std::vector<Piece> filed(pieces.size());
    std::vector<size_t> at(cell_start.begin(), cell_start.end() - 1);
    for (size_t k = 0; k < pieces.size(); ++k) filed[at[static_cast<size_t>(cell_of[k])]++] = pieces[k];
    pieces.swap(filed);
  }
  auto chunk_of = [&](int64_t bytes) {
    int64_t c = lo.chunk_bytes;
    if (bytes / c > lo.max_chunks_per_op) c = (bytes + lo.max_chunks_per_op - 1) / lo.max_chunks_per_op;
    c = (c + 15) / 16 * 16;
    return c;
  };
  // The item of a whole piece; its chunks differ in offsets and bytes only.
  auto whole = [&](const Piece& pc) {
    const Op& o = *pc.op;
    WorkItem w{};
    w.src_off = o.src_off * ub + pc.begin;
    w.dst_off = o.dst_off * ub + pc.begin;
    w.bytes = pc.bytes;
    w.dst_rank = o.dst_rank;
    w.src_buf = static_cast<uint8_t>(o.src_buf);
    w.dst_buf = static_cast<uint8_t>(o.dst_buf);
    w.wait_kind = o.src_buf == Buf::kBalance ? 1 : o.src_buf == Buf::kRail ? 2 : 0;
    w.signal_kind = o.dst_buf == Buf::kBalance ? 1 : o.dst_buf == Buf::kRail ? 2 : 3;
    w.stage = pc.signal_slot;
    w.wait_stage = pc.wait_slot;
    return w;
  };
  struct Slice { double key; uint32_t pc; uint32_t chunk; };
  std::vector<Slice> slices, filed;
  std::vector<uint32_t> bucket;
  std::vector<WorkItem> model;
  std::vector<int64_t> size;
  auto emit_interleaved = [&](const Piece* pcs, size_t n_pcs) {
    if (n_pcs == 0) return;
    if (n_pcs == 1) {  // a stage of a flat plan: one transfer, its chunks in order
      WorkItem w = whole(pcs[0]);
      const int64_t total = pcs[0].bytes, c = chunk_of(total);
      for (int64_t left = total; left > 0; left -= c, w.src_off += c, w.dst_off += c) { w.bytes = std::min(c, left); prog.items.push_back(w); }
      return;
    }
    // Proportional interleave: chunk j of a piece with c chunks gets key (j + 1/2) / c and chunks are
    // issued in key order, so every transfer of the slot advances at a rate proportional to its size
    // and all of them finish together (equal ones degenerate to plain round-robin). A heavy pair
    // is then in flight from the first chunk on instead of trailing alone at the end.
    slices.clear(); model.clear(); size.clear();
    for (size_t k = 0; k < n_pcs; ++k) {
      const int64_t c = chunk_of(pcs[k].bytes), count = (pcs[k].bytes + c - 1) / c;
      model.push_back(whole(pcs[k]));
      size.push_back(c);
      for (int64_t j = 0; j < count; ++j) slices.push_back(Slice{(static_cast<double>(j) + 0.5) / static_cast<double>(count), static_cast<uint32_t>(k), static_cast<uint32_t>(j)});
    }
    // In key order, equal keys in list order. The keys lie in (0, 1), about evenly: filed into as many buckets as there are chunks, what is left to
    // do is an insertion here and there. Lowering the 1026 chunks of a fan-out of eight ranks: 22.7 us with a stable sort, 15.6 so.
    const size_t m = slices.size();
    const double buckets = static_cast<double>(m);
    bucket.assign(m + 1, 0);
    for (const Slice& s : slices) ++bucket[static_cast<size_t>(s.key * buckets) + 1];
    for (size_t q = 1; q <= m; ++q) bucket[q] += bucket[q - 1];
    filed.resize(m);
    for (const Slice& s : slices) filed[bucket[static_cast<size_t>(s.key * buckets)]++] = s;
    for (size_t q = 1; q < m; ++q) {
      const Slice s = filed[q];
      size_t at = q;
      for (; at > 0 && filed[at - 1].key > s.key; --at) filed[at] = filed[at - 1];
      filed[at] = s;
    }
    for (const Slice& s : filed) {
      WorkItem w = model[s.pc];
      const int64_t begin = static_cast<int64_t>(s.chunk) * size[s.pc];
      w.src_off += begin;
      w.dst_off += begin;
      w.bytes = std::min(size[s.pc], w.bytes - begin);
      prog.items.push_back(w);
    }
  };
  {  // one allocation for the whole list
    size_t items = 0;
    for (const Piece& pc : pieces) { const int64_t c = chunk_of(pc.bytes); items += static_cast<size_t>((pc.bytes + c - 1) / c); }
    prog.items.reserve(items);
  }
  for (int c = 0; c < cells; ++c) emit_interleaved(pieces.data() + cell_start[static_cast<size_t>(c)], cell_start[static_cast<size_t>(c) + 1] - cell_start[static_cast<size_t>(c)]);
  return prog;
}

}  // namespace fastb
