#include "plan.h"

#include <algorithm>
#include <stdexcept>

namespace fastb {

namespace {

struct Piece {
  int origin_local, final_local;
  int64_t pair_off, len;
  Buf buf;
  int64_t off;  // units, inside `buf` of the GPU currently holding the piece
};

// Pieces waiting at one (source server, destination server, GPU): a range of one list, taken from the front. A container per
// queue allocates S * S * G times, mostly for a single piece.
struct PieceQueue {
  size_t head = 0, end = 0;
  bool empty() const { return head == end; }
};

// Largest cut <= want that keeps the remainder of `p` aligned inside its segment, or the whole
// piece when want covers it.
int64_t aligned_cut(const Piece& p, int64_t want, int64_t align) {
  if (want >= p.len) return p.len;
  if (align <= 1) return want;
  const int64_t at = p.pair_off + want;
  const int64_t end = (align & (align - 1)) == 0 ? at & -align : at / align * align;  // absolute cut position in the segment; no division per cut
  return end > p.pair_off ? end - p.pair_off : 0;
}

}  // namespace

Plan build_plan(const Matrix& traffic, Topology topo, const PlanOptions& opt) {
  traffic.check_non_negative();
  if (topo.servers < 1 || topo.gpus < 1 || topo.ranks() != traffic.n)
    throw std::invalid_argument("build_plan: servers * gpus must equal the matrix dimension");
  if (opt.split_align < 1) throw std::invalid_argument("build_plan: split_align must be >= 1");

  Plan p;
  p.topo = topo;
  p.opt = opt;
  p.matrix = opt.transpose ? traffic.transposed() : traffic;
  p.matrix_hash = p.matrix.hash();
  const Matrix& M = p.matrix;
  const int n = M.n, S = topo.servers, G = topo.gpus;

  p.in_disp.assign(static_cast<size_t>(n) * n, 0);
  p.out_disp.assign(static_cast<size_t>(n) * n, 0);
  p.buffers.assign(n, RankBuffers{});
  for (int r = 0; r < n; ++r) {
    int64_t a = 0, b = 0;
    for (int q = 0; q < n; ++q) {
      p.in_disp[static_cast<size_t>(r) * n + q] = a;
      a += M.at(r, q);
      p.out_disp[static_cast<size_t>(r) * n + q] = b;
      b += M.at(q, r);
    }
    p.buffers[r].input_units = a;
    p.buffers[r].output_units = b;
  }
  auto in_at = [&](int r, int d) { return p.in_disp[static_cast<size_t>(r) * n + d]; };
  auto out_at = [&](int r, int s) { return p.out_disp[static_cast<size_t>(r) * n + s]; };
  const int only = opt.only_rank;
  if (only >= n) throw std::invalid_argument("build_plan: only_rank out of range");
  auto keep = [only](int src, int dst) { return only < 0 || src == only || dst == only; };
  auto direct = [&](int r, int d, int stage) {
    if (M.at(r, d) == 0 || !keep(r, d)) return;
    p.ops.push_back(Op{Phase::kIntrinsic, Buf::kInput, Buf::kOutput, stage, r, d, r, d, in_at(r, d),
                       out_at(d, r), M.at(r, d), 0});
  };

  p.server_matrix = Matrix(S);

  if (opt.kind == PlanKind::kFanout) {
    for (int step = 0; step < n; ++step)
      for (int r = 0; r < n; ++r) direct(r, (r + step) % n, -1);
    p.num_stages = 0;
    p.rail_tail_start.assign(n, 0);
    return p;
  }
  if (opt.kind == PlanKind::kSpreadOut) {
    for (int step = 0; step < n; ++step)
      for (int r = 0; r < n; ++r) direct(r, (r + step) % n, step);
    p.num_stages = n;
    p.rail_tail_start.assign(n, 0);
    return p;
  }

  // ---- balance: equalise the per-GPU load of every (src server, dst server) tile -------------
  // hold[(s*S+t)*G+i] = pieces GPU i of server s will put on its rail toward server t.
  std::vector<PieceQueue> hold(static_cast<size_t>(S) * S * G);
  std::vector<Piece> pieces;
  pieces.reserve(static_cast<size_t>(n) * n);   // about one piece per rank pair; balancing adds a few
  std::vector<std::vector<Piece>> tile(G);      // the queues of the server pair at hand
  auto hold_at = [&](int s, int t, int i) -> PieceQueue& { return hold[(static_cast<size_t>(s) * S + t) * G + i]; };

  std::vector<int64_t> load(G, 0);
  for (int s = 0; s < S; ++s) {
    for (int t = 0; t < S; ++t) {
      if (s == t) continue;
      std::fill(load.begin(), load.end(), 0);
      for (auto& q : tile) q.clear();
      int64_t sum = 0;
      for (int i = 0; i < G; ++i) {
        for (int j = 0; j < G; ++j) {
          const int64_t x = M.at(s * G + i, t * G + j);
          if (x == 0) continue;
          tile[i].push_back(Piece{i, j, 0, x, Buf::kInput, in_at(s * G + i, t * G + j)});
          load[i] += x;
        }
        sum += load[i];
      }
      const int64_t target = (sum + G - 1) / G;
      bool balance = G > 1;
      if (balance && opt.balance_alpha_beta) {
        double alpha = opt.intra.alpha_us;
        double beta = static_cast<double>(*std::max_element(load.begin(), load.end())) * opt.intra.beta_us_per_mb * opt.mb_per_unit;
        for (int d = 0; d < G; ++d) {
          int64_t mx = 0;
          for (int j = 0; j < G; ++j) mx = std::max(mx, M.at(s * G + j, t * G + (j + d) % G));
          if (mx) { alpha += opt.intra.alpha_us; beta += static_cast<double>(mx) * opt.intra.beta_us_per_mb * opt.mb_per_unit; }
        }
        balance = !(beta / alpha < 2.0);
      }
      for (int big = 0; big < G && balance; ++big) {
        for (int small = 0; small < G && load[big] > target; ++small) {
          if (small == big || load[small] >= target) continue;
          std::vector<Piece>& src = tile[big];
          // Walk the heavy GPU's own pieces (only data still in its input buffer can be relayed).
          for (size_t k = 0; k < src.size() && load[big] > target && load[small] < target;) {
            Piece& pc = src[k];
            if (pc.buf != Buf::kInput) { ++k; continue; }
            const int64_t want = std::min(load[big] - target, target - load[small]);
            const int64_t mv = aligned_cut(pc, want, opt.split_align);
            if (mv == 0) { ++k; continue; }
            const int dst_rank = s * G + small, src_rank = s * G + big;
            int64_t& cursor = p.buffers[dst_rank].balance_units;
            if (keep(src_rank, dst_rank))
              p.ops.push_back(Op{Phase::kBalance, Buf::kInput, Buf::kBalance, -1, src_rank, dst_rank,
                                 src_rank, t * G + pc.final_local, pc.off, cursor, mv, pc.pair_off});
            tile[small].push_back(Piece{pc.origin_local, pc.final_local, pc.pair_off, mv, Buf::kBalance, cursor});
            cursor += mv;
            load[big] -= mv;
            load[small] += mv;
            if (mv == pc.len) {
              src.erase(src.begin() + static_cast<std::ptrdiff_t>(k));
            } else {
              pc.pair_off += mv; pc.off += mv; pc.len -= mv;
              ++k;
            }
          }
        }
      }
      for (int i = 0; i < G; ++i) {
        const size_t head = pieces.size();
        pieces.insert(pieces.end(), tile[i].begin(), tile[i].end());
        hold_at(s, t, i) = PieceQueue{head, pieces.size()};
      }
      p.server_matrix.at(s, t) = *std::max_element(load.begin(), load.end());
    }
  }

  // ---- intra-server traffic ---------------------------------------------------------------------
  for (int s = 0; s < S; ++s)
    for (int step = 0; step < G; ++step)
      for (int i = 0; i < G; ++i) direct(s * G + i, s * G + (i + step) % G, -1);

  // ---- inter-server stages ----------------------------------------------------------------------
  Stage all;                // kSingleBurst: every server pair at once, unlimited budget
  all.weight = -1;
  const Stage* stages = &all;
  int K = 1;
  if (opt.kind == PlanKind::kStaged) {
    int64_t scale = opt.scale > 0 ? opt.scale
                                  : choose_scale(p.server_matrix, G, opt.scale_policy, opt.inter, opt.intra, opt.mb_per_unit);
    if (scale < 1) scale = 1;
    p.decomp = decompose(p.server_matrix, opt.match, scale);
    stages = p.decomp.stages.data();
    K = static_cast<int>(p.decomp.stages.size());
  }

  std::vector<int> last_stage_of_pair(static_cast<size_t>(S) * S, -1);

  // Rail and redistribution ops are collected as they come and filed by stage at the end, so that the
  // final list is [balance][intrinsic][rail 0][redis 0][rail 1][redis 1]...
  std::vector<Op> later;
  later.reserve(std::min<size_t>(static_cast<size_t>(K) * S * G, 4096));

  auto emit_rail = [&](int k, int s, int t, int i, int64_t budget) {
    auto& q = hold_at(s, t, i);
    if (q.empty()) return;
    const int src_rank = s * G + i, dst_rank = t * G + i;
    while (!q.empty() && budget != 0) {
      Piece& pc = pieces[q.head];
      const int64_t take = budget < 0 ? pc.len : aligned_cut(pc, budget, opt.split_align);
      if (take == 0) break;
      const int origin = s * G + pc.origin_local, fin = t * G + pc.final_local;
      if (pc.final_local == i) {
        if (keep(src_rank, dst_rank))
          later.push_back(Op{Phase::kRail, pc.buf, Buf::kOutput, k, src_rank, dst_rank, origin, fin, pc.off,
                            out_at(fin, origin) + pc.pair_off, take, pc.pair_off});
      } else {
        int64_t& cursor = p.buffers[dst_rank].rail_units;
        if (keep(src_rank, dst_rank))
          later.push_back(Op{Phase::kRail, pc.buf, Buf::kRail, k, src_rank, dst_rank, origin, fin, pc.off, cursor,
                            take, pc.pair_off});
        if (keep(dst_rank, fin))
          later.push_back(Op{Phase::kRedistribute, Buf::kRail, Buf::kOutput, k, dst_rank, fin, origin, fin, cursor,
                             out_at(fin, origin) + pc.pair_off, take, pc.pair_off});
        cursor += take;
      }
      if (budget > 0) budget -= take;
      if (take == pc.len) ++q.head;
      else { pc.pair_off += take; pc.off += take; pc.len -= take; }
    }
  };

  for (int k = 0; k < K; ++k) {
    for (int s = 0; s < S; ++s) {
      if (opt.kind == PlanKind::kStaged) {
        const int t = stages[k].to[s];
        if (t == s) continue;
        last_stage_of_pair[static_cast<size_t>(s) * S + t] = k;
        for (int i = 0; i < G; ++i) emit_rail(k, s, t, i, stages[k].weight);
      } else {
        for (int step = 1; step < S; ++step) {
          const int t = (s + step) % S;
          for (int i = 0; i < G; ++i) emit_rail(k, s, t, i, -1);
        }
      }
    }
  }
  p.rail_tail_start.resize(n);
  for (int r = 0; r < n; ++r) p.rail_tail_start[r] = p.buffers[r].rail_units;  // up to here regions follow the stage order
  // Alignment can leave a few units behind a stage budget; ship them with the pair's last stage.
  if (opt.kind == PlanKind::kStaged) {
    for (int s = 0; s < S; ++s)
      for (int t = 0; t < S; ++t) {
        if (s == t) continue;
        for (int i = 0; i < G; ++i) {
          if (hold_at(s, t, i).empty()) continue;
          const int k = last_stage_of_pair[static_cast<size_t>(s) * S + t];
          if (k < 0) throw std::logic_error("build_plan: traffic left without a stage");
          emit_rail(k, s, t, i, -1);
        }
      }
  }
  // Stable counting sort by (stage, rail before redistribution).
  auto slot_of = [](const Op& o) { return static_cast<size_t>(o.stage) * 2 + (o.phase == Phase::kRedistribute ? 1 : 0); };
  std::vector<size_t> at(static_cast<size_t>(K) * 2 + 1, 0);
  for (const Op& o : later) ++at[slot_of(o) + 1];
  for (size_t q = 1; q < at.size(); ++q) at[q] += at[q - 1];
  p.num_stages = K;
  if (std::is_sorted(later.begin(), later.end(), [&](const Op& x, const Op& y) { return slot_of(x) < slot_of(y); })) {   // one GPU per server
    if (p.ops.empty()) p.ops.swap(later);
    else p.ops.insert(p.ops.end(), later.begin(), later.end());
    return p;
  }
  const size_t first = p.ops.size();
  p.ops.resize(first + later.size());
  for (const Op& o : later) p.ops[first + at[slot_of(o)]++] = o;
  return p;
}

Matrix delivered_matrix(const Plan& p) {
  Matrix d(p.matrix.n);
  for (const Op& o : p.ops)
    if (o.dst_buf == Buf::kOutput) d.at(o.origin, o.final_dst) += o.len;
  return d;
}

Matrix stage_matrix(const Plan& p, int stage) {
  Matrix d(p.matrix.n);
  for (const Op& o : p.ops)
    if (o.stage == stage && (o.phase == Phase::kRail || (o.phase == Phase::kIntrinsic && o.stage >= 0)))
      d.at(o.src_rank, o.dst_rank) += o.len;
  return d;
}

}  // namespace fastb
