// Host side of the FP64 GEMM on the tensor cores (kernels_oz.cu): packed layouts, stacked
// panels, tiles and launches of a GemmPlan.
#include <algorithm>
#include <map>
#include <set>

#include "engine.hpp"

namespace mpsxx {

namespace {

// A block as a GEMM operand: element (row, k) at row * rstride + k * kstride.
struct View {
  int rows = 0, k = 0, rstride = 0, kstride = 0;
};

int slices(int k) { return (k + kOzTileK - 1) / kOzTileK; }

// The packs of rows [0, rows) of a block or panel whose tiles start at o.bytes, and their
// room: CTAs of as many rows as fit the pack kernel's registers (row operands: within one
// 128-row tile, column operands: across 32-row tiles).  segs_of(lo, hi) appends the segments
// of rows [lo, hi).
template <class F>
void pack_rows(OzOperand& o, int rows, int k, int scale, bool row_operand, F segs_of) {
  const int nks = slices(k), log2 = row_operand ? 7 : 5, tile = 1 << log2, last = (rows - 1) / tile;
  const int tail = row_operand ? oz_tile_rows(rows, last) : oz_tail_cols(rows, last);
  const int most = std::min(kOzPackRows, std::max(8, kOzPackElems / (nks * kOzTileK) / 8 * 8));
  for (int r0 = 0; r0 < rows;) {
    const int end = row_operand ? std::min(rows, (r0 / tile + 1) * tile) : rows;
    const int parts = (end - r0 + most - 1) / most;
    const int n = std::min(most, ((end - r0 + parts - 1) / parts + 7) / 8 * 8);
    DOzPack pk;
    pk.dst_off = o.bytes;
    pk.seg0 = static_cast<int>(o.h_segs.size());
    segs_of(r0, std::min(r0 + n, rows));
    pk.nseg = static_cast<int>(o.h_segs.size()) - pk.seg0;
    pk.rows = n;
    pk.row0 = r0;
    pk.k = k;
    pk.nks = nks;
    pk.exp0 = o.rows + r0;
    pk.tile_log2 = log2;
    pk.last = last;
    pk.tail = tail;
    pk.scale = scale;
    o.h_packs.push_back(pk);
    r0 += n;
  }
  o.rows += last * tile + tail;
  o.bytes += (int64_t(last) * tile + tail) * nks * (kOzDigits * kOzTileK * 2);
}

// Every used block by itself.  tiled: the blocks' places in a tiled source.
void pack_blocks(OzOperand& o, const Tensor& t, const std::vector<View>& view, const std::vector<int>& scale,
                 bool row_operand, const std::vector<DOzTiled>* tiled = nullptr) {
  o.base.assign(view.size(), -1);
  o.exp0.assign(view.size(), 0);
  o.nks.assign(view.size(), 0);
  for (size_t s = 0; s < view.size(); ++s) {
    const View& v = view[s];
    if (v.rows <= 0 || v.k <= 0) continue;
    o.base[s] = o.bytes;
    o.exp0[s] = o.rows;
    o.nks[s] = slices(v.k);
    pack_rows(o, v.rows, v.k, scale[s], row_operand, [&](int lo, int hi) {
      if (tiled == nullptr) {
        o.h_segs.push_back(DOzSeg{t.offsets[s] + int64_t(lo) * v.rstride, 0, hi - lo, v.rstride, v.kstride});
        return;
      }
      const DOzTiled& p = (*tiled)[s];
      for (int r = lo; r < hi;) {  // runs of rows inside one tile row
        const int at = p.row0 + r, in = at % kOzTileM, run = std::min(hi - r, kOzTileM - in);
        o.h_segs.push_back(DOzSeg{p.base + int64_t(at / kOzTileM) * p.ntn * (kOzTileM * kOzTileN) +
                                      int64_t(in) * kOzTileN,
                                  r - lo, run, kOzTileN, 0});
        r += run;
      }
    });
  }
}

// The powers of two of a plan's contractions, one array per sector of the balancing index (and
// size of the index before it): its tasks and blocks, and the first entry by block slot of A
// and B.  Returns the number of entries; the arrays end at multiples of 16.
int balance(OzGemm& og, const OzBalance& bal, const Tensor& a, const Tensor& b, std::vector<int>& sa, std::vector<int>& sb,
            std::vector<DOzScaleBlock>& blocks) {
  int n = 0;
  const Tensor& of = bal.of;
  std::vector<std::vector<DOzScaleBlock>> by_sector(of.sh.dshape[bal.axis].size());
  for (size_t s = 0; s < of.tags.size(); ++s) {
    int idx[kMaxRank], d[kMaxRank];
    of.sh.index(of.tags[s], idx);
    of.block_dims(static_cast<int32_t>(s), d);
    if (d[0] > 0 && d[1] > 0)
      by_sector[idx[bal.axis]].push_back(bal.axis == 0 ? DOzScaleBlock{of.offsets[s], d[1], d[1], 1}
                                                       : DOzScaleBlock{of.offsets[s], d[0], 1, d[1]});
  }
  std::map<int, std::vector<int>> first;  // by size of the index before: first entry by sector (-1: none)
  auto slots = [&](const Tensor& t, int axis, int w, std::vector<int>& out) {
    out.assign(t.tags.size(), 0);
    const int64_t nsec = t.sh.nsec(axis);
    for (size_t s = 0; s < t.tags.size(); ++s) {
      const int sector = static_cast<int>(t.tags[s] / t.sh.stride[axis] % nsec), dim = t.sh.dshape[axis][sector];
      const int repeat = w < 0 ? 1 : t.sh.dshape[w][t.tags[s] / t.sh.stride[w] % t.sh.nsec(w)];
      if (dim <= 0 || repeat <= 0) continue;
      std::vector<int>& f = first[repeat];
      if (f.empty()) f.assign(nsec, -1);
      out[s] = f[sector] < 0 ? n : f[sector];
      if (f[sector] >= 0) continue;
      f[sector] = n;
      const int b0 = static_cast<int>(blocks.size());
      if (sector < static_cast<int>(by_sector.size()) && of.sh.dshape[bal.axis][sector] == dim)
        blocks.insert(blocks.end(), by_sector[sector].begin(), by_sector[sector].end());
      for (int i0 = 0; i0 < dim; i0 += 32)
        og.h_scale_tasks.push_back(DOzScale{n, dim, repeat, i0, b0, static_cast<int>(blocks.size())});
      n += (dim * repeat + 15) / 16 * 16;
    }
  };
  slots(a, bal.axis_a, bal.w_a, sa);
  slots(b, bal.axis_b, bal.w_b, sb);
  return n;
}

}  // namespace

void build_oz_gemm(Context& ctx, OzGemm& og, const GemmPlan& g, const Tensor& a, const Tensor& b, const OzBalance& bal,
                   bool tiled_out, const OzGemm* from, const GemmPlan* from_plan) {
  og.clear();
  // operand blocks as rows x K
  std::vector<View> va(a.tags.size()), vb(b.tags.size());
  std::set<int32_t> used_a, used_b;
  bool single = true;
  for (const DGemmTask& t : g.h_tasks) {
    single = single && t.p1 - t.p0 == 1;
    for (int p = t.p0; p < t.p1; ++p) {
      const DGemmPair& pr = g.h_pairs[p];
      va[g.pair_a_slot[p]] = g.ta == kNoTrans ? View{t.m, pr.k, pr.lda, 1} : View{t.m, pr.k, 1, pr.lda};
      vb[g.pair_b_slot[p]] = g.tb == kNoTrans ? View{t.n, pr.k, 1, pr.ldb} : View{t.n, pr.k, pr.ldb, 1};
      if (single) {
        used_a.insert(g.pair_a_slot[p]);
        used_b.insert(g.pair_b_slot[p]);
      }
    }
  }
  og.stacked = single;
  og.swap = single && from == nullptr && !tiled_out && used_a.size() < used_b.size();
  og.tiled_out = tiled_out;
  og.tiled_in = from != nullptr;
  if (tiled_out && !single) throw Error(kInternal, "sliced gemm plan: a tiled result needs stacked panels");
  std::vector<DOzTiled> place, pairs_tiled;  // by block slot of a; by pair
  if (from != nullptr) {
    place.assign(a.tags.size(), DOzTiled{0, 0, 0});
    for (size_t ti = 0; ti < from_plan->task_ctag.size(); ++ti) {
      const int32_t s = a.find(from_plan->task_ctag[ti]);
      if (s < 0) throw Error(kInternal, "sliced gemm plan: tiled block missing");
      place[s] = from->task_place[ti];
    }
    for (size_t p = 0; p < g.h_pairs.size(); ++p) {
      pairs_tiled.push_back(place[g.pair_a_slot[p]]);
      if (pairs_tiled.back().ntn == 0) throw Error(kInternal, "sliced gemm plan: tiled block without a place");
    }
    single = false;  // block by block
    og.stacked = false;
  }
  const Tensor& ra = og.swap ? b : a;
  const Tensor& rb = og.swap ? a : b;
  const std::vector<View>& vra = og.swap ? vb : va;
  const std::vector<View>& vrb = og.swap ? va : vb;
  auto slot_a = [&](int p) { return og.swap ? g.pair_b_slot[p] : g.pair_a_slot[p]; };
  auto slot_b = [&](int p) { return og.swap ? g.pair_a_slot[p] : g.pair_b_slot[p]; };
  std::vector<DOzScaleBlock> scale_blocks;
  std::vector<int> sa, sb;  // by block slot: first power of two of the block's contraction
  const int nscales = balance(og, bal, a, b, sa, sb, scale_blocks);
  const std::vector<int>& sra = og.swap ? sb : sa;
  const std::vector<int>& srb = og.swap ? sa : sb;
  og.a.sign = og.swap ? -bal.sign_a : bal.sign_a;
  og.b.sign = -og.a.sign;
  pack_blocks(og.b, rb, vrb, srb, false);
  std::vector<DOzPair> pairs;
  std::vector<int64_t> row_map;
  if (!single) {
    pack_blocks(og.a, ra, vra, sra, true, from != nullptr ? &place : nullptr);
    pairs.resize(g.h_pairs.size());
    for (size_t p = 0; p < pairs.size(); ++p) {
      const int32_t as = slot_a(static_cast<int>(p)), bs = slot_b(static_cast<int>(p));
      if (og.a.nks[as] != og.b.nks[bs] || sra[as] != srb[bs])
        throw Error(kInternal, "sliced gemm plan: operand packing mismatch");
      pairs[p] = DOzPair{og.a.base[as], og.b.base[bs], og.a.exp0[as], og.b.exp0[bs], og.a.nks[as], 0};
    }
    make_tiles(g, kOzTileM, kOzTileN, og.h_tiles, og.h_reduce, og.nslots, kOzTargetTiles);
    for (DTile& t : og.h_tiles) {
      t.h64 = oz_tile_rows(g.h_tasks[t.task].m, t.tm);
      t.nt = oz_tail_cols(g.h_tasks[t.task].n, t.tn);
    }
  } else {
    std::map<int32_t, std::vector<int>> panels;  // column operand block -> tasks in order
    for (size_t ti = 0; ti < g.h_tasks.size(); ++ti)
      panels[slot_b(g.h_tasks[ti].p0)].push_back(static_cast<int>(ti));
    OzOperand& o = og.a;
    for (const auto& kv : panels) {
      const View& vc = vrb[kv.first];
      int64_t rows = 0;
      for (int ti : kv.second) rows += vra[slot_a(g.h_tasks[ti].p0)].rows;
      if (rows > (int64_t(1) << 30) || row_map.size() + rows > 0x7fffff00)
        throw Error(kInternal, "sliced gemm plan: panel too tall");
      const int R = static_cast<int>(rows), panel = static_cast<int>(pairs.size());
      pairs.push_back(DOzPair{o.bytes, og.b.base[kv.first], o.rows, og.b.exp0[kv.first], slices(vc.k),
                              static_cast<int>(row_map.size())});
      const int ntn = (vc.rows + kOzTileN - 1) / kOzTileN;
      if (tiled_out) {
        og.task_place.resize(g.h_tasks.size());
        int at = 0;
        for (int ti : kv.second) {
          og.task_place[ti] = DOzTiled{og.tiled_elems, ntn, at};
          at += vra[slot_a(g.h_tasks[ti].p0)].rows;
        }
        pairs_tiled.push_back(DOzTiled{og.tiled_elems, ntn, 0});
        og.tiled_elems += int64_t((R + kOzTileM - 1) / kOzTileM) * ntn * (kOzTileM * kOzTileN);
      }
      for (int ti : kv.second)
        for (int r = 0; r < vra[slot_a(g.h_tasks[ti].p0)].rows; ++r)
          row_map.push_back((int64_t(ti) << 32) | int64_t(r));
      for (int tr = 0; tr * kOzTileM < R; ++tr) {
        const int rt = oz_tile_rows(R, tr);
        for (int tn = 0; tn < ntn; ++tn)
          og.h_tiles.push_back(DTile{kv.second[0], tr, tn, panel, panel + 1, -1, rt, oz_tail_cols(vc.rows, tn)});
        if (tr * kOzTileM + rt > R)  // padding rows of the last tile
          row_map.insert(row_map.end(), tr * kOzTileM + rt - R, -1);
      }
      size_t j0 = 0;  // first task that reaches the next rows, and its first panel row
      int first = 0;
      pack_rows(o, R, vc.k, srb[kv.first], true, [&](int lo, int hi) {
        while (j0 < kv.second.size() && first + vra[slot_a(g.h_tasks[kv.second[j0]].p0)].rows <= lo)
          first += vra[slot_a(g.h_tasks[kv.second[j0++]].p0)].rows;
        int at = first;
        for (size_t j = j0; j < kv.second.size() && at < hi; ++j) {
          const int32_t as = slot_a(g.h_tasks[kv.second[j]].p0);
          const View& v = vra[as];
          if (v.k != vc.k || sra[as] != srb[kv.first]) throw Error(kInternal, "sliced gemm plan: panel shapes differ");
          const int x = std::max(at, lo), y = std::min(at + v.rows, hi);
          if (x < y)
            o.h_segs.push_back(DOzSeg{ra.offsets[as] + int64_t(x - at) * v.rstride, x - lo, y - x, v.rstride, v.kstride});
          at += v.rows;
        }
      });
    }
  }
  // Tiles to CTAs, heaviest first to the least loaded one: about 8 units (100 clocks) for a
  // K step of a 32-column tile, 6 of a 16-column one, 6 for a group's hand-over.
  std::vector<std::pair<int64_t, int>> order(og.h_tiles.size());
  for (size_t i = 0; i < order.size(); ++i) {
    const DTile& t = og.h_tiles[i];
    int64_t w = 6;
    for (int p = t.p0; p < t.p1; ++p)
      w += int64_t(pairs[p].nks) * (t.nt == kOzTileN ? 8 : 6) + 6 * ((pairs[p].nks + kOzGroupSteps - 1) / kOzGroupSteps);
    order[i] = {-w, static_cast<int>(i)};
  }
  std::stable_sort(order.begin(), order.end());
  int nsm = 0;
  cuda_check(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx.device), "multiprocessor count");
  const int ncta = std::min<int>(std::max(nsm, 1), static_cast<int>(order.size()));
  std::vector<std::vector<int>> list(ncta);
  std::vector<std::pair<int64_t, int>> heap;  // (-load, -CTA): the least loaded on top
  for (int c = 0; c < ncta; ++c) heap.push_back({0, -c});
  std::make_heap(heap.begin(), heap.end());
  for (const auto& o : order) {
    std::pop_heap(heap.begin(), heap.end());
    list[-heap.back().second].push_back(o.second);
    heap.back().first += o.first;
    std::push_heap(heap.begin(), heap.end());
  }
  std::vector<DTile> sorted;
  sorted.reserve(order.size());
  og.h_cta_ptr.assign(1, 0);
  for (const auto& l : list) {
    for (int i : l) sorted.push_back(og.h_tiles[i]);
    og.h_cta_ptr.push_back(static_cast<int>(sorted.size()));
  }
  og.h_tiles.swap(sorted);
  const std::vector<int> none{0};
  const std::vector<int8_t> zeros(nscales, 0);
  Upload up;
  up.add(og.scale_tasks, og.h_scale_tasks);
  up.add(og.scale_blocks, scale_blocks);
  up.add(og.scales, zeros);
  up.add(og.tiles, og.h_tiles);
  up.add(og.cta_ptr, og.h_cta_ptr);
  up.add(og.pairs_tiled, pairs_tiled);
  up.add(og.pairs, pairs);
  up.add(og.row_map, row_map);
  up.add(og.reduce, og.h_reduce);
  for (OzOperand* o : {&og.a, &og.b}) {
    up.add(o->packs, o->h_packs);
    up.add(o->segs, o->h_segs);
    up.add(o->flag, none);
  }
  up.run(og.arrays, ctx.stream);
  og.built = true;
}

bool oz_wanted(const Context& ctx, double flops) {
  return flops >= (ctx.oz_min_flops >= 0.0 ? ctx.oz_min_flops : kOzMinFlops);
}

bool oz_reserve(Context& ctx, const std::vector<OzGemm*>& gs, const std::function<OzScratch()>& build) {
  try {
    const OzScratch scratch = build();
    bool held = true;
    size_t digits = 0, part = 16;
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    for (OzGemm* g : gs) {
      for (OzOperand* o : {&g->a, &g->b}) {
        held = held && o->digits != nullptr;
        digits += up(o->bytes + 16) + up(o->rows * sizeof(int) + 16);
      }
      part = std::max(part, g->partial_bytes());
    }
    size_t need = (held || ctx.oz_mem.capacity() >= digits ? 0 : digits) + (ctx.gemm_part.cap < part ? part : 0);
    if (scratch.buf && scratch.buf->cap < scratch.bytes) need += scratch.bytes;
    if (need > kOzSmallBytes) {
      size_t free_b = 0, total_b = 0;
      cuda_check(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
      const size_t have = free_b + block_cache_bytes();
      if (need > have - have / 8) return false;
    }
    ctx.gemm_part.ensure(part, ctx.stream);
    if (scratch.buf) scratch.buf->ensure(std::max<size_t>(scratch.bytes, 16), ctx.stream);
    if (held) return true;
    uint8_t* at = static_cast<uint8_t*>(ctx.oz_mem.take(digits, ctx.stream));
    for (OzGemm* g : gs)
      for (OzOperand* o : {&g->a, &g->b}) {
        o->drop();
        o->digits = at;
        at += up(o->bytes + 16);
        o->exps = reinterpret_cast<int*>(at);
        at += up(o->rows * sizeof(int) + 16);
      }
  } catch (const Error& e) {
    if (e.code != kAlloc) throw;
    return false;
  }
  return true;
}

OzCall::~OzCall() {
  a_.drop();
  b_.drop();
  ctx_.oz_mem.park();
}

void oz_pack(Context& ctx, const std::vector<OzSource>& what) {
  if (what.size() > kOzPackJobs) throw Error(kInternal, "sliced gemm: too many operands in one packing");
  OzPackJobs jobs{};
  for (const OzSource& w : what) {
    OzOperand& o = *w.o;
    jobs.job[jobs.n++] = OzPackJob{o.packs.get(), o.segs.get(), w.src, o.digits, o.exps, o.flag.get(),
                                   static_cast<int>(o.h_packs.size()), o.seq + 1,
                                   w.balance ? w.balance->scales.get() : nullptr, o.sign};
  }
  launch_oz_pack(jobs, ctx.stream);
  for (const OzSource& w : what) {
    ++w.o->seq;
    w.o->cut = w.balance == nullptr;
  }
  ctx.kernel_launches += 1;
}

void oz_scale(Context& ctx, const std::vector<std::pair<OzGemm*, const double*>>& what) {
  OzScaleJobs jobs{};
  for (const auto& w : what)
    jobs.job[jobs.n++] = OzScaleJob{w.first->scale_tasks.get(), w.first->scale_blocks.get(), w.second,
                                    w.first->scales.p, static_cast<int>(w.first->h_scale_tasks.size())};
  launch_oz_scale(jobs, ctx.stream);
  ctx.kernel_launches += 1;
}

void run_oz_gemm(Context& ctx, OzGemm& og, const GemmPlan& g, double alpha, const double* A, const double* B, double* C,
                 bool assign) {
  OzGemmArgs a{};
  a.Apk = og.a.digits;
  a.Bpk = og.b.digits;
  a.Aexp = og.a.exps;
  a.Bexp = og.b.exps;
  a.flag_a = og.a.flag.get();
  a.flag_b = og.b.flag.get();
  a.seq_a = og.a.seq;
  a.seq_b = og.b.seq;
  a.tiles = og.tiles.get();
  a.cta_ptr = og.cta_ptr.get();
  a.nctas = static_cast<int>(og.h_cta_ptr.size()) - 1;
  a.pairs_tiled = og.pairs_tiled.get();
  a.tiled_out = og.tiled_out;
  a.tiled_in = og.tiled_in;
  a.tasks = g.dtasks.get();
  a.pairs = og.pairs.get();
  a.row_map = og.stacked ? og.row_map.get() : nullptr;
  a.alpha = alpha;
  a.C = C;
  a.partial = ctx.gemm_part.as<double>();
  a.swap = og.swap;
  a.assign = assign;
  a.err = device_err_flag(ctx);
  a.timeout_ns = ctx.device_timeout_ns;
  a.A = A;
  a.B = B;
  a.fpairs = g.pairs.get();
  a.ta = g.ta == kTrans;
  a.tb = g.tb == kTrans;
  launch_gemm_oz(a, ctx.stream);
  launch_oz_reduce(og.reduce.get(), static_cast<int>(og.h_reduce.size()), a, ctx.stream);
  ctx.kernel_launches += 1 + !og.h_reduce.empty();
}

}  // namespace mpsxx
