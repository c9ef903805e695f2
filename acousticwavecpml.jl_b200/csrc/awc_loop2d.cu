// awc_loop2d.cu — tiling and launches of the on-chip 2D time loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "awc_loop2d.cuh"
#include "awc_loop2d.h"

namespace awc {
namespace {

#define LOOP_TRY(ctx, call)                                                               \
  do {                                                                                    \
    const cudaError_t e_ = (call);                                                        \
    if (e_ != cudaSuccess) {                                                              \
      cudaGetLastError();                                                                 \
      return awc::fail(ctx, e_ == cudaErrorMemoryAllocation ? AWC_ERR_OOM : AWC_ERR_CUDA, \
                       cudaGetErrorString(e_));                                           \
    }                                                                                     \
  } while (0)

constexpr int kMaxSmem = 227 * 1024;

int32_t first_right(int64_t n, int64_t h) { return (int32_t)std::max<int64_t>(n - h - 1, h + 1); }

template <typename T>
const void* loop_kernel(int R) {
  switch (R) {
    case 1: return (const void*)loop2d<T, 1>;
    case 2: return (const void*)loop2d<T, 2>;
    case 3: return (const void*)loop2d<T, 3>;
    case 4: return (const void*)loop2d<T, 4>;
    case 5: return (const void*)loop2d<T, 5>;
    case 6: return (const void*)loop2d<T, 6>;
    default: return (const void*)loop2d<T, 8>;
  }
}

// The bands of one axis share no face (a face between a left-band and a
// right-band node would carry two ψ).
bool bands_apart(int64_t n, int64_t h, const int32_t* active) {
  return !(active[0] && active[1]) || n > 2 * h + 2;
}

}  // namespace

bool Loop2D::Shape::operator==(const Shape& o) const {
  return nx == o.nx && ny == o.ny && halo == o.halo && !std::memcmp(active, o.active, sizeof active);
}

Loop2D::~Loop2D() {
  if (blob_) cudaFree(blob_);
  if (table_) cudaFree(table_);
  if (mail_) cudaFree(mail_);
}

namespace {

// Relative cost of one vector of nodes: a plain one, and what an x band and a y
// band add (instructions, counted from the operations).
constexpr int kRow = 45, kRowX = 110, kRowY = 90;

// A tile's rows: y-band rows, plain rows, y-band rows.
struct Rows {
  int n[3] = {};
  int all() const { return n[0] + n[1] + n[2]; }
  bool operator==(const Rows& o) const { return n[0] == o.n[0] && n[1] == o.n[1] && n[2] == o.n[2]; }
};
// The kinds of rows y0 .. y0 + h - 1 of a shot.
Rows tile_rows(int y0, int h, int64_t ny, int halo, const int32_t* active) {
  const BandSlots b = band_slots(y0, h, 1, (int)ny, halo, first_right(ny, halo), active[0] != 0, active[1] != 0);
  Rows r;
  r.n[0] = b.na;
  r.n[2] = b.nb;
  r.n[1] = h - b.na - b.nb;
  return r;
}
// Rows per thread of a tile of cw vector columns and h rows: the fewest that
// need at most LOOP_NT threads (0: more than LOOP_ROWS).
int thread_rows(int cw, int h) {
  const int runs = LOOP_NT / cw;
  if (runs == 0) return 0;
  const int k = (h + runs - 1) / runs;
  return k <= LOOP_ROWS ? k : 0;
}
int band_vectors(int cw, int nvx, const Rows& y) { return nvx * y.all() + (y.n[0] + y.n[2]) * (cw - nvx); }

// Estimated cycles of one step of a tile. A plain row costs a warp about 50
// instructions, 5.5 cycles each when the block has few warps to hide them and
// 1.7 of an issue slot when it has many; a round of band vectors (one per
// thread) 800 to 1600 cycles. Edges sent after the update are waited for, 1700
// cycles; sent before it they cost a round themselves.
double step_cost(int cw, int nvx, const Rows& y, bool exchange) {
  const int h = y.all(), k = thread_rows(cw, h), nb = band_vectors(cw, nvx, y);
  const int threads = (cw * ((h + k - 1) / k) + 31) / 32 * 32;
  const double chain = 5.5 * (60.0 + 50.0 * k);
  const double issue = 1.7 / 4.0 * (threads / 32 * 60.0 + cw * (double)h / 32.0 * 50.0);
  const double rounds = (nb + threads - 1) / threads;
  const double band = nb == 0 ? 0.0 : k == 1 ? 800.0 : 150.0 + 1100.0 * rounds;
  const bool early = k >= LOOP_EARLY_R && 2 * (cw + h) <= threads;
  const double edge = !exchange ? 0.0 : (early ? 1300.0 : 1900.0) + 2.0 * cw + 4.0 * h;
  return 300.0 + std::max(chain, issue) + band + edge;
}

// Cuts n units of the given costs into `parts` consecutive parts of about equal
// cost (tiles of the bands get fewer nodes: the slowest tile sets the pace);
// the parts' first units and n. Empty when a part would have no unit.
std::vector<int> split(const std::vector<int>& cost, int parts) {
  const int n = (int)cost.size();
  int64_t total = 0;
  for (int c : cost) total += c;
  std::vector<int> at{0};
  int64_t have = 0, share = total / parts;
  for (int u = 0; u < n && (int)at.size() < parts; ++u) {
    // the cut nearest to the next equal share
    if (u > at.back() && (have >= share || share - have < have + cost[u] - share)) {
      at.push_back(u);
      share = total * (int64_t)at.size() / parts;
    }
    have += cost[u];
  }
  if ((int)at.size() != parts) return {};
  at.push_back(n);
  return at;
}
// Costs of the vector columns and of the interior rows of a shot.
std::vector<int> column_costs(int64_t nx, int halo, const int32_t* active, int V) {
  const int cv = (int)((nx + V - 1) / V);
  std::vector<int> c((size_t)cv, kRow);
  const BandSlots b = band_slots(0, cv * V, V, (int)nx, halo, first_right(nx, halo), active[0] != 0, active[1] != 0);
  for (int u = 0; u < cv; ++u)
    if (b.slot(u) >= 0) c[u] += kRowX;
  return c;
}
std::vector<int> row_costs(int64_t ny, int halo, const int32_t* active) {
  const Rows y = tile_rows(1, (int)ny - 2, ny, halo, active);
  std::vector<int> c((size_t)ny - 2, kRow + kRowY);
  std::fill(c.begin() + y.n[0], c.begin() + y.n[0] + y.n[1], kRow);
  return c;
}

// Byte offsets of a tile's shared memory (`rows`: the most rows per thread of
// its launch); returns the total.
template <typename T>
int tile_smem(LoopTile& L, int rows) {
  constexpr int V = 16 / (int)sizeof(T);
  int64_t o = 0;
  auto take = [&](int64_t bytes) {
    const int64_t at = o;
    o += (bytes + 15) / 16 * 16;
    return (int32_t)at;
  };
  const int64_t field = (int64_t)(L.h + rows + 1) * (L.w + 2 * V) * (int64_t)sizeof(T);
  const int64_t nb = L.nband, nx = (int64_t)L.nvx * L.h, nyv = (int64_t)(L.ny0 + L.ny1) * (L.w / V);
  L.f[0] = take(field);
  L.f[1] = take(field);
  L.cx = take(4 * (L.w + V) * (int64_t)sizeof(T));
  L.cy = take(4 * ((L.h + V) / V * V) * (int64_t)sizeof(T));
  L.bt = take(4 * nb);
  L.bf = take(16 * nb);
  L.px = take(16 * nx);
  L.px0 = take((int64_t)sizeof(T) * nx);
  L.xx = take(16 * nx);
  L.ylo = take(16 * nyv);
  L.yhi = take(16 * nyv);
  L.xy = take(16 * nyv);
  return (int)std::min<int64_t>(o, 1 << 30);
}

}  // namespace

// The cheapest tiling of a shot for every number of tiles up to max_tiles.
std::vector<Loop2D::Tiling> Loop2D::tilings(const Shape& s, bool f64, int max_tiles, bool even) {
  const int V = f64 ? 2 : 4;
  std::vector<Tiling> best(max_tiles + 1);
  const int cv = (int)((s.nx + V - 1) / V), rows = (int)s.ny - 2;
  const int fx = first_right(s.nx, s.halo);
  std::vector<int> ccost = column_costs(s.nx, s.halo, s.active[0], V), rcost = row_costs(s.ny, s.halo, s.active[1]);
  if (even) {
    std::fill(ccost.begin(), ccost.end(), 1);
    std::fill(rcost.begin(), rcost.end(), 1);
  }
  // cuts of the rows into ty parts with the parts' distinct row patterns: the
  // same for every tx
  struct Cut {
    std::vector<int> yb;
    std::vector<Rows> ys;
    bool done = false;
  };
  std::vector<Cut> cuts(max_tiles + 1);
  auto cut = [&](int ty) -> const Cut& {
    Cut& c = cuts[ty];
    if (c.done) return c;
    c.done = true;
    c.yb = split(rcost, ty);
    for (int t = 0; t < ty && !c.yb.empty(); ++t) {
      const Rows y = tile_rows(1 + c.yb[t], c.yb[t + 1] - c.yb[t], s.ny, s.halo, s.active[1]);
      if (std::find(c.ys.begin(), c.ys.end(), y) == c.ys.end()) c.ys.push_back(y);
    }
    return c;
  };
  std::vector<double> fewer(max_tiles + 1, 1e30);  // lowest cost of fewer tiles so far
  for (int tx = 1; tx <= max_tiles && tx <= cv; ++tx) {
    const std::vector<int> xb = split(ccost, tx);
    // a last tile that starts on the Dirichlet column would send it as its edge
    if (xb.empty() || (tx > 1 && (int64_t)xb[tx - 1] * V >= s.nx - 1)) continue;
    int wide = 0;
    std::vector<std::pair<int, int>> cols;  // distinct (vectors, x-band vectors) of the tile columns
    for (int t = 0; t < tx; ++t) {
      const int ct = xb[t + 1] - xb[t];
      wide = std::max(wide, ct);
      const BandSlots b = band_slots(xb[t] * V, ct * V, V, (int)s.nx, s.halo, fx, s.active[0][0] != 0, s.active[0][1] != 0);
      const std::pair<int, int> k{ct, b.na + b.nb};
      if (std::find(cols.begin(), cols.end(), k) == cols.end()) cols.push_back(k);
    }
    if (wide > LOOP_NT) continue;
    // tile rows: from the fewest that blocks of full threads allow
    const int hmax = LOOP_NT / wide * LOOP_ROWS;
    const int ty_lo = (rows + hmax - 1) / hmax, ty_hi = std::min(max_tiles / tx, rows);
    for (int ty = ty_lo; ty <= ty_hi; ++ty) {
      const std::vector<int>& yb = cut(ty).yb;
      const std::vector<Rows>& ys = cut(ty).ys;
      if (yb.empty()) continue;
      const int k = tx * ty;
      double cost = 0.0;
      bool ok = true;
      for (const auto& c : cols)
        for (const auto& y : ys) {
          if (!ok) break;
          if (thread_rows(c.first, y.all()) == 0) {
            ok = false;
            break;
          }
          cost = std::max(cost, step_cost(c.first, c.second, y, k > 1));
          // not better than another tiling of k tiles, or worse than one of fewer
          if (cost >= best[k].cost || cost > fewer[k]) {
            ok = false;
            break;
          }
          LoopTile L{};
          L.w = c.first * V;
          L.h = y.all();
          L.nvx = c.second;
          L.ny0 = y.n[0];
          L.ny1 = y.n[2];
          L.nband = band_vectors(c.first, c.second, y);
          ok = (f64 ? tile_smem<double>(L, LOOP_ROWS) : tile_smem<float>(L, LOOP_ROWS)) <= kMaxSmem;
        }
      if (!ok) continue;
      Tiling& t = best[k];
      t.tx = tx;
      t.ty = ty;
      t.xb = xb;
      t.yb = yb;
      t.cost = cost;
      for (int q = k + 1; q <= max_tiles && fewer[q] > cost; ++q) fewer[q] = cost;
    }
  }
  for (int k = 2; k <= max_tiles; ++k)  // at most k tiles
    if (best[k - 1].cost < best[k].cost) best[k] = best[k - 1];
  // tiles of equal cost leave the inner ones larger: a shot near the chip's
  // capacity fits in tiles of equal size only
  if (!even && best[max_tiles].tx == 0) return tilings(s, f64, max_tiles, true);
  return best;
}

// Waves: shots packed (largest first) into as few launches as their smallest
// tilings allow, then every wave's shots get the tile counts that minimise
// its slowest shot's step.
bool Loop2D::plan_waves(const awc_ctx* C) {
  const int S = C->loop_blocks, ns = (int)shapes_.size(), V = f64_ ? 2 : 4;
  if (S < 1) return false;
  for (const Shape& sh : shapes_) {
    // a quick bound before the search: every block's threads and rows
    if (!bands_apart(sh.nx, sh.halo, sh.active[0]) || !bands_apart(sh.ny, sh.halo, sh.active[1]) ||
        (sh.nx + V - 1) / V * (sh.ny - 2) > (int64_t)S * LOOP_NT * LOOP_ROWS)
      return false;
  }
  std::vector<std::vector<Tiling>> tab;  // per shot; shots of one shape share the search
  for (int s = 0; s < ns; ++s) {
    int same = -1;
    for (int q = 0; q < s && same < 0; ++q)
      if (shapes_[q] == shapes_[s]) same = q;
    if (same >= 0)
      tab.push_back(tab[same]);
    else
      tab.push_back(tilings(shapes_[s], f64_, S));
    if (tab[s][S].tx == 0) return false;
  }
  auto least = [&](int s) {
    int k = 1;
    while (tab[s][k].tx == 0) ++k;
    return k;
  };
  std::vector<int> order(ns);
  for (int s = 0; s < ns; ++s) order[s] = s;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return least(a) > least(b); });
  std::vector<std::vector<int>> bins;
  std::vector<int> used;
  for (int s : order) {
    const int k = least(s);
    size_t b = 0;
    while (b < bins.size() && used[b] + k > S) ++b;
    if (b == bins.size()) {
      bins.emplace_back();
      used.push_back(0);
    }
    bins[b].push_back(s);
    used[b] += k;
  }
  waves_.clear();
  for (auto& bin : bins) {
    std::vector<int> k(bin.size());
    int left = S;
    for (size_t q = 0; q < bin.size(); ++q) {
      k[q] = least(bin[q]);
      left -= k[q];
    }
    for (;;) {  // more tiles for the slowest shot while there are any left
      size_t worst = 0;
      for (size_t q = 1; q < bin.size(); ++q)
        if (tab[bin[q]][k[q]].cost > tab[bin[worst]][k[worst]].cost) worst = q;
      const auto& tb = tab[bin[worst]];
      int up = k[worst] + 1;
      while (up <= S && !(tb[up].cost < tb[k[worst]].cost)) ++up;
      if (up > S || up - k[worst] > left) break;
      left -= up - k[worst];
      k[worst] = up;
    }
    Wave w;
    for (size_t q = 0; q < bin.size(); ++q) {
      w.shots.push_back(bin[q]);
      w.tiling.push_back(tab[bin[q]][k[q]]);
    }
    waves_.push_back(std::move(w));
  }
  // the wave of the most tiles first: what the device has no room for is refused
  // before anything ran
  auto tiles = [](const Wave& w) {
    int n = 0;
    for (const Tiling& t : w.tiling) n += t.tiles();
    return n;
  };
  std::stable_sort(waves_.begin(), waves_.end(),
                   [&](const Wave& a, const Wave& b) { return tiles(a) > tiles(b); });
  return true;
}

// The tiles of every wave with their edge items (uploaded once per layout),
// mailbox sizes and launch shapes.
template <typename T>
int Loop2D::lay_out(awc_ctx* C) {
  constexpr int V = 16 / (int)sizeof(T), WPV = (int)sizeof(T) / 4;
  std::vector<LoopEdge> edges;
  tiles_.clear();
  int hm = 0, wm = 0;
  int64_t most = 0;
  int64_t count = 0;
  for (Wave& wv : waves_) {
    wv.tile0 = count;
    wv.hmax = wv.wmax = 0;
    wv.ntiles = 0;
    for (const Tiling& t : wv.tiling) {
      for (int k = 0; k < t.tx; ++k) wv.wmax = std::max(wv.wmax, (t.xb[k + 1] - t.xb[k]) * V);
      for (int k = 0; k < t.ty; ++k) wv.hmax = std::max(wv.hmax, t.yb[k + 1] - t.yb[k]);
      wv.ntiles += t.tx * t.ty;
    }
    hm = std::max(hm, wv.hmax);
    wm = std::max(wm, wv.wmax);
    most = std::max(most, wv.ntiles);
    count += wv.ntiles;
  }
  const int64_t words = 2 * (int64_t)(hm + wm) * WPV;  // a slot: four edges
  mail_stride_ = 2 * ((words + 31) / 32 * 32);
  for (Wave& wv : waves_) {
    const int oL = 0, oR = wv.hmax * WPV, oU = 2 * wv.hmax * WPV, oD = (2 * wv.hmax + wv.wmax) * WPV;
    const size_t begin = tiles_.size();
    wv.R = 1;
    wv.first.clear();
    for (size_t q = 0; q < wv.shots.size(); ++q) {
      const Shape& sh = shapes_[wv.shots[q]];
      const Tiling& t = wv.tiling[q];
      const int first = (int)(tiles_.size() - begin);
      wv.first.push_back(first);
      for (int ty = 0; ty < t.ty; ++ty)
        for (int tx = 0; tx < t.tx; ++tx) {
          LoopTile L{};
          L.shot = wv.shots[q];
          L.x0 = t.xb[tx] * V;
          L.w = (t.xb[tx + 1] - t.xb[tx]) * V;
          L.y0 = 1 + t.yb[ty];
          L.h = t.yb[ty + 1] - t.yb[ty];
          const int me = first + ty * t.tx + tx;
          L.nbr[0] = tx > 0 ? me - 1 : -1;
          L.nbr[1] = tx + 1 < t.tx ? me + 1 : -1;
          L.nbr[2] = ty > 0 ? me - t.tx : -1;
          L.nbr[3] = ty + 1 < t.ty ? me + t.tx : -1;
          const BandSlots bx = band_slots(L.x0, L.w, V, (int)sh.nx, sh.halo, first_right(sh.nx, sh.halo),
                                          sh.active[0][0] != 0, sh.active[0][1] != 0);
          const Rows y = tile_rows(L.y0, L.h, sh.ny, sh.halo, sh.active[1]);
          L.nvx = bx.na + bx.nb;
          L.ny0 = y.n[0];
          L.ny1 = y.n[2];
          L.nband = band_vectors(L.w / V, L.nvx, y);
          L.rows = thread_rows(L.w / V, L.h);
          wv.R = std::max(wv.R, L.rows);
          tiles_.push_back(L);
        }
    }
    if (wv.R == 7) wv.R = 8;  // the kernel's instances
    wv.threads = 32;
    wv.smem = 0;
    for (size_t k = begin; k < tiles_.size(); ++k) {
      const LoopTile& L = tiles_[k];
      wv.threads = std::max(wv.threads, (L.w / V * ((L.h + L.rows - 1) / L.rows) + 31) / 32 * 32);
    }
    for (size_t k = begin; k < tiles_.size(); ++k) {
      LoopTile& L = tiles_[k];
      const Shape& sh = shapes_[L.shot];
      wv.smem = std::max(wv.smem, tile_smem<T>(L, wv.R));
      const int cw = L.w / V;
      // edge items, where the update is long enough to hide the trip: at most
      // one per thread
      const int n = (L.nbr[2] >= 0 ? cw : 0) + (L.nbr[3] >= 0 ? cw : 0) + (L.nbr[0] >= 0 ? L.h : 0) +
                    (L.nbr[1] >= 0 ? L.h : 0);
      L.edge0 = (int)edges.size();
      if (wv.R < LOOP_EARLY_R || n > wv.threads) continue;
      L.nedge = n;
      const BandVecs bv{band_slots(L.x0, L.w, V, (int)sh.nx, sh.halo, first_right(sh.nx, sh.halo),
                                   sh.active[0][0] != 0, sh.active[0][1] != 0),
                        cw, L.h, L.ny0, L.ny1};
      auto item = [&](int row, int c, int nbr, int at, int what) {
        edges.push_back(LoopEdge{row << 16 | c, (int)(nbr * mail_stride_) + at, bv.index(row, c), what});
      };
      for (int c = 0; L.nbr[2] >= 0 && c < cw; ++c) item(0, c, L.nbr[2], oD + c * V * WPV, 0);
      for (int c = 0; L.nbr[3] >= 0 && c < cw; ++c) item(L.h - 1, c, L.nbr[3], oU + c * V * WPV, 0);
      for (int r = 0; L.nbr[0] >= 0 && r < L.h; ++r) item(r, 0, L.nbr[0], oR + r * WPV, 1);
      for (int r = 0; L.nbr[1] >= 0 && r < L.h; ++r) item(r, cw - 1, L.nbr[1], oL + r * WPV, 2);
    }
  }
  for (const Wave& wv : waves_)
    LOOP_TRY(C, cudaFuncSetAttribute(loop_kernel<T>(wv.R), cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
  const size_t eb = edges.size() * sizeof(LoopEdge);
  if (table_) cudaFree(table_);
  table_ = nullptr;
  LOOP_TRY(C, cudaMalloc(&table_, eb + 16));
  if (eb) LOOP_TRY(C, cudaMemcpyAsync(table_, edges.data(), eb, cudaMemcpyHostToDevice, C->stream));
  if (mail_) cudaFree(mail_);
  mail_ = nullptr;
  mail_bytes_ = (size_t)(mail_stride_ * most) * 8;
  LOOP_TRY(C, cudaMalloc((void**)&mail_, mail_bytes_));
  LOOP_TRY(C, cudaMemsetAsync(mail_, 0, mail_bytes_, C->stream));
  tag_ = 1;
  LOOP_TRY(C, cudaStreamSynchronize(C->stream));  // host vectors go out of scope
  return AWC_OK;
}

// The shots' descriptors and their source and receiver lists.
template <typename T>
int Loop2D::upload(awc_ctx* C, const std::vector<LoopShotHost>& shots) {
  constexpr int V = 16 / (int)sizeof(T);
  std::vector<LoopTile> tiles = tiles_;
  std::vector<LoopShot<T>> descs(shots.size());
  std::vector<LoopSrc> srcs;
  std::vector<LoopRec> recs;
  for (size_t s = 0; s < shots.size(); ++s) {
    const LoopShotHost& H = shots[s];
    LoopShot<T>& D = descs[s];
    for (int b = 0; b < 3; ++b) D.buf[b] = (T*)H.buf[b];
    D.fact = (const T*)H.fact;
    const int64_t h = H.halo;
    for (int a = 0; a < 2; ++a) {
      const T* blk = (const T*)H.coef + a * (8 * h + 4);
      for (int sd = 0; sd < 2; ++sd) {
        for (int q = 0; q < 2; ++q) D.psi[a][sd][q] = (T*)H.psi[a][sd][q];
        BandSide<T>& B = D.band[a][sd];
        B.psi_old = nullptr;
        B.psi_new = nullptr;
        B.xi = (T*)H.xi[a][sd];
        B.a = blk + sd * h;
        B.bK = blk + 2 * h + sd * h;
        B.ah = blk + 4 * h + sd * (h + 1);
        B.bKh = blk + 4 * h + 2 * (h + 1) + sd * (h + 1);
        D.active[a][sd] = H.active[a][sd];
      }
      D.first_r[a] = first_right(a == 0 ? H.nx : H.ny, h);
      D.inv_d[a] = (T)H.inv_d[a];
      D.inv_d2[a] = (T)H.inv_d2[a];
    }
    D.nx = (int32_t)H.nx;
    D.ny = (int32_t)H.ny;
    D.halo = H.halo;
    D.px = H.px;
    D.src_off = H.src_off;
    D.src_ids = H.src_ids;
    D.stf = (const T*)H.stf;
    D.traces = (T*)H.traces;
    D.nsrc = H.nsrc;
    D.nrec = H.nrec;
  }
  for (const Wave& wv : waves_)
    for (size_t q = 0; q < wv.shots.size(); ++q) {
      const LoopShotHost& H = shots[wv.shots[q]];
      const Tiling& t = wv.tiling[q];
      const size_t base = (size_t)wv.tile0 + wv.first[q];
      // sources and receivers by tile; the cell of node (i, j) in its tile
      std::vector<std::vector<LoopSrc>> ts(t.tiles());
      std::vector<std::vector<LoopRec>> tr(t.tiles());
      for (const IoRim& e : *H.nodes) {
        const int64_t i = e.node % H.px, j = e.node / H.px;
        const int64_t jc = std::min<int64_t>(std::max<int64_t>(j, 1), H.ny - 2);
        const int tx = (int)(std::upper_bound(t.xb.begin(), t.xb.end(), (int)(i / V)) - t.xb.begin()) - 1;
        const int ty = (int)(std::upper_bound(t.yb.begin(), t.yb.end(), (int)(jc - 1)) - t.yb.begin()) - 1;
        const size_t n = (size_t)ty * t.tx + tx;
        LoopTile& L = tiles[base + n];
        const int pitch = L.w + 2 * V, c = (int)(i - L.x0), r = (int)(jc - L.y0);
        const int cell = (int)(j - L.y0 + 1) * pitch + c + V;
        const bool in = i >= 1 && i <= H.nx - 2 && j >= 1 && j <= H.ny - 2;
        if (e.sgrp >= 0) {
          // a source on an edge node: this tile sends its edges after the update
          if (r == 0 || r == L.h - 1 || c == 0 || c == L.w - 1) L.nedge = 0;
          ts[n].push_back(LoopSrc{r / L.rows * (L.w / V) + c / V, cell, e.sgrp,
                                  in ? (int64_t)-1 : e.node});
        }
        if (e.rgrp >= 0)
          for (int32_t k = (*H.rec_off)[e.rgrp]; k < (*H.rec_off)[e.rgrp + 1]; ++k)
            tr[n].push_back(LoopRec{cell, (*H.rec_ids)[k]});
      }
      for (size_t n = 0; n < ts.size(); ++n) {
        LoopTile& L = tiles[base + n];
        std::stable_sort(ts[n].begin(), ts[n].end(),
                         [](const LoopSrc& a, const LoopSrc& b) { return a.owner < b.owner; });
        L.src[0] = (int)srcs.size();
        srcs.insert(srcs.end(), ts[n].begin(), ts[n].end());
        L.src[1] = (int)srcs.size();
        L.rec[0] = (int)recs.size();
        recs.insert(recs.end(), tr[n].begin(), tr[n].end());
        L.rec[1] = (int)recs.size();
      }
    }
  // one blob: tiles, shots, lists (256-byte aligned parts)
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  o_shots_ = up(tiles.size() * sizeof(LoopTile));
  o_srcs_ = o_shots_ + up(descs.size() * sizeof(LoopShot<T>));
  o_recs_ = o_srcs_ + up(srcs.size() * sizeof(LoopSrc));
  const size_t total = o_recs_ + up(recs.size() * sizeof(LoopRec)) + 256;
  std::vector<unsigned char> host(total, 0);
  auto put = [&](size_t at, const void* src, size_t bytes) {
    if (bytes) std::memcpy(host.data() + at, src, bytes);
  };
  put(0, tiles.data(), tiles.size() * sizeof(LoopTile));
  put(o_shots_, descs.data(), descs.size() * sizeof(LoopShot<T>));
  put(o_srcs_, srcs.data(), srcs.size() * sizeof(LoopSrc));
  put(o_recs_, recs.data(), recs.size() * sizeof(LoopRec));
  if (blob_bytes_ < total) {
    if (blob_) cudaFree(blob_);
    blob_ = nullptr;
    blob_bytes_ = 0;
    LOOP_TRY(C, cudaMalloc(&blob_, total));
    blob_bytes_ = total;
  }
  LOOP_TRY(C, cudaMemcpyAsync(blob_, host.data(), total, cudaMemcpyHostToDevice, C->stream));
  LOOP_TRY(C, cudaStreamSynchronize(C->stream));  // host vectors go out of scope
  return AWC_OK;
}

bool Loop2D::fits(const awc_ctx* C, bool f64, const std::vector<LoopShotHost>& shots) {
  std::vector<Shape> shapes;
  for (const LoopShotHost& s : shots)
    shapes.push_back(Shape{s.nx, s.ny, s.halo,
                           {{s.active[0][0], s.active[0][1]}, {s.active[1][0], s.active[1][1]}}});
  if (planned_ && f64 == f64_ && blocks_ == C->loop_blocks && shapes == shapes_)
    return !waves_.empty();
  planned_ = true;
  laid_out_ = false;
  f64_ = f64;
  blocks_ = C->loop_blocks;
  shapes_ = std::move(shapes);
  waves_.clear();
  if (!plan_waves(C)) waves_.clear();
  return !waves_.empty();
}

int Loop2D::prepare(awc_ctx* C, bool f64, const std::vector<LoopShotHost>& shots, int32_t* err_flag) {
  if (!fits(C, f64, shots)) return awc::fail(C, AWC_ERR_INVALID, "internal: the 2D loop does not fit");
  err_ = err_flag;
  if (!laid_out_) {
    if (int rc = f64 ? lay_out<double>(C) : lay_out<float>(C)) return rc;
    laid_out_ = true;
  }
  return f64 ? upload<double>(C, shots) : upload<float>(C, shots);
}

template <typename T>
int Loop2D::launch(awc_ctx* C, const LoopSpan& span, cudaStream_t st) {
  for (const Wave& wv : waves_) {
    if (span.n > 0x7fffffff - 8 || (uint64_t)tag_ + (uint64_t)span.n >= 0xfffffff0ull) {
      // tags would run out: start them again on clean mailboxes
      LOOP_TRY(C, cudaMemsetAsync(mail_, 0, mail_bytes_, st));
      tag_ = 1;
    }
    LoopRun<T> Q{};
    const unsigned char* b = (const unsigned char*)blob_;
    Q.tiles = (const LoopTile*)b + wv.tile0;
    Q.edges = (const LoopEdge*)table_;
    Q.shots = (const LoopShot<T>*)(b + o_shots_);
    Q.srcs = (const LoopSrc*)(b + o_srcs_);
    Q.recs = (const LoopRec*)(b + o_recs_);
    Q.mail = mail_;
    Q.mail_stride = mail_stride_;
    Q.hmax = wv.hmax;
    Q.wmax = wv.wmax;
    for (int q = 0; q < 3; ++q) {
      Q.in[q] = span.in[q];
      Q.out[q] = span.out[q];
    }
    Q.par_in = span.par_in;
    Q.par_out = span.par_out;
    Q.n = (int32_t)span.n;
    Q.it0 = span.it0;
    Q.tag0 = tag_;
    Q.keep = (T*)span.keep;
    Q.keep_stride = span.keep_stride;
    Q.keep_first = span.keep_first;
    Q.keep_count = span.keep_count;
    Q.err = err_;
    Q.wait_ns = span.wait.ns;
    Q.withhold = span.wait.withhold;
    tag_ += (uint32_t)span.n;
    const void* k = loop_kernel<T>(wv.R);
    void* args[] = {&Q};
    const cudaError_t e = cudaLaunchCooperativeKernel(k, dim3((unsigned)wv.ntiles), dim3((unsigned)wv.threads),
                                                      args, (size_t)wv.smem, st);
    if (&wv == &waves_.front() &&
        (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported)) {
      cudaGetLastError();
      waves_.clear();
      return kLoopRefused;
    }
    LOOP_TRY(C, e);
  }
  return AWC_OK;
}

int Loop2D::run(awc_ctx* C, const LoopSpan& span, cudaStream_t st) {
  return f64_ ? launch<double>(C, span, st) : launch<float>(C, span, st);
}

}  // namespace awc
