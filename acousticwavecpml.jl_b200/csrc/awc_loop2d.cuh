// awc_loop2d.cuh — the 2D time loop of whole shots in one launch, with the
// fields held on the chip.
//
// A one-launch-per-step kernel (step2d, step2d_batch*) moves every field
// through L2 or HBM each step and pays a kernel boundary per step: on one
// B200, 3.1 us per step at 241 x 241 in FP64, 7.8 us at 1573 x 787 and 11.6 us
// at 2088 x 1044 in FP32. Here the grid of a shot is cut into tiles, one block
// per tile and per SM; a block keeps its tile's p_t and p_{t-1} (in place of
// which p_{t+1} is written) in shared memory, its fact values in registers and
// the ψ/ξ of its CPML nodes in shared memory, and steps nt times: 1.8, 2.3 and
// 4.7 us per step on the same grids. What bounds it is the chain of a step, with
// at most 16 warps per SM to hide it: issue slots are 16, 37 and 31 % used on the
// three grids, and of the warps' stalls 57, 25 and 22 % are at the block's
// barriers (on small tiles behind the edges' trip through L2, 0.8 us; on full
// ones behind the rounds of band vectors, which the block's threads take after
// the update), 7, 21 and 20 % on shared memory.
// Only the tile's edge nodes leave the SM: after each step they go to the
// neighbour tiles' mailboxes in global memory (L2), every 32-bit word of a
// value paired with the step's tag in one 64-bit store, so the receiver polls
// the data word itself and no fence, flag or kernel boundary stands between
// the store and its use. A mailbox has two slots, by step parity: a tile
// writes the slot of step t + 2 only after it has received its neighbour's
// edges of step t + 1, which that neighbour sent after reading step t.
//
// The blocks wait for one another, so a launch is cooperative (every block
// resident). Every wait is bounded (LoopRun::wait_ns): a thread whose wait runs
// out sets *err and waits no more, nor does any thread that sees *err set while it
// waits; the blocks then run to the end on the edges they have, and the host
// reports the run as failed.
//
// Every node is computed with the functions the per-step kernels use
// (awc_kernels.cuh), on the same operands in the same order, so results are
// bitwise theirs, whatever the tiling.
#pragma once
#include <cstdint>
#include <cstring>

#include "awc_kernels.cuh"

namespace awc {

constexpr int LOOP_NT = 512;  // threads of a block (128 registers each)
constexpr int LOOP_ROWS = 8;  // most rows of a thread
constexpr int LOOP_EARLY_R = 3;  // rows per thread from which a tile's edges are sent first

// A receiver of a tile; a source node, served by thread `owner`, which is the
// one that updates or owns its vector. cell: index into the tile's
// shared-memory field. node: pitched index of a node on the Dirichlet rim,
// -1 for an interior one.
struct LoopRec {
  int32_t cell, id;
};
struct LoopSrc {
  int32_t owner, cell, sgrp;
  int64_t node;
};

// One tile: columns [x0, x0 + w) (x0 and w multiples of a 16-byte vector; the
// Dirichlet columns i = 0 and nx - 1 belong to the outer tiles and are
// masked), interior rows [y0, y0 + h). Built on the host with the list of its
// edge items and its shared-memory layout.
struct LoopTile {
  int32_t shot;
  int32_t x0, y0, w, h;
  int32_t nbr[4];          // tile index of the left, right, upper, lower neighbour, or -1
  int32_t rows;            // rows of a thread (the last run of a column may have fewer)
  int32_t edge0, nedge;    // edge items; none when the edges are sent after the update
  int32_t src[2], rec[2];  // ranges in the entry lists
  int32_t nvx;             // vector columns with x-band nodes
  int32_t ny0, ny1;        // y-band rows at the tile's top and bottom
  int32_t nband;           // vectors with CPML work: nvx * h of the x-band columns, row by
                           // row, then those of the y-band rows in the other columns
  // byte offsets in shared memory: the two fields; the coefficient tables
  // 4 x (w + V) and 4 x (h + V); per band vector its row << 16 | column, fact, and
  // in the x-band ones ψ
  // on the nodes' right faces, on the vector's left face (scalar) and ξ; per
  // vector of a y-band row ψ on its upper and lower faces and ξ
  int32_t f[2], cx, cy, bt, bf, px, px0, xx, ylo, yhi, xy;
};
// An edge item: one vector of the tile whose new value (all of it, or its
// first or last node) goes to mailbox word `mail`. rc: row << 16 | vector.
// band: its number among the band vectors, or -1. what: 0 all, 1 first, 2 last.
struct LoopEdge {
  int32_t rc, mail, band, what;
};

template <typename T>
struct LoopShot {
  T* buf[3];
  const T* fact;
  T* psi[2][2][2];  // [axis][side][parity]
  BandSide<T> band[2][2];  // coefficients and ξ
  int32_t active[2][2];
  int32_t first_r[2];
  int32_t nx, ny, halo;
  int64_t px;
  T inv_d[2], inv_d2[2];
  const int32_t* src_off;
  const int32_t* src_ids;
  const T* stf;  // [nt][nsrc]
  T* traces;     // [nt][nrec]
  int32_t nsrc, nrec;
};

// One launch: n steps from step it0. The state is read from buf[in[0]] (p_t),
// buf[in[1]] (p_{t-1}) and ψ parity par_in, and left in buf[out[0]],
// buf[out[1]] and par_out; in[2] / out[2] is the third buffer, of which only
// the rim's source nodes carry state. keep: when not NULL, step it of
// [keep_first, keep_first + keep_count) also writes its new field (interior
// and rim source nodes) to keep + keep_stride * (it - keep_first).
template <typename T>
struct LoopRun {
  const LoopTile* tiles;
  const LoopEdge* edges;
  const LoopShot<T>* shots;
  const LoopSrc* srcs;
  const LoopRec* recs;
  unsigned long long* mail;
  int64_t mail_stride;  // 64-bit words per tile (both slots)
  int32_t hmax, wmax;   // largest tile of the launch
  int32_t in[3], out[3], par_in, par_out;
  int32_t n;
  int64_t it0;
  uint32_t tag0;
  T* keep;
  int64_t keep_stride, keep_first, keep_count;
  int32_t* err;
  unsigned long long wait_ns;  // limit of a wait for an edge value
  int32_t withhold;            // tests only: the tile that sends no edges, or -1
};

// The units (vector columns or rows) of a tile that hold nodes of an axis's
// active bands: [a0, a0 + na) on the left and [b0, b0 + nb) on the right, in
// units of `unit` nodes from node `first` on, over `count` nodes. They get
// the state slots 0 .. na + nb - 1 in that order.
struct BandSlots {
  int32_t a0 = 0, na = 0, b0 = 0, nb = 0;
  __host__ __device__ int slot(int u) const {
    if (u >= a0 && u < a0 + na) return u - a0;
    if (u >= b0 && u < b0 + nb) return na + u - b0;
    return -1;
  }
  // the t-th unit that has no slot
  __host__ __device__ int other(int t) const {
    if (na > 0 && t >= a0) t += na;
    if (nb > 0 && t >= b0) t += nb;
    return t;
  }
};
__host__ __device__ inline BandSlots band_slots(int first, int count, int unit, int n, int halo,
                                                int first_r, bool act_l, bool act_r) {
  BandSlots s;
  const int last = first + count - 1;
  if (act_l) {  // nodes 1 .. halo
    const int lo = first > 1 ? first : 1, hi = last < halo ? last : halo;
    if (lo <= hi) {
      s.a0 = (lo - first) / unit;
      s.na = (hi - first) / unit - s.a0 + 1;
    }
  }
  if (act_r) {  // nodes first_r .. n - 2
    const int lo = first > first_r ? first : first_r, hi = last < n - 2 ? last : n - 2;
    if (lo <= hi) {
      s.b0 = (lo - first) / unit;
      if (s.na > 0 && s.b0 < s.a0 + s.na) s.b0 = s.a0 + s.na;
      s.nb = (hi - first) / unit - s.b0 + 1;
      if (s.nb < 0) s.nb = 0;
    }
  }
  return s;
}

// Band vector number k of a tile of cw vector columns and h rows: its row and
// column, and back (-1: no CPML work).
struct BandVecs {
  BandSlots bx;
  int cw, h, ny0, ny1;
  __host__ __device__ int nvx() const { return bx.na + bx.nb; }
  __host__ __device__ int count() const { return nvx() * h + (ny0 + ny1) * (cw - nvx()); }
  __host__ __device__ int yrow(int row) const {  // number of a y-band row, or -1
    return row < ny0 ? row : row >= h - ny1 ? ny0 + row - (h - ny1) : -1;
  }
  __host__ __device__ void at(int k, int& row, int& cv) const {
    const int n = nvx();
    if (k < n * h) {
      row = k / n;
      const int q = k - row * n;
      cv = q < bx.na ? bx.a0 + q : bx.b0 + q - bx.na;
    } else {
      const int m = cw - n, y = (k - n * h) / m;
      row = y < ny0 ? y : h - ny1 + y - ny0;
      cv = bx.other(k - n * h - y * m);
    }
  }
  __host__ __device__ int index(int row, int cv) const {
    const int n = nvx(), s = bx.slot(cv), y = yrow(row);
    if (s >= 0) return row * n + s;
    if (y < 0) return -1;
    const int before = (cv >= bx.a0 + bx.na ? bx.na : 0) + (cv >= bx.b0 + bx.nb ? bx.nb : 0);
    return n * h + y * (cw - n) + cv - before;
  }
};

template <typename T>
struct alignas(16) Pack {
  static constexpr int V = 16 / (int)sizeof(T);
  T v[V];
};

// Shared-memory accesses by 32-bit address. They are volatile: the compiler
// keeps them in program order (a block's threads and the receive loop write
// the fields between barriers), ptxas still schedules them by dependence.
__device__ __forceinline__ void lds(uint32_t a, float& x) {
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(a));
}
__device__ __forceinline__ void lds(uint32_t a, double& x) {
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(a));
}
__device__ __forceinline__ void lds(uint32_t a, Pack<float>& x) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(x.v[0]), "=f"(x.v[1]), "=f"(x.v[2]), "=f"(x.v[3])
               : "r"(a));
}
__device__ __forceinline__ void lds(uint32_t a, Pack<double>& x) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x.v[0]), "=d"(x.v[1]) : "r"(a));
}
// x = the value at a where on, else unchanged
__device__ __forceinline__ void lds_if(uint32_t a, int on, float& x) {
  asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p ld.shared.f32 %0, [%1];\n}\n"
               : "+f"(x)
               : "r"(a), "r"(on));
}
__device__ __forceinline__ void sts(uint32_t a, float x) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(x));
}
__device__ __forceinline__ void sts(uint32_t a, double x) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(x));
}
__device__ __forceinline__ void sts(uint32_t a, const Pack<float>& x) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x.v[0]), "f"(x.v[1]),
               "f"(x.v[2]), "f"(x.v[3]));
}
__device__ __forceinline__ void sts(uint32_t a, const Pack<double>& x) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(x.v[0]), "d"(x.v[1]));
}
template <typename T>
__device__ __forceinline__ T get(uint32_t a) {
  T x;
  lds(a, x);
  return x;
}

template <typename T>
__device__ __forceinline__ Pack<T> ldg_pack(const T* p) {
  Pack<T> r;
  const int4 q = __ldg(reinterpret_cast<const int4*>(p));
  memcpy(&r, &q, 16);
  return r;
}

// Edge values travel as 64-bit words {32 bits of the value, tag}: one word
// for a float, two for a double.
__device__ __forceinline__ void mail_put(unsigned long long* q, float x, uint32_t tag) {
  const unsigned long long w = (unsigned long long)__float_as_uint(x) | ((unsigned long long)tag << 32);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(q), "l"(w) : "memory");
}
__device__ __forceinline__ void mail_put(unsigned long long* q, double x, uint32_t tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long hi = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(q), "l"((b & 0xffffffffull) | hi),
               "l"((b >> 32) | hi)
               : "memory");
}
__device__ __forceinline__ unsigned long long mail_get(const unsigned long long* q) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(q) : "memory");
  return w;
}
// Bounded wait for the word of `tag` at q (w: an earlier read of it, or 0, a tag
// that is never used): `limit` ns, or until another
// thread of the launch has raised *err. False when it gives up.
__device__ __forceinline__ bool mail_wait(const unsigned long long* q, uint32_t tag,
                                          unsigned long long& w, const int32_t* err,
                                          unsigned long long limit) {
  unsigned long long t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    if ((uint32_t)(w >> 32) == tag) return true;  // w: 0 or what an earlier read gave
    w = mail_get(q);
    if ((spin & 1023u) == 1023u) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      if (t - t0 > limit || *(volatile const int32_t*)err) return false;
    }
  }
}
__device__ __forceinline__ bool mail_take(const unsigned long long* q, uint32_t tag, float& x,
                                          const int32_t* err, unsigned long long limit,
                                          unsigned long long w = 0) {
  if (!mail_wait(q, tag, w, err, limit)) return false;
  x = __uint_as_float((uint32_t)w);
  return true;
}
__device__ __forceinline__ bool mail_take(const unsigned long long* q, uint32_t tag, double& x,
                                          const int32_t* err, unsigned long long limit,
                                          unsigned long long lo = 0) {
  unsigned long long hi = 0;
  if (!mail_wait(q, tag, lo, err, limit) || !mail_wait(q + 1, tag, hi, err, limit)) return false;
  x = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
  return true;
}

// The update of the V nodes of a vector without CPML: d2x, d2y (kept for the
// band terms) and the leapfrog value, in the operations and order of
// second_diff and leapfrog2d. For floats the y part and the leapfrog run two
// nodes per instruction (packed f32x2, each half rounded like the scalar
// operation): 28 instead of 36 instructions per 4 nodes. The x neighbours of
// a pair straddle register pairs, so the x part stays scalar.
__device__ __forceinline__ void vec_update(const Pack<float>& up, const Pack<float>& c,
                                           const Pack<float>& dn, const Pack<float>& o,
                                           const Pack<float>& f, float xm, float xp, float ix2,
                                           float iy2, Pack<float>& d2x, Pack<float>& d2y,
                                           Pack<float>& nv) {
  // p - 2 c + m with the product fused (2 c is exact): one rounding each
  auto d2 = [&](float m, float v, float p) { return mul_rn(fmaf(-2.f, v, p) + m, ix2); };
  d2x.v[0] = d2(xm, c.v[0], c.v[1]);
  d2x.v[1] = d2(c.v[0], c.v[1], c.v[2]);
  d2x.v[2] = d2(c.v[1], c.v[2], c.v[3]);
  d2x.v[3] = d2(c.v[2], c.v[3], xp);
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    const float2 cc{c.v[q], c.v[q + 1]};
    // (dn - 2 c) + up, times 1/dy²
    float2 d = fma2(cc, float2{-2.f, -2.f}, float2{dn.v[q], dn.v[q + 1]});
    d = mul2_kept(add2(d, float2{up.v[q], up.v[q + 1]}), iy2);
    // 2 c - o as two scalar operations (a packed one has no operand sign)
    const float2 lead{fmaf(2.f, cc.x, -o.v[q]), fmaf(2.f, cc.y, -o.v[q + 1])};
    const float2 sum = add2(float2{d2x.v[q], d2x.v[q + 1]}, d);
    const float2 n = fma2(float2{f.v[q], f.v[q + 1]}, sum, lead);
    d2y.v[q] = d.x;
    d2y.v[q + 1] = d.y;
    nv.v[q] = n.x;
    nv.v[q + 1] = n.y;
  }
}
__device__ __forceinline__ void vec_update(const Pack<double>& up, const Pack<double>& c,
                                           const Pack<double>& dn, const Pack<double>& o,
                                           const Pack<double>& f, double xm, double xp, double ix2,
                                           double iy2, Pack<double>& d2x, Pack<double>& d2y,
                                           Pack<double>& nv) {
  d2x.v[0] = second_diff(xm, c.v[0], c.v[1], ix2);
  d2x.v[1] = second_diff(c.v[0], c.v[1], xp, ix2);
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    d2y.v[v] = second_diff(up.v[v], c.v[v], dn.v[v], iy2);
    nv.v[v] = leapfrog2d(c.v[v], o.v[v], f.v[v], d2x.v[v], d2y.v[v]);
  }
}

// CPML terms of a vector of V nodes, in the operations of psi_face and
// cpml_tail; for floats two nodes per instruction where the operands lie in
// the same register pairs.
// ps = b ps + a (p - c) / d on V faces.
__device__ __forceinline__ void vec_psi(Pack<float>& ps, const Pack<float>& b, const Pack<float>& a,
                                        const Pack<float>& dp, float inv) {
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    const float2 t = mul2(mul2(float2{a.v[q], a.v[q + 1]}, float2{dp.v[q], dp.v[q + 1]}),
                          float2{inv, inv});
    const float2 r = fma2(float2{b.v[q], b.v[q + 1]}, float2{ps.v[q], ps.v[q + 1]}, t);
    ps.v[q] = r.x;
    ps.v[q + 1] = r.y;
  }
}
__device__ __forceinline__ void vec_psi(Pack<double>& ps, const Pack<double>& b,
                                        const Pack<double>& a, const Pack<double>& dp, double inv) {
#pragma unroll
  for (int v = 0; v < 2; ++v) ps.v[v] = psi_face(b.v[v], a.v[v], ps.v[v], dp.v[v], inv);
}
// dj = ψ[q] - ψ[q-1] per node: ξ and the damping term.
__device__ __forceinline__ void vec_tail(const Pack<float>& bk, const Pack<float>& a,
                                         const Pack<float>& dj, Pack<float>& xi,
                                         const Pack<float>& d2, const Pack<float>& f, float inv,
                                         Pack<float>& damp) {
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    const float2 dps = mul2_kept(float2{dj.v[q], dj.v[q + 1]}, inv);
    const float2 s = add2(float2{d2.v[q], d2.v[q + 1]}, dps);
    const float2 x = fma2(float2{bk.v[q], bk.v[q + 1]}, float2{xi.v[q], xi.v[q + 1]},
                          mul2(float2{a.v[q], a.v[q + 1]}, s));
    const float2 g = fma2(float2{f.v[q], f.v[q + 1]}, add2(dps, x),
                          float2{damp.v[q], damp.v[q + 1]});
    xi.v[q] = x.x;
    xi.v[q + 1] = x.y;
    damp.v[q] = g.x;
    damp.v[q + 1] = g.y;
  }
}
__device__ __forceinline__ void vec_tail(const Pack<double>& bk, const Pack<double>& a,
                                         const Pack<double>& dj, Pack<double>& xi,
                                         const Pack<double>& d2, const Pack<double>& f, double inv,
                                         Pack<double>& damp) {
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const double dps = mul_rn(dj.v[v], inv);
    xi.v[v] = fma(bk.v[v], xi.v[v], mul_rn(a.v[v], d2.v[v] + dps));
    damp.v[v] = fma(f.v[v], dps + xi.v[v], damp.v[v]);
  }
}
// a - b
__device__ __forceinline__ Pack<float> vec_sub(const Pack<float>& a, const Pack<float>& b) {
  Pack<float> r;
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    const float2 t = fma2(float2{b.v[q], b.v[q + 1]}, float2{-1.f, -1.f},
                          float2{a.v[q], a.v[q + 1]});
    r.v[q] = t.x;
    r.v[q + 1] = t.y;
  }
  return r;
}
__device__ __forceinline__ Pack<double> vec_sub(const Pack<double>& a, const Pack<double>& b) {
  return Pack<double>{{a.v[0] - b.v[0], a.v[1] - b.v[1]}};
}
// second difference along y
__device__ __forceinline__ Pack<float> vec_d2y(const Pack<float>& up, const Pack<float>& c,
                                               const Pack<float>& dn, float iy2) {
  Pack<float> r;
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    float2 d = fma2(float2{c.v[q], c.v[q + 1]}, float2{-2.f, -2.f}, float2{dn.v[q], dn.v[q + 1]});
    d = mul2_kept(add2(d, float2{up.v[q], up.v[q + 1]}), iy2);
    r.v[q] = d.x;
    r.v[q + 1] = d.y;
  }
  return r;
}
__device__ __forceinline__ Pack<double> vec_d2y(const Pack<double>& up, const Pack<double>& c,
                                                const Pack<double>& dn, double iy2) {
  return Pack<double>{{second_diff(up.v[0], c.v[0], dn.v[0], iy2),
                       second_diff(up.v[1], c.v[1], dn.v[1], iy2)}};
}
template <typename T>
__device__ __forceinline__ Pack<T> splat(T x) {
  Pack<T> r;
#pragma unroll
  for (int v = 0; v < Pack<T>::V; ++v) r.v[v] = x;
  return r;
}
// The x-band terms of one vector: ψ on its left face (s0) and right faces
// (ps), ξ, and the damping of the nodes of mask `in`. ca: shared address of
// the coefficient tables at the vector, cs: bytes from one table to the next.
template <typename T>
__device__ __forceinline__ void vec_xband(uint32_t ca, int cs, const Pack<T>& c, T xm, T xp,
                                          const Pack<T>& f, unsigned in, T ix, T ix2, T& s0,
                                          Pack<T>& ps, Pack<T>& xi, Pack<T>& damp) {
  constexpr int V = Pack<T>::V;
  // faces 0 .. V of the vector; face v + 1 is node v's right one
  const Pack<T> b0 = get<Pack<T>>(ca), a0 = get<Pack<T>>(ca + cs);
  const T be = get<T>(ca + 16), ae = get<T>(ca + cs + 16);
  const Pack<T> nb = get<Pack<T>>(ca + 2 * cs), na = get<Pack<T>>(ca + 3 * cs);
  Pack<T> b, a, dp, d2, dj;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const T l = v == 0 ? xm : c.v[v == 0 ? 0 : v - 1];
    const T r = v == V - 1 ? xp : c.v[v == V - 1 ? v : v + 1];
    b.v[v] = v == V - 1 ? be : b0.v[v == V - 1 ? v : v + 1];
    a.v[v] = v == V - 1 ? ae : a0.v[v == V - 1 ? v : v + 1];
    dp.v[v] = r - c.v[v];
    d2.v[v] = second_diff(l, c.v[v], r, ix2);
  }
  s0 = psi_face(b0.v[0], a0.v[0], s0, c.v[0] - xm, ix);
  vec_psi(ps, b, a, dp, ix);
#pragma unroll
  for (int v = 0; v < V; ++v) dj.v[v] = ps.v[v] - (v == 0 ? s0 : ps.v[v == 0 ? 0 : v - 1]);
  vec_tail(nb, na, dj, xi, d2, f, ix, damp);
  if (in != (1u << V) - 1u) {
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (!(in >> v & 1u)) damp.v[v] = T(0);
  }
}

// R: the most rows a thread of the launch owns. A vector is 16 bytes: 4 floats
// or 2 doubles. Thread t owns the V columns of vector t % cw in the `rows` rows
// from (t / cw) rows on.
template <typename T, int R>
__global__ void __launch_bounds__(LOOP_NT, 1) loop2d(const __grid_constant__ LoopRun<T> Q) {
  constexpr int V = 16 / (int)sizeof(T);
  constexpr int WPV = (int)sizeof(T) / 4;  // mailbox words per value
  constexpr int ES = (int)sizeof(T);
  using P = Pack<T>;
  extern __shared__ __align__(128) unsigned char smem[];
  const LoopTile& tl = Q.tiles[blockIdx.x];
  const LoopShot<T>& S = Q.shots[tl.shot];
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int w = tl.w, h = tl.h, x0 = tl.x0, y0 = tl.y0;
  const int nx = S.nx, ny = S.ny, halo = S.halo;
  const int64_t px = S.px;
  const int cw = w / V, pitch = w + 2 * V;
  const BandVecs bv{band_slots(x0, w, V, nx, halo, S.first_r[0], S.active[0][0] != 0,
                               S.active[0][1] != 0),
                    cw, h, tl.ny0, tl.ny1};
  const int nband = tl.nband, nxv = tl.nvx * h;
  // cur and nxt: the fields of p_t and of p_{t-1}, which becomes p_{t+1}
  const uint32_t sb = smem_u32(smem);
  uint32_t cur = sb + tl.f[0], nxt = sb + tl.f[1];
  // coefficient tables: face c of an axis lies between the tile's nodes c - 1
  // and c; node c of a band uses faces c and c + 1. Zero outside the bands.
  T* const cx = reinterpret_cast<T*>(smem + tl.cx);
  const uint32_t cx_a = sb + tl.cx;
  const int cxs = w + V;  // {bKh, ah} of the faces, {bK, a} of the nodes
  T* const cy = reinterpret_cast<T*>(smem + tl.cy);
  const int cys = (h + V) / V * V;
  const uint32_t bf_a = sb + tl.bf, px_a = sb + tl.px, px0_a = sb + tl.px0, xx_a = sb + tl.xx;
  const int bt_o = tl.bt;
  const uint32_t ylo_a = sb + tl.ylo, yhi_a = sb + tl.yhi, xy_a = sb + tl.xy;
  // ---- load: coefficient tables, fields with their ring, band state --------
  auto table = [&](int a, int c, int g0, int n, T* tab, int stride) {
    const int hl = halo < n - 2 ? halo : n - 2;
    T fb = 0, fa = 0, nb = 0, na = 0;
    const int F = g0 + c - 1, g = g0 + c;
    if (S.active[a][0] && F >= 0 && F <= hl) {
      fb = S.band[a][0].bKh[F];
      fa = S.band[a][0].ah[F];
    } else if (S.active[a][1] && F >= S.first_r[a] - 1 && F <= n - 2) {
      const int q = F - (n - halo - 2);
      fb = S.band[a][1].bKh[q];
      fa = S.band[a][1].ah[q];
    }
    if (S.active[a][0] && g >= 1 && g <= hl) {
      nb = S.band[a][0].bK[g - 1];
      na = S.band[a][0].a[g - 1];
    } else if (S.active[a][1] && g >= S.first_r[a] && g <= n - 2) {
      const int q = g - (n - halo - 2);
      nb = S.band[a][1].bK[q - 1];
      na = S.band[a][1].a[q - 1];
    }
    tab[c] = fb;
    tab[stride + c] = fa;
    tab[2 * stride + c] = nb;
    tab[3 * stride + c] = na;
  };
  for (int c = tid; c <= w; c += nthr) table(0, c, x0, nx, cx, cxs);
  for (int c = tid; c <= h; c += nthr) table(1, c, y0, ny, cy, cys);
  {
    const T* __restrict__ gc = S.buf[Q.in[0]];
    const T* __restrict__ go = S.buf[Q.in[1]];
    for (int e = tid; e < (h + R + 1) * pitch; e += nthr) {
      const int r = e / pitch, c = e - r * pitch;
      const int i = x0 + c - V, j = y0 + r - 1;
      T vc = 0, vo = 0;
      if (i >= 0 && i < nx && r <= h + 1) {
        vc = gc[i + px * j];
        vo = go[i + px * j];
      }
      sts(cur + e * ES, vc);
      sts(nxt + e * ES, vo);
    }
  }
  // which nodes of vector cv are updated, which lie in an active x band
  auto ok_of = [&](int c) {
    unsigned m = 0;
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (x0 + c * V + v >= 1 && x0 + c * V + v <= nx - 2) m |= 1u << v;
    return m;
  };
  const int xl = S.active[0][0] ? min(halo, nx - 2) : 0, xr = S.active[0][1] ? S.first_r[0] : nx;
  auto xin_of = [&](int c) {
    unsigned m = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int i = x0 + c * V + v;
      if ((i >= 1 && i <= xl) || (i >= xr && i <= nx - 2)) m |= 1u << v;
    }
    return m;
  };
  // side (0, 1) and entry q of a band node c of an axis of n nodes
  auto side_q = [&](int c, int n, int& q) {
    if (c <= halo) {
      q = c;
      return 0;
    }
    q = c - (n - halo - 2);
    return 1;
  };
  for (int k = tid; k < nband; k += nthr) {
    int row, c;
    bv.at(k, row, c);
    reinterpret_cast<int*>(smem + tl.bt)[k] = row << 16 | c;
    const int i = x0 + c * V, j = y0 + row;
    const unsigned ok = ok_of(c);
    P f = splat(T(0));
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (ok >> v & 1u) f.v[v] = S.fact[i + v + px * j];
    sts(bf_a + k * 16, f);
    if (k < nxv) {
      const unsigned xin = xin_of(c);
      P ps = splat(T(0)), xi = splat(T(0));
      T p0 = 0;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (!(xin >> v & 1u)) continue;
        int q;
        const int sd = side_q(i + v, nx, q);
        const T* psi = S.psi[0][sd][Q.par_in] + (int64_t)(halo + 1) * j;
        ps.v[v] = psi[q];
        (v == 0 ? p0 : ps.v[v == 0 ? 0 : v - 1]) = psi[q - 1];
        xi.v[v] = S.band[0][sd].xi[(int64_t)halo * j + q - 1];
      }
      sts(px_a + k * 16, ps);
      sts(xx_a + k * 16, xi);
      sts(px0_a + k * ES, p0);
    }
    const int y = bv.yrow(row);
    if (y >= 0) {
      int q;
      const int sd = side_q(j, ny, q);
      const T* psi = S.psi[1][sd][Q.par_in] + px * (q - 1) + i;
      const T* x = S.band[1][sd].xi + px * (q - 1) + i;
      P lo = splat(T(0)), hi = splat(T(0)), xi = splat(T(0));
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (ok >> v & 1u) {
          lo.v[v] = psi[v];
          hi.v[v] = psi[px + v];
          xi.v[v] = x[v];
        }
      const int at = (y * cw + c) * 16;
      sts(ylo_a + at, lo);
      sts(yhi_a + at, hi);
      sts(xy_a + at, xi);
    }
  }
  const int trow = tl.rows;
  const bool live = tid < cw * ((h + trow - 1) / trow);
  const int cv = live ? tid % cw : 0, r0 = live ? tid / cw * trow : 0;  // idle threads shadow the first
  const int nrow = live ? min(trow, h - r0) : 0;
  const int i0 = x0 + cv * V;
  const unsigned okm = ok_of(cv);
  const bool full = okm == (1u << V) - 1u, fix = !full && nrow > 0;
  P f[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int v = 0; v < V; ++v)
      f[r].v[v] = (r < nrow && (okm >> v & 1u)) ? S.fact[i0 + v + px * (y0 + r0 + r)] : T(0);
  // this thread's source nodes [s0, s1), in the sorted list; rim nodes of the
  // tile's own rows (the columns i = 0 and nx - 1) belong to the thread that
  // owns their vector, the others to any thread
  int s0 = tl.src[1], s1 = tl.src[1];
  for (int e = tl.src[0]; e < tl.src[1]; ++e)
    if (Q.srcs[e].owner == tid) {
      if (s0 == tl.src[1]) s0 = e;
      s1 = e + 1;
    }
  const bool any_src = tl.src[1] > tl.src[0];
  // The common case, one source node with one source: its amplitude is loaded
  // a step ahead and a rim node's three buffers are kept in registers, so no
  // load stands between the update and the edge sends.
  int one_cell = -1;
  int64_t one_node = -1;
  const T* one_amp = S.stf;
  T amp = 0, rim0 = 0, rim1 = 0, rim2 = 0;  // the rim node's values, oldest first
  if (s1 - s0 == 1) {
    const LoopSrc sr = Q.srcs[s0];
    const int k = S.src_off[sr.sgrp];
    if (S.src_off[sr.sgrp + 1] == k + 1) {
      one_cell = sr.cell;
      one_node = sr.node;
      one_amp = S.stf + Q.it0 * S.nsrc + S.src_ids[k];
      amp = *one_amp;
      s0 = s1;
      if (one_node >= 0) {
        rim0 = S.buf[Q.in[2]][one_node];
        rim1 = S.buf[Q.in[1]][one_node];
        rim2 = S.buf[Q.in[0]][one_node];
      }
    }
  }
  const int nsrc = S.nsrc, nrec = S.nrec;
  // receivers: one per thread in registers, any further ones from the list
  const int rec1 = tl.rec[1];
  int rec_e = tl.rec[0] + tid, rec_cell = -1;
  T* rec_to = nullptr;
  if (rec_e < rec1) {
    rec_cell = Q.recs[rec_e].cell;
    rec_to = S.traces + Q.it0 * nrec + Q.recs[rec_e].id;
  }
  rec_e += nthr;
  const bool any_rec = tl.rec[1] > tl.rec[0];
  const T ix2 = S.inv_d2[0], iy2 = S.inv_d2[1], ix = S.inv_d[0], iy = S.inv_d[1];
  const int rows = __reduce_max_sync(0xffffffffu, nrow);  // of the warp's threads
  const int base = (r0 + 1) * pitch + cv * V + V;  // the thread's first node
  const int dp = pitch * ES;
  // x neighbours from the adjacent lanes (floats), except across a warp's or
  // a row's end
  const int lane = tid & 31;
  const int cl = __shfl_up_sync(0xffffffffu, base, 1), cr = __shfl_down_sync(0xffffffffu, base, 1);
  const int lds_l = lane == 0 || cl != base - V, lds_r = lane == 31 || cr != base + V;
  // edges: where this thread's go, where the first ring value it fetches is
  // (mailbox words as 32-bit numbers)
  const int slot_words = (int)(Q.mail_stride / 2);
  const int oL = 0, oR = Q.hmax * WPV, oU = 2 * Q.hmax * WPV, oD = (2 * Q.hmax + Q.wmax) * WPV;
  const int nU = tl.nbr[2] >= 0 ? w : 0, nD = tl.nbr[3] >= 0 ? w : 0;
  const int nL = tl.nbr[0] >= 0 ? h : 0, nR = tl.nbr[1] >= 0 ? h : 0;
  const int nring = nU + nD + nL + nR;
  const int inbox = (int)blockIdx.x * (int)Q.mail_stride;
  auto ring = [&](int k, int& cell) -> int {  // ring value k: its cell and mailbox word
    if (k < nU) {
      cell = V + k;
      return oU + k * WPV;
    }
    if ((k -= nU) < nD) {
      cell = (h + 1) * pitch + V + k;
      return oD + k * WPV;
    }
    if ((k -= nD) < nL) {
      cell = (k + 1) * pitch + V - 1;
      return oL + k * WPV;
    }
    k -= nL;
    cell = (k + 1) * pitch + V + w;
    return oR + k * WPV;
  };
  int ring_cell = 0;
  const int ring_at = inbox + (tid < nring ? ring(tid, ring_cell) : 0);
  const bool early = R >= LOOP_EARLY_R && tl.nedge > 0;
  const bool mute = (int)blockIdx.x == Q.withhold;
  // late sends: the mailbox words of this thread's edges, -1 without one
  const bool send = nring && !early && nrow > 0 && !mute;
  const int to_u = send && nU && r0 == 0 ? (int)(tl.nbr[2] * Q.mail_stride) + oD + cv * V * WPV : -1;
  const int to_d = send && nD && r0 + nrow == h ? (int)(tl.nbr[3] * Q.mail_stride) + oU + cv * V * WPV : -1;
  const int to_l = send && nL && cv == 0 ? (int)(tl.nbr[0] * Q.mail_stride) + oR + r0 * WPV : -1;
  const int to_r = send && nR && cv == cw - 1 ? (int)(tl.nbr[1] * Q.mail_stride) + oL + r0 * WPV : -1;
  const bool edge = to_u >= 0 || to_d >= 0 || to_l >= 0 || to_r >= 0;
  // With several rows per thread the edges are computed first, by all threads
  // (an item each), and sent before the tile's own update, which then hides
  // their trip. Items only read the state; the update computes the same values
  // again. The Dirichlet columns of an upper or lower row are sent too; nothing
  // reads them.
  LoopEdge im{};
  int it_base = -1;
  unsigned it_xin = 0;
  if (early && tid < tl.nedge && !mute) {
    im = Q.edges[tl.edge0 + tid];
    it_base = ((im.rc >> 16) + 1) * pitch + (im.rc & 0xffff) * V + V;
    it_xin = xin_of(im.rc & 0xffff);
  }
  const T* __restrict__ fact = S.fact + x0 + px * y0;  // of the tile's first node
  const int ipx = (int)px;
  // The CPML terms of band vector k (row, vector c; centre value cc, its
  // neighbours read from cur): the damping, and the new state when `put`.
  auto band_terms = [&](int k, int row, int c, uint32_t at, const P& cc, unsigned ok, unsigned xin,
                        bool put) -> P {
    const P fk = get<P>(bf_a + k * 16);
    P damp = splat(T(0));
    if (k < nxv) {
      const T xm = get<T>(at - ES), xp = get<T>(at + V * ES);
      P ps = get<P>(px_a + k * 16), xo = get<P>(xx_a + k * 16);
      T p0 = get<T>(px0_a + k * ES);
      vec_xband(cx_a + c * 16, cxs * ES, cc, xm, xp, fk, xin, ix, ix2, p0, ps, xo, damp);
      if (put) {
        sts(px0_a + k * ES, p0);
        sts(px_a + k * 16, ps);
        sts(xx_a + k * 16, xo);
      }
    }
    const int y = bv.yrow(row);
    if (y >= 0) {
      const P up = get<P>(at - dp), dn = get<P>(at + dp);
      const int e = (y * cw + c) * 16;
      P lo = get<P>(ylo_a + e), hi = get<P>(yhi_a + e), xo = get<P>(xy_a + e);
      vec_psi(lo, splat(cy[row]), splat(cy[cys + row]), vec_sub(cc, up), iy);
      vec_psi(hi, splat(cy[row + 1]), splat(cy[cys + row + 1]), vec_sub(dn, cc), iy);
      vec_tail(splat(cy[2 * cys + row]), splat(cy[3 * cys + row]), vec_sub(hi, lo), xo,
               vec_d2y(up, cc, dn, iy2), fk, iy, damp);
      if (put) {
        sts(ylo_a + e, lo);
        sts(yhi_a + e, hi);
        sts(xy_a + e, xo);
      }
    }
    if (ok != (1u << V) - 1u) {  // the Dirichlet columns take none
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (!(ok >> v & 1u)) damp.v[v] = T(0);
    }
    return damp;
  };
  // The band vectors this thread works on: with one row per thread its own,
  // inside the update; else numbers tid, tid + nthr, ... after it, spread over
  // the block (as the owners' own they made the band threads of a full tile
  // take 8200 cycles where the others took 3200).
  int bk = -1, brow = 0, bc = 0;
  unsigned bok = 0, bxin = 0;
  if (R == 1) {
    if (nrow > 0) bk = bv.index(r0, cv);
    brow = r0;
    bc = cv;
  } else if (tid < nband) {
    bk = tid;
    bv.at(bk, brow, bc);
  }
  if (bk >= 0) {
    bok = ok_of(bc);
    bxin = xin_of(bc);
  }
  const int bcell = (brow + 1) * pitch + bc * V + V;
  const bool settle = any_src || (nring && !early);
  bool dead = false;  // a wait ran out: no more waiting, the host reports it
  __syncthreads();

  for (int s = 0; s < Q.n; ++s) {
    // receivers of the field the last step left (p_it)
    if (any_rec && s > 0) {
      if (rec_cell >= 0) {
        *rec_to = get<T>(cur + rec_cell * ES);
        rec_to += nrec;
      }
      for (int e = rec_e; e < rec1; e += nthr)
        S.traces[(Q.it0 + s - 1) * nrec + Q.recs[e].id] = get<T>(cur + Q.recs[e].cell * ES);
    }
    const uint32_t tag = Q.tag0 + (uint32_t)s;
    const int slot = (s & 1) * slot_words;
    const bool more = s + 1 < Q.n;
    if (early && more) {
      if (it_base >= 0) {
        const int row = im.rc >> 16, c = im.rc & 0xffff;
        const uint32_t b = cur + it_base * ES;
        const P fi = ldg_pack<T>(fact + c * V + ipx * row);
        const P cc = get<P>(b), up = get<P>(b - dp), dn = get<P>(b + dp);
        const P o = get<P>(nxt + it_base * ES);
        const T xm = get<T>(b - ES), xp = get<T>(b + V * ES);
        P nv, d2x, d2y;
        vec_update(up, cc, dn, o, fi, xm, xp, ix2, iy2, d2x, d2y, nv);
        if (im.band >= 0) {
          const P damp = band_terms(im.band, row, c, b, cc, (1u << V) - 1u, it_xin, false);
#pragma unroll
          for (int v = 0; v < V; ++v) nv.v[v] += damp.v[v];
        }
        unsigned long long* m = Q.mail + (slot + im.mail);
        if (im.what == 0) {
#pragma unroll
          for (int v = 0; v < V; ++v) mail_put(m + v * WPV, nv.v[v], tag);
        } else {
          mail_put(m, im.what == 1 ? nv.v[0] : nv.v[V - 1], tag);
        }
      }
      __syncthreads();  // the update below overwrites what the items read
    }
    unsigned long long ahead = 0;  // the first ring value, asked for ahead of its use
    {
      // leapfrog of the thread's rows, without CPML terms; all that row r + 1
      // reads is loaded while row r is computed
      const uint32_t cb = cur + base * ES, ob = nxt + base * ES;
      P q[R + 2], o[R];
      T xm[R], xp[R];
      auto neighbours = [&](int r, uint32_t a, const P& c) {  // of row r's vector c, at a
        if constexpr (sizeof(T) == 4) {
          xm[r] = __shfl_up_sync(0xffffffffu, c.v[V - 1], 1);
          xp[r] = __shfl_down_sync(0xffffffffu, c.v[0], 1);
          lds_if(a - ES, lds_l, xm[r]);
          lds_if(a + V * ES, lds_r, xp[r]);
        } else {
          lds(a - ES, xm[r]);
          lds(a + V * ES, xp[r]);
        }
      };
      lds(cb, q[1]);
      lds(cb - dp, q[0]);
      lds(ob, o[0]);
      lds(cb + dp, q[2]);
      neighbours(0, cb, q[1]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r > 0 && r >= rows) break;
        const uint32_t rc = cb + r * dp, ro = ob + r * dp;
        if (r + 1 < R) {
          constexpr int last = R + 1;
          lds(rc + 2 * dp, q[r + 3 < last ? r + 3 : last]);
          lds(ro + dp, o[r + 1 < R ? r + 1 : r]);
          neighbours(r + 1 < R ? r + 1 : r, rc + dp, q[r + 2]);
        }
        P nv, d2x, d2y;
        vec_update(q[r], q[r + 1], q[r + 2], o[r], f[r], xm[r], xp[r], ix2, iy2, d2x, d2y, nv);
        if (R == 1 && bk >= 0) {
          const P damp = band_terms(bk, brow, bc, rc, q[1], bok, bxin, true);
#pragma unroll
          for (int v = 0; v < V; ++v) nv.v[v] += damp.v[v];
        }
        if (r < nrow) sts(ro, nv);
      }
      if (fix) {  // Dirichlet columns hold 0 (where no source sits)
        for (int r = 0; r < nrow; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v)
            if (!(okm >> v & 1u)) sts(ob + r * dp + v * ES, T(0));
      }
    }
    if (R >= LOOP_EARLY_R && early && more && tid < nring) ahead = mail_get(Q.mail + (ring_at + slot));
    if (R > 1 && nband > 0) {
      // CPML: the damping term is added to the stored leapfrog value, as the
      // per-step kernels add it
      __syncthreads();
      if (bk >= 0) {
        const uint32_t at = cur + bcell * ES, to = nxt + bcell * ES;
        const P cc = get<P>(at);
        const P damp = band_terms(bk, brow, bc, at, cc, bok, bxin, true);
        P nv = get<P>(to);
#pragma unroll
        for (int v = 0; v < V; ++v) nv.v[v] += damp.v[v];
        sts(to, nv);
        for (int k = bk + nthr; k < nband; k += nthr) {
          const int rc = reinterpret_cast<const int*>(smem + bt_o)[k], row = rc >> 16, c = rc & 0xffff;
          const int cell = (row + 1) * pitch + c * V + V;
          const P c2 = get<P>(cur + cell * ES);
          const P d2 = band_terms(k, row, c, cur + cell * ES, c2, ok_of(c), xin_of(c), true);
          P n2 = get<P>(nxt + cell * ES);
#pragma unroll
          for (int v = 0; v < V; ++v) n2.v[v] += d2.v[v];
          sts(nxt + cell * ES, n2);
        }
      }
      if (settle) __syncthreads();  // owners read their nodes below
    }
    if (any_src) {
      if (one_cell >= 0) {
        const T v = (one_node >= 0 ? rim0 : get<T>(nxt + one_cell * ES)) + amp;
        sts(nxt + one_cell * ES, v);
        if (one_node >= 0) {
          rim0 = rim1;
          rim1 = rim2;
          rim2 = v;
          S.buf[Q.in[2 - s % 3]][one_node] = v;
          const int64_t m = Q.it0 + s - Q.keep_first;
          if (Q.keep && m >= 0 && m < Q.keep_count) Q.keep[Q.keep_stride * m + one_node] = v;
        }
        one_amp += nsrc;
        if (s + 1 < Q.n) amp = *one_amp;
      }
      for (int e = s0; e < s1; ++e) {
        const LoopSrc sr = Q.srcs[e];
        const int64_t it = Q.it0 + s;
        // a rim node's new value is the one of three steps ago plus the
        // source: its three buffers live in global memory (in[2], in[1],
        // in[0], in[2], ...), touched by this thread alone
        T* b = sr.node >= 0 ? S.buf[Q.in[2 - s % 3]] + sr.node : nullptr;
        T v = b ? *b : get<T>(nxt + sr.cell * ES);
        const T* row = S.stf + it * nsrc;
        for (int k = S.src_off[sr.sgrp]; k < S.src_off[sr.sgrp + 1]; ++k) v += row[S.src_ids[k]];
        if (b) *b = v;
        sts(nxt + sr.cell * ES, v);
        if (sr.node >= 0 && Q.keep && it >= Q.keep_first && it < Q.keep_first + Q.keep_count)
          Q.keep[Q.keep_stride * (it - Q.keep_first) + sr.node] = v;
      }
    }
    if (nring && more) {
      if (edge) {  // this thread's edge nodes to the neighbours' inboxes
        const uint32_t own = nxt + base * ES;
        if (to_u >= 0) {
          const P e = get<P>(own);
          unsigned long long* q = Q.mail + (to_u + slot);
#pragma unroll
          for (int v = 0; v < V; ++v) mail_put(q + v * WPV, e.v[v], tag);
        }
        if (to_d >= 0) {
          const P e = get<P>(own + (nrow - 1) * dp);
          unsigned long long* q = Q.mail + (to_d + slot);
#pragma unroll
          for (int v = 0; v < V; ++v) mail_put(q + v * WPV, e.v[v], tag);
        }
        if (to_l >= 0)
          for (int r = 0; r < nrow; ++r)
            mail_put(Q.mail + (to_l + slot + r * WPV), get<T>(own + r * dp), tag);
        if (to_r >= 0)
          for (int r = 0; r < nrow; ++r)
            mail_put(Q.mail + (to_r + slot + r * WPV), get<T>(own + r * dp + (V - 1) * ES), tag);
      }
      // the neighbours' edges into this tile's ring
      if (tid < nring && !dead) {
        T x;
        if (mail_take(Q.mail + (ring_at + slot), tag, x, Q.err, Q.wait_ns, ahead))
          sts(nxt + ring_cell * ES, x);
        else
          dead = true;
        for (int e = tid + nthr; e < nring && !dead; e += nthr) {
          int cell;
          const int word = ring(e, cell);
          if (mail_take(Q.mail + (inbox + slot + word), tag, x, Q.err, Q.wait_ns))
            sts(nxt + cell * ES, x);
          else
            dead = true;
        }
        if (dead) atomicExch(Q.err, 1);
      }
    }
    if (Q.keep) {
      const int64_t it = Q.it0 + s;
      if (it >= Q.keep_first && it < Q.keep_first + Q.keep_count) {
        if (R > 1 && nband > 0 && !settle) __syncthreads();  // other threads' band terms
        T* g = Q.keep + Q.keep_stride * (it - Q.keep_first) + i0 + px * (y0 + r0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (r >= nrow) break;
          const P own = get<P>(nxt + (base + r * pitch) * ES);
          if (full) {
            *reinterpret_cast<P*>(g + px * r) = own;
          } else {
#pragma unroll
            for (int v = 0; v < V; ++v)
              if (okm >> v & 1u) g[px * r + v] = own.v[v];
          }
        }
      }
    }
    __syncthreads();
    const uint32_t t = cur;
    cur = nxt;
    nxt = t;
  }

  // ---- store: the last receivers, p_t, p_{t-1} and the band state -----------
  for (int e = tl.rec[0] + tid; e < tl.rec[1]; e += nthr) {
    const LoopRec rc = Q.recs[e];
    S.traces[(Q.it0 + Q.n - 1) * S.nrec + rc.id] = get<T>(cur + rc.cell * ES);
  }
  T* gc = S.buf[Q.out[0]];
  T* go = S.buf[Q.out[1]];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (r >= nrow) break;
    const int64_t g = i0 + px * (y0 + r0 + r);
    const P pc = get<P>(cur + (base + r * pitch) * ES), po = get<P>(nxt + (base + r * pitch) * ES);
    if (full) {
      *reinterpret_cast<P*>(gc + g) = pc;
      *reinterpret_cast<P*>(go + g) = po;
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (okm >> v & 1u) {
          gc[g + v] = pc.v[v];
          go[g + v] = po.v[v];
        }
    }
  }
  for (int k = tid; k < nband; k += nthr) {
    int row, c;
    bv.at(k, row, c);
    const int i = x0 + c * V, j = y0 + row;
    if (k < nxv) {
      const unsigned xin = xin_of(c);
      const P ps = get<P>(px_a + k * 16), xo = get<P>(xx_a + k * 16);
      const T p0 = get<T>(px0_a + k * ES);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (!(xin >> v & 1u)) continue;
        int q;
        const int sd = side_q(i + v, nx, q);
        T* psi = S.psi[0][sd][Q.par_out] + (int64_t)(halo + 1) * j;
        psi[q] = ps.v[v];
        if (i + v == 1 || i + v == S.first_r[0])
          psi[q - 1] = v == 0 ? p0 : ps.v[v == 0 ? 0 : v - 1];
        S.band[0][sd].xi[(int64_t)halo * j + q - 1] = xo.v[v];
      }
    }
    const int y = bv.yrow(row);
    if (y >= 0) {
      const unsigned ok = ok_of(c);
      int q;
      const int sd = side_q(j, ny, q);
      T* psi = S.psi[1][sd][Q.par_out] + i;
      T* xi = S.band[1][sd].xi + px * (q - 1) + i;
      const bool first = j == 1 || j == S.first_r[1];
      const int at = (y * cw + c) * 16;
      const P lo = get<P>(ylo_a + at), hi = get<P>(yhi_a + at), xo = get<P>(xy_a + at);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (!(ok >> v & 1u)) continue;
        psi[px * q + v] = hi.v[v];
        if (first) psi[px * (q - 1) + v] = lo.v[v];
        xi[v] = xo.v[v];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// One 2D step of a grid too large for the chip: warp w of a block owns a strip
// of 32 vectors x R rows and issues every load of it (R + 2 pressure rows, R
// rows of p_{t-1} and of fact, a vector per lane) before any arithmetic; x
// neighbours come from the adjacent lanes. Bound by HBM: 16 bytes per node and
// step in FP32. At 5210 x 2604 a step takes 47 us (4.6 TB/s) where one node per
// thread (step2d) takes 88; strips of 1 and 4 rows 55 us, 8 warps of 4 rows 55.
constexpr int STRIP_WARPS = 4, STRIP_R = 2;
template <typename T>
__global__ void __launch_bounds__(32 * STRIP_WARPS) step2d_strip(StepParams<T> P) {
  using K = Pack<T>;
  constexpr int V = K::V, R = STRIP_R, TX = 32 * V, TY = STRIP_WARPS * R;
  const int lane = threadIdx.x, w = threadIdx.y;
  const int nx = P.nx, ny = P.ny, halo = P.halo;
  const int blk = blockIdx.x + gridDim.x * blockIdx.y;
  if (blk == 0 && P.do_rim && P.io.nrim > 0) rim_io(P.io, P.pnew, P.it);
  const int xw = blockIdx.x * TX, i = xw + lane * V;
  const int j0 = 1 + blockIdx.y * TY + w * R;
  if (j0 > ny - 2) return;  // whole warp
  const int64_t px = P.px;
  const T* __restrict__ pcur = P.pcur;
  // lanes past the row's end load its last vector, rows past the grid its last
  // rows; what they compute is not stored
  const int64_t il = min((int64_t)i, px - V);
  K q[R + 2], o[R], f[R];
  T xe[R];
#pragma unroll
  for (int r = 0; r < R + 2; ++r) q[r] = ldg_pack<T>(pcur + il + px * min(j0 - 1 + r, ny - 1));
  const int64_t ie = lane == 0 ? max(i - 1, 0) : min((int64_t)i + V, px - 1);
  const bool edge = lane == 0 || lane == 31;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t row = px * min(j0 + r, ny - 2);
    o[r] = ldg_pack<T>(P.pold + il + row);
    f[r] = ldg_pack<T>(P.fact + il + row);
    xe[r] = edge ? __ldg(pcur + ie + row) : T(0);
  }
  unsigned ok = 0;
#pragma unroll
  for (int v = 0; v < V; ++v)
    if (i + v >= 1 && i + v <= nx - 2) ok |= 1u << v;
  const bool xband = (P.active[0][0] && xw <= halo) || (P.active[0][1] && xw + TX - 1 >= nx - halo - 1);
  const bool yband = (P.active[1][0] && j0 <= halo) || (P.active[1][1] && j0 + R - 1 >= ny - halo - 1);
  const int e0 = P.io.blk_off[blk], e1 = P.io.blk_off[blk + 1];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = j0 + r;
    const K& c = q[r + 1];
    T xm = __shfl_up_sync(0xffffffffu, c.v[V - 1], 1), xp = __shfl_down_sync(0xffffffffu, c.v[0], 1);
    if (lane == 0) xm = xe[r];
    if (lane == 31) xp = xe[r];
    K nv, d2x, d2y;
    vec_update(q[r], c, q[r + 2], o[r], f[r], xm, xp, P.inv_d2[0], P.inv_d2[1], d2x, d2y, nv);
    if (j > ny - 2) continue;
    if (xband || yband) {
      // all of the row's ψ and ξ are loaded before any is used
      T damp[V], ps[V], pm[V], xo[V];
      K yq, ym, yx;
      int side[V], qx[V], qy = 0;
      bool fx[V], fy = false;
      int by = yband ? band_of(j, ny, halo, P.first_r[1], qy, fy) : 0;
      if (by != 0 && !P.active[1][by - 1]) by = 0;
      const bool in = ok != 0;  // the lane's vector lies in the grid's pitched row
      if (by != 0 && in) {
        const BandSide<T>& B = P.band[1][by - 1];
        yq = *reinterpret_cast<const K*>(B.psi_old + px * qy + i);
        ym = *reinterpret_cast<const K*>(B.psi_old + px * (qy - 1) + i);
        yx = *reinterpret_cast<const K*>(B.xi + px * (qy - 1) + i);
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        damp[v] = T(0);
        side[v] = xband && (ok >> v & 1u) ? band_of(i + v, nx, halo, P.first_r[0], qx[v], fx[v]) : 0;
        if (side[v] != 0 && !P.active[0][side[v] - 1]) side[v] = 0;
        if (side[v] == 0) continue;
        const BandSide<T>& B = P.band[0][side[v] - 1];
        ps[v] = B.psi_old[(int64_t)(halo + 1) * j + qx[v]];
        pm[v] = B.psi_old[(int64_t)(halo + 1) * j + qx[v] - 1];
        xo[v] = B.xi[(int64_t)halo * j + qx[v] - 1];
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (side[v] == 0) continue;
        const BandSide<T>& B = P.band[0][side[v] - 1];
        T sq, sm, xn;
        cpml_axis(band_coef(B, qx[v]), ps[v], pm[v], xo[v], v == 0 ? xm : c.v[v == 0 ? 0 : v - 1],
                  c.v[v], v == V - 1 ? xp : c.v[v == V - 1 ? v : v + 1], d2x.v[v], f[r].v[v],
                  P.inv_d[0], sq, sm, xn, damp[v]);
        B.psi_new[(int64_t)(halo + 1) * j + qx[v]] = sq;
        if (fx[v]) B.psi_new[(int64_t)(halo + 1) * j + qx[v] - 1] = sm;
        B.xi[(int64_t)halo * j + qx[v] - 1] = xn;
      }
      if (by != 0 && in) {
        const BandSide<T>& B = P.band[1][by - 1];
        const BandCoef<T> cf = band_coef(B, qy);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          T sq, sm, xn;
          cpml_axis(cf, yq.v[v], ym.v[v], yx.v[v], q[r].v[v], c.v[v], q[r + 2].v[v], d2y.v[v],
                    f[r].v[v], P.inv_d[1], sq, sm, xn, damp[v]);
          yq.v[v] = sq;
          ym.v[v] = sm;
          yx.v[v] = xn;
        }
        // the Dirichlet columns' entries are written too; nothing reads them
        *reinterpret_cast<K*>(B.psi_new + px * qy + i) = yq;
        if (fy) *reinterpret_cast<K*>(B.psi_new + px * (qy - 1) + i) = ym;
        *reinterpret_cast<K*>(B.xi + px * (qy - 1) + i) = yx;
      }
#pragma unroll
      for (int v = 0; v < V; ++v) nv.v[v] += damp[v];
    }
    for (int e = e0; e < e1; ++e) {
      const int4 en = P.io.ent[e];
      const int lx = en.x % TX - lane * V;
      if (en.x / TX != w * R + r || lx < 0 || lx >= V) continue;
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (v == lx) nv.v[v] = node_io(P.io, P.it, en.z, en.w, nv.v[v]);
    }
    T* out = P.pnew + i + px * j;
    if (ok == (1u << V) - 1u) {
      *reinterpret_cast<K*>(out) = nv;
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (ok >> v & 1u) out[v] = nv.v[v];
    }
  }
}

}  // namespace awc
