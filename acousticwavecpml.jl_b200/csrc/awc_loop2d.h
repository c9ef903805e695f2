// awc_loop2d.h — host side of the on-chip 2D time loop (awc_loop2d.cuh):
// tiling of a set of shots, device lists, launches. Internal.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "awc_ctx.h"
#include "awc_kernels.cuh"
#include "awc_loop2d.cuh"

namespace awc {

// What the loop needs of one shot: sizes, which band sides are live, device
// pointers of its state (fields, fact, ψ, ξ, packed coefficients, source
// functions, traces), and its source/receiver nodes on the host.
struct LoopShotHost {
  int64_t nx = 0, ny = 0, px = 0;
  int32_t halo = 0;
  int32_t active[2][2] = {};
  double inv_d[2] = {}, inv_d2[2] = {};
  void* buf[3] = {};
  const void* fact = nullptr;
  void* psi[2][2][2] = {};
  void* xi[2][2] = {};
  const void* coef = nullptr;
  const int32_t* src_off = nullptr;
  const int32_t* src_ids = nullptr;
  const void* stf = nullptr;
  void* traces = nullptr;
  int32_t nsrc = 0, nrec = 0;
  const std::vector<IoRim>* nodes = nullptr;  // node, source group, receiver group
  const std::vector<int32_t>* rec_off = nullptr;  // receiver groups (host copy)
  const std::vector<int32_t>* rec_ids = nullptr;
};

// Limit of a wait for an edge value, and the tile of each launch that sends no
// edges (tests of the timeout; -1: none).
struct LoopWait {
  unsigned long long ns = 4096000000ull;
  int32_t withhold = -1;
};

// Where the state of the first and last step lives (buffer numbers of p_t,
// p_{t-1} and the third field; ψ parity), and the fields to keep (see
// LoopRun).
struct LoopSpan {
  int64_t it0 = 0, n = 0;
  int32_t in[3] = {}, out[3] = {}, par_in = 0, par_out = 0;
  void* keep = nullptr;
  int64_t keep_stride = 0, keep_first = 0, keep_count = 0;
  LoopWait wait;
};

// A set of shots that run through the loop: one launch per wave of shots
// whose tiles fill the SMs together.
class Loop2D {
 public:
  ~Loop2D();
  // Tiles the shots (when their shapes changed; no device work). False when
  // one cannot run this way: its tiles do not fit on the chip, or the two
  // bands of an axis share a face.
  bool fits(const awc_ctx* C, bool f64, const std::vector<LoopShotHost>& shots);
  // Device tables of the tiling (when it changed) and the shots' lists.
  int prepare(awc_ctx* C, bool f64, const std::vector<LoopShotHost>& shots, int32_t* err_flag);
  // Enqueues n steps of every shot on st. kLoopRefused: the device had no room for
  // all blocks of a launch at once; nothing ran, and fits() is false from now on.
  int run(awc_ctx* C, const LoopSpan& span, cudaStream_t st);
  int64_t launches() const { return (int64_t)waves_.size(); }

 private:
  struct Tiling {
    int tx = 0, ty = 0;
    std::vector<int> xb, yb;  // first vector column / interior row of each tile, and the end
    double cost = 1e30;
    int tiles() const { return tx * ty; }
  };
  struct Shape {
    int64_t nx, ny;
    int32_t halo, active[2][2];
    bool operator==(const Shape& o) const;
  };
  struct Wave {
    int R = 1, threads = 32, smem = 0, hmax = 0, wmax = 0;
    int64_t tile0 = 0, ntiles = 0;
    std::vector<int> shots, first;  // the shots, and each one's first tile in the wave
    std::vector<Tiling> tiling;
  };
  static std::vector<Tiling> tilings(const Shape& s, bool f64, int max_tiles, bool even = false);
  template <typename T>
  int lay_out(awc_ctx* C);
  template <typename T>
  int upload(awc_ctx* C, const std::vector<LoopShotHost>& shots);
  template <typename T>
  int launch(awc_ctx* C, const LoopSpan& span, cudaStream_t st);
  bool plan_waves(const awc_ctx* C);

  bool f64_ = false, planned_ = false, laid_out_ = false;
  int blocks_ = 0;  // most blocks of a launch the tiling was made for
  std::vector<Shape> shapes_;
  std::vector<Wave> waves_;
  std::vector<LoopTile> tiles_;               // without the shots' lists
  int64_t mail_stride_ = 0;
  int32_t* err_ = nullptr;
  void* table_ = nullptr;  // edge items
  void* blob_ = nullptr;  // tiles, shots, entry lists
  size_t blob_bytes_ = 0;
  size_t o_shots_ = 0, o_srcs_ = 0, o_recs_ = 0;
  unsigned long long* mail_ = nullptr;
  size_t mail_bytes_ = 0;
  uint32_t tag_ = 1;
};

// Runs shorter than this use the per-step kernels: a loop launch loads and
// stores the whole state, which costs about as much as a few steps.
constexpr int64_t kLoopMinSteps = 8;
// What Loop2D::run returns beside the library's status codes.
constexpr int kLoopRefused = 1;

}  // namespace awc
