// kernels.cu -- instantiates the pmhd kernels for every precision policy and
// tile height and exposes them through a KernelTable.  Built twice by the
// Makefile:
//   -DPMHD_KNS=exact -fmad=false                  -> kernel_table_exact()
//   -DPMHD_KNS=fast  -fmad=true -prec-div=false -prec-sqrt=false
//                                                 -> kernel_table_fast()
#include <mutex>

#include "stage_kernels.cuh"

namespace pmhd {
namespace PMHD_KNS {

#include "hancock_kernel.cuh"  // no includes of its own; lives in this namespace

// 32 x 19 tiles may cover fewer rows (tile_rows).
template <int TY>
constexpr bool kPartial = TY == kTileShapes[0];

using StageFn = void (*)(Member, Batch, int, int, unsigned);

template <class Pol, bool HLLD, int TY, bool BATCHED>
static StageFn stage_fn(int stage, bool partial) {
  if constexpr (kPartial<TY>)
    if (partial) return stage == 1 ? stage_kernel<Pol, 1, HLLD, TY, BATCHED, true> : stage_kernel<Pol, 2, HLLD, TY, BATCHED, true>;
  return stage == 1 ? stage_kernel<Pol, 1, HLLD, TY, BATCHED, false> : stage_kernel<Pol, 2, HLLD, TY, BATCHED, false>;
}

template <class Pol, bool HLLD, int TY, bool BATCHED>
static cudaError_t set_smem_attr() {
  cudaError_t e = cudaSuccess;
  for (int partial = 0; partial <= (kPartial<TY> ? 1 : 0); partial++)
    for (int stage = 1; stage <= 2 && e == cudaSuccess; stage++)
      e = cudaFuncSetAttribute(stage_fn<Pol, HLLD, TY, BATCHED>(stage, partial != 0),
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Smem<Pol, TY>::total);
  return e;
}

template <class Pol, int TY, bool BATCHES>
static cudaError_t init_pol_ty(int hlld, bool batched) {
  if constexpr (BATCHES)
    if (batched) return hlld ? set_smem_attr<Pol, true, TY, true>() : set_smem_attr<Pol, false, TY, true>();
  if (batched) return cudaErrorNotSupported;
  return hlld ? set_smem_attr<Pol, true, TY, false>() : set_smem_attr<Pol, false, TY, false>();
}

// The policy has the shapes past kNumBatchShapes: the performance build's binary64.
template <class Pol>
constexpr bool kAllShapes = PMHD_FAST_FLUX != 0 && !Pol::kMixed && sizeof(typename Pol::R) == 8;

template <class Pol>
static cudaError_t init_pol(int hlld, int ty_idx, bool batched) {
  if (ty_idx == 0) return init_pol_ty<Pol, kTileShapes[0], true>(hlld, batched);
  if (ty_idx == 1) return init_pol_ty<Pol, kTileShapes[1], true>(hlld, batched);
  if constexpr (kAllShapes<Pol>) {
    if (ty_idx == 2) return init_pol_ty<Pol, kTileShapes[2], false>(hlld, batched);
    if (ty_idx == 3) return init_pol_ty<Pol, kTileShapes[3], false>(hlld, batched);
    if (ty_idx == 4) return init_pol_ty<Pol, kTileShapes[4], false>(hlld, batched);
  }
  return cudaErrorNotSupported;
}

static cudaError_t init_stage(int precision, int hlld, int ty_idx, int batched) {
  switch (precision) {
    case PREC_FP64: return init_pol<PolF64>(hlld, ty_idx, batched != 0);
    case PREC_FP32: return init_pol<PolF32>(hlld, ty_idx, batched != 0);
    case PREC_MIXED: return init_pol<PolMixed>(hlld, ty_idx, batched != 0);
    default: return cudaErrorInvalidValue;
  }
}

template <class Pol, bool HLLD>
static cudaError_t init_hancock_pol() {
  const int smem = (int)sizeof(HancockTileOf<Pol>);
  if constexpr (HancockPersistent<Pol>::on)
    return cudaFuncSetAttribute(hancock_persistent_kernel<Pol, HLLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  else
    return cudaFuncSetAttribute(hancock_kernel<Pol, HLLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

static cudaError_t init_hancock(int precision, int hlld) {
  switch (precision) {
    case PREC_FP64: return hlld ? init_hancock_pol<PolF64, true>() : init_hancock_pol<PolF64, false>();
    case PREC_FP32: return hlld ? init_hancock_pol<PolF32, true>() : init_hancock_pol<PolF32, false>();
    case PREC_MIXED: return hlld ? init_hancock_pol<PolMixed, true>() : init_hancock_pol<PolMixed, false>();
    default: return cudaErrorInvalidValue;
  }
}

static int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 1;
}

template <class Pol, bool HLLD, int TY, bool BATCHED>
static int occupancy() {
  static int per_sm = -1;
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  if (per_sm < 0) {
    int nb = 0;
    set_smem_attr<Pol, HLLD, TY, BATCHED>();  // without it the answer is 0
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, stage_kernel<Pol, 1, HLLD, TY, BATCHED, false>, Geo<TY>::NT,
                                                  Smem<Pol, TY>::total);
    per_sm = nb > 0 ? nb : 1;
  }
  return per_sm;
}

// Tiles per run of a batched launch of `ntiles` tiles on `grid` CTAs.  A run
// flushes a member's counts and reads the next one's descriptor and control slot,
// so short lists are one run a CTA (16 members of 64^2 .. 256^2, 700 tiles on 148
// CTAs: 113 us a step, 123 as runs of one, 324 as 44 runs of 16); longer ones take
// the longest power of two whose busiest CTA gets at most 1/16 more tiles than it
// would with runs of one (the 512-member benchmark ensemble, 73,000 tiles: 16; 48
// members of 64^2 .. 512^2: 880 us with 4, 894 with 11, where full tiles gather in
// some CTAs and the grids' short edge tiles in others).
static int batch_run(int ntiles, int grid) {
  const long long even = ((long long)ntiles + grid - 1) / grid;
  if (even <= kBatchRunMax) return even > 1 ? (int)even : 1;
  for (int run = kBatchRunMax; run > 1; run /= 2) {
    const long long units = ((long long)ntiles + run - 1) / run;
    const long long most = (units + grid - 1) / grid * run;
    if (16 * most <= 17 * even) return run;
  }
  return 1;
}

template <class Pol, bool HLLD, int TY, bool BATCHED>
static cudaError_t launch_one(int stage, const Batch& b, const Member& m0, int parity, int run, int grid,
                              cudaStream_t s) {
  const size_t smem = Smem<Pol, TY>::total;
  const StageFn kernel = stage_fn<Pol, HLLD, TY, BATCHED>(stage, b.rows < tile_height(0));
  kernel<<<grid, Geo<TY>::NT, smem, s>>>(m0, b, parity, run, ((1u << 28) + run - 1) / run);
  return cudaGetLastError();
}

template <class Pol, int TY, bool BATCHES>
static int occ_pol_ty(int hlld, bool batched) {
  if constexpr (BATCHES)
    if (batched) return hlld ? occupancy<Pol, true, TY, true>() : occupancy<Pol, false, TY, true>();
  return hlld ? occupancy<Pol, true, TY, false>() : occupancy<Pol, false, TY, false>();
}

template <class Pol, int TY, bool BATCHES>
static cudaError_t launch_stage_pol(int hlld, int stage, const Batch& b, const Member* single, int parity, int grid,
                                    cudaStream_t s) {
  if (b.ntiles <= 0) return cudaSuccess;
  const bool batched = single == nullptr;
  if (batched && !BATCHES) return cudaErrorNotSupported;
  if (grid <= 0) grid = sm_count() * occ_pol_ty<Pol, TY, BATCHES>(hlld, batched);
  const int run = batched ? batch_run(b.ntiles, grid) : 1;
  const int units = (b.ntiles + run - 1) / run;  // runs of tiles
  if (grid > units) grid = units;
  static const Member empty = {};
  const Member& m0 = batched ? empty : *single;
  if constexpr (BATCHES) {
    if (batched) {
      return hlld ? launch_one<Pol, true, TY, true>(stage, b, m0, parity, run, grid, s)
                  : launch_one<Pol, false, TY, true>(stage, b, m0, parity, run, grid, s);
    }
  }
  return hlld ? launch_one<Pol, true, TY, false>(stage, b, m0, parity, run, grid, s)
              : launch_one<Pol, false, TY, false>(stage, b, m0, parity, run, grid, s);
}

template <class Pol>
static cudaError_t launch_stage_ty(int hlld, int stage, int ty_idx, const Batch& b, const Member* single, int parity,
                                   int grid, cudaStream_t s) {
  if (ty_idx == 0) return launch_stage_pol<Pol, kTileShapes[0], true>(hlld, stage, b, single, parity, grid, s);
  if (ty_idx == 1) return launch_stage_pol<Pol, kTileShapes[1], true>(hlld, stage, b, single, parity, grid, s);
  if constexpr (kAllShapes<Pol>) {
    if (ty_idx == 2) return launch_stage_pol<Pol, kTileShapes[2], false>(hlld, stage, b, single, parity, grid, s);
    if (ty_idx == 3) return launch_stage_pol<Pol, kTileShapes[3], false>(hlld, stage, b, single, parity, grid, s);
    if (ty_idx == 4) return launch_stage_pol<Pol, kTileShapes[4], false>(hlld, stage, b, single, parity, grid, s);
  }
  return cudaErrorNotSupported;
}

static cudaError_t launch_stage(int precision, int hlld, int stage, int ty_idx, const Batch& b, const Member* single,
                                int parity, int grid, cudaStream_t s) {
  switch (precision) {
    case PREC_FP64: return launch_stage_ty<PolF64>(hlld, stage, ty_idx, b, single, parity, grid, s);
    case PREC_FP32: return launch_stage_ty<PolF32>(hlld, stage, ty_idx, b, single, parity, grid, s);
    case PREC_MIXED: return launch_stage_ty<PolMixed>(hlld, stage, ty_idx, b, single, parity, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

template <class Pol>
static int occ_pol(int hlld, int ty_idx, bool batched) {
  if constexpr (kAllShapes<Pol>) {
    if (ty_idx == 2) return occ_pol_ty<Pol, kTileShapes[2], false>(hlld, batched);
    if (ty_idx == 3) return occ_pol_ty<Pol, kTileShapes[3], false>(hlld, batched);
    if (ty_idx == 4) return occ_pol_ty<Pol, kTileShapes[4], false>(hlld, batched);
  }
  return ty_idx == 0 ? occ_pol_ty<Pol, kTileShapes[0], true>(hlld, batched)
                     : occ_pol_ty<Pol, kTileShapes[1], true>(hlld, batched);
}

static int ctas_per_sm(int precision, int hlld, int ty_idx, int batched) {
  switch (precision) {
    case PREC_FP64: return occ_pol<PolF64>(hlld, ty_idx, batched != 0);
    case PREC_FP32: return occ_pol<PolF32>(hlld, ty_idx, batched != 0);
    default: return occ_pol<PolMixed>(hlld, ty_idx, batched != 0);
  }
}

// Tile shape of a single grid: the smallest split shape that gives every tile an SM
// of its own, if there is one (a stage is then one tile's dependent chain; 64^2
// binary64, us a step: 33 with 32 x 19 tiles, 20 / 14 / 12 with split 32 x 8 / 4 / 2;
// 192^2: 34 and 20 with split 32 x 8), else 32 x 19.  Only the performance
// build's binary64: the compiler contracts binary32 fluxes differently for every
// shape, and binary32 and mixed results of grids and ensembles stay together.
static int default_shape(int precision, int nx, int ny) {
  if (!PMHD_FAST_FLUX || precision != PREC_FP64) return 0;
  for (int idx = kNumTileShapes - 1; idx >= kNumBatchShapes; idx--)
    if (num_tiles(nx, ny, tile_height(idx)) <= sm_count()) return idx;
  return 0;
}

// Cell rows per tile of a list of grids: the fewest with which the persistent
// CTAs, one per SM, take no more rounds than with full 32 x 19 tiles -- a tile's
// time falls with its rows, and the SMs a short last round leaves idle take part --
// but not 17 or 18: with rows + 1 flux warps a scheduler still has its five, and a
// runtime height and more halo rows cost more than the other phases save (full tiles'
// time over that of fewer rows, ten sizes each, binary32 / mixed / binary64: 17 rows
// 0.96 - 1.01 / 0.97 - 1.03 / 0.96 - 1.02, 18 rows 0.96 - 1.00 / 0.96 - 1.01 / 0.96 - 1.00;
// 16 rows 0.98 - 1.01 / 0.99 - 1.03 / 0.98 - 1.03, kept for their mean of 1.01; 15 rows,
// four warps a scheduler, 1.05 - 1.12 in all).  Mixed, us a step, of few rows against
// full tiles: 64^2 14.6 / 22.4, 128^2 16.1 / 22.4, 320^2 32.0 / 38.2.
// The parity build's bits do not depend on the rows.  The performance build's can,
// through tiny slopes: the tiles at the domain's edge reconstruct by minmod(), whose
// product underflows where minmod_fast() has a value, and the rows move those tiles.
static int tile_rows(int idx, const int (*sizes)[2], int n) {
  const int height = tile_height(idx);
  if (idx != 0) return height;
  auto tiles = [&](int rows) {
    long long t = 0;
    for (int k = 0; k < n; k++) t += num_tiles(sizes[k][0], sizes[k][1], rows);
    return t;
  };
  const long long sms = sm_count(), budget = (tiles(height) + sms - 1) / sms * sms;
  for (int rows = 2; rows < height - 2; rows++)
    if (tiles(rows) <= budget) return rows;
  return height;
}

static int grid_for(long long n) {
  long long b = (n + NTA - 1) / NTA;
  if (b > 148 * 64) b = 148 * 64;
  return (int)(b < 1 ? 1 : b);
}

static cudaError_t launch_speed(int precision, const void* u, long long plane, int nx, int ny, int pitch,
                                double gamma, Ctrl* ctrl, int slot, cudaStream_t s) {
  const int g = grid_for((long long)nx * ny);
  switch (precision) {
    case PREC_FP64:
      speed_kernel<PolF64><<<g, NTA, 0, s>>>(static_cast<const double*>(u), plane, nx, ny, pitch, gamma, ctrl, slot);
      break;
    case PREC_FP32:
      speed_kernel<PolF32><<<g, NTA, 0, s>>>(static_cast<const float*>(u), plane, nx, ny, pitch, gamma, ctrl, slot);
      break;
    case PREC_MIXED:
      speed_kernel<PolMixed><<<g, NTA, 0, s>>>(static_cast<const double*>(u), plane, nx, ny, pitch, gamma, ctrl,
                                              slot);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

static cudaError_t launch_aos_to_soa(int precision, const void* aos, int layout, void* u, long long plane, int nx,
                                     int ny, int pitch, const int bc[4], cudaStream_t s) {
  const int g = grid_for((long long)nx * ny);
  if (precision == PREC_FP32)
    aos_to_soa_kernel<float><<<g, NTA, 0, s>>>(static_cast<const float*>(aos), layout, static_cast<float*>(u), plane,
                                               nx, ny, pitch, bc[0], bc[1], bc[2], bc[3]);
  else
    aos_to_soa_kernel<double><<<g, NTA, 0, s>>>(static_cast<const double*>(aos), layout, static_cast<double*>(u),
                                                plane, nx, ny, pitch, bc[0], bc[1], bc[2], bc[3]);
  return cudaGetLastError();
}

static cudaError_t launch_soa_to_aos(int precision, const void* u, long long plane, int nx, int ny, int pitch,
                                     int layout, void* aos, cudaStream_t s) {
  const long long n = layout == 0 ? (long long)nx * ny : (long long)(nx + 4) * (ny + 4);
  const int g = grid_for(n);
  if (precision == PREC_FP32)
    soa_to_aos_kernel<float><<<g, NTA, 0, s>>>(static_cast<const float*>(u), plane, nx, ny, pitch, layout,
                                               static_cast<float*>(aos));
  else
    soa_to_aos_kernel<double><<<g, NTA, 0, s>>>(static_cast<const double*>(u), plane, nx, ny, pitch, layout,
                                                static_cast<double*>(aos));
  return cudaGetLastError();
}

// Resident CTAs per SM of the persistent Hancock kernel.
template <class Pol, bool HLLD>
static int hancock_occupancy() {
  static int per_sm = -1;
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  if (per_sm < 0) {
    int nb = 0;
    init_hancock_pol<Pol, HLLD>();  // without it the answer is 0
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, hancock_persistent_kernel<Pol, HLLD>, 256,
                                                  sizeof(HancockTileOf<Pol>));
    per_sm = nb > 0 ? nb : 1;
  }
  return per_sm;
}

template <class Pol>
static cudaError_t hancock_pol(int hlld, int part, const Member& m, int parity, cudaStream_t s) {
  if (part == 0) {
    hancock_begin_kernel<Pol><<<1, 32, 0, s>>>(m, parity);
    return cudaGetLastError();
  }
  constexpr int TYH = HancockTileOf<Pol>::TYH;
  const int ntiles = ((m.nx + TX - 1) / TX) * ((m.ny + TYH - 1) / TYH);
  const size_t smem = sizeof(HancockTileOf<Pol>);
  if constexpr (HancockPersistent<Pol>::on) {
    // Persistent: the SMs x the resident CTAs, at most one per tile.
    int grid = sm_count() * (hlld ? hancock_occupancy<Pol, true>() : hancock_occupancy<Pol, false>());
    if (grid > ntiles) grid = ntiles;
    if (hlld)
      hancock_persistent_kernel<Pol, true><<<grid, 256, smem, s>>>(m, parity);
    else
      hancock_persistent_kernel<Pol, false><<<grid, 256, smem, s>>>(m, parity);
  } else {
    if (hlld)
      hancock_kernel<Pol, true><<<ntiles, HancockTileOf<Pol>::NT, smem, s>>>(m, parity);
    else
      hancock_kernel<Pol, false><<<ntiles, HancockTileOf<Pol>::NT, smem, s>>>(m, parity);
  }
  return cudaGetLastError();
}

static cudaError_t launch_hancock(int precision, int hlld, int part, const Member& m, int parity, cudaStream_t s) {
  switch (precision) {
    case PREC_FP64: return hancock_pol<PolF64>(hlld, part, m, parity, s);
    case PREC_FP32: return hancock_pol<PolF32>(hlld, part, m, parity, s);
    case PREC_MIXED: return hancock_pol<PolMixed>(hlld, part, m, parity, s);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace PMHD_KNS

#define PMHD_STR2(x) #x
#define PMHD_STR(x) PMHD_STR2(x)
#define PMHD_TABLE_FN2(n) kernel_table_##n
#define PMHD_TABLE_FN(n) PMHD_TABLE_FN2(n)

const KernelTable& PMHD_TABLE_FN(PMHD_KNS)() {
  static const KernelTable t = {PMHD_STR(PMHD_KNS),          PMHD_KNS::init_stage,
                                PMHD_KNS::init_hancock,      PMHD_KNS::launch_stage,      PMHD_KNS::ctas_per_sm,
                                PMHD_KNS::launch_speed,      PMHD_KNS::launch_aos_to_soa,
                                PMHD_KNS::launch_soa_to_aos, PMHD_KNS::default_shape,
                                PMHD_KNS::tile_rows,         PMHD_KNS::launch_hancock};
  return t;
}

}  // namespace pmhd
