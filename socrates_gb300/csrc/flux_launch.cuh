// flux_launch.cuh -- dispatch of the templated flux kernel over the tile
// shapes (lanes per solve P, layers per lane CH) it is instantiated for.
#pragma once

#include <algorithm>
#include <cstdio>
#include "flux_kernel.cuh"
#include "flux_tau_kernel.cuh"
#include "region_rows.h"

namespace socgpu {

template <int P_, int CH_>
struct Shape { static constexpr int P = P_, CH = CH_; };

// Whether batch p runs on the mixed kernels in optical-depth form.
template <class R, bool MCICA>
constexpr bool tau_form(const FluxParams &p) { return sizeof(R) == 4 && !(MCICA && p.region); }

constexpr int kRegionCtasPerSm = 4, kRegionWarps = 4;

inline TauChip tau_chip() {
  int dev = 0, n = 0, cta = 0, sm = 0, kept = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&cta, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&kept, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  return TauChip{n, (size_t)cta, (size_t)sm, (size_t)kept};
}

// The kernel of shape S built for mb resident CTAs (tau_min_ctas of them where
// no other is built).
template <bool NOSCAT, bool MCICA, int SRC, class S>
auto tau_single(int mb) {
  constexpr int least = tau_min_ctas(S::CH), most = tau_dense_ctas(S::P, S::CH, MCICA);
  if constexpr (most >= 4) if (mb == 4) return tau_kernel<S::P, S::CH, NOSCAT, MCICA, SRC, 4>;
  if constexpr (most >= 3) if (mb == 3) return tau_kernel<S::P, S::CH, NOSCAT, MCICA, SRC, 3>;
  return tau_kernel<S::P, S::CH, NOSCAT, MCICA, SRC, least>;
}
template <bool NOSCAT, bool MCICA, int SRC, class S>
auto tau_batched(int mb) {
  constexpr int least = tau_min_ctas(S::CH), most = tau_dense_ctas(S::P, S::CH, MCICA);
  if constexpr (most >= 4) if (mb == 4) return tau_kernel_batched<S::P, S::CH, NOSCAT, MCICA, SRC, 4>;
  if constexpr (most >= 3) if (mb == 3) return tau_kernel_batched<S::P, S::CH, NOSCAT, MCICA, SRC, 3>;
  return tau_kernel_batched<S::P, S::CH, NOSCAT, MCICA, SRC, least>;
}

// Threads that solve a cloud-region column's g-points at a time: whole warps
// for the calls of up to 64 g-points.
inline int region_rt(const FluxParams &p) { return std::min(kRegionRt, (p.g_end - p.g_begin + 15) / 16 * 16); }

// Resident CTAs of a cloud-region launch: four of four warps to an SM (solar,
// 1025 x 70 x 48: 904 us; two of eight warps 1232, four of two 987).
template <class K>
int region_ctas(K kern, int threads, size_t bytes) {
  int per_sm = 0, dev = 0, n_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, bytes) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
  }
  return std::min(per_sm, kRegionCtasPerSm) * n_sm;
}

// One batch on the mixed kernel of shape S.
template <bool NOSCAT, bool MCICA, int SRC, class S>
int launch_tau(const FluxParams &p, const TileConfig &cfg, cudaStream_t st, char *msg, size_t len) {
  FluxParams q = p;
  int warps = cfg.warps_per_cta, mb = 0;
  const TauChip chip = tau_chip();
  const TauShape shape = tau_choose(&q, 1, S::P * S::CH, S::P, warps, MCICA, tau_dense_ctas(S::P, S::CH, MCICA), chip);
  if (shape.warps) {
    warps = shape.warps;
    mb = shape.mb;
  } else {
    if (warps == 0) warps = 8;
    while (!tau_fit(q, S::P * S::CH, S::P, warps, MCICA, chip)) {
      if (warps == 1) {
        snprintf(msg, len, "one band of %d layers needs %u bytes of shared memory (limit %zu)", p.n_layer, q.tau.stride,
                 chip.cta);
        return SOCGPU_I_ERR_RANGE;
      }
      warps /= 2;
    }
  }
  const size_t bytes = tau_bytes(q);
  auto kern = tau_single<NOSCAT, MCICA, SRC, S>(mb);
  cudaError_t e = allow_shared((const void *)kern, bytes, 0);
  if (e != cudaSuccess) {
    snprintf(msg, len, "shared memory request of %zu bytes refused: %s", bytes, cudaGetErrorString(e));
    return SOCGPU_I_ERR_RANGE;
  }
  if (p.n_profile <= 0) return 0;
  kern<<<(p.n_profile + q.tau.cols - 1) / q.tau.cols, warps * 32, bytes, st>>>(q);
  count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    snprintf(msg, len, "flux kernel launch failed: %s", cudaGetErrorString(e));
    return SOCGPU_I_ABORT_CALCULATION;
  }
  return 0;
}

// One kernel class on the mixed kernel of shape S: every item's layout, the
// work in column groups, and a persistent grid.
template <bool NOSCAT, bool MCICA, int SRC, class S>
int prepare_tau(BatchGroup &g, char *msg, size_t len) {
  for (int i = 0; i < g.n_items; ++i)
    if (g.items[i].n_layer > S::P * S::CH) {
      snprintf(msg, len, "batch %d has %d layers, more than the %d of its tile", i, g.items[i].n_layer, S::P * S::CH);
      return SOCGPU_I_ERR_RANGE;
    }
  TauChip chip = tau_chip();
  const size_t optin = chip.cta;
  // the kernel's static shared memory (its parameter copy) counts too
  auto static_of = [&](const void *kern) {
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, kern) == cudaSuccess) return (long long)fa.sharedSizeBytes;
    cudaGetLastError();
    snprintf(msg, len, "attributes of the batched kernel not available");
    return -1LL;
  };
  auto kern = tau_batched<NOSCAT, MCICA, SRC, S>(0);
  const long long fixed = static_of((const void *)kern);
  if (fixed < 0) return SOCGPU_I_ABORT_CALCULATION;
  chip.cta = optin - std::min(optin, (size_t)fixed);
  chip.besides += (size_t)fixed;
  int warps = g.tile.warps_per_cta;
  const TauShape shape = tau_choose(g.items, g.n_items, S::P * S::CH, S::P, warps, MCICA,
                                    tau_dense_ctas(S::P, S::CH, MCICA), chip);
  if (shape.warps) {
    warps = shape.warps;
    kern = tau_batched<NOSCAT, MCICA, SRC, S>(shape.mb);
  } else if (warps == 0) {
    warps = 8;
  }
  size_t bytes = 0;
  long long alone = 0;                  // CTAs with one column
  for (int i = 0; i < g.n_items; ++i) {
    FluxParams &p = g.items[i];
    if (!shape.warps && !tau_fit(p, S::P * S::CH, S::P, warps, MCICA, chip)) {
      snprintf(msg, len, "batch %d: one band needs %u bytes of shared memory (limit %zu)", i, p.tau.stride, chip.cta);
      return SOCGPU_I_ERR_RANGE;
    }
    bytes = std::max(bytes, tau_bytes(p));
    g.col_start[i + 1] = g.col_start[i] + (p.n_profile + p.tau.cols - 1) / p.tau.cols;
    if (p.tau.cols == 1) alone += p.n_profile;
  }
  g.total = g.col_start[g.n_items];
  if (!shape.warps && warps == 8 && 2 * alone > g.total && tau_narrow(g.total, chip))
    kern = tau_batched<NOSCAT, MCICA, SRC, S>(3);
  cudaError_t e = allow_shared((const void *)kern, bytes, (size_t)fixed);
  if (e != cudaSuccess) {
    snprintf(msg, len, "shared memory request of %zu bytes refused: %s", bytes, cudaGetErrorString(e));
    return SOCGPU_I_ERR_RANGE;
  }
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, bytes);
  if (e != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    snprintf(msg, len, "no CTA of %d threads and %zu bytes fits an SM", warps * 32, bytes);
    return SOCGPU_I_ERR_RANGE;
  }
  g.kernel = (const void *)kern;
  g.smem = bytes;
  g.threads = warps * 32;
  g.grid = (int)std::min<long long>(g.total, (long long)per_sm * chip.n_sm);
  return 0;
}

template <class R, bool MIX, bool NOSCAT, bool MCICA, int SRC, class S>
int try_launch(const FluxParams &p, const TileConfig &cfg, cudaStream_t st, char *msg, size_t len,
               bool &done) {
  if (done || cfg.lanes_per_solve != S::P || S::P * S::CH < p.n_layer) return 0;
  if (cfg.chunk && cfg.chunk != S::CH) return 0;
  // the smallest chunk of this P that covers the column is chosen by the
  // caller's ordering of shapes (ascending CH)
  done = true;
  if constexpr (sizeof(R) == 4) {
    if (tau_form<R, MCICA>(p)) return launch_tau<NOSCAT, MCICA, SRC, S>(p, cfg, st, msg, len);
  }
  if constexpr (sizeof(R) == 8 || MCICA) {
  const int nb = p.last_band - p.first_band + 1;
  int max_smem = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  // widest band batch (then most warps) whose staging fits in shared memory
  // (no warps are given for mixed equivalent extinction: cloud regions here)
  const int given = cfg.warps_per_cta > 0 ? cfg.warps_per_cta : 8;
  int warps = MCICA && p.region ? std::min(given, kRegionWarps) : given, batch = nb;
  SmemLayout lay{};
  FluxParams q = p;
  for (;;) {
    lay = make_layout<R>(q, S::P * S::CH, S::P, batch, warps * 32 / S::P, MCICA,
                         FluxKernel<R, MIX, S::P, S::CH, NOSCAT, MCICA, SRC>::kRawFetch);
    if ((long long)lay.bytes <= max_smem) break;
    if (batch > 1) { --batch; continue; }
    if (warps > 1) { warps /= 2; batch = nb; continue; }
    if (lay.ksi_on) { q.no_ksi = 1; batch = nb; continue; }
    snprintf(msg, len, "one band of %d layers needs %zu bytes of shared memory (limit %d)", p.n_layer, lay.bytes,
             max_smem);
    return SOCGPU_I_ERR_RANGE;
  }
  const int threads = warps * 32;
  q.band_batch = batch;
  auto kern = flux_kernel<R, MIX, S::P, S::CH, NOSCAT, MCICA, SRC>;
  cudaError_t e = allow_shared((const void *)kern, lay.bytes, 0);
  if (e != cudaSuccess) {
    snprintf(msg, len, "shared memory request of %zu bytes refused: %s", lay.bytes, cudaGetErrorString(e));
    return SOCGPU_I_ERR_RANGE;
  }
  if (p.n_profile <= 0) return 0;
  int grid = p.n_profile;
  if (MCICA && p.region) {
    q.region_rt = region_rt(p);
    q.region_stride = region_cta_bytes<R>(q);
    long long ctas = region_grid(std::min(grid, region_ctas(kern, threads, lay.bytes)), q.region_stride);
    const bool rows = take_rows(ctas, q.region_stride, [&](size_t bytes) {
      if (scratch_alloc(&q.region_scr, bytes, st) == cudaSuccess) return true;
      cudaGetLastError();
      return false;
    });
    grid = (int)ctas;
    if (!rows) {
      snprintf(msg, len, "no device memory for the cloud regions' rows");
      return SOCGPU_I_ABORT_CALCULATION;
    }
  }
  kern<<<grid, threads, lay.bytes, st>>>(q);
  count_launch();
  e = cudaGetLastError();
  if (MCICA && p.region) scratch_free(q.region_scr, st);
  if (e != cudaSuccess) {
    snprintf(msg, len, "flux kernel launch failed: %s", cudaGetErrorString(e));
    return SOCGPU_I_ABORT_CALCULATION;
  }
  }
  return 0;
}

// Prepare one kernel class of a multi-batch launch for shape S: the band
// batch of every item so that all fit one shared-memory size, the kernel
// attribute, and a persistent grid of the resident CTAs of every SM.
template <class R, bool MIX, bool NOSCAT, bool MCICA, int SRC, class S>
int try_prepare(BatchGroup &g, char *msg, size_t len, bool &done) {
  if (done || g.tile.lanes_per_solve != S::P || g.tile.chunk != S::CH) return 0;
  done = true;
  if constexpr (sizeof(R) == 4) {
    // a class holds cloud regions only, or none (its key says which)
    if (g.n_items == 0 || tau_form<R, MCICA>(g.items[0])) return prepare_tau<NOSCAT, MCICA, SRC, S>(g, msg, len);
  }
  if constexpr (sizeof(R) == 8 || MCICA) {
  int max_smem = 0, dev = 0, n_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  const bool region = MCICA && g.n_items > 0 && g.items[0].region;
  const int given = g.tile.warps_per_cta > 0 ? g.tile.warps_per_cta : 8;
  int warps = region ? std::min(given, kRegionWarps) : given;
  auto bytes_of = [&](const FluxParams &p, int batch) {
    return make_layout<R>(p, S::P * S::CH, S::P, batch, warps * 32 / S::P, MCICA,
                          FluxKernel<R, MIX, S::P, S::CH, NOSCAT, MCICA, SRC>::kRawFetch).bytes;
  };
  auto kern = flux_kernel_batched<R, MIX, S::P, S::CH, NOSCAT, MCICA, SRC>;
  // the kernel's static shared memory (its parameter copy) counts against
  // the same per-CTA limit
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) {
    cudaGetLastError();
    snprintf(msg, len, "attributes of the batched kernel not available");
    return SOCGPU_I_ABORT_CALCULATION;
  }
  const size_t dyn_cap = (size_t)max_smem > fa.sharedSizeBytes ? (size_t)max_smem - fa.sharedSizeBytes : 0;
  // the launch's shared memory: the largest whole-spectrum staging of any
  // item, capped at the device limit; items that need more stage their bands
  // in batches
  size_t smem = 0;
  for (int i = 0; i < g.n_items; ++i) {
    FluxParams &p = g.items[i];
    if (p.n_layer > S::P * S::CH) {
      snprintf(msg, len, "batch %d has %d layers, more than the %d of its tile", i, p.n_layer, S::P * S::CH);
      return SOCGPU_I_ERR_RANGE;
    }
    // fewer warps for all, then no ksi_0 row, where one band does not fit
    while (bytes_of(p, 1) > dyn_cap && warps > 1) warps /= 2;
    p.no_ksi = bytes_of(p, 1) > dyn_cap;
    if (bytes_of(p, 1) > dyn_cap) {
      snprintf(msg, len, "batch %d: one band needs %zu bytes of shared memory (limit %zu)", i, bytes_of(p, 1), dyn_cap);
      return SOCGPU_I_ERR_RANGE;
    }
  }
  for (int i = 0; i < g.n_items; ++i) {
    const FluxParams &p = g.items[i];
    smem = std::max(smem, bytes_of(p, p.last_band - p.first_band + 1));
  }
  smem = std::min(smem, dyn_cap);
  for (int i = 0; i < g.n_items; ++i) {
    FluxParams &p = g.items[i];
    int batch = p.last_band - p.first_band + 1;
    while (batch > 1 && bytes_of(p, batch) > smem) --batch;
    p.band_batch = batch;
  }
  const size_t dyn = smem;
  cudaError_t e = allow_shared((const void *)kern, dyn, fa.sharedSizeBytes);
  if (e != cudaSuccess) {
    snprintf(msg, len, "shared memory request of %zu bytes refused: %s", dyn, cudaGetErrorString(e));
    return SOCGPU_I_ERR_RANGE;
  }
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, dyn);
  if (e != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    snprintf(msg, len, "no CTA of %d threads and %zu bytes fits an SM", warps * 32, dyn);
    return SOCGPU_I_ERR_RANGE;
  }
  g.kernel = (const void *)kern;
  g.smem = dyn;
  g.threads = warps * 32;
  g.grid = (int)std::min<long long>(g.total, (long long)per_sm * n_sm);
  if (region) {
    // the resident CTAs' rows, sized for the widest item
    size_t cta = 0;
    for (int i = 0; i < g.n_items; ++i) {
      g.items[i].region_rt = region_rt(g.items[i]);
      cta = std::max(cta, region_cta_bytes<R>(g.items[i]));
    }
    for (int i = 0; i < g.n_items; ++i) g.items[i].region_stride = cta;
    g.grid = (int)region_grid(std::min<long long>(g.total, (long long)std::min(per_sm, kRegionCtasPerSm) * n_sm), cta);
    g.scratch = cta * g.grid;
  }
  }
  return 0;
}

template <class R, bool MIX, bool NOSCAT, bool MCICA, int SRC, class... Shapes>
int prepare_shapes(BatchGroup &g, char *msg, size_t len) {
  bool done = false;
  int status = 0;
  ((status = status ? status : try_prepare<R, MIX, NOSCAT, MCICA, SRC, Shapes>(g, msg, len, done)), ...);
  if (!done && status == 0) {
    snprintf(msg, len, "no kernel instantiated for %d lanes per solve and %d layers per lane",
             g.tile.lanes_per_solve, g.tile.chunk);
    return SOCGPU_I_ERR_RANGE;
  }
  return status;
}

template <class R, bool MIX, bool NOSCAT, bool MCICA, int SRC, class... Shapes>
int launch_shapes(const FluxParams &p, const TileConfig &cfg, cudaStream_t st, char *msg, size_t len) {
  bool done = false;
  int status = 0;
  ((status = status ? status : try_launch<R, MIX, NOSCAT, MCICA, SRC, Shapes>(p, cfg, st, msg, len, done)), ...);
  if (!done && status == 0) {
    snprintf(msg, len, "no kernel instantiated for %d lanes per solve and %d layers", cfg.lanes_per_solve,
             p.n_layer);
    return SOCGPU_I_ERR_RANGE;
  }
  return status;
}


// The kernels of one source (SOCGPU_IP_SOLAR or SOCGPU_IP_INFRA_RED) over the
// chunk list; the build compiles the two sources as separate objects and the
// infra-red object's entry points hand solar work to the solar one.
template <class R, bool MIX, bool NOSCAT, bool MCICA, int SRC, int P, int... CH>
int launch_chunks(const FluxParams &p, const TileConfig &cfg, cudaStream_t st, char *msg, size_t len) {
  return launch_shapes<R, MIX, NOSCAT, MCICA, SRC, Shape<P, CH>...>(p, cfg, st, msg, len);
}

template <class R, bool MIX, bool NOSCAT, bool MCICA, int SRC, int P, int... CH>
int prepare_chunks(BatchGroup &g, char *msg, size_t len) {
  for (int i = 0; i < g.n_items; ++i)
    if (g.items[i].isolir != SRC) {
      snprintf(msg, len, "a kernel class mixes solar and infra-red batches");
      return SOCGPU_I_ERR_FATAL;
    }
  return prepare_shapes<R, MIX, NOSCAT, MCICA, SRC, Shape<P, CH>...>(g, msg, len);
}

// Load every kernel of the chunk list onto the device now (cudaFuncGetAttributes
// loads a lazily-loaded function): a first launch that loads its module can
// wait for kernels already running, which a request server must not do.
template <class R, bool MIX, bool NOSCAT, bool MCICA, int SRC, int P, int... CH>
int preload_chunks() {
  cudaFuncAttributes a{};
  bool ok = true;
  if constexpr (sizeof(R) == 8 || MCICA) {
    ((ok = ok && cudaFuncGetAttributes(&a, flux_kernel<R, MIX, P, CH, NOSCAT, MCICA, SRC>) == cudaSuccess), ...);
    ((ok = ok && cudaFuncGetAttributes(&a, flux_kernel_batched<R, MIX, P, CH, NOSCAT, MCICA, SRC>) == cudaSuccess),
     ...);
  }
  if constexpr (sizeof(R) == 4) {
    for (int mb = 0; mb <= 4; ++mb) {
      ((ok = ok && cudaFuncGetAttributes(&a, tau_single<NOSCAT, MCICA, SRC, Shape<P, CH>>(mb)) == cudaSuccess), ...);
      ((ok = ok && cudaFuncGetAttributes(&a, tau_batched<NOSCAT, MCICA, SRC, Shape<P, CH>>(mb)) == cudaSuccess), ...);
    }
  }
  if (!ok) cudaGetLastError();
  return ok ? 0 : SOCGPU_I_ABORT_CALCULATION;
}

}  // namespace socgpu
