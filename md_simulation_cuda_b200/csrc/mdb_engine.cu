// Host engine of libmdb200 (see mdb_engine.h) and the kernel instantiations.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <sys/stat.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <fstream>
#include <mutex>
#include <sstream>
#include <string>

#include "mdb_engine.h"
#include "mdb_band.cuh"
#include "mdb_band_steps.cuh"
#include "mdb_kernels.cuh"
#include "mdb_steps.cuh"
#include "mdb_util.h"

namespace mdb {

namespace {

// Kernel of a force phase (FM_*; py: periodic y); ln: the launch holds systems
// with several lanes per slot.
void* force_fn(int fm, bool py, bool ln) {
#define MDB_F(M)                                                                 \
  return ln ? (py ? (void*)k_force<M, true, true> : (void*)k_force<M, false, true>) \
            : (py ? (void*)k_force<M, true, false> : (void*)k_force<M, false, false>)
  switch (fm) {
    case FM_INIT: MDB_F(FM_INIT);
    case FM_NVE: MDB_F(FM_NVE);
    case FM_NH: MDB_F(FM_NH);
    case FM_NPH: MDB_F(FM_NPH);
    case FM_PISTON: MDB_F(FM_PISTON);
    // FIRE systems keep one lane per slot
    case FM_FIRE: return py ? (void*)k_force<FM_FIRE, true, false> : (void*)k_force<FM_FIRE, false, false>;
    default: MDB_F(FM_OBS);
  }
#undef MDB_F
}

void* force_band_fn(int fm, bool py) {
#define MDB_F(M) return py ? (void*)k_force_band<M, true> : (void*)k_force_band<M, false>
  switch (fm) {
    case FM_INIT: MDB_F(FM_INIT);
    case FM_NVE: MDB_F(FM_NVE);
    case FM_NH: MDB_F(FM_NH);
    case FM_NPH: MDB_F(FM_NPH);
    case FM_PISTON: MDB_F(FM_PISTON);
    case FM_FIRE: MDB_F(FM_FIRE);
    default: MDB_F(FM_OBS);
  }
#undef MDB_F
}

}  // namespace

Engine::Kernel Engine::force_kernel(int fm, bool py) const {
  if (banded_)
    return {force_band_fn(fm, py), nblocks_, kThreads,
            sizeof(float4) * (2 * kBandCap + kBandRoom)};
  return {force_fn(fm, py, lanes_), nblocks_, kThreads, 0};
}

Engine::Kernel Engine::list_kernel() const {
  if (banded_) return {(void*)k_rb_band, nlist_grid_, kThreads, sizeof(float4) * (kBandCap + kBandRoom)};
  return {(void*)k_rb_nlist, nlist_grid_, kThreads, 0};
}

namespace {

// Kernel of a drift phase (DM_*); ln: the launch holds systems with several
// lanes per slot.
void* drift_fn(int dm, bool ln) {
  switch (dm) {
    case DM_NVE: return ln ? (void*)k_drift<DM_NVE, true> : (void*)k_drift<DM_NVE, false>;
    case DM_NH: return ln ? (void*)k_drift<DM_NH, true> : (void*)k_drift<DM_NH, false>;
    case DM_NPH: return ln ? (void*)k_drift<DM_NPH, true> : (void*)k_drift<DM_NPH, false>;
    case DM_PISTON: return ln ? (void*)k_drift<DM_PISTON, true> : (void*)k_drift<DM_PISTON, false>;
    default: return (void*)k_drift<DM_FIRE, false>;
  }
}

}  // namespace

Engine::Kernel Engine::drift_kernel(int dm) const {
  return {drift_fn(dm, lanes_), nblocks_, kThreads, 0};
}

void* steps_fn(int dm, bool ln) {
#define MDB_S(D, F) \
  return ln ? (void*)k_run_steps<D, F, true> : (void*)k_run_steps<D, F, false>
  switch (dm) {
    case DM_NVE: MDB_S(DM_NVE, FM_NVE);
    case DM_NH: MDB_S(DM_NH, FM_NH);
    case DM_NPH: MDB_S(DM_NPH, FM_NPH);
    case DM_PISTON: MDB_S(DM_PISTON, FM_PISTON);
    // FIRE systems keep one lane per slot
    default: return (void*)k_run_steps<DM_FIRE, FM_FIRE, false>;
  }
#undef MDB_S
}

void* band_steps_fn(int dm) {
  switch (dm) {
    case DM_NVE: return (void*)k_run_band<DM_NVE, FM_NVE>;
    case DM_NH: return (void*)k_run_band<DM_NH, FM_NH>;
    case DM_NPH: return (void*)k_run_band<DM_NPH, FM_NPH>;
    case DM_PISTON: return (void*)k_run_band<DM_PISTON, FM_PISTON>;
    default: return (void*)k_run_band<DM_FIRE, FM_FIRE>;
  }
}

namespace {

double next_pow2(double x) {
  double b = 1.0;
  while (b < x) b *= 2.0;
  return b;
}

}  // namespace

int64_t resident_limit(int device) {
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  return (int64_t)nsm * 2 * kThreads;  // two blocks an SM, one slot a thread
}

Engine::Engine(const mdb_options_t& opt) {
  device_ = opt.device;
  skin_ = opt.skin > 0.0 ? opt.skin : 0.0;  // 0: chosen at build from the systems' kinds
  use_graphs_ = opt.use_graphs != 0;
  max_nbr_ = opt.max_neighbors > 0 ? opt.max_neighbors : (opt.max_neighbors < 0 ? 0 : 48);
  stream_priority_ = opt.stream_priority > 0 ? opt.stream_priority : 0;
  fire_prec_ = opt.fire_precision;
  autotune_ = opt.autotune;
  step_kernel_ = opt.step_kernel;
  lanes_opt_ = opt.lanes;
  // MDB_EAGER=1 issues every phase as a separate launch (profilers cannot
  // see kernel nodes of graphs that contain conditional nodes).
  const char* eager = getenv("MDB_EAGER");
  if (eager && eager[0] == '1') use_graphs_ = false;
}

Engine::~Engine() {
  cudaSetDevice(device_);
  if (stream_) cudaStreamSynchronize(stream_);  // destructor: not counted
  drop_graphs();
  free_proto();
  for (void* p : allocs_) cudaFree(p);
  if (d_prof_) cudaFree(d_prof_);
  if (stream_) cudaStreamDestroy(stream_);
}

void Engine::drop_graphs() {
  for (auto& kv : graphs_) {
    if (kv.second.second) cudaGraphExecDestroy(kv.second.second);
    if (kv.second.first) cudaGraphDestroy(kv.second.first);
  }
  graphs_.clear();
}

int Engine::ensure_device() {
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0)
    return set_error(MDB_ERR_NODEVICE, "no CUDA device available");
  if (device_ < 0 || device_ >= ndev) return set_error(MDB_ERR_ARG, "invalid CUDA device ordinal");
  MDB_CUDA(cudaSetDevice(device_));
  if (!stream_) {
    if (stream_priority_ > 0) {
      // numerically lower is higher priority; "greatest" is the highest
      int least = 0, greatest = 0;
      MDB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
      const int p = std::max(greatest, least - stream_priority_);
      MDB_CUDA(cudaStreamCreateWithPriority(&stream_, cudaStreamNonBlocking, p));
    } else {
      MDB_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    }
  }
  return MDB_OK;
}

int Engine::add_system(SystemSpec&& spec) {
  if (built_) return set_error(MDB_ERR_STATE, "systems can only be added before build()");
  if (spec.frame.empty()) return set_error(MDB_ERR_ARG, "a system needs at least one particle");
  if (spec.frame.size() > (size_t)INT32_MAX / 2)
    return set_error(MDB_ERR_CAPACITY, "too many particles in one system");
  const mdb_config_t& c = spec.cfg;
  if (!(c.box_w_global > 0.0) || !(c.box_h_global > 0.0) || !isfinite(c.box_w_global) ||
      !isfinite(c.box_h_global))
    return set_error(MDB_ERR_BOX, "box_w_global and box_h_global must be positive");
  if (!(c.cutoff > 0.0) || !(c.dt > 0.0) || !isfinite(c.dt))
    return set_error(MDB_ERR_CONFIG, "cutoff and dt must be positive");
  if (!(c.MASS_A > 0.0) || !(c.MASS_B > 0.0))
    return set_error(MDB_ERR_CONFIG, "MASS_A and MASS_B must be positive");
  if (!(c.SIGMA_AA > 0.0) || !(c.SIGMA_BB > 0.0) || !(c.SIGMA_AB > 0.0))
    return set_error(MDB_ERR_CONFIG, "SIGMA_* must be positive");
  specs_.push_back(std::move(spec));
  return MDB_OK;
}

int Engine::alloc(void** p, size_t bytes) {
  MDB_CUDA(cudaMalloc(p, bytes < 16 ? 16 : bytes));
  allocs_.push_back(*p);
  bytes_ += (int64_t)(bytes < 16 ? 16 : bytes);
  return MDB_OK;
}

int Engine::alloc_slot_lists() {
  if (max_nbr_ <= 0) return MDB_OK;
  if (dev_.nl16)
    return alloc((void**)&dev_.nlist16, sizeof(*dev_.nlist16) * (size_t)max_nbr_ * ntot_);
  return alloc((void**)&dev_.nlist, sizeof(*dev_.nlist) * (size_t)max_nbr_ * ntot_);
}

// The list build is instruction-bound with per-slot costs that vary (list
// lengths, minimum-image slots): one wave of resident blocks, grid-stride, so
// that no SM is left with a partial second wave.
void Engine::set_list_grid() {
  int nsm = 148, per_sm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device_);
  const Kernel lk = list_kernel();
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lk.fn, kThreads, lk.smem) !=
          cudaSuccess ||
      per_sm <= 0) {
    (void)cudaGetLastError();
    nlist_grid_ = rb_grid_;
  } else {
    nlist_grid_ = std::max(1, std::min(dev_.nchunks, nsm * per_sm));
  }
}

// A band holds 1,408 positions: enough for a chunk of a system whose cells hold up
// to some 25 particles (a cutoff of 5 at density 0.8), not for the chunks that
// span two rows of a longer cutoff, and there is none for all-pairs systems. A
// chunk without one scans its stencil from global memory, which is slow enough
// that a few hold a force phase up; then the lists of slot offsets and their
// kernels are the faster ones. (Estimated for a system of its mean density: a chunk
// that spans two rows takes from four of them its 256 slots and about three cells
// more. The frame's own count only says where it is far from uniform: a lattice's
// rows of cells hold two or three of its own rows, and fit or don't until it melts.) 16 systems of 9,000 a step, bands / slot lists, us: cutoff 5
// 52 / 62, 7 162 / 93, 9 249 / 132, 15 748 / 413; all-pairs strips of 3,000
// 549 / 321. 262,144 particles: cutoff 5 65 / 83, 5.5 (1% of the
// chunks) 200 / 107, 7 (7%) 347 / 149.
bool Engine::bands_fit() const {
  double mean = 0.0, all_pairs = 0.0;
  for (const SysParams& P : hsp_) {
    const double cols = std::max(1.0, floor(P.Lx0 / P.r_cell));
    const double rows = std::max(1.0, floor(P.Ly0 / P.r_cell));
    const double cell = P.n / (cols * rows), row = P.n / rows;
    if (cols < 3.0 || rows < 3.0)
      all_pairs += P.n;
    else if (4.0 * row > kBandCap && 4.0 * (kThreads + 3.0 * cell) > 0.95 * kBandCap)
      mean += P.n * std::min(1.0, kThreads / row);
  }
  return all_pairs * kBandUnfitNow <= (double)ntot_ && mean * kBandUnfitMean <= (double)ntot_;
}

int Engine::use_slot_lists() {
  BatchGlobal g;
  MDB_CUDA(cudaMemcpyAsync(&g, dev_.bg, sizeof(g), cudaMemcpyDeviceToHost, stream_));
  MDB_CUDA(wait_host());
  if (g.unbanded * (double)kBandUnfitNow <= (double)ntot_) return MDB_OK;
  const size_t bytes[2] = {sizeof(Band) * (size_t)dev_.nchunks,
                           sizeof(uint2) * (size_t)((max_nbr_ + 3) / 4) * ntot_};
  void* const gone[2] = {dev_.bands, dev_.lists};
  dev_.bands = nullptr;
  dev_.lists = nullptr;
  for (int k = 0; k < 2; ++k) {
    if (!gone[k]) continue;
    allocs_.erase(std::find(allocs_.begin(), allocs_.end(), gone[k]));
    bytes_ -= (int64_t)std::max<size_t>(16, bytes[k]);
    MDB_CUDA(cudaFree(gone[k]));
  }
  banded_ = band_steps_ = false;
  if (int rc = alloc_slot_lists()) return rc;
  set_list_grid();
  return rebuild_now(-1, true);
}

int Engine::build() {
  if (built_) return set_error(MDB_ERR_STATE, "engine already built");
  if (specs_.empty()) return set_error(MDB_ERR_STATE, "no systems");
  int rc = ensure_device();
  if (rc) return rc;
  const int ns = (int)specs_.size();
  hsp_.resize(ns);
  std::vector<SysState> hst(ns);
  if (!(skin_ > 0.0)) {
    // Automatic skin (measured on B200): MD steps move particles slowly and
    // the list build is the expensive part, so a wide skin (fewer rebuilds)
    // pays; FIRE moves them fast and evaluates small systems many times, so
    // a narrow one does. Skin 0.45 vs 0.3: NVT slab N=1M 0.147 -> 0.141 ms per
    // step, NPH N=4M 0.449 -> ~0.446; FIRE mix at 0.2 vs 0.3: +3%.
    bool all_fire = true;
    for (const SystemSpec& sp : specs_) all_fire = all_fire && sp.kind == K_FIRE;
    skin_ = all_fire ? kSkinFire : kSkinMD;
  }
  int64_t p0 = 0, c0 = 0;
  int b0 = 0, ch0 = 0, t0 = 0;
  int64_t maxn = 0;
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device_);
  // A block covers kThreads * items slots of one system; large systems take
  // several particles per thread so that one wave of ~4 blocks per SM covers
  // them: every block is resident from the start (the force phase spreads
  // each block's chunks over the system, which balances only within a wave),
  // fewer block partials, a short reduction tail.
  const int64_t wave = (int64_t)nsm * 4 * kThreads;
  constexpr int kMaxItems = 4096;
  // MDB_ITEMS=<k> fixes the particles per thread (tuning aid; 0 = automatic).
  const char* items_env = getenv("MDB_ITEMS");
  const int items_fixed = items_env ? atoi(items_env) : 0;
  for (int s = 0; s < ns; ++s) {
    const SystemSpec& sp = specs_[s];
    const mdb_config_t& c = sp.cfg;
    SysParams& P = hsp_[s];
    memset(&P, 0, sizeof(P));
    const int32_t n = (int32_t)sp.frame.size();
    maxn = std::max<int64_t>(maxn, n);
    P.p0 = p0;
    P.n = n;
    // lanes per slot: split for small MD systems when the handle asks for it
    // (simulation handles resolve MDB_LANES_AUTO to split, batches to one)
    P.lanes = (sp.kind != K_FIRE && lanes_opt_ == MDB_LANES_SPLIT && n <= kLanesMaxN) ? kLanes : 1;
    const int spb = kThreads / P.lanes;  // slots per block and pass
    P.items = items_fixed > 0
                  ? std::min(items_fixed, kMaxItems)
                  : (int)std::min<int64_t>(kMaxItems, std::max<int64_t>(1, (n + wave - 1) / wave));
    if (P.lanes > 1) P.items = 1;
    if (P.lanes > 1) lanes_ = true;
    P.nb = (n + spb * P.items - 1) / (spb * P.items);
    P.b0 = b0;
    P.ch0 = ch0;
    P.t0 = t0;
    P.kind = sp.kind;
    P.sig[0] = c.SIGMA_AA;
    P.sig[1] = c.SIGMA_BB;
    P.sig[2] = c.SIGMA_AB;
    P.eps[0] = c.EPSILON_AA;
    P.eps[1] = c.EPSILON_BB;
    P.eps[2] = c.EPSILON_AB;
    const double inv_c = 1.0 / c.cutoff;
    const double csr2 = inv_c * inv_c;
    const double csr6 = csr2 * csr2 * csr2;
    const double csr12 = csr6 * csr6;
    const float cutoff_f = (float)c.cutoff;
    for (int k = 0; k < 3; ++k) {
      P.Vc[k] = P.eps[k] * (4.0 * (csr12 - csr6));
      const float sf = (float)P.sig[k];
      const float ef = (float)P.eps[k];
      P.fsig2[k] = sf * sf;
      P.feps24[k] = 24.0f * ef;
      P.feps4[k] = 4.0f * ef;
      const float rcf = cutoff_f * sf;
      P.frc2[k] = rcf * rcf;
    }
    P.massA = c.MASS_A;
    P.massB = c.MASS_B;
    P.cutoff = c.cutoff;
    P.rc_max = c.cutoff * std::max(P.sig[0], std::max(P.sig[1], P.sig[2]));
    P.skin = skin_;
    P.r_cell = P.rc_max + skin_;
    for (int k = 0; k < 3; ++k) {
      const double rl = c.cutoff * P.sig[k] + skin_;
      P.frl2[k] = (float)(rl * rl);
    }
    P.dt = c.dt;
    P.Q = c.Q;
    P.T0 = c.T_target;
    P.g_dof = 2.0 * (double)c.n_particles_global - 2.0;
    P.W = c.barostat_mass > 1e-12 ? c.barostat_mass : 1e-12;
    P.k_piston = c.k_piston;
    P.hmin = c.barostat_height_min_ratio;
    P.hmax = c.barostat_height_max_ratio;
    P.Lx0 = c.box_w_global;
    P.Ly0 = c.box_h_global;
    P.rate_init = c.barostat_area_rate_init;
    const double grow = std::max(1.0, P.hmax);
    const double mx = 8.0 + 0.02 * P.Lx0, my = 8.0 + 0.02 * P.Ly0;
    P.offx = next_pow2(grow * P.Lx0 + 2.0 * mx) + mx;
    P.offy = next_pow2(grow * P.Ly0 + 2.0 * my) + my;
    P.ccap_x = std::max(1, (int)floor(grow * P.Lx0 / P.r_cell) + 1);
    P.ccap_y = std::max(1, (int)floor(grow * P.Ly0 / P.r_cell) + 1);
    P.c0 = c0;
    P.f_dt_max = sp.fire.dt_max;
    P.f_alpha0 = sp.fire.alpha0;
    P.f_inc = sp.fire.f_inc;
    P.f_dec = sp.fire.f_dec;
    P.f_Nmin = sp.fire.N_min;
    P.f_tol = sp.tol;
    P.f_max_steps = sp.max_steps;
    // FIRE pair arithmetic: FP32 pair terms leave a noise floor near 1e-6 in
    // max |a|, so the automatic mode switches a system to FP64 pair terms
    // once its max |a| is below 1e-3 (the switch is sticky).
    P.f_hp_below = fire_prec_ == MDB_FIRE_FP32 ? -1.0
                   : fire_prec_ == MDB_FIRE_FP64 ? HUGE_VAL : kFireFp64Below;
    P.target_steps = sp.target_steps;
    SysState& S = hst[s];
    memset(&S, 0, sizeof(S));
    S.Lx = c.box_w_global;
    S.Ly = c.box_h_global;
    S.aspect = 1.0;
    S.periodic_y = 1;
    S.fl = std::max(1e-12, P.hmin * P.Ly0);
    S.ce = std::max(S.fl, P.hmax * P.Ly0);
    S.need_rebuild = 1;
    S.ncx = S.ncy = 1;
    S.allpairs = 1;
    S.f_dt = sp.fire.dt_init;
    S.f_alpha = sp.fire.alpha0;
    S.f_fp64 = (sp.kind == K_FIRE && fire_prec_ == MDB_FIRE_FP64) ? 1 : 0;
    S.rb_last = kNoRebuildYet;
    p0 += n;
    b0 += P.nb;
    ch0 += (n + kThreads - 1) / kThreads;
    c0 += (int64_t)P.ccap_x * P.ccap_y;
    t0 += (int)(((int64_t)P.ccap_x * P.ccap_y + kScanTile - 1) / kScanTile);
  }
  ntot_ = p0;
  nblocks_ = b0;
  ncells_ = c0;
  if (ntot_ >= (int64_t)INT32_MAX || ncells_ >= (int64_t)INT32_MAX)
    return set_error(MDB_ERR_CAPACITY, "batch exceeds 2^31 particles or cells");

#define MDB_ALLOC(ptr, count)                                                 \
  do {                                                                        \
    int rc_ = alloc((void**)&(ptr), sizeof(*(ptr)) * (size_t)(count));       \
    if (rc_) return rc_;                                                      \
  } while (0)
  Dev& D = dev_;
  memset(&D, 0, sizeof(D));
  int32_t* sob;
  SysParams* dsp;
  MDB_ALLOC(sob, nblocks_);
  MDB_ALLOC(dsp, ns);
  D.sys_of_block = sob;
  D.sp = dsp;
  MDB_ALLOC(D.st, ns);
  MDB_ALLOC(D.bg, 1);
  MDB_ALLOC(D.pos, 2 * ntot_);
  MDB_ALLOC(D.vel, 2 * ntot_);
  MDB_ALLOC(D.acc, 2 * ntot_);
  MDB_ALLOC(D.type, 2 * ntot_);
  MDB_ALLOC(D.theta, 2 * ntot_);
  MDB_ALLOC(D.orig, 2 * ntot_);
  MDB_ALLOC(D.pff, ntot_);
  MDB_ALLOC(D.sb, ntot_);
  MDB_ALLOC(D.cell_of, ntot_);
  MDB_ALLOC(D.key, ntot_);
  MDB_ALLOC(D.rank, ntot_);
  MDB_ALLOC(D.perm, ntot_);
  D.max_nbr = max_nbr_;
  MDB_ALLOC(D.ncount, ntot_);
  // 16-bit list offsets when the stencil of every system spans well under
  // 32768 slots (about two cell rows); a particle whose offsets still do not
  // fit falls back to scanning its stencil.
  D.nl16 = 1;
  for (int s = 0; s < ns; ++s) {
    const double rows = std::max(1.0, floor(hsp_[s].Ly0 / hsp_[s].r_cell));
    if (3.0 * hsp_[s].n / rows >= 30000.0) D.nl16 = 0;
  }
  D.nsys = ns;
  D.nblocks = nblocks_;
  D.ntot = ntot_;
  D.ncells = ncells_;
  rc = choose_multi_step();
  if (rc) return rc;
  // Systems that do not run in the resident steps kernel take the staged bands
  // (one lane per slot), where these fit.
  banded_ = !multi_step_ && !lanes_ && bands_fit();
  band_steps_ = band_steps_ && banded_;
  int32_t *soc = nullptr, *sot = nullptr;
  D.nchunks = ch0;
  D.ntiles = t0;
  MDB_ALLOC(soc, ch0);
  MDB_ALLOC(sot, t0);
  MDB_ALLOC(D.tcount, t0);
  D.sys_of_chunk = soc;
  D.sys_of_tile = sot;
  if (banded_) {
    MDB_ALLOC(D.bands, ch0);
    if (max_nbr_ > 0) MDB_ALLOC(D.lists, (int64_t)((max_nbr_ + 3) / 4) * ntot_);
  } else {
    rc = alloc_slot_lists();
    if (rc) return rc;
  }
  MDB_ALLOC(D.ccount, ncells_);
  MDB_ALLOC(D.cstart, ncells_ + 1);
  MDB_ALLOC(D.part, (int64_t)nblocks_ * kNP);
  MDB_ALLOC(D.partm, (int64_t)nblocks_ * 4);
  aos_cap_ = maxn;
  {
    int rc2 = alloc(&d_aos_, sizeof(mdb_particle_t) * (size_t)maxn);
    if (rc2) return rc2;
    rc2 = alloc(&d_obs_, sizeof(mdb_observables_t));
    if (rc2) return rc2;
  }
#undef MDB_ALLOC
  D.use_cond = 0;
  rb_grid_ = std::max(1, std::min(ch0, nsm * 8));
  scan_grid_ = std::max(1, std::min(t0, nsm * 4));
  D.pf_rows = kListPrefetchRows;
  set_list_grid();

  // block table, per-slot system ids, parameters, state
  std::vector<int32_t> hsob(nblocks_), hsoc(ch0), hsot(t0);
  for (int s = 0; s < ns; ++s) {
    const int chunks = (s + 1 < ns ? hsp_[s + 1].ch0 : ch0) - hsp_[s].ch0;
    const int tiles = (s + 1 < ns ? hsp_[s + 1].t0 : t0) - hsp_[s].t0;
    for (int k = 0; k < chunks; ++k) hsoc[hsp_[s].ch0 + k] = s;
    for (int k = 0; k < tiles; ++k) hsot[hsp_[s].t0 + k] = s;
    for (int b = 0; b < hsp_[s].nb; ++b) hsob[hsp_[s].b0 + b] = s;
  }
  MDB_CUDA(cudaMemcpyAsync(sob, hsob.data(), sizeof(int32_t) * hsob.size(),
                           cudaMemcpyHostToDevice, stream_));
  MDB_CUDA(cudaMemcpyAsync(soc, hsoc.data(), sizeof(int32_t) * hsoc.size(),
                           cudaMemcpyHostToDevice, stream_));
  MDB_CUDA(cudaMemcpyAsync(sot, hsot.data(), sizeof(int32_t) * hsot.size(),
                           cudaMemcpyHostToDevice, stream_));
  MDB_CUDA(cudaMemcpyAsync(dsp, hsp_.data(), sizeof(SysParams) * ns, cudaMemcpyHostToDevice,
                           stream_));
  MDB_CUDA(cudaMemcpyAsync(D.st, hst.data(), sizeof(SysState) * ns, cudaMemcpyHostToDevice,
                           stream_));
  BatchGlobal bg{};
  bg.nsys = ns;
  MDB_CUDA(cudaMemcpyAsync(D.bg, &bg, sizeof(bg), cudaMemcpyHostToDevice, stream_));
  MDB_CUDA(cudaMemsetAsync(D.part, 0, sizeof(double) * (size_t)nblocks_ * kNP, stream_));
  MDB_CUDA(cudaMemsetAsync(D.partm, 0, sizeof(double) * (size_t)nblocks_ * 4, stream_));
  MDB_CUDA(cudaMemsetAsync(D.ccount, 0, sizeof(int32_t) * (size_t)ncells_, stream_));
  MDB_CUDA(cudaMemsetAsync(D.tcount, 0, sizeof(int32_t) * (size_t)t0, stream_));
  MDB_CUDA(cudaMemsetAsync(D.cell_of, 0, sizeof(int32_t) * (size_t)ntot_, stream_));
  MDB_CUDA(wait_host());
  built_ = true;
  for (int s = 0; s < ns; ++s) {
    rc = set_frame(s, specs_[s].frame.data());
    if (rc) return rc;
    if (specs_[s].fire_prepare) {
      const int g = (int)std::min<int64_t>((hsp_[s].n + kThreads - 1) / kThreads, 1024);
      k_fire_prepare<<<g, kThreads, 0, stream_>>>(dev_, hsp_[s].p0, hsp_[s].n, s);
      MDB_CUDA(cudaGetLastError());
      launches_ += 1;
    }
  }
  rc = rebuild_now(-1);
  if (rc) return rc;
  if (banded_) {
    rc = use_slot_lists();
    if (rc) return rc;
  }
  int items_max = 1;
  for (int s = 0; s < ns; ++s) items_max = std::max(items_max, (int)hsp_[s].items);
  schedule_.list_prefetch_rows = dev_.pf_rows;
  schedule_.nlist_grid = nlist_grid_;
  schedule_.rebuild_grid = rb_grid_;
  schedule_.items = items_max;
  schedule_.skin = skin_;
  return autotune_ ? tune() : MDB_OK;
}

// Steps of a single system in one launch need all of its blocks on the device
// at once. At one slot per thread, two blocks an SM (up to 75,776 particles on
// 148 SMs): the resident steps kernel (mdb_steps.cuh), state in registers. Above
// that: the steps kernel over staged bands (mdb_band_steps.cuh), one wave of
// four blocks an SM, which every size fits (its slots per thread grow). AUTO and
// MULTI take them for calls of any length: launches, reduction tails and
// barriers dominate a step of the small systems and are a quarter of it at
// 262,144.
int Engine::choose_multi_step() {
  multi_step_ = band_steps_ = false;
  multi_cap_ = 0;
  schedule_.multi_step = 0;
  schedule_.multi_step_blocks = 0;
  if (nsys() != 1 || !use_graphs_ || step_kernel_ == MDB_STEPS_PER_PHASE) return MDB_OK;
  int nsm = 0;
  MDB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device_));
  int coop = 0;
  MDB_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device_));
  if (!coop) return MDB_OK;
  const bool fire = hsp_[0].kind == K_FIRE;
  // blocks of a kernel family that fit at once (the least over its modes)
  auto capacity = [&](bool bands, size_t smem, int* out) -> int {
    int per_sm = 1 << 30;
    for (int dm : {DM_NVE, DM_NH, DM_NPH, DM_PISTON, DM_FIRE}) {
      if (fire != (dm == DM_FIRE)) continue;
      int b = 0;
      MDB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &b, bands ? band_steps_fn(dm) : steps_fn(dm, lanes_), kThreads, smem));
      per_sm = std::min(per_sm, b);
    }
    *out = per_sm * nsm;
    return MDB_OK;
  };
  // Shared list columns: 16-bit offsets, up to 40 KB a block (80 entries per
  // thread); longer or 32-bit lists are read from global memory.
  const int per = (max_nbr_ + hsp_[0].lanes - 1) / hsp_[0].lanes;
  const int rows = (per + kListGroup - 1) / kListGroup * kListGroup;
  steps_.list_rows = (dev_.nl16 && rows > 0 && rows <= 80) ? rows : 0;
  steps_smem_ = sizeof(int16_t) * kThreads * (size_t)steps_.list_rows;
  int rc = capacity(false, steps_smem_, &multi_cap_);
  if (rc) return rc;
  multi_step_ = hsp_[0].items == 1 && nblocks_ <= multi_cap_;
  schedule_.multi_step = multi_step_ ? 1 : 0;
  schedule_.multi_step_blocks = multi_cap_;
  if (!multi_step_ && !lanes_) {
    steps_smem_ = sizeof(float4) * (2 * kBandCap + kBandRoom);
    int cap = 0;
    rc = capacity(true, steps_smem_, &cap);
    if (rc) return rc;
    band_steps_ = nblocks_ <= cap;
  }
  if (!multi_step_ && !band_steps_) return MDB_OK;
  // one zeroed allocation: positions (second buffer), block sums, maxima,
  // sequence, tile counts
  const size_t pos = multi_step_ ? sizeof(float4) * (size_t)ntot_ : 0;
  const size_t part = sizeof(double) * 2 * kNP * (size_t)nblocks_;
  const size_t mx = sizeof(unsigned long long) * 16;
  const size_t cnt = sizeof(int32_t) * (size_t)(nblocks_ + 3);
  const size_t bytes = pos + part + mx + cnt;
  char* base = nullptr;
  MDB_CUDA(cudaMalloc((void**)&base, bytes));
  allocs_.push_back(base);
  bytes_ += (int64_t)bytes;
  MDB_CUDA(cudaMemsetAsync(base, 0, bytes, stream_));
  steps_.pff1 = (float4*)base;
  steps_.part = (double*)(base + pos);
  steps_.max = (unsigned long long*)(base + pos + part);
  steps_.seq = (uint32_t*)(base + pos + part + mx);
  steps_.tile = (int32_t*)(steps_.seq + 3);
  dev_.progress = steps_.seq + 2;
  // For tests, MDB_EXCHANGE_POLLS=<polls> makes blocks look after that many polls
  // whether others get on; with @<block> only that block, which also waits for an
  // arrival that never comes in a launch's last exchange.
  steps_.polls = kExchangePolls;
  steps_.late_block = -1;
  const char* polls = getenv("MDB_EXCHANGE_POLLS");
  if (polls && polls[0]) {
    steps_.polls = (uint32_t)std::min<unsigned long>(strtoul(polls, nullptr, 10), kExchangePolls);
    const char* at = strchr(polls, '@');
    if (at) steps_.late_block = atoi(at + 1);
  }
  return MDB_OK;
}

// n steps (FIRE: iterations) in cooperative launches. A launch holds its blocks'
// places until it ends, over staged bands the whole device, whatever the priority of
// the streams that wait. So its steps are those of about a millisecond, by a rule on
// the size (measured us a step: 5.0 at 900 particles, 14.8 at 60,013; 33 at 262,144,
// 97 at 1,048,576; launches of 0.3 ms cost a step 2% there, of 1 ms less than 0.5%).
// 200 steps of 4,096 particles at a higher priority, 1.4 ms alone, took 7.6 ms beside
// launches of 64 steps of 1,048,576 particles, 3.4 beside these, 1.7 beside one kernel
// per phase (MDB_STEPS_PER_PHASE).
int Engine::run_resident(int dm, int64_t n) {
  Dev d = dev_;
  d.use_cond = 0;
  StepsMem m = steps_;
  const double us = multi_step_ ? 5.0 + ntot_ / 6000.0 : 8.0 + ntot_ / 11500.0;
  const int64_t most =
      std::max<int64_t>(1, std::min<int64_t>(multi_step_ ? 256 : 64, (int64_t)(1000.0 / us)));
  for (int64_t left = n; left > 0;) {
    int64_t k = std::min(left, most);
    void* args[] = {&d, &m, &k};
    MDB_CUDA(cudaLaunchCooperativeKernel(multi_step_ ? steps_fn(dm, lanes_) : band_steps_fn(dm),
                                         dim3(nblocks_), dim3(kThreads), args, steps_smem_,
                                         stream_));
    launches_ += 1;
    count_launches(1);
    left -= k;
  }
  return MDB_OK;
}

int Engine::launch(void* fn, int grid, int block, const Dev& d, size_t smem) {
  Dev copy = d;
  void* args[] = {&copy};
  MDB_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(block), args, smem, stream_));
  launches_ += 1;
  count_launches(1);
  return MDB_OK;
}

int Engine::launch_rebuild_eager() {
  const Dev& d = dev_;
  int rc;
  if ((rc = launch((void*)k_rb_bin, rb_grid_, kThreads, d))) return rc;
  if ((rc = launch((void*)k_rb_scan, scan_grid_, kScanBlock, d))) return rc;
  if ((rc = launch((void*)k_rb_scatter, rb_grid_, kThreads, d))) return rc;
  if ((rc = launch((void*)k_rb_permute, rb_grid_, kThreads, d))) return rc;
  if ((rc = launch(list_kernel(), d))) return rc;
  return MDB_OK;
}

int Engine::rebuild_now(int periodic_y, bool again) {
  if (!built_) return set_error(MDB_ERR_STATE, "engine not built");
  MDB_CUDA(cudaSetDevice(device_));
  k_force_rebuild<<<1, kThreads, 0, stream_>>>(dev_, periodic_y, again ? 1 : 0);
  MDB_CUDA(cudaGetLastError());
  launches_ += 1;
  count_launches(1);
  return launch_rebuild_eager();
}

int Engine::set_pext(double p) {
  MDB_CUDA(cudaSetDevice(device_));
  k_set_pext<<<1, kThreads, 0, stream_>>>(dev_, p);
  MDB_CUDA(cudaGetLastError());
  launches_ += 1;
  count_launches(1);
  return MDB_OK;
}

int Engine::force(int fm, bool py) {
  MDB_CUDA(cudaSetDevice(device_));
  return launch(force_kernel(fm, py), dev_);
}

int Engine::reduce_K() {
  MDB_CUDA(cudaSetDevice(device_));
  return launch((void*)k_reduce_K, nblocks_, kThreads, dev_);
}

int Engine::add_kernel_node(cudaGraph_t g, const cudaGraphNode_t* deps, int ndeps, void* fn,
                            int grid, int block, const Dev& d, cudaGraphNode_t* out, size_t smem) {
  Dev copy = d;
  void* args[] = {&copy};
  cudaKernelNodeParams kp = {};
  kp.func = fn;
  kp.gridDim = dim3(grid);
  kp.blockDim = dim3(block);
  kp.sharedMemBytes = (unsigned)smem;
  kp.kernelParams = args;
  kp.extra = nullptr;
  MDB_CUDA(cudaGraphAddKernelNode(out, g, deps, (size_t)ndeps, &kp));
  return MDB_OK;
}

int Engine::add_rebuild_body(cudaGraph_t body, const Dev& d) {
  const Kernel ks[] = {{(void*)k_rb_bin, rb_grid_, kThreads, 0},
                       {(void*)k_rb_scan, scan_grid_, kScanBlock, 0},
                       {(void*)k_rb_scatter, rb_grid_, kThreads, 0},
                       {(void*)k_rb_permute, rb_grid_, kThreads, 0},
                       list_kernel()};
  cudaGraphNode_t prev = nullptr;
  for (const Kernel& k : ks) {
    cudaGraphNode_t node;
    const int rc = add_kernel_node(body, prev ? &prev : nullptr, prev ? 1 : 0, k, d, &node);
    if (rc) return rc;
    prev = node;
  }
  return MDB_OK;
}

int Engine::add_cond_rebuild(cudaGraph_t g, cudaGraphNode_t dep, cudaGraphConditionalHandle h,
                             cudaGraphNode_t* out) {
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeIf;
  cp.conditional.size = 1;
  MDB_CUDA(cudaGraphAddNode(out, g, &dep, 1, &cp));
  Dev d = dev_;
  d.use_cond = 0;
  return add_rebuild_body(cp.conditional.phGraph_out[0], d);
}

// kind 0: MD steps (drift, cond rebuild, force); kind 1: FIRE iterations
// (force, drift, cond rebuild).
int Engine::get_graph(int kind, int dm, int fm, bool py, int chunk, cudaGraphExec_t* exec) {
  auto key = std::make_tuple(kind, dm, fm, py ? 1 : 0, chunk);
  auto it = graphs_.find(key);
  if (it != graphs_.end()) {
    *exec = it->second.second;
    return MDB_OK;
  }
  cudaGraph_t g;
  MDB_CUDA(cudaGraphCreate(&g, 0));
  cudaGraphNode_t prev = nullptr;
  int rc = MDB_OK;
  for (int k = 0; k < chunk && rc == MDB_OK; ++k) {
    // No reset of the condition at each launch (cudaGraphCondAssignDefault
    // cost ~4 us per step node): the drift kernel's last block sets it on
    // every step before the conditional node reads it.
    cudaGraphConditionalHandle h;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, g, 0, 0);
    if (e != cudaSuccess) {
      rc = cuda_error(e, "cudaGraphConditionalHandleCreate");
      break;
    }
    Dev dd = dev_;
    dd.cond = h;
    dd.use_cond = 1;
    cudaGraphNode_t nd, nc, nf;
    if (kind == 0) {
      rc = add_kernel_node(g, prev ? &prev : nullptr, prev ? 1 : 0, drift_kernel(dm), dd, &nd);
      if (!rc) rc = add_cond_rebuild(g, nd, h, &nc);
      if (!rc) rc = add_kernel_node(g, &nc, 1, force_kernel(fm, py), dev_, &nf);
      prev = nf;
    } else {
      rc = add_kernel_node(g, prev ? &prev : nullptr, prev ? 1 : 0, force_kernel(FM_FIRE, true), dev_, &nf);
      if (!rc) rc = add_kernel_node(g, &nf, 1, drift_kernel(DM_FIRE), dd, &nd);
      if (!rc) rc = add_cond_rebuild(g, nd, h, &nc);
      prev = nc;
    }
  }
  if (rc != MDB_OK) {
    cudaGraphDestroy(g);
    return rc;
  }
  cudaGraphExec_t ex;
  cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(g);
    return cuda_error(e, "cudaGraphInstantiate");
  }
  graphs_[key] = std::make_pair(g, ex);
  *exec = ex;
  return MDB_OK;
}

int Engine::run_md(int dm, int fm, bool py, int64_t nsteps) {
  if (!built_) return set_error(MDB_ERR_STATE, "engine not built");
  MDB_CUDA(cudaSetDevice(device_));
  if ((multi_step_ || band_steps_) && py == (dm != DM_PISTON)) return run_resident(dm, nsteps);
  int64_t left = nsteps;
  if (use_graphs_) {
    static const int kChunks[] = {64, 8, 1};
    for (int c : kChunks) {
      while (left >= c) {
        cudaGraphExec_t ex;
        int rc = get_graph(0, dm, fm, py, c, &ex);
        if (rc) {
          use_graphs_ = false;  // fall back to eager launches
          break;
        }
        MDB_CUDA(cudaGraphLaunch(ex, stream_));
        launches_ += 2LL * c;
        count_launches(2LL * c);
        left -= c;
      }
      if (!use_graphs_) break;
    }
  }
  for (; left > 0; --left) {
    int rc;
    if ((rc = launch(drift_kernel(dm), dev_))) return rc;
    if ((rc = launch_rebuild_eager())) return rc;
    if ((rc = launch(force_kernel(fm, py), dev_))) return rc;
  }
  return MDB_OK;
}

int Engine::run_md_timed(int dm, int fm, bool py, int64_t nsteps, double* ms) {
  if (!built_) return set_error(MDB_ERR_STATE, "engine not built");
  MDB_CUDA(cudaSetDevice(device_));
  cudaEvent_t ev[4];
  for (int k = 0; k < 4; ++k) MDB_CUDA(cudaEventCreate(&ev[k]));
  double acc[3] = {0.0, 0.0, 0.0};
  int rc = MDB_OK;
  for (int64_t s = 0; s < nsteps && rc == MDB_OK; ++s) {
    cudaEventRecord(ev[0], stream_);
    rc = launch(drift_kernel(dm), dev_);
    cudaEventRecord(ev[1], stream_);
    if (!rc) rc = launch_rebuild_eager();
    cudaEventRecord(ev[2], stream_);
    if (!rc) rc = launch(force_kernel(fm, py), dev_);
    cudaEventRecord(ev[3], stream_);
    cudaError_t e = cudaEventSynchronize(ev[3]);
    if (e != cudaSuccess) {
      rc = cuda_error(e, "cudaEventSynchronize");
      break;
    }
    for (int k = 0; k < 3; ++k) {
      float t = 0.f;
      cudaEventElapsedTime(&t, ev[k], ev[k + 1]);
      acc[k] += t;
    }
  }
  for (int k = 0; k < 4; ++k) cudaEventDestroy(ev[k]);
  for (int k = 0; k < 3; ++k) ms[k] = acc[k];
  return rc;
}

int Engine::run_fire(int64_t iters) {
  if (!built_) return set_error(MDB_ERR_STATE, "engine not built");
  MDB_CUDA(cudaSetDevice(device_));
  if (multi_step_ || band_steps_) return run_resident(DM_FIRE, iters);
  int64_t left = iters;
  if (use_graphs_) {
    static const int kChunks[] = {100, 10, 1};
    for (int c : kChunks) {
      while (left >= c) {
        cudaGraphExec_t ex;
        int rc = get_graph(1, DM_FIRE, FM_FIRE, true, c, &ex);
        if (rc) {
          use_graphs_ = false;
          break;
        }
        MDB_CUDA(cudaGraphLaunch(ex, stream_));
        launches_ += 2LL * c;
        count_launches(2LL * c);
        left -= c;
      }
      if (!use_graphs_) break;
    }
  }
  for (; left > 0; --left) {
    int rc;
    if ((rc = launch(force_kernel(FM_FIRE, true), dev_))) return rc;
    if ((rc = launch(drift_kernel(DM_FIRE), dev_))) return rc;
    if ((rc = launch_rebuild_eager())) return rc;
  }
  return MDB_OK;
}

int Engine::get_state(int s, SysState* out) {
  MDB_CUDA(cudaSetDevice(device_));
  MDB_CUDA(cudaMemcpyAsync(out, dev_.st + s, sizeof(SysState), cudaMemcpyDeviceToHost, stream_));
  MDB_CUDA(wait_host());
  return MDB_OK;
}

int Engine::get_states(std::vector<SysState>& out) {
  MDB_CUDA(cudaSetDevice(device_));
  out.resize(specs_.size());
  MDB_CUDA(cudaMemcpyAsync(out.data(), dev_.st, sizeof(SysState) * out.size(),
                           cudaMemcpyDeviceToHost, stream_));
  MDB_CUDA(wait_host());
  return MDB_OK;
}

int Engine::put_state(int s, const SysState& st) {
  MDB_CUDA(cudaSetDevice(device_));
  // (as a kernel argument, which the launch copies: the caller may let go of `st`
  // at once, and nothing waits)
  k_put_state<<<1, 1, 0, stream_>>>(dev_, s, st);
  MDB_CUDA(cudaGetLastError());
  launches_ += 1;
  count_launches(1);
  return MDB_OK;
}

int Engine::get_frame(int s, mdb_particle_t* out) {
  MDB_CUDA(cudaSetDevice(device_));
  const SysParams& P = hsp_[s];
  const int g = (int)std::min<int64_t>((P.n + kThreads - 1) / kThreads, 4096);
  k_export<<<g, kThreads, 0, stream_>>>(dev_, (DevParticle*)d_aos_, P.p0, P.n, s);
  MDB_CUDA(cudaGetLastError());
  launches_ += 1;
  count_launches(1);
  MDB_CUDA(cudaMemcpyAsync(out, d_aos_, sizeof(mdb_particle_t) * (size_t)P.n,
                           cudaMemcpyDeviceToHost, stream_));
  MDB_CUDA(wait_host());
  return MDB_OK;
}

int Engine::profiles(int s, int nb, bool py, double* ptens, int32_t* counts) {
  MDB_CUDA(cudaSetDevice(device_));
  // bins on the device: 3 nb sums, then 2 nb counts; kept, and grown on demand
  const size_t bytes = (sizeof(unsigned long long) * 3 + sizeof(int) * 2) * (size_t)nb;
  if (prof_bytes_ < bytes) {
    if (d_prof_) cudaFree(d_prof_);  // (every call waits for its kernels below)
    d_prof_ = nullptr;
    bytes_ -= (int64_t)prof_bytes_;
    prof_bytes_ = 0;
    MDB_CUDA(cudaMalloc(&d_prof_, bytes));
    prof_bytes_ = bytes;
    bytes_ += (int64_t)bytes;
  }
  unsigned long long* d_acc = (unsigned long long*)d_prof_;
  int* d_cnt = (int*)(d_acc + 3 * (size_t)nb);
  MDB_CUDA(cudaMemsetAsync(d_prof_, 0, bytes, stream_));
  const SysParams& P = hsp_[s];
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((P.n + kThreads - 1) / kThreads, 4096));
  if (counts) {
    k_count_profile<<<g, kThreads, 0, stream_>>>(dev_, s, nb, d_cnt);
    MDB_CUDA(cudaGetLastError());
    launches_ += 1;
    count_launches(1);
  }
  std::vector<long long> acc(ptens ? (size_t)3 * nb : 0);
  if (ptens) {
    // a window reaches as far as a pair's midpoint is from its particle (half
    // the largest cutoff), within 48 KB of shared memory; finer bins than that
    // covers add to the global bins one by one
    const double reach = 0.5 * P.rc_max * (double)nb / P.Ly0;
    const int win = 2 * (int)std::min(3.0, std::max(1.0, ceil(reach))) + 1;
    const size_t smem = sizeof(unsigned long long) * 3 * (size_t)win * kThreads;
    if (py)
      k_pressure_profile<true><<<g, kThreads, smem, stream_>>>(dev_, s, nb, win, d_acc);
    else
      k_pressure_profile<false><<<g, kThreads, smem, stream_>>>(dev_, s, nb, win, d_acc);
    MDB_CUDA(cudaGetLastError());
    launches_ += 1;
    count_launches(1);
    MDB_CUDA(cudaMemcpyAsync(acc.data(), d_acc, sizeof(long long) * acc.size(),
                             cudaMemcpyDeviceToHost, stream_));
  }
  if (counts)
    MDB_CUDA(cudaMemcpyAsync(counts, d_cnt, sizeof(int) * 2 * (size_t)nb, cudaMemcpyDeviceToHost,
                             stream_));
  MDB_CUDA(wait_host());
  for (size_t k = 0; k < acc.size(); ++k) ptens[k] = (double)acc[k] / kProfileFix;
  return MDB_OK;
}

int Engine::observables_async(int s, double t, int piston_active, mdb_observables_t* host) {
  MDB_CUDA(cudaSetDevice(device_));
  k_observables<<<1, 1, 0, stream_>>>(dev_, s, t, piston_active, (mdb_observables_t*)d_obs_);
  MDB_CUDA(cudaGetLastError());
  launches_ += 1;
  count_launches(1);
  MDB_CUDA(cudaMemcpyAsync(host, d_obs_, sizeof(mdb_observables_t), cudaMemcpyDeviceToHost,
                           stream_));
  return MDB_OK;
}

int Engine::export_async(int s, mdb_particle_t* host) {
  MDB_CUDA(cudaSetDevice(device_));
  const SysParams& P = hsp_[s];
  const int g = (int)std::min<int64_t>((P.n + kThreads - 1) / kThreads, 4096);
  k_export<<<g, kThreads, 0, stream_>>>(dev_, (DevParticle*)d_aos_, P.p0, P.n, s);
  MDB_CUDA(cudaGetLastError());
  launches_ += 1;
  count_launches(1);
  MDB_CUDA(cudaMemcpyAsync(host, d_aos_, sizeof(mdb_particle_t) * (size_t)P.n,
                           cudaMemcpyDeviceToHost, stream_));
  return MDB_OK;
}

int Engine::set_frame(int s, const mdb_particle_t* in) {
  MDB_CUDA(cudaSetDevice(device_));
  const SysParams& P = hsp_[s];
  MDB_CUDA(cudaMemcpyAsync(d_aos_, in, sizeof(mdb_particle_t) * (size_t)P.n,
                           cudaMemcpyHostToDevice, stream_));
  const int g = (int)std::min<int64_t>((P.n + kThreads - 1) / kThreads, 4096);
  k_import<<<g, kThreads, 0, stream_>>>(dev_, (const DevParticle*)d_aos_, P.p0, P.n, s);
  MDB_CUDA(cudaGetLastError());
  launches_ += 1;
  count_launches(1);
  return MDB_OK;
}

int Engine::debug_cells(int s, int32_t* orig, int32_t* cell) {
  MDB_CUDA(cudaSetDevice(device_));
  const SysParams& P = hsp_[s];
  SysState S;
  if (int rc = get_state(s, &S)) return rc;
  MDB_CUDA(cudaMemcpyAsync(orig, dev_.orig + (S.buf ? ntot_ : 0) + P.p0, sizeof(int32_t) * (size_t)P.n,
                           cudaMemcpyDeviceToHost, stream_));
  MDB_CUDA(cudaMemcpyAsync(cell, dev_.cell_of + P.p0, sizeof(int32_t) * (size_t)P.n,
                           cudaMemcpyDeviceToHost, stream_));
  MDB_CUDA(wait_host());
  return MDB_OK;
}

int Engine::sync() {
  MDB_CUDA(cudaSetDevice(device_));
  MDB_CUDA(wait_host());
  return MDB_OK;
}

int Engine::idle(bool* out) {
  MDB_CUDA(cudaSetDevice(device_));
  const cudaError_t e = cudaStreamQuery(stream_);
  if (e == cudaSuccess) {
    *out = true;
    return MDB_OK;
  }
  if (e == cudaErrorNotReady) {
    *out = false;
    return MDB_OK;
  }
  return cuda_error(e, "cudaStreamQuery");
}

// ------------------------------------------------------------- autotuner --
// The schedule knobs tuned here change where and when work runs, never what
// is computed: the prefetch depth only moves list rows into L1 earlier, and
// the rebuild kernels are grid-stride loops over independent slots and cells
// whose order is fixed by the stable sort. Candidates are timed on the
// workload's own force phase (Nose-Hoover for MD handles, FIRE for FIRE
// batches), after which the velocities, accelerations and every system's
// scalar state are put back (positions do not move), and on rebuilds at
// unchanged positions, which keep every slot where it is (the sort is stable
// and the cells are unchanged).
namespace {

std::mutex g_cache_mu;

std::string cache_path() {
  const char* p = getenv("MDB_SCHEDULE_CACHE");
  if (p && p[0]) return p;
  const char* home = getenv("HOME");
  const std::string dir = std::string(home && home[0] ? home : "/tmp") + "/.cache";
  mkdir(dir.c_str(), 0755);
  const std::string d2 = dir + "/md_simulation_cuda_b200";
  mkdir(d2.c_str(), 0755);
  return d2 + "/schedule.txt";
}

bool cache_lookup(const std::string& key, int* pf, int* nlg, int* rbg) {
  std::lock_guard<std::mutex> lk(g_cache_mu);
  std::ifstream in(cache_path());
  if (!in) return false;
  std::string line;
  bool found = false;
  while (std::getline(in, line)) {
    const size_t tab = line.find('\t');
    if (tab == std::string::npos || line.compare(0, tab, key) != 0 || tab != key.size()) continue;
    std::istringstream vs(line.substr(tab + 1));
    int a, b, c;
    // (several processes may append to the file at once: a line that does not
    // hold a plausible schedule is skipped)
    if ((vs >> a >> b >> c) && a >= 0 && a <= 32 && b >= 1 && b <= (1 << 20) && c >= 1 &&
        c <= (1 << 20)) {
      *pf = a;
      *nlg = b;
      *rbg = c;
      found = true;  // the last entry for the key wins
    }
  }
  return found;
}

void cache_store(const std::string& key, int pf, int nlg, int rbg) {
  std::lock_guard<std::mutex> lk(g_cache_mu);
  // one write of the whole line (appends of a short line are atomic between
  // processes)
  std::ostringstream line;
  line << key << '\t' << pf << ' ' << nlg << ' ' << rbg << '\n';
  std::ofstream out(cache_path(), std::ios::app);
  if (out) {
    const std::string t = line.str();
    out.write(t.data(), (std::streamsize)t.size());
  }
}

int bucket(int64_t x) {  // log2 bucket of a size
  int b = 0;
  while (x > 1) {
    x >>= 1;
    ++b;
  }
  return b;
}

}  // namespace

int Engine::time_force(int fm, int reps, double* ms) {
  cudaEvent_t a, b;
  MDB_CUDA(cudaEventCreate(&a));
  MDB_CUDA(cudaEventCreate(&b));
  int rc = launch(force_kernel(fm, true), dev_);  // warm
  double best = 1e30;
  for (int r = 0; !rc && r < reps; ++r) {
    cudaEventRecord(a, stream_);
    rc = launch(force_kernel(fm, true), dev_);
    cudaEventRecord(b, stream_);
    cudaEventSynchronize(b);
    float t = 0.f;
    cudaEventElapsedTime(&t, a, b);
    best = std::min(best, (double)t);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  *ms = best;
  return rc;
}

int Engine::time_rebuild(int reps, double* ms) {
  cudaEvent_t a, b;
  MDB_CUDA(cudaEventCreate(&a));
  MDB_CUDA(cudaEventCreate(&b));
  int rc = rebuild_now(-1);  // warm
  double best = 1e30;
  for (int r = 0; !rc && r < reps; ++r) {
    cudaEventRecord(a, stream_);
    rc = rebuild_now(-1);
    cudaEventRecord(b, stream_);
    cudaEventSynchronize(b);
    float t = 0.f;
    cudaEventElapsedTime(&t, a, b);
    best = std::min(best, (double)t);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  *ms = best;
  return rc;
}

int Engine::tune() {
  const auto t0 = std::chrono::steady_clock::now();
  cudaDeviceProp prop;
  MDB_CUDA(cudaGetDeviceProperties(&prop, device_));
  const int nsm = prop.multiProcessorCount;
  int kinds = 0;
  for (const SystemSpec& sp : specs_) kinds |= 1 << sp.kind;
  // (the kernels that the schedule was timed on, and a number that goes up with them:
  // a line of other kernels does not fit)
  const char* form = multi_step_ ? "resident" : band_steps_ ? "bandsteps" : banded_ ? "bands"
                     : lanes_ ? "lanes" : "lists";
  char keyb[512];
  snprintf(keyb, sizeof(keyb), "2|%s|%s|sm%d|sys%d|n%d|cells%d|nbr%d|nl16_%d|skin%.3f|kinds%d",
           form, prop.name, nsm, bucket((int64_t)specs_.size()), bucket(ntot_), bucket(ncells_),
           max_nbr_, dev_.nl16, skin_, kinds);
  const std::string key(keyb);
  int pf = dev_.pf_rows, nlg = nlist_grid_, rbg = rb_grid_;
  if (cache_lookup(key, &pf, &nlg, &rbg)) {
    dev_.pf_rows = pf;
    nlist_grid_ = std::max(1, nlg);
    rb_grid_ = std::max(1, rbg);
    schedule_.from_cache = 1;
  } else if (multi_step_) {
    // (the resident steps kernel reads none of these: the built-in schedule stands)
    cache_store(key, dev_.pf_rows, nlist_grid_, rb_grid_);
  } else {
    // force phase: list prefetch depth, timed on the workload's force kernel
    // with the velocities (kicked by it) and the scalar state put back after
    const bool all_fire = (kinds == (1 << K_FIRE));
    const int fm = all_fire ? FM_FIRE : FM_NH;
    std::vector<SysState> snap;
    if (int rc = get_states(snap)) return rc;
    // (kept in the half of each array that is not in use; the rebuilds so far were of
    // all systems, so it is the same half for every one)
    const size_t bytes = sizeof(double2) * (size_t)ntot_;
    const int64_t used = snap[0].buf ? ntot_ : 0, idle = ntot_ - used;
    for (const SysState& S : snap)
      if (S.buf != snap[0].buf) return set_error(MDB_ERR_STATE, "systems in unlike halves");
    for (double2* p : {dev_.vel, dev_.acc})
      MDB_CUDA(cudaMemcpyAsync(p + idle, p + used, bytes, cudaMemcpyDeviceToDevice, stream_));
    double best = 1e30;
    int best_pf = dev_.pf_rows;
    for (int cand : {28, 16, 8, 0}) {
      dev_.pf_rows = cand;
      double ms = 0.0;
      const int rc = time_force(fm, 3, &ms);
      if (rc) return rc;
      if (ms < best * 0.98) {  // keep the earlier (deeper) choice within 2%
        best = ms;
        best_pf = cand;
      }
    }
    dev_.pf_rows = best_pf;
    for (double2* p : {dev_.vel, dev_.acc})
      MDB_CUDA(cudaMemcpyAsync(p + used, p + idle, bytes, cudaMemcpyDeviceToDevice, stream_));
    MDB_CUDA(cudaMemcpyAsync(dev_.st, snap.data(), sizeof(SysState) * snap.size(),
                             cudaMemcpyHostToDevice, stream_));
    MDB_CUDA(wait_host());
    // rebuild: list-build grid, then the grid of the other rebuild kernels (the
    // steps kernel over staged bands rebuilds on its own blocks)
    const int one_wave = nlist_grid_;
    const int cap = std::max(1, dev_.nchunks);
    best = 1e30;
    int best_nlg = one_wave;
    const bool grids = !band_steps_;
    for (int cand : {one_wave, std::min(cap, 2 * one_wave), std::max(1, one_wave / 2)}) {
      if (!grids) break;
      nlist_grid_ = cand;
      double ms = 0.0;
      const int rc = time_rebuild(2, &ms);
      if (rc) return rc;
      if (ms < best * 0.98) {
        best = ms;
        best_nlg = cand;
      }
    }
    nlist_grid_ = best_nlg;
    best = 1e30;
    int best_rbg = rb_grid_;
    for (int cand : {rb_grid_, std::min(cap, nsm * 16), std::min(cap, nsm * 4)}) {
      if (!grids) break;
      rb_grid_ = std::max(1, cand);
      double ms = 0.0;
      const int rc = time_rebuild(2, &ms);
      if (rc) return rc;
      if (ms < best * 0.98) {
        best = ms;
        best_rbg = rb_grid_;
      }
    }
    rb_grid_ = best_rbg;
    cache_store(key, dev_.pf_rows, nlist_grid_, rb_grid_);
  }
  MDB_CUDA(wait_host());
  schedule_.list_prefetch_rows = dev_.pf_rows;
  schedule_.nlist_grid = nlist_grid_;
  schedule_.rebuild_grid = rb_grid_;
  schedule_.tuned = 1;
  schedule_.tune_ms =
      std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return MDB_OK;
}

}  // namespace mdb
