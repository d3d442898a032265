// Resident steps over staged bands: many steps (or FIRE iterations) of a single
// system of more particles than the resident steps kernel holds in registers,
// in one cooperative launch.
//
// The blocks of such a system are one wave (four of 256 threads an SM, several
// slots a thread), all on the device at once. With one launch per phase a step
// of 262,144 particles took 17.5 us in the drift and 26.6 us in the force phase,
// of which the bytes and instructions account for about half: each launch starts
// with a chain of dependent loads (system, scalars, first chunk) on an empty
// device and ends in a last block's tail. Here the phases are the loops of
// k_drift and of k_force_band between two exchanges (mdb_steps.cuh): the scalars
// stay in shared memory, and a rebuild runs its passes in place. The blocks,
// chunks, sums and their order are those of the per-phase kernels: the same
// result bits.
#pragma once

#include "mdb_band.cuh"
#include "mdb_steps.cuh"

namespace mdb {

// Orders generic accesses before it and bulk copies after it (and the reverse).
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

struct BandSteps {
  StepsShared steps;
  BandShared band;
  Band list_band;
  uint64_t list_full;
};

// A rebuild inside the kernel: the passes of k_rb_*, an exchange after each.
// Out of line: it runs once in some twenty steps.
__device__ __noinline__ void band_rebuild(Dev D, StepsMem M, BandSteps* sh, float4* sh_band,
                                          uint32_t* seq_io, uint32_t* list_parity) {
  uint32_t seq = *seq_io;
  Totals in, out;
  // (an exchange that gave up ends the kernel: no pass runs on partial results)
  auto all_arrived = [&]() {
    exchange<0, 0, 0>(M, sh->steps, seq, in, out);
    *seq_io = seq;
    return sh->steps.abort == 0;
  };
  SysState& S = sh->steps.S;
  if (threadIdx.x == 0) {
    set_cell_grid(sh->steps.P, &S);
    S.need_rebuild = 1;
  }
  __syncthreads();
  // the passes read the system's state from global memory
  if (blockIdx.x == 0) {
    store_state(D, S);
    if (threadIdx.x == 0) D.st->nl_overflow = 0;
  }
  if (!all_arrived()) return;
  rb_bin(D);
  if (!all_arrived()) return;
  rb_scan(D);
  if (!all_arrived()) return;
  rb_scatter(D);
  if (!all_arrived()) return;
  rb_permute(D, false);
  fence_async();
  if (!all_arrived()) return;
  fence_async();
  if (!rb_band(D, sh_band, sh->list_band, sh->list_full, *list_parity, false))
    sh->steps.abort = 1;
  if (blockIdx.x == 0)
    for (int t = threadIdx.x; t < D.ntiles; t += kThreads) D.tcount[t] = 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    S.need_rebuild = 0;
    S.buf ^= 1;
    S.rebuilds += 1;
    S.rb_last = rebuild_clock(sh->steps.P, S);
  }
  // (lists and counts are read by other blocks' chunks)
  all_arrived();
}

// Runs up to `todo` steps (FIRE: iterations) of the engine's single system.
// Grid: the system's blocks, all resident (cooperative launch).
template <int DMd, int FM>
__global__ void __launch_bounds__(kThreads, 4) k_run_band(Dev D, StepsMem M, int64_t todo) {
  constexpr bool PY = DMd != DM_PISTON;
  constexpr bool FIRE = DMd == DM_FIRE;
  constexpr bool kBoxMoves = (DMd == DM_NPH || DMd == DM_PISTON);
  constexpr int kDNS = (DMd == DM_NH) ? 1 : 0;
  constexpr int kFNS = ForceRed<FM>::NS;
  extern __shared__ __align__(128) float4 sh_band[];  // [2][kBandCap] and room
  __shared__ BandSteps sh;
  const int tid = threadIdx.x;
  load_state(D, sh.steps);
  if (tid == 0) {
    mbar_init(sh.band.full + 0, 1);
    mbar_init(sh.band.full + 1, 1);
    mbar_init(sh.band.empty + 0, kThreads / 32);
    mbar_init(sh.band.empty + 1, kThreads / 32);
    mbar_init(&sh.list_full, 1);
    sh.band.lost = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  uint32_t seq = *M.seq;
  const uint32_t seq0 = seq;
  __syncthreads();
  const SysParams& P = sh.steps.P;
  SysState& S = sh.steps.S;
  uint32_t pass = 0, list_parity = 0;
  Totals in, out;
  int bad = 0;
  if (tid == 0) {
    drift_prelude<DMd>(P, S, sh.steps.dc, sh.steps.ds);
    sh.steps.lim =
        rebuild_limits<DMd>(sh.steps.dc.Lx, sh.steps.dc.Ly, drift_tail_scalars(P, S));
  }
  __syncthreads();

  int64_t done = 0;
  while (done < todo) {
    if (S.done != 0 || S.err != 0) break;
    if (FIRE && (S.f_conv != 0 || S.f_step >= P.f_max_steps)) {
      __syncthreads();
      if (tid == 0) S.f_drift = 0;
      break;
    }
    // One pass is a step: drift, rebuild, force. A FIRE iteration is force,
    // drift, rebuild.
#pragma unroll
    for (int phase = 0; phase < 2; ++phase) {
      if ((phase == 0) != FIRE) {
        // ---- drift: the block's slots are one contiguous stretch
        if (sh.steps.ds.boxbad) {
          __syncthreads();
          if (tid == 0) {
            S.err = 5;  // MDB_ERR_BOX
            sh.steps.stop = 1;
          }
          __syncthreads();
          break;
        }
        const int64_t half = half_of(D, &S);
        const int64_t end = P.p0 + P.n;
        const int64_t first = P.p0 + (int64_t)blockIdx.x * P.items * kThreads + tid;
        double ks = 0.0, mdx = 0.0, mdy = 0.0, mjump = 0.0;
        float fdx = 0.f, fdy = 0.f;
#pragma unroll 1
        for (int it = 0; it < P.items; ++it) {
          const int64_t i = first + (int64_t)it * kThreads;
          if (i >= end) break;
          double2 x = D.pos[half + i], v = D.vel[half + i];
          const int t = D.type[half + i];
          drift_move<DMd>(sh.steps.dc, x, v, D.acc[half + i], t, D.sb[i], ks, mdx, mdy, mjump, fdx,
                          fdy, bad);
          D.pos[half + i] = x;
          D.vel[half + i] = v;
          D.pff[i] = encode_ff(x.x, x.y, t, sh.steps.dc.offx, sh.steps.dc.offy);
        }
        fence_async();  // the positions are read by bulk copies
        in.sum[0] = ks;
        in.max32[0] = __float_as_uint(fdx);
        in.max32[1] = PY ? __float_as_uint(fdy) : 0u;
        in.max64 = PY ? 0ull : (unsigned long long)__double_as_longlong(mdy);
        in.max32[2] = mjump <= sh.steps.lim.jump ? 0u : 1u;
        exchange<kDNS, 3, PY ? 0 : 1>(M, sh.steps, seq, in, out);
        if (tid == 0) {
          const double tmx[3] = {
              (double)__uint_as_float(out.max32[0]) * sh.steps.dc.Lx,
              PY ? (double)__uint_as_float(out.max32[1]) * sh.steps.dc.Ly
                 : __longlong_as_double((long long)out.max64),
              out.max32[2] != 0u ? __longlong_as_double(0x7ff0000000000000LL) : 0.0};
          sh.steps.need = drift_tail<DMd>(&S, sh.steps.dc, sh.steps.ds, drift_tail_scalars(P, S),
                                          sh.steps.lim, out.sum, tmx);
        }
        __syncthreads();
        if (sh.steps.abort) break;
        if (sh.steps.need) {
          band_rebuild(D, M, &sh, sh_band, &seq, &list_parity);
          if (sh.steps.abort) break;
          if (tid == 0) {
            sh.steps.need = 0;
            sh.steps.lim =
                rebuild_limits<DMd>(sh.steps.dc.Lx, sh.steps.dc.Ly, drift_tail_scalars(P, S));
          }
          __syncthreads();
        }
      } else {
        // ---- force
        fence_async();
        const double Lx = S.Lx, Ly = S.Ly;
        ForceFinish<FM, PY> fin;
        if (FIRE && S.f_fp64 != 0) {
          fin = band_items_hp<FM, PY, false>(D, &P, &S, &sh.band, sh_band, blockIdx.x, P.items,
                                             &pass);
        } else {
          fin.init();
          band_items<FM, PY, false, false>(D, P, S, sh.band, sh_band, blockIdx.x, P.items, pass,
                                           fin);
        }
        bad |= fin.bad;
#pragma unroll
        for (int k = 0; k < kFNS; ++k) in.sum[k] = fin.red[k];
        if (FIRE) {
          in.max64 = (unsigned long long)__double_as_longlong(fin.mx[0]);
          in.max32[0] = fin.mx[1] > 0.0 ? 1u : 0u;
        }
        // (without sums too: the next drift overwrites the positions that slower
        // blocks still read, and reads velocities that other blocks have kicked)
        exchange<kFNS, FIRE ? 1 : 0, FIRE ? 1 : 0>(M, sh.steps, seq, in, out);
        if (tid == 0) {
          const ForceTail tin = force_tail_inputs<FM>(P, &S);
          const double tmx[3] = {FIRE ? __longlong_as_double((long long)out.max64) : 0.0,
                                 FIRE && out.max32[0] != 0u ? 1.0 : 0.0, 0.0};
          const int conv =
              force_tail<FM, PY>(&S, tin, Lx, Ly, 0.5 * P.dt, out.sum, tmx);
          if (FIRE) S.f_drift = conv ? 0 : 1;
          // scalars of the drift that follows (its limits change with the box)
          drift_prelude<DMd, kBoxMoves>(P, S, sh.steps.dc, sh.steps.ds);
          if (kBoxMoves)
            sh.steps.lim =
                rebuild_limits<DMd>(sh.steps.dc.Lx, sh.steps.dc.Ly, drift_tail_scalars(P, S));
          if (sh.band.lost) sh.steps.abort = 1;
        }
        __syncthreads();
        if (sh.steps.abort) break;
        if (FIRE && S.f_drift == 0) break;  // converged
      }
    }
    if (sh.steps.abort || sh.steps.stop) break;
    ++done;
  }
  if (bad) atomicOr(&D.st->nonfinite, 1);
  if (sh.steps.abort) {
    if (tid == 0) atomicExch(&D.st->err, 6);  // MDB_ERR_CUDA: an exchange or a copy gave up
    return;
  }
  __syncthreads();
  // (every block has read D.st and M.seq: see k_run_steps)
  if (blockIdx.x == 0) {
    store_state(D, S);
    if (tid == 0 && seq != seq0) *M.seq = seq;
  }
}

}  // namespace mdb
