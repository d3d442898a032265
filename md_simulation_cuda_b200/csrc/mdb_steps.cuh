// Resident steps kernel: many steps (or FIRE iterations) of a single system
// whose blocks all fit on the device at once, in one cooperative launch, with
// the cell-list rebuilds inside it.
//
// What bounds a step of such a system is latency: a few thousand particles
// give each SM a warp or two per scheduler, and what a step costs is the
// length of its dependent chain (loads, the pair loop, the reductions, the
// synchronisation of the blocks), not bytes or operations. So
//   * a thread keeps its slot's position, velocity, acceleration, type and
//     rebuild position in registers between rebuilds and its neighbour list in
//     shared memory; only the float-float positions go through global memory
//     (two buffers in turn, so the next drift may write while slower blocks
//     still gather);
//   * every block keeps a copy of the system's scalars (SysState) in shared
//     memory and updates it with the same operations on the same operands, so
//     no block waits for another one's scalar update;
//   * the reduction of a phase and the barrier after it are one exchange: each
//     block writes its partial sums and counts itself in, and every block that
//     sees the full count adds all partials up itself, in the fixed order of
//     reduce_system: no last block whose tail the others wait for, and no
//     second barrier after it. Maxima need no order: they go through one
//     atomic each;
//   * NVE needs nothing from other blocks between a force phase and the next
//     drift, so its steps hold one exchange instead of two.
// The arithmetic, the order of every sum and the blocks are those of the
// per-phase kernels (k_drift, k_rb_*, k_force): the results are the same bits.
//
// Measured on B200 against the phases as block functions with a last-block tail
// and a grid barrier each, in a graph loop that left the kernel for every
// rebuild (us per step, one call of many steps, rebuilds included): NVE 4,096
// particles 17.2 -> 5.0, Nose-Hoover slab 60,013 31 -> 14.8; against one launch
// per phase (piston, FIRE and one-step calls had no other): piston 20,011
// 30.6 -> 11.2, 20 one-step NVE calls of 900 particles 495 -> 250 us. What is
// left of a Nose-Hoover step at 4,096 (8.2 us, ~15,000 cycles): exchanges 9,000,
// pair sums 2,300, drift 1,300, rebuilds 1,600, scalars 1,000.
#pragma once

#include <stddef.h>

#include "mdb_kernels.cuh"

namespace mdb {

// Shared list columns are padded to a multiple of this with the slot's own
// offset, which the pair term skips (r^2 = 0): the pair loop then takes whole
// groups, with all of a group's gathers in flight at once.
constexpr int kListGroup = 8;
// Polls of an exchange (each is a round trip to L2, so some 1.5 s) before it looks
// whether the blocks it waits for have got on with a long scan (mark_progress); it
// gives up when nothing has moved since it last looked.
constexpr uint32_t kExchangePolls = 1u << 22;

// What a block keeps in shared memory beside its lists.
struct StepsShared {
  SysParams P;
  SysState S;
  DriftCtx dc;
  DriftScalars ds;
  RebuildLimits lim;
  PairBox box;
  double ksum[kThreads / kLanes];
  int scan[kThreads / 32];
  double sums[kNP][kThreads / 32];
  uint32_t max32[3][kThreads / 32];
  unsigned long long max64[kThreads / 32];
  int need, stop, abort;
};

// The system's parameters and state into shared memory (a block barrier before
// their first use is the caller's).
__device__ __forceinline__ void load_state(const Dev& D, StepsShared& sh) {
  for (int k = threadIdx.x; k < (int)(sizeof(SysParams) / 4); k += kThreads)
    ((uint32_t*)&sh.P)[k] = ((const uint32_t*)D.sp)[k];
  for (int k = threadIdx.x; k < (int)(sizeof(SysState) / 4); k += kThreads)
    ((uint32_t*)&sh.S)[k] = ((const uint32_t*)D.st)[k];
  if (threadIdx.x == 0) {
    sh.need = 0;
    sh.stop = 0;
    sh.abort = 0;
  }
}
// The state back to global memory (one block), but for what other blocks write
// there themselves: counts, flags and errors. An error is final for the handle
// and never lowered: a block that gave up an exchange has set it, perhaps one
// that this block saw through.
__device__ __forceinline__ void store_state(const Dev& D, const SysState& S) {
  for (int k = threadIdx.x; k < (int)(sizeof(SysState) / 4); k += kThreads) {
    const size_t at = (size_t)k * 4;
    if (at == offsetof(SysState, nonfinite) || at == offsetof(SysState, nl_overflow) ||
        at == offsetof(SysState, err))
      continue;
    ((uint32_t*)D.st)[k] = ((const uint32_t*)&S)[k];
  }
  if (threadIdx.x == 0 && S.err != 0) atomicCAS(&D.st->err, 0, S.err);
}

// What the threads of a block bring to an exchange, and thread 0 takes from
// it: sums, maxima of 32-bit values (non-negative floats as bits, flags) and
// one maximum of 64-bit ones (a non-negative double as bits).
struct Totals {
  double sum[kNP];
  uint32_t max32[3];
  unsigned long long max64;
};

// The sum of a block's eight warp sums, by the tree of block_reduce.
__device__ __forceinline__ double warps_sum(const double (&w)[kThreads / 32]) {
  static_assert(kThreads == 256, "eight warps");
  return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}

// One exchange between all blocks: the block's writes before it are visible
// to every block after it, and thread 0 of each block holds the system's NS
// sums, N32 32-bit and N64 64-bit maxima in out. The sums are added up as
// reduce_system adds them (thread t takes blocks t, t + kThreads, ..., then the
// block tree). One thread per block polls one counter: polling every block's
// own flag instead (all to all) cost 8,700 cycles at 148 blocks against 2,600.
// The partials alternate between two buffers and the maxima between four (the
// one used two exchanges ago is cleared here), so a block may be one exchange
// ahead of another. A wait that gives up sets sh.abort, after which the kernel ends
// with the system's error flag set; it does not wait again.
template <int NS, int N32, int N64>
__device__ __forceinline__ void exchange(const StepsMem& M, StepsShared& sh, uint32_t& seq,
                                         const Totals& in, Totals& out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N32; ++k) {
    const uint32_t v = __reduce_max_sync(0xffffffffu, in.max32[k]);
    if (lane == 0) sh.max32[k][warp] = v;
  }
  if (N64 > 0) {
    unsigned long long v = in.max64;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o);
      v = w > v ? w : v;
    }
    if (lane == 0) sh.max64[warp] = v;
  }
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    const double v = warp_sum(in.sum[k]);
    if (lane == 0) sh.sums[k][warp] = v;
  }
  __syncthreads();
  ++seq;
  const int nb = gridDim.x;
  double* part = M.part + (size_t)(seq & 1u) * kNP * nb;
  unsigned long long* mslot = M.max + (seq & 3u) * 4;
  if (warp == 0) {
    uint32_t v32[3];
#pragma unroll
    for (int k = 0; k < N32; ++k)
      v32[k] = __reduce_max_sync(0xffffffffu, lane < kThreads / 32 ? sh.max32[k][lane] : 0u);
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < NS; ++k) part[(size_t)k * nb + blockIdx.x] = warps_sum(sh.sums[k]);
#pragma unroll
      for (int k = 0; k < N32; ++k)
        if (v32[k] != 0u) atomicMax((unsigned int*)(mslot + k), v32[k]);
      if (N64 > 0) {
        unsigned long long v = sh.max64[0];
#pragma unroll
        for (int w = 1; w < kThreads / 32; ++w) v = sh.max64[w] > v ? sh.max64[w] : v;
        if (v != 0ull) atomicMax(mslot + 3, v);
      }
      // counts the block in; the release covers the block's writes (ordered
      // before by the block barrier)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(M.seq + 1) : "memory");
      uint32_t target = seq * (uint32_t)nb;
      const uint32_t most =
          M.late_block < 0 || M.late_block == (int)blockIdx.x ? M.polls : kExchangePolls;
      if (M.late_block == (int)blockIdx.x) ++target;
      uint32_t got, polls = 0, seen = 0;
      bool looked = false;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(M.seq + 1) : "memory");
        if ((int32_t)(got - target) >= 0) break;
        if (++polls < most) continue;
        const uint32_t now = *(volatile uint32_t*)(M.seq + 2);
        if (looked && now == seen) {
          sh.abort = 1;
          break;
        }
        looked = true;
        seen = now;
        polls = 0;
      }
    }
  }
  // (a block barrier, not only a warp's: it also brings warp 0 together after
  // its first lane's polling)
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x >= kThreads - 4)
    M.max[((seq + 2) & 3u) * 4 + (threadIdx.x - (kThreads - 4))] = 0ull;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < N32; ++k) out.max32[k] = (uint32_t)__ldcg(mslot + k);
    if (N64 > 0) out.max64 = __ldcg(mslot + 3);
  }
  if (NS > 0) {
    double v[NS > 0 ? NS : 1];
    const int q = threadIdx.x;
#pragma unroll
    for (int k = 0; k < NS; ++k) v[k] = q < nb ? __ldcg(part + (size_t)k * nb + q) : 0.0;
    for (int r = q + kThreads; r < nb; r += kThreads) {
#pragma unroll
      for (int k = 0; k < NS; ++k) v[k] += __ldcg(part + (size_t)k * nb + r);
    }
#pragma unroll
    for (int k = 0; k < NS; ++k) {
      v[k] = warp_sum(v[k]);
      if (lane == 0) sh.sums[k][warp] = v[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int k = 0; k < NS; ++k) out.sum[k] = warps_sum(sh.sums[k]);
    }
  }
}

// Pair sums of one slot that slot_list does not cover: stencil or whole-system
// scans, lists in global memory, and FP64 pair terms (rows >= 0: over the
// shared list column col where the slot has a list). Out of line: its registers do not count against the steps
// loop.
template <int FM, bool PY, int L>
__device__ __noinline__ void slot_sum_general(const Dev& D, const float4* pff, const SysParams& P,
                                              const SysState& S, int64_t i, double Lx, double Ly,
                                              int lane, bool hp, const int16_t* col, int rows,
                                              int nc, double* out) {
  constexpr bool kVirial = (FM == FM_NPH);
  constexpr bool kFloor = (FM == FM_FIRE);
  double fx, fy, w, u, an;
  if (FM == FM_FIRE && hp && rows >= 0 && nc >= 0) {
    const PairCtxD c = pair_ctx_hp(P, ld_pos<false>(pff + i), Lx, Ly);
    const int li = (int)(i - P.p0), n = P.n;
    const bool inner = (nc & kListInterior) != 0;
    fx = fy = w = u = an = 0.0;
    for (int k = 0; k < rows; ++k) {  // (a padding entry is the slot itself: r^2 = 0)
      int t = col[k * kThreads];
      if (inner) {
        pair_one_hp<PY, false, kVirial, false>(ld_pos<false>(pff + i + t), c, fx, fy, w, u, an);
      } else {
        t += li;
        t += (t < 0) ? n : 0;
        t -= (t >= n) ? n : 0;
        pair_one_hp<PY, false, kVirial, true>(ld_pos<false>(pff + P.p0 + t), c, fx, fy, w, u, an);
      }
    }
    w = 0.5 * w;
  } else if (FM == FM_FIRE && hp) {
    particle_force_hp<PY, false, kVirial, false>(D, pff, P, S, i, Lx, Ly, fx, fy, w, u, an);
  } else {
    int tci;
    particle_force<PY, false, kVirial, kFloor, false, L>(D, pff, P, S, i, Lx, Ly, fx, fy, w, u, an,
                                                         tci, lane);
  }
  out[0] = fx;
  out[1] = fy;
  out[2] = w;
}

// Pair sums over a shared list column of `rows` entries (a multiple of
// kListGroup). MIC = false: interior list, offsets from the slot itself.
template <bool PY, bool VIRIAL, bool MIC, bool FLOOR>
__device__ __forceinline__ void slot_list(const float4* __restrict__ pff, const int16_t* col,
                                          int rows, int64_t i, int li, int n, const PairCtx& c,
                                          float2& fs, float2& fc, float& ws, float& wc) {
  const float4* __restrict__ base = MIC ? pff + (i - li) : pff + i;
  double u = 0.0, an = 0.0;
  auto gather = [&](int k, float4 (&q)[kListGroup]) {
#pragma unroll
    for (int e = 0; e < kListGroup; ++e) {
      int t = col[(k + e) * kThreads];
      if (MIC) {
        t += li;
        t += (t < 0) ? n : 0;
        t -= (t >= n) ? n : 0;
      }
      q[e] = ld_pos<false>(base + t);
    }
  };
  for (int k = 0; k < rows; k += kListGroup) {
    float4 q[kListGroup];
    gather(k, q);
#pragma unroll
    for (int e = 0; e < kListGroup; ++e)
      pair_one<PY, false, VIRIAL, MIC, FLOOR>(q[e], c, fs, fc, ws, wc, u, an);
  }
}

// Neighbour list of slot k (the entries and order of build_list), shared by
// the L lanes of the slot: the lanes test consecutive candidates and a ballot
// gives each accepted one its place. Called by whole warps (a ballot over the
// lanes of one slot would run the warp's slots one after the other); `on`: the
// thread's slot gets a list. Entries go to row e / L of lane e % L in
// the shared columns (the kernel writes these to the global list when it ends:
// once, and whole rows at a time) or else to the global list. Returns the count
// (more than max_nbr: no list).
// (The minimum image is taken for interior slots as well: its shift is zero
// there and changes no bit. One copy of this code instead of two: it runs once
// in ~20 steps and is bound by fetching its instructions.)
template <bool PY, int L>
__device__ __forceinline__ int steps_build_list(const Dev& D, const float4* pff,
                                                const SysParams& P, const SysState& S, int64_t k,
                                                int cell, int lane, bool on, int16_t* cols,
                                                bool shared, int& nowrap) {
  PairCtx c;
  const float4 qi = ld_pos<false>(pff + k);
  set_pair_box<PY>(c, qi, S.Lx, S.Ly);
  const uint32_t tci = ff_class(qi);
  const uint32_t ts = (tci == 2u) ? 99u : tci;
  const float rl2s = P.frl2[tci == 2u ? 2 : tci], rl2ab = P.frl2[2];
  const int ncx = S.ncx, ncy = S.ncy;
  const int cx = cell % ncx, cy = cell / ncx;
  const int maxn = D.max_nbr;
  const int half = (P.n + 1) / 2;
  const unsigned lane0 = (threadIdx.x & 31) & ~(unsigned)(L - 1);
  // The candidate ranges (up to two per stencil row, in visiting order), all
  // loaded before the first is used, then walked as one sequence so that every
  // batch of loads is full: the build is bound by its dependent loads.
  int r0[6], r1[6];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    int yy = cy + r - 1;
    bool row_ok = on;
    if (PY) {
      if (yy < 0) yy += ncy;
      if (yy >= ncy) yy -= ncy;
    } else if (yy < 0 || yy >= ncy) {
      row_ok = false;
    }
    r0[2 * r] = r1[2 * r] = r0[2 * r + 1] = r1[2 * r + 1] = 0;
    if (row_ok) {
      const int32_t* cs = D.cstart + P.c0 + (int64_t)yy * ncx;
      const bool mid = cx > 0 && cx < ncx - 1;
      r0[2 * r] = ld_idx<false>(cs + (mid ? cx - 1 : (cx == 0 ? 0 : ncx - 2)));
      r1[2 * r] = ld_idx<false>(cs + (mid ? cx + 2 : (cx == 0 ? 2 : ncx)));
      if (!mid) {
        r0[2 * r + 1] = ld_idx<false>(cs + (cx == 0 ? ncx - 1 : 0));
        r1[2 * r + 1] = ld_idx<false>(cs + (cx == 0 ? ncx : 1));
      }
    }
  }
  // candidate m of the sequence is slot m + off[r] for m below end[r]
  int end[6], off[6], total = 0;
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    off[r] = r0[r] - total;
    total += r1[r] - r0[r];
    end[r] = total;
  }
  int cnt = 0;
  nowrap = 1;
  bool over = false;
  constexpr int U = L > 1 ? 4 : 8;
  const int most = __reduce_max_sync(0xffffffffu, (unsigned)total);
  for (int m0 = 0; m0 < most; m0 += L * U) {
    int jj[U];
    float4 qq[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int m = m0 + u * L + lane;
      int o = off[5];
#pragma unroll
      for (int r = 4; r >= 0; --r) o = m < end[r] ? off[r] : o;
      jj[u] = m < total ? m + o : (int)k;
      qq[u] = ld_pos<false>(pff + jj[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float2 dd;
      const float r2 = pair_r2<true>(qq[u], c, dd);
      const float rl2 = (ff_class(qq[u]) == ts) ? rl2s : rl2ab;
      const bool in = jj[u] != (int)k && r2 < rl2;
      int e = cnt;
      if (L > 1) {
        const unsigned got = (__ballot_sync(0xffffffffu, in) >> lane0) & ((1u << L) - 1u);
        e += __popc(got & ((1u << lane) - 1u));
        cnt += __popc(got);
      } else {
        cnt += in ? 1 : 0;
      }
      if (in) {
        int d = jj[u] - (int)k;  // offset modulo n into [-n/2, n/2)
        if (d >= half) {
          d -= P.n;
          nowrap = 0;
        }
        if (d < -half) {
          d += P.n;
          nowrap = 0;
        }
        if (D.nl16 && (d > 32767 || d < -32768)) {
          over = true;
        } else if (e < maxn) {
          if (shared)
            cols[(e / L) * kThreads + (e % L)] = (int16_t)d;
          else if (D.nl16)
            D.nlist16[(int64_t)e * D.ntot + k] = (int16_t)d;
          else
            D.nlist[(int64_t)e * D.ntot + k] = d;
        }
      }
    }
  }
  if (L > 1) {
    const unsigned slot = ((1u << L) - 1u) << lane0;
    nowrap = (__ballot_sync(0xffffffffu, nowrap == 0) & slot) == 0u ? 1 : 0;
    over = (__ballot_sync(0xffffffffu, over) & slot) != 0u;
  }
  return over ? maxn + 1 : cnt;
}

// Runs up to `todo` steps (FIRE: iterations) of the engine's single system.
// Grid: the system's blocks, all resident (cooperative launch). One slot per
// thread, or per kLanes threads (LN).
template <int DMd, int FM, bool LN>
__global__ void __launch_bounds__(kThreads, 2) k_run_steps(Dev D, StepsMem M, int64_t todo) {
  constexpr bool PY = DMd != DM_PISTON;
  constexpr bool FIRE = DMd == DM_FIRE;
  constexpr int L = LN ? kLanes : 1;
  constexpr int spb = kThreads / L;
  constexpr bool kVirial = (FM == FM_NPH);
  constexpr bool kBoxMoves = (DMd == DM_NPH || DMd == DM_PISTON);
  constexpr int kDNS = (DMd == DM_NH) ? 1 : 0;
  constexpr int kFNS = ForceRed<FM>::NS;
  __shared__ StepsShared sh;
  extern __shared__ int16_t sh_lists[];  // [list_rows][kThreads]
  const int tid = threadIdx.x;
  const int lane = tid % L;
  const int li = blockIdx.x * spb + tid / L;
  const bool act = li < (int)D.ntot;  // (the engine's one system)
  const bool shared_list = M.list_rows > 0;
  // What does not depend on the system's state is loaded first: a call of one
  // step is mostly this chain of loads (20 calls of one step, 900 particles:
  // 281 -> 250 us; a list entry at a time cost a trip to L2 each).
  int nc = 0;
  int16_t head[kListGroup];
  if (act) {
    nc = D.ncount[li];
    if (shared_list) {
#pragma unroll
      for (int k = 0; k < kListGroup; ++k)
        head[k] = k * L + lane < D.max_nbr ? D.nlist16[(int64_t)(k * L + lane) * D.ntot + li]
                                           : (int16_t)0;
    }
  }
  load_state(D, sh);
  uint32_t seq = *M.seq;
  const uint32_t seq0 = seq;
  __syncthreads();
  const SysParams& P = sh.P;
  SysState& S = sh.S;
  const int64_t i = P.p0 + li;
  const bool own = act && lane == 0;
  const int64_t rebuilds0 = S.rebuilds;
  const int64_t half = half_of(D, &S);  // (the sort in here is in place)
  int16_t* col = sh_lists + tid;

  // the slot's state, in registers from here on
  double2 x = make_double2(0.0, 0.0), v = x, a = x;
  float2 sb = make_float2(0.f, 0.f);
  float4 qi = make_float4(0.f, 0.f, 0.f, 0.f);
  int t = 0, rows = 0;
  if (act) {
    x = D.pos[half + i];
    v = D.vel[half + i];
    a = D.acc[half + i];
    t = D.type[half + i];
    sb = D.sb[i];
    qi = D.pff[i];
  }
  // pads this thread's list column to whole groups
  auto pad_column = [&]() {
    const int nn = nc >= 0 ? (nc & (kListInterior - 1)) : 0;
    const int kk = nn > lane ? (nn - lane + L - 1) / L : 0;
    rows = (kk + kListGroup - 1) / kListGroup * kListGroup;
    for (int k = kk; k < rows; ++k) col[k * kThreads] = 0;
    return kk;
  };
  if (act && shared_list) {
    const int kk = pad_column();
#pragma unroll
    for (int k = 0; k < kListGroup; ++k)
      if (k < kk) col[k * kThreads] = head[k];
    for (int k0 = kListGroup; k0 < kk; k0 += kListGroup) {
#pragma unroll
      for (int k = 0; k < kListGroup; ++k)
        if (k0 + k < kk) head[k] = D.nlist16[(int64_t)((k0 + k) * L + lane) * D.ntot + i];
#pragma unroll
      for (int k = 0; k < kListGroup; ++k)
        if (k0 + k < kk) col[(k0 + k) * kThreads] = head[k];
    }
  }
  const float4* cur = D.pff;  // positions of the last drift or rebuild
  Totals in, out;
  int bad = 0;

  if (tid == 0) {
    drift_prelude<DMd>(P, S, sh.dc, sh.ds);
    sh.lim = rebuild_limits<DMd>(sh.dc.Lx, sh.dc.Ly, drift_tail_scalars(P, S));
    sh.box = pair_box<PY>(S.Lx, S.Ly);
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
        // ---- drift
        if (sh.ds.boxbad) {
          __syncthreads();
          if (tid == 0) {
            S.err = 5;  // MDB_ERR_BOX
            sh.stop = 1;
          }
          __syncthreads();
          break;
        }
        in.sum[0] = 0.0;
        in.max32[0] = in.max32[1] = in.max32[2] = 0u;
        in.max64 = 0ull;
        if (act) {
          double mdx = 0.0, mdy = 0.0, mjump = 0.0;
          float fdx = 0.f, fdy = 0.f;
          drift_move<DMd>(sh.dc, x, v, a, t, sb, in.sum[0], mdx, mdy, mjump, fdx, fdy, bad);
          qi = encode_ff(x.x, x.y, t, sh.dc.offx, sh.dc.offy);
          // maxima of the fractional displacements (the box length is
          // multiplied in after: the same bits), of the walled y axis itself,
          // and whether the jump exceeds its limit
          in.max32[0] = __float_as_uint(fdx);
          if (PY)
            in.max32[1] = __float_as_uint(fdy);
          else
            in.max64 = (unsigned long long)__double_as_longlong(mdy);
          in.max32[2] = mjump <= sh.lim.jump ? 0u : 1u;
        }
        float4* nxt = (cur == D.pff) ? M.pff1 : D.pff;
        if (own) nxt[i] = qi;
        cur = nxt;
        if (LN && kDNS > 0) {
          // k_drift sums slot by slot (thread t: slot t): put the sums there
          if (lane == 0) sh.ksum[tid / L] = in.sum[0];
          __syncthreads();
          in.sum[0] = tid < spb ? sh.ksum[tid] : 0.0;
        }
        exchange<kDNS, 3, PY ? 0 : 1>(M, sh, seq, in, out);
        if (tid == 0) {
          const double tmx[3] = {
              (double)__uint_as_float(out.max32[0]) * sh.dc.Lx,
              PY ? (double)__uint_as_float(out.max32[1]) * sh.dc.Ly
                 : __longlong_as_double((long long)out.max64),
              out.max32[2] != 0u ? __longlong_as_double(0x7ff0000000000000LL) : 0.0};
          sh.need = drift_tail<DMd>(&S, sh.dc, sh.ds, drift_tail_scalars(P, S), sh.lim, out.sum, tmx);
          if (kBoxMoves) sh.box = pair_box<PY>(S.Lx, S.Ly);
        }
        __syncthreads();
        if (sh.abort) break;
        if (sh.need) {
          // ---- rebuild (the passes of k_rb_*, on the slots' own threads)
          if (tid == 0) {
            set_cell_grid(P, &S);
            if (blockIdx.x == 0) D.st->nl_overflow = 0;
          }
          __syncthreads();
          // bin: the rank of the arrival in its cell is arbitrary
          const int ncell = S.ncx * S.ncy;
          const int per = (ncell + (int)gridDim.x - 1) / (int)gridDim.x;  // cells per block
          int key = 0, rank = 0, orig = 0;
          double theta = 0.0;
          if (own) {
            key = bin_axis(x.y * S.inv_wy, S.ncy) * S.ncx + bin_axis(x.x * S.inv_wx, S.ncx);
            rank = atomicAdd(D.ccount + P.c0 + key, 1);
            // one add per warp and tile: neighbouring slots share tiles, and
            // single adds queued for 40,000 cycles at 60,000 slots
            const int tile = key / per;
            const unsigned same = __match_any_sync(__activemask(), tile);
            if ((tid & 31) == __ffs(same) - 1) atomicAdd(M.tile + tile, __popc(same));
            orig = D.orig[half + i];
            theta = D.theta[half + i];
          }
          exchange<0, 0, 0>(M, sh, seq, in, out);
          if (sh.abort) break;
          // scan: this block's cells after the particles of all cells before
          {
            int before = 0;
            for (int q = tid; q < (int)blockIdx.x; q += kThreads) before += __ldcg(M.tile + q);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
            if ((tid & 31) == 0) sh.scan[tid >> 5] = before;
            __syncthreads();
            int carry = 0;
#pragma unroll
            for (int w = 0; w < kThreads / 32; ++w) carry += sh.scan[w];
            __syncthreads();
            const int c0 = (int)blockIdx.x * per;
            const int c1 = min(ncell, c0 + per);
            for (int cb = c0; cb < c1; cb += kThreads) {
              const int cc = cb + tid;
              const int cn = cc < c1 ? __ldcg(D.ccount + P.c0 + cc) : 0;
              int xs = cn;
#pragma unroll
              for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, xs, o);
                if ((tid & 31) >= o) xs += y;
              }
              if ((tid & 31) == 31) sh.scan[tid >> 5] = xs;
              __syncthreads();
              int base = carry, all = 0;
#pragma unroll
              for (int w = 0; w < kThreads / 32; ++w) {
                if (w < (tid >> 5)) base += sh.scan[w];
                all += sh.scan[w];
              }
              if (cc < c1) {
                D.cstart[P.c0 + cc] = (int)P.p0 + base + xs - cn;
                D.ccount[P.c0 + cc] = 0;
              }
              carry += all;
              __syncthreads();
            }
            if (c0 < ncell && c1 == ncell && tid == 0) D.cstart[P.c0 + ncell] = (int)P.p0 + P.n;
          }
          exchange<0, 0, 0>(M, sh, seq, in, out);
          if (sh.abort) break;
          if (tid == 0) M.tile[blockIdx.x] = 0;
          int ca = 0, ce = 0;
          if (own) {
            ca = ld_idx<false>(D.cstart + P.c0 + key);
            ce = ld_idx<false>(D.cstart + P.c0 + key + 1);
            D.perm[ca + rank] = (int)i;
          }
          exchange<0, 0, 0>(M, sh, seq, in, out);
          if (sh.abort) break;
          if (own) {
            // the stable place in the cell: after the lower source slots
            int before = 0;
            for (int k = ca; k < ce; k += 8) {
              int other[8];
#pragma unroll
              for (int e = 0; e < 8; ++e)
                other[e] = k + e < ce ? ld_idx<false>(D.perm + k + e) : (int)i;
#pragma unroll
              for (int e = 0; e < 8; ++e) before += other[e] < (int)i ? 1 : 0;
            }
            const int64_t dst = ca + before;
            D.pos[half + dst] = x;
            D.vel[half + dst] = v;
            D.acc[half + dst] = a;
            D.type[half + dst] = t;
            D.theta[half + dst] = theta;
            D.orig[half + dst] = orig;
            D.cell_of[dst] = key;
            D.pff[dst] = qi;
            M.pff1[dst] = qi;
            const float sx = (float)(x.x * (1.0 / S.Lx));
            const float sy = S.periodic_y ? (float)(x.y * (1.0 / S.Ly)) : (float)x.y;
            D.sb[dst] = make_float2(sx, sy);
          }
          exchange<0, 0, 0>(M, sh, seq, in, out);
          if (sh.abort) break;
          const int64_t clock = rebuild_clock(P, S);
          const bool recent = clock - S.rb_last < kListMinReuse;
          nc = -1;
          if (!S.allpairs && D.max_nbr > 0 && !recent) {  // (the same for every block)
            const int64_t k = act ? i : P.p0;
            const int cell = __ldcg(D.cell_of + k);
            const int cx = cell % S.ncx, cy = cell / S.ncx;
            // interior cells: see k_rb_nlist
            const bool inner = cx >= 2 && cx <= S.ncx - 3 &&
                               (!S.periodic_y || (cy >= 2 && cy <= S.ncy - 3));
            int nowrap = 0;
            const int cnt = steps_build_list<PY, L>(D, cur, P, S, k, cell, lane, act,
                                                    sh_lists + (tid - lane), shared_list, nowrap);
            if (cnt > D.max_nbr) {
              if (own) atomicAdd(&D.st->nl_overflow, 1);
            } else {
              nc = cnt | ((inner && nowrap) ? kListInterior : 0);
            }
          }
          if (act) {
            x = __ldcg(D.pos + half + i);
            v = __ldcg(D.vel + half + i);
            a = __ldcg(D.acc + half + i);
            t = __ldcg(D.type + half + i);
            sb = __ldcg(D.sb + i);
            qi = __ldcg(cur + i);
            if (lane == 0) D.ncount[i] = nc;
            if (shared_list) pad_column();
          }
          __syncthreads();
          if (tid == 0) {
            S.rebuilds += 1;
            S.rb_last = clock;
            sh.need = 0;
            sh.lim = rebuild_limits<DMd>(sh.dc.Lx, sh.dc.Ly, drift_tail_scalars(P, S));
          }
          __syncthreads();
        }
      } else {
        // ---- force
        ForceFinish<FM, PY> fin;
        fin.init();
        const double Lx = S.Lx, Ly = S.Ly;
        const double h = 0.5 * P.dt;
        const double xi2 = (FM == FM_NH) ? S.xi : 0.0;
        const double fdt = FIRE ? S.f_dt : 0.0;
        double fx = 0.0, fy = 0.0, w = 0.0;
        const int tci = (int)ff_class(qi);
        if (act) {
          const bool hp = FIRE && S.f_fp64 != 0;
          if (shared_list && nc >= 0 && !hp) {
            PairCtx c;
            c.ih = make_float2(qi.x, qi.y);
            c.il = make_float2(qi.z, qi.w);
            c.nLh = sh.box.nLh;
            c.nLl = sh.box.nLl;
            c.invL = sh.box.invL;
            set_pair_class<FIRE>(c, P, tci);
            float2 fs = make_float2(0.f, 0.f), fc = make_float2(0.f, 0.f);
            float ws = 0.f, wc = 0.f;
            if (nc & kListInterior)
              slot_list<PY, kVirial, false, FIRE>(cur, col, rows, i, li, P.n, c, fs, fc, ws, wc);
            else
              slot_list<PY, kVirial, true, FIRE>(cur, col, rows, i, li, P.n, c, fs, fc, ws, wc);
            fx = (double)fs.x - (double)fc.x;
            fy = (double)fs.y - (double)fc.y;
            w = 0.5 * ((double)ws - (double)wc);
          } else {
            double out[3];
            slot_sum_general<FM, PY, L>(D, cur, P, S, i, Lx, Ly, lane, hp, col,
                                        shared_list ? rows : -1, nc, out);
            fx = out[0];
            fy = out[1];
            w = out[2];
          }
        }
        if (L > 1) {
          // the fixed butterfly of k_force: every lane ends with the same bits
#pragma unroll
          for (int o = 1; o < L; o <<= 1) {
            fx += __shfl_xor_sync(0xffffffffu, fx, o);
            fy += __shfl_xor_sync(0xffffffffu, fy, o);
            if (kVirial) w += __shfl_xor_sync(0xffffffffu, w, o);
          }
        }
        if (act) fin.kick(P, Ly, h, xi2, fdt, x.y, fx, fy, w, 0.0, 0.0, tci, v, a);
        bad |= fin.bad;
        if (L > 1 && lane != 0) {
#pragma unroll
          for (int k = 0; k < kNP; ++k) fin.red[k] = 0.0;  // one lane counts for the slot
        }
        if (kFNS > 0) {
#pragma unroll
          for (int k = 0; k < kFNS; ++k) in.sum[k] = fin.red[k];
          if (FIRE) {
            in.max64 = (unsigned long long)__double_as_longlong(fin.mx[0]);
            in.max32[0] = fin.mx[1] > 0.0 ? 1u : 0u;
          }
          exchange<kFNS, FIRE ? 1 : 0, FIRE ? 1 : 0>(M, sh, seq, in, out);
        } else {
          __syncthreads();
        }
        if (tid == 0) {
          const ForceTail tin = force_tail_inputs<FM>(P, &S);
          const double tmx[3] = {FIRE ? __longlong_as_double((long long)out.max64) : 0.0,
                                 FIRE && out.max32[0] != 0u ? 1.0 : 0.0, 0.0};
          const int conv = force_tail<FM, PY>(&S, tin, Lx, Ly, h, out.sum, tmx);
          if (FIRE) S.f_drift = conv ? 0 : 1;
          // scalars of the drift that follows (its limits change with the box)
          drift_prelude<DMd, kBoxMoves>(P, S, sh.dc, sh.ds);
          if (kBoxMoves)
            sh.lim = rebuild_limits<DMd>(sh.dc.Lx, sh.dc.Ly, drift_tail_scalars(P, S));
        }
        __syncthreads();
        if (sh.abort) break;
        if (FIRE && S.f_drift == 0) break;  // converged
      }
    }
    if (sh.abort || sh.stop) break;
    ++done;
  }
  if (bad) atomicOr(&D.st->nonfinite, 1);
  if (sh.abort) {
    // MDB_ERR_CUDA: an exchange gave up. (The slots stay as they are: others may
    // have finished a rebuild that this block has not.)
    if (tid == 0) atomicExch(&D.st->err, 6);
    return;
  }
  if (own) {
    D.pos[half + i] = x;
    D.vel[half + i] = v;
    D.acc[half + i] = a;
    D.pff[i] = qi;
  }
  if (act && shared_list && S.rebuilds != rebuilds0) {
    const int nn = nc >= 0 ? (nc & (kListInterior - 1)) : 0;
    for (int k = 0; k * L + lane < nn; ++k)
      D.nlist16[(int64_t)(k * L + lane) * D.ntot + i] = col[k * kThreads];
  }
  __syncthreads();
  // Every block has read D.st and M.seq (it took part in an exchange) unless
  // there was none, in which case nothing a block acts on has changed.
  if (blockIdx.x == 0) {
    store_state(D, S);
    if (tid == 0 && seq != seq0) *M.seq = seq;
  }
}

}  // namespace mdb
