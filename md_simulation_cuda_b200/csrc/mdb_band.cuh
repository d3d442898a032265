// Force phase and list build over staged bands: for systems too large for the
// resident steps kernel and for batches.
//
// A chunk is 256 consecutive slots of a system. Slots are sorted by cell, cells
// by rows, so what a chunk's particles can meet are a few contiguous slot
// ranges: the chunk's own stretch of its cell row and the same stretch of the
// rows above and below, one cell wider on each side (four rows in two pieces
// each where the chunk runs over the end of a row; whole rows where those are
// short). This band, ~850 positions of 16 bytes, is what the block copies into
// shared memory with one bulk copy per range (cp.async.bulk, completion on an
// mbarrier), the next chunk's band while it works on this one.
//
// Why: the force phase was bound by waiting, not by issue (55% of the cycles) or
// bytes (15% of HBM): each list entry is an index load and then a gather through
// L1 that missed to L2 in 28% of its sectors, and a slot's last entries were
// taken one at a time. From a staged band a gather costs ~30 cycles, an entry
// is a 16-bit index into the band (no wrap, no 64-bit address), four entries
// arrive in one 8-byte load, and lists are padded to groups of four with the
// slot itself (r^2 = 0, which the pair term skips), so that no lane runs a
// remainder loop. The candidates, their order and the arithmetic are those of
// k_force: the results are the same bits.
#pragma once

#include "mdb_kernels.cuh"

namespace mdb {

// ------------------------------------------------------------------- bands --

// First and one-past-last cell of piece r of the band of a chunk whose slots lie
// in the cells from (x0, y0) to (x1, y1) of an ncx x ncy grid; the number of
// pieces through nr. Pieces are disjoint runs of cells in slot order, and every
// run of stencil cells that a slot of the chunk visits lies inside one of them:
//  * full: whole rows y0 - 1 .. y1 + 1 (every row when that covers the grid),
//    as one run, split where it passes the periodic edge;
//  * one row: the cells x0 - 1 .. x1 + 1 of three rows, and for an end cell of
//    the row the cell across the edge;
//  * two rows (y1 = y0 + 1): of four rows the cells 0 .. x1 + 1 and
//    x0 - 1 .. ncx - 1. (Of a periodic side of three rows the fourth is the first
//    again; a side of fewer has no cell lists.)
//  * more rows: its rows whole, as one run, and of the rows before and after them
//    the cells x0 - 1 .. ncx - 1 and 0, and 0 .. x1 + 1 and ncx - 1. (A lattice's
//    rows of cells are as unequal as 256 and 384 particles: as whole rows, the
//    chunks of an eighth of 16,384 did not fit.)
// Rows beyond a walled y axis are empty. A box three or four cells high takes the
// row pieces too: its rows are long, and as whole rows they left its chunks
// without lists (16 systems of 9,000 particles in strips of four rows: 55 us a
// step, 32 with lists).
struct BandShape {
  int x0, y0, x1, y1, ncx, ncy;
  bool py, full;
};
__device__ __forceinline__ int band_pieces(const BandShape& s) {
  if (s.full) return 3;
  if (s.y1 > s.y0 + 1) return 5;
  return s.y1 == s.y0 ? 6 : 8;
}
__device__ __forceinline__ bool band_piece(const BandShape& s, int r, int* c0, int* c1) {
  if (s.full) {
    int lo = s.y0 - 1, hi = s.y1 + 1;
    if (hi - lo + 1 >= s.ncy || !s.py) {
      lo = max(lo, 0);
      hi = min(hi, s.ncy - 1);
      if (s.py) {
        lo = 0;
        hi = s.ncy - 1;
      }
      *c0 = lo * s.ncx;
      *c1 = (hi + 1) * s.ncx;
      return r == 0;
    }
    // rows below the edge, in the grid, above the edge
    if (r == 0) {
      *c0 = (lo + s.ncy) * s.ncx;
      *c1 = s.ncy * s.ncx;
      return lo < 0;
    }
    if (r == 1) {
      *c0 = max(lo, 0) * s.ncx;
      *c1 = (min(hi, s.ncy - 1) + 1) * s.ncx;
      return true;
    }
    *c0 = 0;
    *c1 = (hi - s.ncy + 1) * s.ncx;
    return hi >= s.ncy;
  }
  int y, a, b;
  bool some = true;
  if (s.y1 == s.y0) {
    y = s.y0 - 1 + r / 2;
    const int lo = max(s.x0 - 1, 0), hi = min(s.x1 + 1, s.ncx - 1);
    if ((r & 1) == 0) {
      a = lo;
      b = hi;
    } else {
      // the cell across the edge, unless the run holds it
      a = b = (s.x0 == 0) ? s.ncx - 1 : 0;
      some = (s.x0 == 0 || s.x1 == s.ncx - 1) && !(a >= lo && a <= hi);
    }
  } else if (s.y1 > s.y0 + 1) {
    if (r == 2) {
      *c0 = s.y0 * s.ncx;
      *c1 = (s.y1 + 1) * s.ncx;
      return true;
    }
    y = r < 2 ? s.y0 - 1 : s.y1 + 1;
    if (r < 2) {
      a = r == 0 ? max(s.x0 - 1, 0) : 0;
      b = r == 0 ? s.ncx - 1 : 0;
      some = r == 0 || s.x0 > 1;
    } else {
      a = r == 3 ? 0 : s.ncx - 1;
      b = r == 3 ? min(s.x1 + 1, s.ncx - 1) : s.ncx - 1;
      some = r == 3 || s.x1 < s.ncx - 2;
    }
  } else {
    y = s.y0 - 1 + r / 2;
    const int left = min(s.x1 + 1, s.ncx - 1), right = max(s.x0 - 1, 0);
    const bool joined = right <= left + 1;
    if ((r & 1) == 0) {
      a = 0;
      b = joined ? s.ncx - 1 : left;
    } else {
      a = right;
      b = s.ncx - 1;
      some = !joined;
    }
  }
  if (s.py && s.ncy == 3 && s.y1 == s.y0 + 1 && r >= 6) some = false;
  if (y < 0 || y >= s.ncy) {
    if (!s.py) some = false;
    y += (y < 0) ? s.ncy : -s.ncy;
  }
  *c0 = y * s.ncx + a;
  *c1 = y * s.ncx + b + 1;
  return some;
}

// Computed by warp 0 of a block for the chunk that starts at slot cs: the
// band's ranges into *b (shared or global memory). total = 0: no band (it
// would exceed kBandCap).
__device__ __forceinline__ void make_band(const Dev& D, const SysParams& P, const SysState& S,
                                          int64_t cs, Band* b) {
  const int lane = threadIdx.x & 31;
  const int64_t last = min(cs + kThreads, P.p0 + P.n) - 1;
  BandShape s;
  s.ncx = S.ncx;
  s.ncy = S.ncy;
  s.py = S.periodic_y != 0;
  const int f = D.cell_of[cs], l = D.cell_of[last];
  s.x0 = f % s.ncx;
  s.y0 = f / s.ncx;
  s.x1 = l % s.ncx;
  s.y1 = l / s.ncx;
  const int32_t* cst = D.cstart + P.c0;
  // whole rows when they fit (one run), or when the rows before and after the
  // chunk's meet
  {
    const int lo = max(s.y0 - 1, 0), hi = min(s.y1 + 1, s.ncy - 1);
    int rows = cst[(hi + 1) * s.ncx] - cst[lo * s.ncx];
    if (s.py && s.y0 == 0) rows += cst[s.ncy * s.ncx] - cst[(s.ncy - 1) * s.ncx];
    if (s.py && s.y1 == s.ncy - 1) rows += cst[s.ncx] - cst[0];
    s.full = rows <= kBandCap || (s.py && s.y1 > s.y0 + 1 && s.y1 - s.y0 + 3 > s.ncy);
  }
  const int np = band_pieces(s);
  int start = 0, len = 0;
  if (lane < np) {
    int c0, c1;
    if (band_piece(s, lane, &c0, &c1)) {
      start = cst[c0];
      len = cst[c1] - start;
    }
  }
  int end = len;
#pragma unroll
  for (int o = 1; o < kBandRanges; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += y;
  }
  const int total = __shfl_sync(0xffffffffu, end, kBandRanges - 1);
  const bool fits = total <= kBandCap;
  if (lane < kBandRanges) {
    b->start[lane] = start;
    b->len[lane] = fits ? len : 0;
    b->off[lane] = end - len;
  }
  if (lane == 0) b->total = fits ? total : 0;
}

// Place in the band of slot j (which some range holds).
__device__ __forceinline__ int band_place(const Band& b, int j) {
  int at = 0;
#pragma unroll
  for (int r = 0; r < kBandRanges; ++r) {
    const int d = j - b.start[r];
    if (d >= 0 && d < b.len[r]) at = b.off[r] + d;
  }
  return at;
}

// ---------------------------------------------------------- rebuild: lists --

// The list of the slot at place `self` of a staged band (cell cx, cy), whole
// groups of four to out, padded with the slot's own place. Returns the count
// (the groups are written as far as max_nbr reaches).
//
// Two passes over each run of candidates: a test that only sets a bit, then a
// loop over the set bits. About 19 of 63 candidates are near, but in a warp
// nearly every candidate is near for some lane: appending inside the test ran
// the append code 63 times per slot instead of ~25 (the whole list kernel
// 242 -> 137 us at 1,048,576 particles).
template <bool MIC>
__device__ __forceinline__ int build_band_list(const Dev& D, const SysParams& P, const SysState& S,
                                               const Band& band, const float4* pos, int self,
                                               int cx, int cy, bool py, uint2* out) {
  const int ncx = S.ncx, ncy = S.ncy;
  PairCtx c;
  const float4 qi = pos[self];
  c.ih = make_float2(qi.x, qi.y);
  c.il = make_float2(qi.z, qi.w);
  if (MIC) {
    const PairBox bx = py ? pair_box<true>(S.Lx, S.Ly) : pair_box<false>(S.Lx, S.Ly);
    c.nLh = bx.nLh;
    c.nLl = bx.nLl;
    c.invL = bx.invL;
  }
  const uint32_t tci = ff_class(qi);
  const uint32_t tsz = (tci == 1u) ? 1u : 0u;  // (see pair_one)
  const float rl2s = P.frl2[tci == 2u ? 2 : tci], rl2ab = P.frl2[2];
  const int groups = (D.max_nbr + 3) >> 2;
  const int32_t* cst = D.cstart + P.c0;
  int cnt = 0;
  uint64_t acc = 0;  // the group being filled
  auto append = [&](int place) {
    acc = (acc >> 16) | ((uint64_t)place << 48);
    ++cnt;
    if ((cnt & 3) == 0 && (cnt >> 2) <= groups) {
      *out = make_uint2((uint32_t)acc, (uint32_t)(acc >> 32));
      out += D.ntot;
    }
  };
  // one run of stencil cells: slots [a, e), contiguous in the band
  auto scan = [&](int a, int e) {
    int at = band_place(band, a);
    for (int left = e - a; left > 0; left -= 32, at += 32) {
      const int len = min(left, 32);
      uint32_t near = 0;
      for (int m = 0; m < len; m += 4) {
        // (up to three places past the run are read: the band has that much
        // room, and their bits are cleared below)
        uint32_t four = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 q = pos[at + m + u];
          float2 dd;
          const float r2 = pair_r2<MIC>(q, c, dd);
          const bool same = (((__float_as_uint(q.z) ^ tsz) | __float_as_uint(q.w)) & 1u) == 0u;
          if (r2 < (same ? rl2s : rl2ab)) four |= 1u << u;
        }
        near |= four << m;
      }
      if (len < 32) near &= (1u << len) - 1u;
      const int own = self - at;
      if (own >= 0 && own < 32) near &= ~(1u << own);
      while (near != 0u) {
        append(at + __ffs(near) - 1);
        near &= near - 1u;
      }
    }
  };
  for (int dr = -1; dr <= 1; ++dr) {
    int yy = cy + dr;
    if (py) {
      if (yy < 0) yy += ncy;
      if (yy >= ncy) yy -= ncy;
    } else if (yy < 0 || yy >= ncy) {
      continue;
    }
    const int32_t* row = cst + (int64_t)yy * ncx;
    // (interior slots have the one run)
    const bool mid = !MIC || (cx > 0 && cx < ncx - 1);
    scan(row[mid ? cx - 1 : (cx == 0 ? 0 : ncx - 2)], row[mid ? cx + 2 : (cx == 0 ? 2 : ncx)]);
    if (!mid) scan(row[cx == 0 ? ncx - 1 : 0], row[cx == 0 ? ncx : 1]);
  }
  const int n = cnt;
  while ((cnt & 3) != 0) append(self);
  return n;
}

// Bands of every chunk of the systems that rebuild, and their slots' lists:
// entry e of slot k is the place of its partner in the chunk's band, 16 bits at
// lists[((e / 4) * ntot + k) * 4 + e % 4], whole groups of four padded with the
// slot's own place. One block per chunk in turn; the candidates are read from
// the staged band. The entries, their order and the count are those of
// build_list.
// (full: an mbarrier for one arrival, parity its current phase. False: a copy
// never arrived.)
__device__ __forceinline__ bool rb_band(const Dev& D, float4* sh_band, Band& band, uint64_t& full,
                                        uint32_t& parity, bool forced) {
  bool all = true;
  for (int q = blockIdx.x; q < D.nchunks; q += gridDim.x) {
    const int s = D.sys_of_chunk[q];
    if (!sys_rebuilds(D, s)) continue;  // (the whole block)
    const SysParams& P = D.sp[s];
    SysState* S = D.st + s;
    const int64_t cs = P.p0 + (int64_t)(q - P.ch0) * kThreads;
    const int64_t k = cs + threadIdx.x;
    const bool act = k < P.p0 + P.n;
    // a system that rebuilds again within kListMinReuse steps scans its cell
    // stencil instead of a list it would hardly reuse
    const bool recent = !forced && rebuild_clock(P, *S) - S->rb_last < kListMinReuse;
    const bool lists = !S->allpairs && D.max_nbr > 0 && !recent;
    if (threadIdx.x < 32) {
      if (!S->allpairs) {
        make_band(D, P, *S, cs, &band);
      } else if (threadIdx.x < kBandRanges) {
        band.start[threadIdx.x] = band.len[threadIdx.x] = band.off[threadIdx.x] = 0;
        if (threadIdx.x == 0) band.total = 0;
      }
    }
    __syncthreads();
    if (threadIdx.x < (int)(sizeof(Band) / 4))
      ((int32_t*)(D.bands + q))[threadIdx.x] = ((const int32_t*)&band)[threadIdx.x];
    if (band.total == 0 || !lists) {
      if (act) D.ncount[k] = -1;
      if (threadIdx.x == 0) {
        const int slots = (int)min((int64_t)kThreads, P.p0 + P.n - cs);
        if (lists) atomicAdd(&S->nl_overflow, slots);  // they scan their stencils
        if (forced && band.total == 0) atomicAdd(&D.bg->unbanded, slots);
      }
      __syncthreads();  // (the band is rewritten for the next chunk)
      continue;
    }
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0) mbar_expect(&full, (uint32_t)band.total * 16u);
      __syncwarp();
      if (threadIdx.x < kBandRanges && band.len[threadIdx.x] > 0)
        copy_bulk(sh_band + band.off[threadIdx.x], D.pff + band.start[threadIdx.x],
                       band.len[threadIdx.x], &full);
    }
    const bool here = mbar_wait(&full, parity);
    parity ^= 1u;
    all = all && here;
    if (!here) {
      if (act) D.ncount[k] = -1;
    } else if (act) {
      const int cell = D.cell_of[k];
      const int cx = cell % S->ncx, cy = cell / S->ncx;
      const bool py = S->periodic_y != 0;
      const bool interior =
          cx >= 2 && cx <= S->ncx - 3 && (!py || (cy >= 2 && cy <= S->ncy - 3));
      const int self = band_place(band, (int)k);
      const int cnt =
          interior
              ? build_band_list<false>(D, P, *S, band, sh_band, self, cx, cy, py, D.lists + k)
              : build_band_list<true>(D, P, *S, band, sh_band, self, cx, cy, py, D.lists + k);
      if (cnt > D.max_nbr) {
        D.ncount[k] = -1;  // too many neighbours: the force loop scans the stencil
        atomicAdd(&S->nl_overflow, 1);
      } else {
        D.ncount[k] = cnt | (interior ? kListInterior : 0);
      }
    }
    __syncthreads();  // every thread is done with the band
  }
  return all;
}

__global__ void __launch_bounds__(kThreads, 4) k_rb_band(Dev D) {
  if (!rebuild_requested(D)) return;
  extern __shared__ __align__(128) float4 sh_band[];
  __shared__ Band band;
  __shared__ __align__(8) uint64_t full;
  const bool forced = *((volatile int*)&D.bg->forced) != 0;
  if (threadIdx.x == 0) mbar_init(&full, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  uint32_t parity = 0;
  if (!rb_band(D, sh_band, band, full, parity, forced)) {
    for (int s = 0; s < D.nsys; ++s) D.st[s].err = 6;  // MDB_ERR_CUDA: a copy never arrived
  }
  rebuild_finish(D, forced);
}

// ------------------------------------------------------------- force phase --

// A group of list entries (NC: see ld_idx).
template <bool NC>
__device__ __forceinline__ uint2 ld_group(const uint2* p) {
  if (NC) return __ldg(p);
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// Pair sums over a slot's list in the staged band.
template <bool PY, bool ENERGY, bool VIRIAL, bool MIC, bool FLOOR, bool NC>
__device__ __forceinline__ void band_list(const float4* __restrict__ band,
                                          const uint2* __restrict__ list, int64_t ntot, int groups,
                                          const PairCtx& c, float2& fs, float2& fc, float& ws,
                                          float& wc, double& u, double& an) {
  uint2 e = groups > 0 ? ld_group<NC>(list) : make_uint2(0u, 0u);
  for (int g = 0; g < groups; ++g) {
    const float4 q0 = band[e.x & 0xffffu], q1 = band[e.x >> 16];
    const float4 q2 = band[e.y & 0xffffu], q3 = band[e.y >> 16];
    list += ntot;
    if (g + 1 < groups) e = ld_group<NC>(list);  // the next group's entries
    pair_one<PY, ENERGY, VIRIAL, MIC, FLOOR>(q0, c, fs, fc, ws, wc, u, an);
    pair_one<PY, ENERGY, VIRIAL, MIC, FLOOR>(q1, c, fs, fc, ws, wc, u, an);
    pair_one<PY, ENERGY, VIRIAL, MIC, FLOOR>(q2, c, fs, fc, ws, wc, u, an);
    pair_one<PY, ENERGY, VIRIAL, MIC, FLOOR>(q3, c, fs, fc, ws, wc, u, an);
  }
}

// The same with FP64 pair terms.
template <bool PY, bool ENERGY, bool VIRIAL, bool MIC, bool NC>
__device__ __forceinline__ void band_list_hp(const float4* band, const uint2* __restrict__ list,
                                             int64_t ntot, int groups, const PairCtxD& c,
                                             double& fx, double& fy, double& w, double& u,
                                             double& an) {
  for (int g = 0; g < groups; ++g, list += ntot) {
    const uint2 e = ld_group<NC>(list);
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      const uint32_t at = ((k < 2 ? e.x : e.y) >> (16 * (k & 1))) & 0xffffu;
      pair_one_hp<PY, ENERGY, VIRIAL, MIC>(band[at], c, fx, fy, w, u, an);
    }
  }
}

// Shared state of a block of k_force_band beside its two bands.
struct BandShared {
  Band bands[2];
  uint64_t full[2], empty[2];
  int lost;  // a wait ran out of tries
};

// Run r of the stencil of cell (cx, cy), in visiting order: two runs a row, the
// second across the periodic x edge. Global slots [a, e); false: no such run.
template <bool PY, bool NC>
__device__ __forceinline__ bool stencil_run(const int32_t* cst, int ncx, int ncy, int cx, int cy,
                                            int r, int* a, int* e) {
  int y = cy - 1 + (r >> 1);
  if (PY) {
    if (y < 0) y += ncy;
    if (y >= ncy) y -= ncy;
  } else if (y < 0 || y >= ncy) {
    return false;
  }
  const int32_t* row = cst + (int64_t)y * ncx;
  const bool mid = cx > 0 && cx < ncx - 1;
  if ((r & 1) != 0) {
    if (mid) return false;
    *a = ld_idx<NC>(row + (cx == 0 ? ncx - 1 : 0));
    *e = ld_idx<NC>(row + (cx == 0 ? ncx : 1));
    return true;
  }
  *a = ld_idx<NC>(row + (mid ? cx - 1 : (cx == 0 ? 0 : ncx - 2)));
  *e = ld_idx<NC>(row + (mid ? cx + 2 : (cx == 0 ? 2 : ncx)));
  return true;
}

// The chunks of one block: pair sums and what follows them, into fin. HP: FP64
// pair terms (a FIRE system past its switch point, and its observations). pass
// counts the passes run on sh's barriers so far: it gives the buffer and the
// barriers' parities.
template <int FM, bool PY, bool HP, bool NC>
__device__ __forceinline__ void band_items(const Dev& D, const SysParams& P, const SysState& S,
                                           BandShared& sh, float4* sh_band, int q_first, int items,
                                           uint32_t& pass, ForceFinish<FM, PY>& fin) {
  constexpr bool kEnergy = (FM == FM_OBS);
  constexpr bool kVirial = (FM == FM_OBS || FM == FM_NPH);
  constexpr bool kFloor = (FM == FM_FIRE || FM == FM_OBS || FM == FM_INIT);
  const int nb = P.nb;
  const int64_t end = P.p0 + P.n;
  const int64_t half = half_of(D, &S);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Chunk of a pass: pass it takes chunk it * nb + rot, rot advancing by half
  // the blocks per pass (a block's chunks spread over the system, each pass
  // still covering one contiguous stretch).
  int rot = q_first;
  auto next_rot = [&](int r) {
    r += nb / 2;
    return r >= nb ? r - nb : r;
  };
  // Starts the copy of a chunk's band into buffer buf (warp 0).
  auto stage = [&](int q, int buf) {
    Band* bd = sh.bands + buf;
    const Band* g = D.bands + P.ch0 + q;
    int st = 0, ln = 0, of = 0;
    if (lane < kBandRanges) {
      st = g->start[lane];
      ln = g->len[lane];
      of = g->off[lane];
      bd->start[lane] = st;
      bd->len[lane] = ln;
      bd->off[lane] = of;
    }
    const int total = g->total;
    if (lane == 0) bd->total = total;
    __syncwarp();
    // (the arrival also releases the ranges to the warps that wait for the copy)
    if (lane == 0) mbar_expect(sh.full + buf, (uint32_t)total * 16u);
    __syncwarp();
    if (lane < kBandRanges && ln > 0)
      copy_bulk(sh_band + buf * kBandCap + of, D.pff + st, ln, sh.full + buf);
  };
  if (warp == 0 && items > 0) stage(q_first, (int)(pass & 1u));
  const double Lx = S.Lx, Ly = S.Ly;
  const double h = 0.5 * P.dt;
  const double xi2 = (FM == FM_NH) ? S.xi : 0.0;
  const double fdt = (FM == FM_FIRE) ? S.f_dt : 0.0;
#pragma unroll 1
  for (int it = 0; it < items; ++it, ++pass) {
    const int buf = (int)(pass & 1u);
    const int64_t cs = P.p0 + (int64_t)(it * nb + rot) * kThreads;
    if (cs >= end) break;  // (every thread of the block agrees)
    const int64_t i = cs + threadIdx.x;
    const bool act = i < end;
    const int nc = act ? ld_idx<NC>(D.ncount + i) : -1;
    rot = next_rot(rot);
    {
      const int q = (it + 1) * nb + rot;
      const int64_t ncs = P.p0 + (int64_t)q * kThreads;
      if (it + 1 < items && ncs < end) {
        if (warp == 0) {
          // the other buffer: free once every warp has left the pass before
          if (pass > 0 && !mbar_wait(sh.empty + (buf ^ 1), ((pass - 1) >> 1) & 1u)) sh.lost = 1;
          stage(q, buf ^ 1);
        }
        // L1 prefetch of the next chunk's list groups (32 slots of a group are
        // two lines), counts and velocities
        const int64_t wslot = ncs + (threadIdx.x & ~31);
        if (wslot < end) {
          if (lane * 2 < D.pf_rows && (lane >> 1) * 4 < D.max_nbr)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(D.lists + (int64_t)(lane >> 1) * D.ntot +
                                                           wslot + (lane & 1) * 16));
          if (ncs + threadIdx.x < end) {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(D.ncount + ncs + threadIdx.x));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(D.vel + half + ncs + threadIdx.x));
          }
        }
      }
    }
    if (!mbar_wait(sh.full + buf, (pass >> 1) & 1u)) sh.lost = 1;
    const float4* band = sh_band + buf * kBandCap;
    double fx = 0.0, fy = 0.0, w = 0.0, u = 0.0, an = 0.0;
    int tci = 0;
    if (act) {
      const bool staged = sh.bands[buf].total > 0;
      const float4 qi = staged ? band[band_place(sh.bands[buf], (int)i)] : ld_pos<NC>(D.pff + i);
      tci = (int)ff_class(qi);
      PairCtx c;
      PairCtxD cd;
      float2 fs = make_float2(0.f, 0.f), fc = make_float2(0.f, 0.f);
      float ws = 0.f, wc = 0.f;
      if (HP) {
        cd = pair_ctx_hp(P, qi, Lx, Ly);
      } else {
        c.ih = make_float2(qi.x, qi.y);
        c.il = make_float2(qi.z, qi.w);
        set_pair_class<kFloor>(c, P, tci);
      }
      const int groups = ((nc & (kListInterior - 1)) + 3) >> 2;
      if (nc >= 0 && (nc & kListInterior) != 0) {
        if (HP)
          band_list_hp<PY, kEnergy, kVirial, false, NC>(band, D.lists + i, D.ntot, groups, cd, fx, fy,
                                                    w, u, an);
        else
          band_list<PY, kEnergy, kVirial, false, kFloor, NC>(band, D.lists + i, D.ntot, groups, c, fs,
                                                         fc, ws, wc, u, an);
      } else {
        if (!HP) set_pair_box<PY>(c, qi, Lx, Ly);
        if (nc >= 0) {
          if (HP)
            band_list_hp<PY, kEnergy, kVirial, true, NC>(band, D.lists + i, D.ntot, groups, cd, fx, fy,
                                                     w, u, an);
          else
            band_list<PY, kEnergy, kVirial, true, kFloor, NC>(band, D.lists + i, D.ntot, groups, c, fs,
                                                          fc, ws, wc, u, an);
        } else {
          // no list: the stencil's runs from the band (or, without one, from
          // global memory), or the whole system
          // (A slot whose position is not finite has no pairs: every test fails. The
          // walled y axis is not wrapped, so it can be infinite.)
          const bool some = isfinite(qi.x) && isfinite(qi.y);
          const int cell = S.allpairs ? 0 : ld_idx<NC>(D.cell_of + i);
          const int cx = cell % S.ncx, cy = cell / S.ncx;
          // the minimum image for the warps that hold a slot within two cells of
          // a periodic edge (its shift is zero for the others: see k_rb_nlist)
          const bool image =
              __any_sync(__activemask(), cx < 2 || cx > S.ncx - 3 ||
                                             (S.periodic_y && (cy < 2 || cy > S.ncy - 3)));
#pragma unroll 1
          for (int r = some ? 0 : 6; r < 6; ++r) {
            int a, e;
            if (S.allpairs) {
              if (r > 0) break;
              a = (int)P.p0;
              e = (int)end;
            } else if (!stencil_run<PY, NC>(D.cstart + P.c0, S.ncx, S.ncy, cx, cy, r, &a, &e)) {
              continue;
            }
            if constexpr (HP) {
              const float4* src = staged ? band + band_place(sh.bands[buf], a) : D.pff + a;
              for (int m = 0; m < e - a;) {
                const int end = NC ? e - a : min(e - a, m + kScanPiece);
#pragma unroll 1
                for (; m < end; ++m)
                  pair_one_hp<PY, kEnergy, kVirial, true>(src[m], cd, fx, fy, w, u, an);
                if (!NC && end < e - a) mark_progress(D);
              }
            } else if (staged) {
              const float4* src = band + band_place(sh.bands[buf], a);
              if (image)
                pair_run<kEnergy, kVirial, true, kFloor>(src, e - a, c, fs, fc, ws, wc, u, an);
              else
                pair_run<kEnergy, kVirial, false, kFloor>(src, e - a, c, fs, fc, ws, wc, u, an);
            } else {
              for (int m = a; m < e;) {
                const int end = NC ? e : min(e, m + kScanPiece);
#pragma unroll 1
                for (; m < end; ++m)
                  pair_one<PY, kEnergy, kVirial, true, kFloor>(ld_pos<NC>(D.pff + m), c, fs, fc,
                                                               ws, wc, u, an);
                if (!NC && end < e) mark_progress(D);
              }
            }
          }
        }
      }
      if (HP) {
        w = 0.5 * w;
      } else {
        fx = (double)fs.x - (double)fc.x;
        fy = (double)fs.y - (double)fc.y;
        w = 0.5 * ((double)ws - (double)wc);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(sh.empty + buf);  // this warp has left the band
    if (act) fin(D, P, Ly, h, xi2, fdt, half + i, fx, fy, w, u, an, tci);
  }
}

// The FP64 form out of line: its registers do not count against the FP32 loop.
template <int FM, bool PY, bool NC>
__device__ __noinline__ ForceFinish<FM, PY> band_items_hp(Dev D, const SysParams* P,
                                                          const SysState* S, BandShared* sh,
                                                          float4* sh_band, int q_first, int items,
                                                          uint32_t* pass) {
  ForceFinish<FM, PY> fin;
  fin.init();
  uint32_t at = *pass;
  band_items<FM, PY, true, NC>(D, *P, *S, *sh, sh_band, q_first, items, at, fin);
  *pass = at;
  return fin;
}

// The force phase of k_force over staged bands: the same blocks, chunks,
// reductions and scalar tail.
template <int FM, bool PY>
__global__ void __launch_bounds__(kThreads, 4) k_force_band(Dev D) {
  extern __shared__ __align__(128) float4 sh_band[];  // [2][kBandCap]
  __shared__ BandShared sh;
  const int b = blockIdx.x;
  const int s = D.nsys == 1 ? 0 : D.sys_of_block[b];
  const SysParams& P = D.sp[s];
  SysState* S = D.st + s;
  constexpr bool kHpCapable = (FM == FM_FIRE || FM == FM_OBS || FM == FM_INIT);
  constexpr int kNS = ForceRed<FM>::NS, kNM = ForceRed<FM>::NM;
  if (threadIdx.x == 0) {
    mbar_init(sh.full + 0, 1);
    mbar_init(sh.full + 1, 1);
    mbar_init(sh.empty + 0, kThreads / 32);
    mbar_init(sh.empty + 1, kThreads / 32);
    sh.lost = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  // a finished batch system is still observed (FM_OBS) and re-evaluated (FM_INIT)
  const bool skip = (FM != FM_OBS && FM != FM_INIT && S->done != 0) || (S->err != 0) ||
                    (FM == FM_FIRE && (S->f_conv != 0 || S->f_step >= P.f_max_steps));
  const double Lx = S->Lx, Ly = S->Ly;
  const int items = skip ? 0 : P.items;
  __syncthreads();
  ForceFinish<FM, PY> fin;
  uint32_t pass = 0;
  if (kHpCapable && S->f_fp64 != 0) {
    fin = band_items_hp<FM, PY, true>(D, &P, S, &sh, sh_band, b - P.b0, items, &pass);
  } else {
    fin.init();
    band_items<FM, PY, false, true>(D, P, *S, sh, sh_band, b - P.b0, items, pass, fin);
  }
  if (fin.bad) atomicOr(&S->nonfinite, 1);
  ForceTail tin;
  if (threadIdx.x == 0) tin = force_tail_inputs<FM>(P, S);
  double tot[kNP];
  double tmx[3];
  if (!reduce_system<kNS, kNM>(D, P, S, fin.red, fin.mx, tot, tmx)) {
    if (threadIdx.x == 0 && sh.lost) S->err = 6;  // MDB_ERR_CUDA: a band never arrived
    return;
  }
  if (threadIdx.x != 0) return;
  int conv = 0;
  if (!skip) conv = force_tail<FM, PY>(S, tin, Lx, Ly, 0.5 * P.dt, tot, tmx);
  // (a system that was converged at launch is skipped)
  if (FM == FM_FIRE) S->f_drift = (!skip && !conv) ? 1 : 0;
  if (sh.lost) S->err = 6;
  S->counter = 0u;
}

}  // namespace mdb
