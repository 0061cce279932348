// Software-pipelined step kernel for FP64 storage with F64X arithmetic (any
// box; link words for walls and solids; no per-cell fields).
//
// The F64X collision is about 1.1k instructions per D3Q19 cell and 1.9k per D3Q27
// cell, so the plain one-cell-per-thread kernel spends its time either issuing or
// waiting on its 19/27 loads.  Here every warp is persistent and works on tiles of
// 32 consecutive cells: while it collides tile k it already has the loads of tile
// k+1 in flight as cp.async copies (8 bytes per thread and direction) into its own
// two-stage shared-memory buffer, so the loads hold no registers and their latency
// overlaps the collision.  Each thread reads back only what it copied itself, so
// cp.async.wait_group is the only synchronisation needed.
//
// AA (in place) stays race-free under the prefetch: the locations a cell's
// thread reads are exactly the ones it writes (even step: its own slots; odd
// step: slot s at x - c_s and slot opp(s) at x + c_s form the same set, a
// bounced-back direction reading and writing the own cell), so a
// prefetch of another tile never sees a write of this one.
#pragma once

#include <atomic>

#include "lbm_launch.cuh"
#include "lbm_step.cuh"

namespace lbm {

// Warps per block and blocks per SM.  What limits them is the L1 that the
// shared memory leaves: every 8-byte cp.async passes through it, and its lines
// bound the copies in flight.  At 256x128x128, with the blocks' shared memory
// in the smallest carve-out that holds it (164 KB, 92 KB of L1), in the next
// (196 KB) or in the largest (228 KB, 28 KB of L1):
//   D3Q19 AA even / odd step   197 / 211 us,  -,               246 / 293 us
//   D3Q27 AA even / odd step   283 / 342 us,  295 / 356 us,    362 / 438 us
//   D3Q27 AB push / pull step  302 / 309 us,  316 / 305 us,    375 / 395 us
// So D3Q19 runs 16 warps in two blocks (128 registers) and D3Q27 12 warps (168
// registers; 16 warps need 228 KB), and the launch asks for the carve-out.  The
// 12 warps come in two forms:
//   REST   three blocks, with the rest population, which every kind reads from the
//          own cell, in a register (as three blocks with all 27 staged they take
//          165 KB): odd 324 us, pull 295 us, even 291 us, push 303 us (links 317);
//   else   one block, all directions staged: odd 342, pull 309, even 281, push
//          302 us (links 308).
// AA odd and AB run the first; AA even the second, but the first for grids of fewer
// than 16 tiles per warp, where a step overlaps the next by the block (48^3: 11.5 us
// a step against 13.6).  D3Q19 with a rest register: 201 / 219 us, so not there.
template <int Q, bool REST>
constexpr int async_warps() { return Q == 19 ? 8 : (REST ? 4 : 12); }
template <int Q, bool REST>
constexpr int async_min_blocks() { return Q == 19 ? 2 : (REST ? 3 : 1); }
// Directions staged in shared memory per tile.
template <int Q, bool REST>
constexpr int async_rows() { return REST ? Q - 1 : Q; }
// Whether a block's warps take adjacent tiles at the same time, one barrier per
// tile.  A D3Q27 AB step moves 54 streams; once its warps have drifted apart, each
// 256-byte piece of a stream comes at a time of its own, and DRAM falls from 6.1
// to 4.2 TB/s: the 256x128x128 pull channel took 291 or 423 us a step, from one run
// to the next and within a run, and push 303 or 413 us.  Kept together in fours: 297
// us whatever came before (box 292 -> 299).  AA reads and writes one set of 27
// streams and does not fall; the barrier costs it 10 %.
template <int Q, int KIND>
constexpr bool async_together() { return Q == 27 && (KIND == K_AB_PUSH || KIND == K_AB_PULL); }
constexpr int kAsyncStages = 2;
constexpr int kBlockReserve = 1024;          // shared memory the system takes per block
constexpr int kMaxSharedPerSM = 228 * 1024;

// The smallest shared-memory carve-out (percent) that holds `blocks` blocks.
constexpr int carveout_percent(int blocks, size_t smem)
{
   return (int)((blocks * (smem + kBlockReserve) * 100 + kMaxSharedPerSM - 1) / kMaxSharedPerSM);
}

template <int Q, bool REST>
constexpr size_t async_smem_bytes()
{
   return (size_t)async_warps<Q, REST>() * kAsyncStages * async_rows<Q, REST>() * 32 * sizeof(unsigned long long);
}

// Tiles of 32 consecutive cells, whatever rows they lie in: tile t covers the cells
// c in [32 t, 32 t + 32) below ncell.  Every lane has a cell then, and every tile
// starts on 256 bytes; with tiles that ended at their rows, rows of 161 cells left
// 16 % of the lanes idle (D3Q27 AB pull channel 161x75x93, two steps: 196 us).
// Divisions by a run-time d use q = umulhi64(n, m) with m = ceil(2^64 / d) (exact for
// n, d < 2^32); d = 1 is m = 0.
struct AsyncGeom {
   uint32_t ntiles, ncell;
   uint64_t m_nx, m_ny;
};

__device__ __forceinline__ uint32_t div_magic(uint32_t n, uint32_t d, uint64_t m)
{
   return m ? (uint32_t)__umul64hi((uint64_t)n, m) : n;
}

// Returns false for a lane past the last cell.
__device__ __forceinline__ bool tile_cell(const KParams& p, const AsyncGeom& ag, uint32_t t, int lane,
                                          CellIndex& ci)
{
   const uint32_t c = t * 32u + (uint32_t)lane;
   const uint32_t row = div_magic(c, (uint32_t)p.nx, ag.m_nx);
   const int x = (int)(c - row * (uint32_t)p.nx);
   const uint32_t z = div_magic(row, (uint32_t)p.ny, ag.m_ny);
   const int y = (int)(row - z * (uint32_t)p.ny);
   ci.c = (int64_t)c;
   ci.dxm = (x == 0) ? p.nx - 1 : -1;
   ci.dxp = (x == p.nx - 1) ? -(p.nx - 1) : 1;
   ci.dym = (y == 0) ? (p.ny - 1) * p.nx : -p.nx;
   ci.dyp = (y == p.ny - 1) ? -(p.ny - 1) * p.nx : p.nx;
   const int nxy = p.nx * p.ny;
   ci.dzm = (z == 0) ? (p.nz - 1) * nxy : -nxy;
   ci.dzp = ((int)z == p.nz - 1) ? -(p.nz - 1) * nxy : nxy;
   return c < ag.ncell;
}

__device__ __forceinline__ void cp_async8(uint32_t smem, const void* g)
{
   asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// Base pointer of every direction plane of the source and target buffers,
// passed by value so each sits in the kernel's parameter bank: an access is
// then one wide multiply-add of a 32-bit cell index (fewer than 2^31 cells;
// the periodic wrap keeps neighbour indices inside the box) onto a
// parameter-bank pointer.
struct PlanePtrs {
   const unsigned long long* src[27];
   unsigned long long* dst[27];
};

// Lane state of a tile: its cell, its link word (0 without walls) and
// whether it updates anything (a cell, not solid).
struct TileLane {
   CellIndex ci;
   uint32_t lk;
   bool active;
};

// Link word of this lane's cell in tile t (the solid bit past the last cell).
__device__ __forceinline__ uint32_t tile_link(const KParams& p, const AsyncGeom& ag, uint32_t t, int lane)
{
   const uint32_t c = t * 32u + (uint32_t)lane;
   return c < ag.ncell ? __ldg(p.links + c) : kSolidBit;
}

// lk: the tile's link words, loaded one tile ahead so the load's latency
// hides behind a collision.
// RAGGED: the cell count is not a multiple of 32, so the last tile has lanes
// without a cell (with LINKS their link word says so, and RAGGED is not looked at).
template <bool LINKS, bool RAGGED>
__device__ __forceinline__ void tile_lane(const KParams& p, const AsyncGeom& ag, uint32_t t, int lane, uint32_t lk,
                                          TileLane& tl)
{
   const bool inside = tile_cell(p, ag, t, lane, tl.ci);
   tl.lk = LINKS ? lk : 0u;
   tl.active = LINKS ? !(lk & kSolidBit) : (RAGGED ? inside : true);
}

// Whether any cell of the tile has a blocked neighbour (warp-uniform; every
// lane calls it).  A tile without one runs its neighbour reads and writes
// without the bounce-back selects, about six instructions per direction: on the
// 256x128x128 channel the D3Q27 push step 336 -> 322 us, pull 332 -> 324 us, the
// D3Q19 pull step 221 -> 216 us (with four-warp blocks).
__device__ __forceinline__ bool tile_linked(uint32_t lk)
{
   return __any_sync(0xFFFFFFFFu, (lk & ~kSolidBit) != 0u);
}

template <int Q, int KIND, bool LINKS, bool REST>
__device__ __forceinline__ void async_issue_cell(const PlanePtrs& pp, const TileLane& tl, int lane, uint32_t sbuf)
{
   const uint32_t c = (uint32_t)tl.ci.c;
#pragma unroll
   for (int s = 0; s < async_rows<Q, REST>(); s++) {
      const Access a = read_access<Q, KIND, LINKS>(tl.ci, tl.lk, s);
      cp_async8(sbuf + (uint32_t)(s * 32 + lane) * 8u, pp.src[a.slot] + (c + (uint32_t)a.off));
   }
}

// The copies of a tile's populations (REST: the rest one into a register).
template <int Q, int KIND, bool LINKS, bool RAGGED, bool REST>
__device__ __forceinline__ void async_issue(const PlanePtrs& pp, const TileLane& tl, int lane, uint32_t sbuf, uint64_t& rest)
{
   constexpr bool kGathers = KIND == K_AA_ODD || KIND == K_AB_PULL;
   const bool linked = LINKS && kGathers && tile_linked(tl.lk);
   if ((LINKS || RAGGED) && !tl.active) return;
   if constexpr (REST) rest = pp.src[lat_rest(Q)][(uint32_t)tl.ci.c];
   if (LINKS && kGathers && linked) async_issue_cell<Q, KIND, LINKS, REST>(pp, tl, lane, sbuf);
   else async_issue_cell<Q, KIND, false, REST>(pp, tl, lane, sbuf);
}

// Stores each output straight to its target slot.  AA stays race-free with
// stores that may be overwritten later by the same thread (the fast path's
// outputs when a range check fails): the locations are this cell's own.
template <int Q, int KIND, bool LINKS>
struct StoreEmit {
   const PlanePtrs& pp;
   const CellIndex& ci;
   uint32_t lk;
   __device__ __forceinline__ void operator()(int s, uint64_t v) const
   {
      const Access a = write_access<Q, KIND, LINKS>(ci, lk, s);
      pp.dst[a.slot][(uint32_t)ci.c + (uint32_t)a.off] = v;
   }
};

template <int Q, int KIND, bool LINKS, bool RAGGED, int FORCE, bool REST>
__global__ void __launch_bounds__(async_warps<Q, REST>() * 32, async_min_blocks<Q, REST>()) step_async_kernel(const KParams p, const AsyncGeom ag,
                                                                      const PlanePtrs pp)
{
   extern __shared__ __align__(16) unsigned long long async_smem[];
   const int lane = threadIdx.x & 31;
   const int warp = threadIdx.x >> 5;
   const uint32_t kWarps = blockDim.x >> 5;
   const uint32_t nw = gridDim.x * kWarps;
   const uint32_t ntiles = ag.ntiles;
   wait_prior_grid();
   constexpr int kRows = async_rows<Q, REST>();
   unsigned long long* mine = async_smem + (size_t)warp * kAsyncStages * kRows * 32;
   const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(mine);
   constexpr uint32_t kStageBytes = kRows * 32 * 8;
   if constexpr (async_together<Q, KIND>()) {
      // The block's warps take kWarps consecutive tiles together: group g is the
      // tiles g kWarps + warp.  Three groups in a fixed order, then one counter,
      // which the block's first thread asks one group ahead.  Everything about
      // groups is block-uniform, a warp past the last tile only skips the work.
      __shared__ uint32_t next_group[2];
      const uint32_t nb = gridDim.x, ngroups = (ntiles + kWarps - 1) / kWarps;
      const bool fed = feed_on(ntiles, nw);
      uint32_t pend = 0;
      if (fed && threadIdx.x == 0) pend = atomicAdd(p.sched, 1u);
      uint32_t g = blockIdx.x, it = 0;
      if (g < ngroups) {
         uint32_t g1 = g + nb < ngroups ? g + nb : ngroups, g2 = g + 2u * nb < ngroups ? g + 2u * nb : ngroups;
         auto tile = [&](uint32_t gg) { const uint32_t tt = gg * kWarps + warp; return gg < ngroups && tt < ntiles ? tt : ntiles; };
         uint32_t t = tile(g), t1 = tile(g1), t2 = tile(g2);
         TileLane cur;
         cur.active = false;
         cur.lk = kSolidBit;
         uint64_t rest = 0, rest_next = 0;
         if (t < ntiles) {
            tile_lane<LINKS, RAGGED>(p, ag, t, lane, LINKS ? tile_link(p, ag, t, lane) : 0u, cur);
            async_issue<Q, KIND, LINKS, RAGGED, REST>(pp, cur, lane, sbase, rest);
         }
         uint32_t lk_ahead = (LINKS && t1 < ntiles) ? tile_link(p, ag, t1, lane) : 0u;
         cp_async_commit();
         int stage = 0;
         for (;;) {
            TileLane nxt = cur;
            if (t1 < ntiles) {
               tile_lane<LINKS, RAGGED>(p, ag, t1, lane, lk_ahead, nxt);
               if (LINKS && t2 < ntiles) lk_ahead = tile_link(p, ag, t2, lane);
               async_issue<Q, KIND, LINKS, RAGGED, REST>(pp, nxt, lane, sbase + (stage ^ 1) * kStageBytes, rest_next);
            }
            cp_async_commit();
            cp_async_wait_prev();
            constexpr bool kScatters = KIND == K_AA_ODD || KIND == K_AB_PUSH;
            const unsigned long long* in = mine + stage * kRows * 32 + lane;
            if (t < ntiles) {
               const bool linked = LINKS && kScatters && tile_linked(cur.lk);
               if (!(LINKS || RAGGED) || cur.active) {
                  if (LINKS && kScatters && linked) {
                     StoreEmit<Q, KIND, LINKS> emit{pp, cur.ci, cur.lk};
                     collide_f64x_shared_emit<Q, FORCE, REST>(in, rest, p, emit);
                  } else {
                     StoreEmit<Q, KIND, false> emit{pp, cur.ci, 0u};
                     collide_f64x_shared_emit<Q, FORCE, REST>(in, rest, p, emit);
                  }
               }
            }
            if (g1 >= ngroups) break;
            g = g1;
            g1 = g2;
            if (g2 < ngroups) {
               if (fed) {
                  if (threadIdx.x == 0) {
                     const uint64_t n = 3ull * nb + pend;
                     next_group[it & 1] = n < ngroups ? (uint32_t)n : ngroups;
                     if (n < ngroups) pend = atomicAdd(p.sched, 1u);
                  }
                  __syncthreads();
                  g2 = next_group[it & 1];
               } else {
                  g2 = g2 + nb < ngroups ? g2 + nb : ngroups;
                  __syncthreads();
               }
            }
            it++;
            t = t1;
            t1 = t2;
            t2 = tile(g2);
            cur = nxt;
            rest = rest_next;
            stage ^= 1;
         }
      }
      if (fed) feed_done(p.sched);
   } else {
      // tiles: three per warp in a fixed order, then the launch's tile feed (8
      // counters for the D3Q19 tiles, which it hands out fastest); t is collided
      // while t1's populations are in flight and t2's link words are loaded
      const bool fed = feed_on(ntiles, nw);
      TileFeed feed{0u, 0u, 1u, false};
      if (fed) feed = feed_start(p.sched, 3u * nw, ntiles, blockIdx.x * kWarps + warp, nw, Q == 19 ? kFeedGroups : 1u, lane);
      uint32_t t = blockIdx.x * kWarps + warp;
      if (t < ntiles) {
         uint32_t t1 = t + nw < ntiles ? t + nw : ntiles;
         uint32_t t2 = t + 2u * nw < ntiles ? t + 2u * nw : ntiles;
         TileLane cur;
         tile_lane<LINKS, RAGGED>(p, ag, t, lane, LINKS ? tile_link(p, ag, t, lane) : 0u, cur);
         uint32_t lk_ahead = (LINKS && t1 < ntiles) ? tile_link(p, ag, t1, lane) : 0u;
         uint64_t rest = 0, rest_next = 0;
         async_issue<Q, KIND, LINKS, RAGGED, REST>(pp, cur, lane, sbase, rest);
         cp_async_commit();
         int stage = 0;
         for (;;) {
            TileLane nxt = cur;
            if (t1 < ntiles) {
               tile_lane<LINKS, RAGGED>(p, ag, t1, lane, lk_ahead, nxt);
               if (LINKS && t2 < ntiles) lk_ahead = tile_link(p, ag, t2, lane);
               async_issue<Q, KIND, LINKS, RAGGED, REST>(pp, nxt, lane, sbase + (stage ^ 1) * kStageBytes, rest_next);
            }
            cp_async_commit();
            cp_async_wait_prev();
            // each output is stored as the collision makes it, and the update
            // re-reads its inputs from shared memory: neither the Q input nor the
            // Q output patterns stay in registers
            constexpr bool kScatters = KIND == K_AA_ODD || KIND == K_AB_PUSH;
            const unsigned long long* in = mine + stage * kRows * 32 + lane;
            const bool linked = LINKS && kScatters && tile_linked(cur.lk);
            if (!(LINKS || RAGGED) || cur.active) {
               if (LINKS && kScatters && linked) {
                  StoreEmit<Q, KIND, LINKS> emit{pp, cur.ci, cur.lk};
                  collide_f64x_shared_emit<Q, FORCE, REST>(in, rest, p, emit);
               } else {
                  StoreEmit<Q, KIND, false> emit{pp, cur.ci, 0u};
                  collide_f64x_shared_emit<Q, FORCE, REST>(in, rest, p, emit);
               }
            }
            if (t1 >= ntiles) break;
            t = t1;
            t1 = t2;
            t2 = feed_after(feed, fed, t2, p.sched, 3u * nw, ntiles, nw, lane);
            cur = nxt;
            rest = rest_next;
            stage ^= 1;
         }
      }
      if (fed) feed_done(p.sched);
   }
}

inline AsyncGeom async_geom(int nx, int ny, int nz)
{
   AsyncGeom g;
   g.ncell = (uint32_t)nx * (uint32_t)ny * (uint32_t)nz;   // below 2^31
   g.ntiles = g.ncell / 32u + (g.ncell % 32u ? 1u : 0u);
   g.m_nx = nx == 1 ? 0 : (~0ull / (uint64_t)nx) + 1;
   g.m_ny = ny == 1 ? 0 : (~0ull / (uint64_t)ny) + 1;
   return g;
}

// Blocks and warps per block of a launch on nsm SMs, per_sm blocks of max_warps on
// each at most.  A grid with fewer tiles than that many warps runs smaller blocks
// on as many SMs, not full blocks on a few (D3Q27 AB pull, 24x21x38: 798 tiles, 67
// blocks of 12 warps left 85 of the 152 SMs idle: 5.5 us, 4.2 us spread).
struct AsyncLaunch {
   unsigned blocks, warps;
};
inline AsyncLaunch async_launch(uint32_t ntiles, uint32_t nsm, uint32_t per_sm, uint32_t max_warps)
{
   const uint32_t each = (ntiles + nsm - 1) / nsm;
   const uint32_t w = each < max_warps ? (each ? each : 1u) : max_warps;
   const uint32_t need = (ntiles + w - 1) / w;
   const uint32_t resident = nsm * per_sm;
   return {need < resident ? need : resident, w};
}

// Persistent grid: as many blocks as fit on the device at once (queried once
// per device and kernel; the shared-memory opt-in is set at the same time).
template <int Q, int KIND, bool LINKS, bool RAGGED, int FORCE, bool REST>
cudaError_t launch_async_kernel(const KParams& p, const AsyncGeom& ag, const void* src, void* dst, cudaStream_t stream)
{
   // Persistent grid size per device ordinal, set once (the value is the same
   // whichever thread computes it first).
   static std::atomic<int> grid_of_device[64];
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) return e;
   if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
   auto kern = step_async_kernel<Q, KIND, LINKS, RAGGED, FORCE, REST>;
   constexpr int kWarps = async_warps<Q, REST>();
   constexpr size_t smem = async_smem_bytes<Q, REST>();
   int cached = grid_of_device[dev].load(std::memory_order_relaxed);
   if (cached == 0) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                               carveout_percent(async_min_blocks<Q, REST>(), smem));
      if (e != cudaSuccess) return e;
      int per_sm = 0, nsm = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWarps * 32, smem);
      if (e != cudaSuccess) return e;
      e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return e;
      if (per_sm < async_min_blocks<Q, REST>()) return cudaErrorInvalidConfiguration;
      cached = async_min_blocks<Q, REST>() * nsm;   // no more than the carve-out is meant for
      grid_of_device[dev].store(cached, std::memory_order_relaxed);
   }
   const AsyncLaunch L = async_launch(ag.ntiles, (uint32_t)cached / async_min_blocks<Q, REST>(), async_min_blocks<Q, REST>(),
                                      kWarps);
   PlanePtrs pp;
   for (int s = 0; s < 27; s++) {
      const int k = s < Q ? s : 0;
      pp.src[s] = static_cast<const unsigned long long*>(src) + (int64_t)k * p.plane;
      pp.dst[s] = static_cast<unsigned long long*>(dst) + (int64_t)k * p.plane;
   }
   return launch_overlapped(kern, dim3(L.blocks), dim3(L.warps * 32), smem / kWarps * L.warps, stream, p, ag, pp);
}

// Rule for REST (at async_warps).
template <int Q, int KIND, bool LINKS, bool RAGGED, int FORCE>
cudaError_t launch_async_form(const KParams& p, const AsyncGeom& ag, const void* src, void* dst, cudaStream_t stream)
{
   if constexpr (Q == 27) {
      if constexpr (KIND != K_AA_EVEN || FORCE == kForceOther) {
         return launch_async_kernel<Q, KIND, LINKS, RAGGED, FORCE, true>(p, ag, src, dst, stream);
      } else {
         int dev = 0, nsm = 0;
         cudaError_t e = cudaGetDevice(&dev);
         if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
         if (e != cudaSuccess) return e;
         if ((uint64_t)ag.ntiles < (uint64_t)kFeedMinTiles * 12u * (uint64_t)nsm)
            return launch_async_kernel<Q, KIND, LINKS, RAGGED, FORCE, true>(p, ag, src, dst, stream);
      }
   }
   if constexpr (Q == 19 || (KIND == K_AA_EVEN && FORCE != kForceOther))
      return launch_async_kernel<Q, KIND, LINKS, RAGGED, FORCE, false>(p, ag, src, dst, stream);
}

// links: the grid has link words.  Kernels exist for no force and the velocity
// shift with and without a ragged last tile; the other forcing forms run the
// ragged form for every cell count.
template <int Q, int KIND>
cudaError_t launch_async_kind(bool links, const KParams& p, const AsyncGeom& ag, const void* src, void* dst,
                              cudaStream_t stream)
{
   const bool ragged = ag.ncell % 32u != 0u;
   if (p.forced == 0) {
      if (links) return launch_async_form<Q, KIND, true, false, 0>(p, ag, src, dst, stream);
      return ragged ? launch_async_form<Q, KIND, false, true, 0>(p, ag, src, dst, stream)
                    : launch_async_form<Q, KIND, false, false, 0>(p, ag, src, dst, stream);
   }
   if (p.forced == 3) {
      if (links) return launch_async_form<Q, KIND, true, false, 3>(p, ag, src, dst, stream);
      return ragged ? launch_async_form<Q, KIND, false, true, 3>(p, ag, src, dst, stream)
                    : launch_async_form<Q, KIND, false, false, 3>(p, ag, src, dst, stream);
   }
   return links ? launch_async_form<Q, KIND, true, false, kForceOther>(p, ag, src, dst, stream)
                : launch_async_form<Q, KIND, false, true, kForceOther>(p, ag, src, dst, stream);
}

// launch_async_kind for a kind known at run time; instantiated in
// lbm_step_q*_aa.cu and lbm_step_q*_ab.cu, so the library builds in parallel.
template <int Q>
cudaError_t launch_async_aa(int kind, bool links, const KParams& p, const AsyncGeom& ag, const void* src, void* dst,
                            cudaStream_t stream);
template <int Q>
cudaError_t launch_async_ab(int kind, bool links, const KParams& p, const AsyncGeom& ag, const void* src, void* dst,
                            cudaStream_t stream);

}  // namespace lbm
