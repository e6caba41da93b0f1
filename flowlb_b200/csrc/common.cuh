// common.cuh -- kernel parameters and population access shared by all passes.
//
// Layout in HBM (structure of arrays, the reference layout, one population
// buffer):
//   f      9N  S   slot s of cell c at f[c + s*N] (slot[s] below points at
//                  f + s*N); updated in place by the esoteric-pull pattern:
//                  a cell loads and stores the same 9 addresses, so no second
//                  buffer is needed
//   rho     N  C   density of the incoming populations of the last step
//   u      2N  C   force-shifted velocity, u_x then u_y
//   flags  2xN u8  cell types; two buffers, the flag-stencil pass reads one
//                  and writes the other
//   nbmask  N  u8  bit k-1 set when neighbour k is a wall (half-way walls)
//   mass, excess, phi  N  M   free-surface cell mass, excess share, fill level
//   recon  8N  C   populations rebuilt by FS_1 toward gas (reference mode only)
// S/C/M: storage / arithmetic / mass types.
#pragma once

#include <utility>

#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "lattice.cuh"

namespace flb {

constexpr int kBlock = 256;

struct KParams {
  uint32_t nx, ny, N;
  void* f;
  void* slot[9];  // f + s*N, typed by the kernel
  void* rho;
  void* u;
  uint8_t* flags;      // current flags
  uint8_t* flags_out;  // flag-stencil pass output
  const uint8_t* nbmask;
  void* mass;
  void* excess;
  void* phi;
  void* recon;
  uint8_t* recon_mask;
  const void* rho_snap;
  const void* u_snap;
  float inv_tau, fx, fy;
  float cF[9];  // cx[i]*Fx + cy[i]*Fy, computed on the host in float as the reference does per cell
  float f16_scale, f16_inv;
  double inlet_ux, inlet_uy;
  int use_force, subgrid, collision, fs_cons;
  // 1 when flags_out holds the previous step's post-stream-collide flags and
  // the mass fields come from the previous full step (see k_fs234)
  int trust_prev;
  float u_max;  // velocity limiter, 0 = off
  // fused SRT arithmetic (collide_fused), float constants computed on the host:
  // 1-w, -3k, F/2, F (zero without forcing), and per direction pair q (odd
  // direction 2q+1) 3k c.F and 9k c.F, with k = 1 - w/2
  float fu_omc, fu_nk3, fu_hfx, fu_hfy, fu_fx, fu_fy;
  float fu_g[4], fu_h[4];
  float fu_sw[3];  // FP16S deviation form: f16_scale * w for directions 0, 1..4, 5..8
  int has_io;      // the case has inlet or outlet cells
  // time step of the FP16S stochastic rounding: the step with parity q reads
  // tstep[q] and writes tstep[q ^ 1] = t + 1 (graph replays see the current t)
  uint32_t* tstep;
  // single phase: chunk map of plain fluid cells, 4 cells per bit (k_plain_chunks); null otherwise
  const uint32_t* plain;
  // -F/2 for the packed arithmetic; last and 16 bytes long, so that the fields
  // before and what follows the struct in the batch's case records stay where
  // wide shared-memory loads reach them (8 bytes before fu_g: the persistent
  // batch kernel 212 ms against 200 for 600 steps of 256 cases)
  float fu_nhfx, fu_nhfy, fu_pad[2];
};

// Whether the n*4 cells from cell c (a multiple of 4n, n = 1 or 2) are all
// plain fluid cells with no wall neighbour.
template <int n>
__device__ __forceinline__ bool plain_cells(const uint32_t* plain, uint32_t c) {
  const uint32_t word = plain[c >> 7], bit = (c >> 2) & 31u;
  constexpr uint32_t m = (1u << n) - 1u;
  return ((word >> bit) & m) == m;
}

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// Free-surface steps work on super-tiles of kSTW x kSTH cells.  Only the
// super-tiles a pass can change are visited: the flag pass, as it finishes a
// super-tile, appends to the next step's lists the super-tiles that step must
// visit (NextLists), and the next step's passes loop over the lists in a
// persistent grid.  all = 1 visits every super-tile (first step after the
// state was set from outside).
// 64 x 8 cells: with 128 x 8 the about 320 super-tiles of a 2048x512 dam break
// were one round and a bit of blocks, and small grids ran on a few SMs
// (measured with the forms of k_fs.cu and k_sc.cu, us per step, 128 -> 64 wide:
// 101x101 17.8 -> 13.8, 2048x512 26.7 -> 23.4, 8192x2048 239 -> 232).
constexpr uint32_t kSTW = 64, kSTH = 8;
struct TileList {
  const uint32_t* list;
  const uint32_t* count;
  uint32_t ntiles, nsx;
  int all;
};

// Programmatic dependent launch.  The free-surface step kernels are launched
// with launch_pdl, so the next kernel on the stream (also inside a CUDA graph)
// may be scheduled while this one drains.  Each such kernel calls pdl_wait()
// before its first read of anything the previous kernel wrote (it returns once
// that kernel has completed and its writes are visible; it returns at once
// when the kernel was launched without the attribute), then pdl_trigger() to
// let its own successor be scheduled.  Its pointer parameters are not
// __restrict__: the qualifier says that nothing else writes the array while the
// kernel runs, and allows a load to be moved above the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Where the flag pass of the step at t appends the super-tiles of step t+1:
// FS_1 and stream-collide visit those holding fluid or interface cells
// (list_sc); the flag pass also visits a neighbour of such a super-tile when
// one of those cells lies within the stencil chain's reach of their shared
// edge or corner, and, once more, those that held such cells a step earlier
// (list_fs; bits marks the super-tiles already in it, so each is listed once).
// The lengths and the marks start at zero: FS_1 of the same step clears them
// (ListClear), after the previous step's passes have finished reading that
// parity's lists.
struct NextLists {
  uint32_t* list_sc;
  uint32_t* list_fs;
  uint32_t* counts;  // [2]: lengths of list_sc and list_fs
  uint32_t* bits;    // (ntiles + 31) / 32 words
  uint32_t nsx, nsy;
  uint32_t thin;     // the last super-tile column (1) or row (2) is narrower than the flag pass's reach
};
struct ListClear {
  uint32_t* counts;  // [2]
  uint32_t* bits;
  uint32_t nwords;
};

// FS_1's first block clears the lengths and marks the flag pass of the same
// step appends to (called after pdl_wait).
__device__ __forceinline__ void clear_next_lists(const ListClear& lc) {
  if (blockIdx.x != 0 || !lc.counts) return;
  if (threadIdx.x < 2) lc.counts[threadIdx.x] = 0u;
  for (uint32_t i = threadIdx.x; i < lc.nwords; i += blockDim.x) lc.bits[i] = 0u;
}

// A launch of several single-phase steps (k_mt.cu): T steps from t, on windows
// of W x H cells of which OW x OH are output; columns start pad cells left of
// the output.  The state is read through KParams and written to dst.
struct MtArgs {
  void* dst;
  uint32_t t;
  int T, W, H, OW, OH, pad;
  int bx, tiles;  // windows per row of windows, and in all
  int vec;      // rows move in groups of four cells (nx % 4 == 0)
  int wm;       // the last step writes density and velocity
  int threads;
  int pairs;    // FP32 fused: two cells per thread with packed arithmetic
};

// What the persistent free-surface step (k_fsp.cu) needs besides the step
// parameters: the lists and their lengths of both parities (read by the step
// of that parity, built by the step before), the activity words, and its
// grid barrier.
struct FspArgs {
  uint32_t* list[2][2];  // [parity][0: FS_1 and stream-collide, 1: flag pass]
  uint32_t* lcount;      // [parity][2] list lengths
  uint32_t* lbits;       // [parity][nwords] marks of the flag-pass lists
  uint32_t nwords;
  uint32_t* nz;
  uint32_t nsx, nsy;
  uint32_t thin;         // NextLists::thin
  uint32_t* bar;         // grid barrier arrivals, zeroed before each launch
  uint32_t* err;         // set when a barrier wait gave up
  uint32_t steps;        // even: the run starts at an even t with flag buffer 0 current
  uint32_t wait_limit;   // polls before a barrier wait gives up
  uint32_t skip_cta;     // failure injection: this CTA never arrives (0xffffffff: none)
  uint64_t* trace;       // null, or 3*steps+1 slots: CTA 0's exit time of each barrier (ns)
};

// A list holds at most ntiles entries; the length is clamped so that no state
// (a launch that gave up part-way, for instance) can make a pass read past it.
__device__ __forceinline__ uint32_t tile_count(const TileList& tl) {
  return tl.all ? tl.ntiles : min(__ldcg(tl.count), tl.ntiles);
}
__device__ __forceinline__ uint32_t tile_at(const TileList& tl, uint32_t i) { return tl.all ? i : tl.list[i]; }
// An entry of the FS_1 / stream-collide list: the super-tile, and kDeepTile when
// it is deep: it lies inside the grid, and its cells and their neighbours are
// all plain fluid (no wall next to them), so those passes read no flag or wall
// mask there and wrap no neighbour.  The flag pass sets it from the window it
// reads anyway.  Only on grids of more than kSmallTiles super-tiles: the passes of a small grid run their code about once per block
// and a second form of the cell costs them its instructions (1001x401 22.7 ->
// 23.5 us per step, 300x120 13.3 -> 13.8).  Measured on a B200, us per step
// without | with: 2048x512 FP32 23.4 | 22.6, FP64 28.0 | 26.5, 4001x1201 144 |
// 140, 8192x2048 FP32 232 | 206, FP16S 227 | 197.
constexpr uint32_t kDeepTile = 0x80000000u;

// The parameters of an odd step for a kernel compiled for even ones: the two
// slots of every direction pair trade places.  The free-surface kernels are
// compiled for one parity only: a step runs each pass's long, mostly
// straight-line code once per block, and the passes of both parities together
// did not stay in the SMs' instruction caches from step to step (on a tile of
// its own the flag stencil took 5,000 cycles, nearly all of it waiting for
// instructions).
constexpr bool kFsOdd = false;  // the parity they are compiled for
inline KParams as_even(const KParams& kp, uint32_t odd) {
  KParams q = kp;
  if (odd)
    for (int i = 1; i < 9; i += 2) std::swap(q.slot[i], q.slot[i + 1]);
  return q;
}

template <class S>
__device__ __forceinline__ S* slotp(const KParams& p, int s) {
  return static_cast<S*>(p.slot[s]);
}

// Slot holding incoming population i of a cell (i odd: own cell, slot a;
// i+1: neighbour i's cell, slot b), cellCalculations.cuh:185-196.
template <bool ODD>
__device__ __forceinline__ constexpr int slot_a(int i) { return ODD ? i : i + 1; }
template <bool ODD>
__device__ __forceinline__ constexpr int slot_b(int i) { return ODD ? i + 1 : i; }

// loadf plus the half-way wall: a population that would arrive from a wall
// neighbour is read from where this cell stored the opposite population last
// step, i.e. it comes back reflected after one step.  nbm bit k-1 = neighbour
// k is a wall.
template <class S, class C, bool HW, bool ODD, class K = Codec<S, C>>
__device__ __forceinline__ void load_in(const KParams& p, uint32_t idx, const uint32_t* nb, uint32_t nbm, C* f) {
  const float inv = p.f16_inv;
  f[0] = K::ld(slotp<S>(p, 0), idx, 0, inv);
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    const int a = slot_a<ODD>(i), b = slot_b<ODD>(i);
    if (HW && ((nbm >> i) & 1u)) f[i] = K::ld(slotp<S>(p, b), idx, i, inv);
    else f[i] = K::ld(slotp<S>(p, a), idx, i, inv);
    if (HW && ((nbm >> (i - 1)) & 1u)) f[i + 1] = K::ld(slotp<S>(p, a), nb[i], i + 1, inv);
    else f[i + 1] = K::ld(slotp<S>(p, b), nb[i], i + 1, inv);
  }
}

// The half-way wall part of load_in alone: f holds what load_in reads when
// no neighbour is a wall, and the populations that arrive from a wall
// neighbour (nbm) are replaced by their reflections.
template <class S, class C, bool ODD, class K = Codec<S, C>>
__device__ __forceinline__ void reload_reflected(const KParams& p, uint32_t idx, const uint32_t* nb, uint32_t nbm,
                                                 C* f) {
  const float inv = p.f16_inv;
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    const int a = slot_a<ODD>(i), b = slot_b<ODD>(i);
    if ((nbm >> i) & 1u) f[i] = K::ld(slotp<S>(p, b), idx, i, inv);
    if ((nbm >> (i - 1)) & 1u) f[i + 1] = K::ld(slotp<S>(p, a), nb[i], i + 1, inv);
  }
}

// loadOutgoingf, cellCalculations.cuh:207-217.
template <class S, class C, bool ODD>
__device__ __forceinline__ void load_out(const KParams& p, uint32_t idx, const uint32_t* nb, C* out) {
  const float inv = p.f16_inv;
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    out[i] = Codec<S, C>::ld(slotp<S>(p, slot_a<ODD>(i)), nb[i], i, inv);
    out[i + 1] = Codec<S, C>::ld(slotp<S>(p, slot_b<ODD>(i)), idx, i + 1, inv);
  }
}

// storef, cellCalculations.cuh:228-238.
template <class S, class C, bool ODD, class K = Codec<S, C>>
__device__ __forceinline__ void store_post(const KParams& p, uint32_t idx, const uint32_t* nb, const C* f) {
  const float sc = p.f16_scale;
  K::st(slotp<S>(p, 0), idx, 0, f[0], sc);
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    K::st(slotp<S>(p, slot_b<ODD>(i)), nb[i], i, f[i], sc);
    K::st(slotp<S>(p, slot_a<ODD>(i)), idx, i + 1, f[i + 1], sc);
  }
}

// Runtime-parity wrappers for passes that are not on the step's hot path.
template <class S, class C, bool HW>
__device__ __forceinline__ void load_in_rt(const KParams& p, uint32_t odd, uint32_t idx, const uint32_t* nb,
                                           uint32_t nbm, C* f) {
  if (odd) load_in<S, C, HW, true>(p, idx, nb, nbm, f);
  else load_in<S, C, HW, false>(p, idx, nb, nbm, f);
}

}  // namespace flb
