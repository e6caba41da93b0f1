// k_fs.cu -- the free-surface passes as separate kernels: FS_1
// (lbmKernel2D.cu:14-121) and FS_2, FS_3, FS_4 fused into one shared-memory
// flag-stencil kernel (lbmKernel2D.cu:124-303) that also lists the next
// step's super-tiles.  The per-cell and per-tile code is in fs_cells.cuh.
// Compiled for one step parity (as_even).
#include <type_traits>

#include "fs_cells.cuh"
#include "launch.h"

namespace flb {

// FS_1 on the listed super-tiles, one row of a super-tile per warp.  With two
// cells per thread (256-thread blocks, three per SM at 85 registers) about 440
// listed super-tiles are one round; one cell per thread (512 threads) makes the
// pass shorter where there are few.  Measured on a B200, us per step with two |
// one: 101x101 17.2 | 14.9, 300x120 16.4 | 15.0, 1001x401 26.3 | 25.4, 2048x512
// 24.2 | 27.6, 8192x2048 232 | 264; the line is kSmallTiles.  One cell: two
// blocks per SM at 64 registers, where the FP64 mass arithmetic spills (136
// bytes, FP64 storage 350); grids of up to kTinyTiles super-tiles, whose listed
// ones fit one block per SM, take 128: 300x120 14.4 -> 13.4, 601x301 16.2 -> 15.0
// (but 1001x401 22.8 -> 24.1).  Two cells, three blocks per SM | four at 64
// registers | five at 48: 2048x512 FP32 22.4 | 22.5 | 23.6, FP64 25.8 | 26.3 |
// 31.7, 4001x1201 50.8 | 51.6 | 53.6.  The block's next super-tile is not
// prefetched into L2: with the short form of the plain-fluid super-tiles that
// cost more than it hid (8192x2048 FP32 196 against 184, FP16S 183 against 172,
// 4001x1201 58 against 54).
constexpr int kFs1Block = 256;   // two cells per thread (x and x + 32 of a row), three blocks per SM
constexpr int kFs1Small = 512;   // one cell per thread, two blocks per SM, or one
// lc: the next step's list lengths and marks, cleared here for this step's
// flag pass.
template <class S, class C, class M, bool HW, int BLOCK, int MB, bool DEEP>
__global__ void __launch_bounds__(BLOCK, MB) k_fs1(const __grid_constant__ KParams p,
                                                                       const TileList tl, const ListClear lc) {
  pdl_wait();
  pdl_trigger();
  clear_next_lists(lc);
  constexpr uint32_t kCpr = BLOCK / 32 / kSTH;         // warps per row of a super-tile
  constexpr uint32_t kCells = kSTW / (32u * kCpr);     // cells per thread and super-tile
  static_assert(kCells * 32u * kCpr == kSTW && kCells <= 2u, "FS_1: one or two cells per thread and super-tile");
  // the block's first entry is loaded with the length (the list holds at least
  // a grid of entries, whatever its length)
  uint32_t t = tile_at(tl, blockIdx.x);
  const uint32_t n = tile_count(tl);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t row = warp % kSTH, chunk = warp / kSTH;
  const uint32_t nx = p.nx;
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x, t = i < n ? tile_at(tl, i) : 0u) {
    const bool deep = DEEP && (t & kDeepTile);
    t &= ~kDeepTile;
    const uint32_t y = (t / tl.nsx) * kSTH + row;
    if (y >= p.ny) continue;
    const uint32_t xa = (t % tl.nsx) * kSTW + chunk * 32u + lane, xc = xa + 32u * kCpr;
    if (deep) {
      // the loads of both cells before either store
      M m[kCells];
#pragma unroll
      for (uint32_t k = 0; k < kCells; k++) m[k] = fs1_deep_cell<S, C, M>(p, xa + 32u * kCpr * k + y * nx);
#pragma unroll
      for (uint32_t k = 0; k < kCells; k++) static_cast<M*>(p.mass)[xa + 32u * kCpr * k + y * nx] = m[k];
      continue;
    }
    // the cells' flags and wall masks first: one round trip for both
    uint8_t fa = kGas, fc = kGas;
    uint32_t ma = 0, mc = 0;
    if (xa < nx) {
      fa = p.flags[xa + y * nx];
      if (HW) ma = p.nbmask[xa + y * nx];
    }
    if (kCells == 2u && xc < nx) {
      fc = p.flags[xc + y * nx];
      if (HW) mc = p.nbmask[xc + y * nx];
    }
    if (xa < nx) fs1_cell<S, C, M, HW>(p, xa, y, fa, ma);
    if (kCells == 2u && xc < nx) fs1_cell<S, C, M, HW>(p, xc, y, fc, mc);
  }
}

// Writes the populations FS_1 parked in recon (reference mode) into their
// incoming slots, as the reference FS_1 kernel does itself.  Only the
// isolated-pass path uses it; a full step hands them to stream-collide.
template <class S, class C>
__global__ void k_apply_recon(const __grid_constant__ KParams p, uint32_t odd) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t y = blockIdx.y;
  if (x >= p.nx) return;
  const uint32_t N = p.N, idx = x + y * p.nx;
  const uint8_t flag = p.flags[idx];
  if ((flag & (kFGI | kGas | kWall | kInlet)) != kInterface) return;
  const uint32_t m = p.recon_mask[idx];
  if (!m) return;
  uint32_t nb[9];
  neighbours(x, y, p.nx, p.ny, nb);
  const C* rec = static_cast<const C*>(p.recon);
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    const int a = odd ? i : i + 1, b = odd ? i + 1 : i;
    if ((m >> (i - 1)) & 1u) Codec<S, C>::st(slotp<S>(p, a), idx, i, rec[(uint32_t)(i - 1) * N + idx], p.f16_scale);
    if ((m >> i) & 1u) Codec<S, C>::st(slotp<S>(p, b), nb[i], i + 1, rec[(uint32_t)i * N + idx], p.f16_scale);
  }
  p.recon_mask[idx] = 0;
}

// The listed super-tiles: each block runs the flag pass on a super-tile,
// records its activity word in nz and appends to the next step's lists.
// TW x 8 tiles, CPT cells per thread, MB blocks resident per SM: with one cell
// per thread two on grids of up to kTinyTiles super-tiles (three spill at 40
// registers: 300x120 14.4 against 13.4 us per step with FS_1's form), three
// above (1001x401 22.8 against 23.4); with two cells four (five spill at 48:
// 2048x512 23.5 against 22.5), and five on grids of more than kLargeTiles
// super-tiles, most of them plain fluid in many rounds (8192x2048 FP32 174
// against 177, FP16S 168 against 172; 4001x1201 51.6 either way).
template <class S, class C, class M, int TW, int CPT, int MB, bool THIN>
__global__ void __launch_bounds__(TW* kTY / CPT, MB)
    k_fs234(const __grid_constant__ KParams p, const TileList tl, uint32_t* __restrict__ nz, const NextLists nl) {
  __shared__ FlagMasks<TW> sm;
  __shared__ uint32_t wact_sm[TW * kTY / CPT / 32];
  // the list was built by the previous step (FS_1 waited for it), so it is
  // read before waiting for stream-collide, whose flags the pass needs
  const uint32_t n = tile_count(tl);
  pdl_wait();
  pdl_trigger();
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x)
    fs234_super_tile<S, C, M, TW, CPT, (CPT > 1), THIN>(p, tile_at(tl, i), tl.nsx, nz, nl, sm, wact_sm);
}

// ---- launchers -------------------------------------------------------------------
template <class S, class C, class M>
void launch_fs1(const KParams& kp, cudaStream_t st, uint32_t odd, bool hw, const TileList& tl, uint32_t grid,
                const ListClear& lc) {
  const KParams q = as_even(kp, odd);
  auto go = [&](auto block, auto mb) {
    constexpr int BLOCK = decltype(block)::value, MB = decltype(mb)::value;
    constexpr bool DEEP = BLOCK == kFs1Block;
    if (hw) launch_pdl(k_fs1<S, C, M, true, BLOCK, MB, DEEP>, grid, BLOCK, st, q, tl, lc);
    else launch_pdl(k_fs1<S, C, M, false, BLOCK, MB, DEEP>, grid, BLOCK, st, q, tl, lc);
  };
  using std::integral_constant;
  if (tl.ntiles <= kTinyTiles) go(integral_constant<int, kFs1Small>{}, integral_constant<int, 1>{});
  else if (tl.ntiles <= kSmallTiles) go(integral_constant<int, kFs1Small>{}, integral_constant<int, 2>{});
  else go(integral_constant<int, kFs1Block>{}, integral_constant<int, 3>{});
}

template <class S, class C, class M>
void launch_apply_recon(const KParams& kp, cudaStream_t st, uint32_t odd) {
  k_apply_recon<S, C><<<dim3((kp.nx + kBlock - 1) / kBlock, kp.ny), kBlock, 0, st>>>(kp, odd);
}

// The flag pass, which also lists the next step's super-tiles, in one of its
// launch forms (FsForm: tile width and cells per thread).  On grids of up to
// kWideTiles super-tiles it is launched so that it may start while
// stream-collide drains (programmatic dependent launch); above, with an
// ordinary launch (measured faster on the 8192x2048 dam break).  Returns the
// number of kernels launched.
template <class S, class C, class M, int TW, int CPT, int MB>
void launch_fs234_form(const KParams& kp, cudaStream_t st, uint32_t odd, const TileList& tl, uint32_t grid,
                       uint32_t* nz, const NextLists& nl) {
  constexpr int threads = TW * kTY / CPT;
  const KParams q = as_even(kp, odd);
  auto go = [&](auto thin) {
    constexpr bool THIN = decltype(thin)::value;
    if (tl.ntiles <= kWideTiles) launch_pdl(k_fs234<S, C, M, TW, CPT, MB, THIN>, grid, threads, st, q, tl, nz, nl);
    else k_fs234<S, C, M, TW, CPT, MB, THIN><<<grid, threads, 0, st>>>(q, tl, nz, nl);
  };
  if (nl.thin) go(std::true_type{});
  else go(std::false_type{});
}

template <class S, class C, class M>
int launch_fs234(const KParams& kp, cudaStream_t st, uint32_t odd, const TileList& tl, uint32_t grid, uint32_t* nz,
                 const NextLists& nl, int form) {
  switch (form) {
    case FS_FORM_W32: launch_fs234_form<S, C, M, 32, 1, 6>(kp, st, odd, tl, grid, nz, nl); break;
    case FS_FORM_W64X1:
      if (tl.ntiles <= kTinyTiles) launch_fs234_form<S, C, M, 64, 1, 2>(kp, st, odd, tl, grid, nz, nl);
      else launch_fs234_form<S, C, M, 64, 1, 3>(kp, st, odd, tl, grid, nz, nl);
      break;
    default:
      if (tl.ntiles <= kLargeTiles) launch_fs234_form<S, C, M, 64, 2, 4>(kp, st, odd, tl, grid, nz, nl);
      else launch_fs234_form<S, C, M, 64, 2, 5>(kp, st, odd, tl, grid, nz, nl);
      break;
  }
  return 1;
}

// Resident blocks per SM: the launch bounds above.
int fs1_blocks_per_sm(uint32_t ntiles) { return ntiles <= kTinyTiles ? 1 : ntiles <= kSmallTiles ? 2 : 3; }
int fs234_blocks_per_sm(int form, uint32_t ntiles) {
  return form == FS_FORM_W32 ? 6 : form == FS_FORM_W64X1 ? (ntiles <= kTinyTiles ? 2 : 3)
                               : ntiles <= kLargeTiles ? 4 : 5;
}

#define FLB_INSTANTIATE(S, C, M)                                                                                  \
  template void launch_fs1<S, C, M>(const KParams&, cudaStream_t, uint32_t, bool, const TileList&, uint32_t,       \
                                    const ListClear&);                                                     \
  template void launch_apply_recon<S, C, M>(const KParams&, cudaStream_t, uint32_t);                             \
  template int launch_fs234<S, C, M>(const KParams&, cudaStream_t, uint32_t, const TileList&, uint32_t, uint32_t*,   \
                                     const NextLists&, int);
FLB_FOR_EACH_VARIANT(FLB_INSTANTIATE)
#undef FLB_INSTANTIATE

}  // namespace flb
