// k_mt.cu -- several single-phase time steps per launch (no counterpart in
// the reference, which launches every step's kernel on the whole grid).
//
// A block takes a window of the grid, its output and a halo of as many cells
// as there are steps, into shared memory, steps it there in place by the same
// esoteric pull as the one-step kernels, one row and column less on every side
// per step, and writes the output to the second population buffer.  Every
// value stored is the one the one-step kernels store, those of cells that are
// not updated included, so the buffers are interchangeable at any step.
//
// Why: one step per launch is bound by HBM on large grids (72 bytes per
// cell and step in FP32: 8192x2048 182 us, 1.02 of the copy) and by the launch
// and one latency chain on small ones (256x64: 4.1 us).  With T steps per
// launch a cell moves about 24 bytes per step and the launch is shared.  The
// halo costs recomputed cells and reads: at T = 4 and 64 x 22 windows (output
// 56 x 14) 1.39 cell updates per output cell and step.
// Measured on a B200 (FP32, fused arithmetic): 8192x2048 182 -> 107 us,
// 1024x256 4.6 -> 2.9, 256x64 4.1 -> 1.05; FP64 8192x2048 426 -> 270.  What
// bounds it now is shared memory (a warp's 64 cells move 48 wavefronts per
// step) and issue, with the load and store phases of the three resident blocks
// only partly under the others' steps.  Measured and not kept: windows in
// registers (rows exchanged by shuffles; 8192x2048 116 us), a sweep down the
// rows with the intermediate states in registers (104-118 us, FP32 and
// half-way walls only), one persistent block per SM loading its next window
// while it steps the current one (140 us), one cell per thread (147 us).
#include <atomic>
#include <type_traits>

#include "launch.h"
#include "pair.cuh"
#include "sc_cell.cuh"

namespace flb {

template <int B>
__device__ __forceinline__ void cp_async(void* sm, const void* g) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(sm);
  if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(g) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(a), "l"(g), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ uint32_t wrap_u(int v, uint32_t n) {
  if ((uint32_t)v < n) return (uint32_t)v;
  v += v < 0 ? (int)n : -(int)n;
  if ((uint32_t)v < n) return (uint32_t)v;
  return (uint32_t)(((v % (int)n) + (int)n) % (int)n);
}

// Code of a cell in shared memory: bits 0..7 its wall mask, bit 8 not updated.
constexpr uint32_t kIdle = 0x100u;

// The window in shared memory: row y holds its nine slots one after the other,
// RS values each, so that every slot of a cell and of its neighbours lies at a
// compile-time distance from the cell's own address.
template <class S, int W>
struct Win {
  static constexpr int RS = W + 4;      // values per slot and row (the pair path writes up to two past W)
  static constexpr int RP = 9 * RS;     // row pitch
  __host__ __device__ static constexpr int at(int s, int dx, int dy) { return s * RS + dx + dy * RP; }
  // distance to slot s of the neighbour toward i
  __host__ __device__ static constexpr int nb(int s, int i) { return at(s, cx(i), cy(i)); }
  __host__ __device__ static constexpr size_t bytes(int H) {
    return (((size_t)H * RP + 4) * sizeof(S) + (size_t)H * W * sizeof(uint16_t) + 15) / 16 * 16;
  }
};

// ---- one cell per thread ----------------------------------------------------
template <class S, class C, int W, bool DEV, bool FU, bool WM, bool ODD>
__device__ __forceinline__ void mt_cell(const KParams& p, S* q, uint32_t nbm, uint32_t gidx, uint32_t t) {
  using K = typename std::conditional<DEV, RawHalf, Codec<S, C>>::type;
  using L = Win<S, W>;
  const float inv = p.f16_inv, sc = p.f16_scale;
  C f[9];
  f[0] = K::ld(q, 0, 0, inv);
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    f[i] = K::ld(q + L::at(slot_a<ODD>(i), 0, 0), 0, i, inv);
    f[i + 1] = K::ld(q + L::nb(slot_b<ODD>(i), i), 0, i + 1, inv);
  }
  if (nbm) {
    // all eight reflections are loaded, then selected: one round trip
    C r[9];
#pragma unroll
    for (int i = 1; i < 9; i += 2) {
      r[i] = K::ld(q + L::at(slot_b<ODD>(i), 0, 0), 0, i, inv);
      r[i + 1] = K::ld(q + L::nb(slot_a<ODD>(i), i), 0, i + 1, inv);
    }
#pragma unroll
    for (int i = 1; i < 9; i += 2) {
      f[i] = ((nbm >> i) & 1u) ? r[i] : f[i];
      f[i + 1] = ((nbm >> (i - 1)) & 1u) ? r[i + 1] : f[i + 1];
    }
  }
  collide_cell<C, double, false, WM, FU, DEV, S>(p, gidx, 0u, 0u, kFluid, 0u, f, t);
  K::st(q, 0, 0, f[0], sc);
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    K::st(q + L::nb(slot_b<ODD>(i), i), 0, i, f[i], sc);
    K::st(q + L::at(slot_a<ODD>(i), 0, 0), 0, i + 1, f[i + 1], sc);
  }
}

// ---- two cells per thread, packed FP32 arithmetic ----------------------------
// Cells (x, x + 1), x even in the window; cd: their two codes; in0, in1: which
// of them lie in the step's columns (the other's result is not used).
template <int W, bool WM, bool ODD>
__device__ __forceinline__ void mt_pair(const KParams& p, float* q, uint32_t cd, uint32_t g0,
                                        uint32_t g1, bool in0, bool in1) {
  using L = Win<float, W>;
  f2 f[9];
  f[0] = ld_pair(q);
#pragma unroll
  for (int i = 1; i < 9; i += 2) {
    f[i] = ld_pair(q + L::at(slot_a<ODD>(i), 0, 0));
    const float* n = q + L::nb(slot_b<ODD>(i), i);
    f[i + 1] = i == 3 ? ld_pair(n) : pack(n[0], n[1]);
  }
  if (cd) {
    // all the reflections are loaded, then selected: one round trip
    f2 r[9];
#pragma unroll
    for (int i = 1; i < 9; i += 2) {
      r[i] = ld_pair(q + L::at(slot_b<ODD>(i), 0, 0));
      const float* n = q + L::nb(slot_a<ODD>(i), i);
      r[i + 1] = i == 3 ? ld_pair(n) : pack(n[0], n[1]);
    }
#pragma unroll
    for (int i = 1; i < 9; i += 2) {
      f[i] = pack((cd >> i) & 1u ? lo(r[i]) : lo(f[i]), (cd >> (16 + i)) & 1u ? hi(r[i]) : hi(f[i]));
      f[i + 1] = pack((cd >> (i - 1)) & 1u ? lo(r[i + 1]) : lo(f[i + 1]),
                      (cd >> (15 + i)) & 1u ? hi(r[i + 1]) : hi(f[i + 1]));
    }
  }
  const PairMacro m = collide_fused_pair(f, p);
  const bool act0 = !(cd & kIdle), act1 = !(cd & (kIdle << 16));
  if (WM) {
    float* R = static_cast<float*>(p.rho);
    float* U = static_cast<float*>(p.u);
    if (act0 && in0) {
      R[g0] = lo(m.rho);
      U[g0] = lo(m.ux);
      U[g0 + p.N] = lo(m.uy);
    }
    if (act1 && in1) {
      R[g1] = hi(m.rho);
      U[g1] = hi(m.ux);
      U[g1 + p.N] = hi(m.uy);
    }
  }
  if (act0 && act1) {
    st_pair(q, f[0]);
#pragma unroll
    for (int i = 1; i < 9; i += 2) {
      float* n = q + L::nb(slot_b<ODD>(i), i);
      if (i == 3) {
        st_pair(n, f[i]);
      } else {
        n[0] = lo(f[i]);
        n[1] = hi(f[i]);
      }
      st_pair(q + L::at(slot_a<ODD>(i), 0, 0), f[i + 1]);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 2; c++) {
      if (!(c ? act1 : act0)) continue;
      q[c] = c ? hi(f[0]) : lo(f[0]);
#pragma unroll
      for (int i = 1; i < 9; i += 2) {
        q[L::nb(slot_b<ODD>(i), i) + c] = c ? hi(f[i]) : lo(f[i]);
        q[L::at(slot_a<ODD>(i), c, 0)] = c ? hi(f[i + 1]) : lo(f[i + 1]);
      }
    }
  }
}

// One step over rows ylo..yhi, columns xlo..xhi of the window.
template <class S, class C, int W, bool PK, bool DEV, bool FU, bool WM, bool ODD>
__device__ __forceinline__ void mt_step(const KParams& p, S* sm, const uint16_t* code, int xlo, int xhi, int ylo,
                                        int yhi, int gx0, int gy0, uint32_t t) {
  using L = Win<S, W>;
  constexpr int CW = PK ? 2 : 1, PW = W / CW;  // cells per thread, threads per row
  constexpr int SEG = PW >= 32 ? PW / 32 : 1, RPW = PW >= 32 ? 1 : 32 / PW;  // segments per row, rows per warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x >> 5) / SEG;
  if (SEG > 1 && warp >= nw * SEG) return;
  const int x = (RPW > 1 ? lane % PW : lane + (SEG > 1 ? warp % SEG * 32 : 0)) * CW;
  if (x + CW - 1 < xlo || x > xhi) return;
  const int y0 = ylo + warp / SEG * RPW + (RPW > 1 ? lane / PW : 0), dy = nw * RPW;
  S* q = sm + y0 * L::RP + x;
  const uint16_t* cq = code + y0 * W + x;
  for (int y = y0; y <= yhi; y += dy, q += dy * L::RP, cq += dy * W) {
    uint32_t cd;
    if constexpr (PK) cd = *reinterpret_cast<const uint32_t*>(cq);
    else cd = *cq;
    if (cd & kIdle && (!PK || cd & (kIdle << 16))) continue;
    uint32_t row = 0, g0 = 0, g1 = 0;
    if (DEV || WM) {
      row = wrap_u(gy0 + y, p.ny) * p.nx;
      g0 = row + wrap_u(gx0 + x, p.nx);
      if (PK) g1 = row + wrap_u(gx0 + x + 1, p.nx);
    }
    if constexpr (PK) mt_pair<W, WM, ODD>(p, q, cd, g0, g1, x >= xlo, x + 1 <= xhi);
    else mt_cell<S, C, W, DEV, FU, WM, ODD>(p, q, cd, g0, t);
  }
}

template <class S, class C, bool FU, int W, bool VEC, bool PK>
__global__ void __launch_bounds__(sizeof(C) == 8 ? 512 : 1024, 1) k_mt(const __grid_constant__ KParams p, const __grid_constant__ MtArgs a) {
  constexpr bool DEV = kDev<S, false, FU>;
  using L = Win<S, W>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int H = a.H, T = a.T, pad = a.pad;
  const int tid = threadIdx.x, nthr = blockDim.x;
  constexpr int V = VEC ? 4 : 1, WV = W / V;
  S* sm = reinterpret_cast<S*>(smem);
  uint16_t* code = reinterpret_cast<uint16_t*>(sm + (uint32_t)(H * L::RP) + 4u);
  const int ox = (int)(blockIdx.x % (uint32_t)a.bx) * a.OW, oy = (int)(blockIdx.x / (uint32_t)a.bx) * a.OH;
  const int ow = min(a.OW, (int)p.nx - ox), oh = min(a.OH, (int)p.ny - oy);
  const int gx0 = ox - pad, gy0 = oy - T;  // cell (0, 0) of the window
  const int hh = oh + 2 * T;               // rows of the window in use
  pdl_wait();
  pdl_trigger();
  for (int k = tid; k < hh * WV; k += nthr) {
    const int y = k / WV, x = (k % WV) * V;
    if (x > pad + ow + T) continue;
    const uint32_t g = wrap_u(gx0 + x, p.nx) + wrap_u(gy0 + y, p.ny) * p.nx;
    S* q = sm + y * L::RP + x;
#pragma unroll
    for (int s = 0; s < 9; s++) {
      const S* src = slotp<S>(p, s) + g;
      if constexpr (sizeof(S) * V == 2) {
        q[s * L::RS] = *src;
      } else if constexpr (sizeof(S) * V == 32) {
        cp_async<16>(q + s * L::RS, src);
        cp_async<16>(q + s * L::RS + 2, src + 2);
      } else {
        cp_async<(int)(sizeof(S) * V)>(q + s * L::RS, src);
      }
    }
    if constexpr (VEC) {
      const uint32_t fl = *reinterpret_cast<const uint32_t*>(p.flags + g);
      const uint32_t nm = p.nbmask ? *reinterpret_cast<const uint32_t*>(p.nbmask + g) : 0u;
      const uint32_t idle = __vcmpne4(fl & 0x0a0a0a0au, 0u) & 0x01010101u;
      uint2 c;
      c.x = __byte_perm(nm, idle, 0x5140);
      c.y = __byte_perm(nm, idle, 0x7362);
      *reinterpret_cast<uint2*>(code + y * W + x) = c;
    } else {
      uint32_t cd = (p.flags[g] & (kGas | kWall)) ? kIdle : 0u;
      if (p.nbmask) cd |= p.nbmask[g];
      code[y * W + x] = (uint16_t)cd;
    }
  }
  cp_async_wait();
  __syncthreads();
  const int par = (int)(a.t & 1u);
  for (int k = 1; k <= T; k++) {
    const int xlo = pad - T + k - 1, xhi = pad + ow - 1 + T - k, ylo = k, yhi = hh - 1 - k;
    const uint32_t t = a.t + (uint32_t)(k - 1);
    const bool odd = ((par + k - 1) & 1) != 0;
    if (k == T && a.wm) {
      if (odd) mt_step<S, C, W, PK, DEV, FU, true, true>(p, sm, code, xlo, xhi, ylo, yhi, gx0, gy0, t);
      else mt_step<S, C, W, PK, DEV, FU, true, false>(p, sm, code, xlo, xhi, ylo, yhi, gx0, gy0, t);
    } else {
      if (odd) mt_step<S, C, W, PK, DEV, FU, false, true>(p, sm, code, xlo, xhi, ylo, yhi, gx0, gy0, t);
      else mt_step<S, C, W, PK, DEV, FU, false, false>(p, sm, code, xlo, xhi, ylo, yhi, gx0, gy0, t);
    }
    __syncthreads();
  }
  // slot b of the pair (i, i+1) of a cell is written by the cell at -e_i: its
  // rows are those of the output tile shifted by e_i
  const bool lodd = ((par + T - 1) & 1) != 0;  // parity of the last step
  for (int k = tid; k < oh * WV; k += nthr) {
    const int y = T + k / WV, x = (k % WV) * V;
    if (x < pad || x >= pad + ow) continue;
    const uint32_t gx = (uint32_t)(gx0 + x);
    const uint32_t r0 = (uint32_t)(gy0 + y), rp = (r0 + 1u == p.ny ? 0u : r0 + 1u), rm = (r0 == 0u ? p.ny - 1u : r0 - 1u);
#pragma unroll
    for (int s = 0; s < 9; s++) {
      const int i = s == 0 ? 0 : (s - 1) | 1;
      const bool isb = s != 0 && ((s == i) != lodd);  // s is slot b of its pair in the last step
      const int ey = isb ? cy(i) : 0;
      const uint32_t gy = ey == 0 ? r0 : (ey > 0 ? rp : rm);
      S* dst = static_cast<S*>(a.dst) + (size_t)s * p.N + gx + gy * p.nx;
      const S* src = sm + (y + ey) * L::RP + s * L::RS + x;
      if constexpr (sizeof(S) * V == 32) {
        reinterpret_cast<uint4*>(dst)[0] = reinterpret_cast<const uint4*>(src)[0];
        reinterpret_cast<uint4*>(dst)[1] = reinterpret_cast<const uint4*>(src)[1];
      } else if constexpr (sizeof(S) * V == 16) {
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
      } else if constexpr (VEC) {
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(src);
      } else {
        *dst = *src;
      }
    }
  }
  if (DEV && tid == 0 && blockIdx.x == 0) p.tstep[(a.t + (uint32_t)T) & 1u] = a.t + (uint32_t)T;
}

template <class S, class C, bool FU, int W, bool VEC, bool PK>
static cudaError_t launch_mt_k(const KParams& kp, const MtArgs& a, cudaStream_t st) {
  auto kern = k_mt<S, C, FU, W, VEC, PK>;
  const size_t smem = Win<S, W>::bytes(a.H);
  if (smem > 48u * 1024u) {
    // once per kernel and device (setting it again does no harm)
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;
    if (!(done.load(std::memory_order_relaxed) & bit)) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return e;
      done.fetch_or(bit, std::memory_order_relaxed);
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = a.tiles;
  cfg.blockDim = a.threads;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, kp, a);
}

template <class S, class C, class M>
cudaError_t launch_mt(const KParams& kp, const MtArgs& a, cudaStream_t st, bool fu) {
  auto go = [&](auto f, auto v) -> cudaError_t {
    constexpr bool F = decltype(f)::value, V = decltype(v)::value;
    if constexpr (F && std::is_same<S, float>::value) {
      if (a.pairs)
        return a.W == 32 ? launch_mt_k<S, C, F, 32, V, true>(kp, a, st) : launch_mt_k<S, C, F, 64, V, true>(kp, a, st);
    }
    return a.W == 32 ? launch_mt_k<S, C, F, 32, V, false>(kp, a, st) : launch_mt_k<S, C, F, 64, V, false>(kp, a, st);
  };
  using T = std::true_type;
  using N = std::false_type;
  if (fu) return a.vec ? go(T{}, T{}) : go(T{}, N{});
  return a.vec ? go(N{}, T{}) : go(N{}, N{});
}

#define FLB_INSTANTIATE(S, C, M) \
  template cudaError_t launch_mt<S, C, M>(const KParams&, const MtArgs&, cudaStream_t, bool);
FLB_INSTANTIATE(double, double, double)
FLB_INSTANTIATE(float, float, double)
FLB_INSTANTIATE(__half, float, double)
#undef FLB_INSTANTIATE

}  // namespace flb
