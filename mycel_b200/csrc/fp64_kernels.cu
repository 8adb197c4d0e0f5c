// Plain FP64 path: reproduces Mycel.Core's arithmetic on sm_100a.
// This translation unit is compiled with -fmad=false: no a*b+c is contracted, as in the reference (RyuJIT).
//
// Kernels and the reference code whose rounding sequence they reproduce:
//   k_matvec64      FemOperator.ApplyK/ApplyA (Fem/FemOperator.cs:196-294, MultiplyElementUnsafe :379-422).
//                   Node-centric gather: one thread per node sums its <= 8 element contributions in the
//                   8-colour order the reference scatters them, each contribution computed with the
//                   reference's scale-then-dot order (ue = x*E; four lane chains; Vector256.Sum). In the
//                   PCG it also forms the direction (ProcessUpdatePChunk, Fem/PcgSolver.cs:529-553).
//   k_diag          FemOperator.AssembleDiagonal (:143-172), same colour order; Jacobi inverse (JacobiPreconditioner.cs:25).
//   k_dot_exact     PcgSolver DotParallel/ProcessDotChunk (Fem/PcgSolver.cs:385-450): one CTA per 8192-block,
//                   producer warps stage products in shared memory, lanes 0-3 of warp 0 run the four
//                   sequential lane chains, the last CTA adds the block partials in block order.
//   k_xr_exact      ProcessUpdateXrNormChunk + ProcessApplyPrecDotChunk (:452-527) fused: two chain sets.
//   k_filter_*      DensityFilter (Optimization/DensityFilter.cs:34-303) as a stencil in the reference's
//                   neighbour order (jz, jy, jx ascending), weights (rmin - dist) * invHs_row.
//   k_sens          SensitivityAnalysis (Optimization/SensitivityAnalysis.cs:98-144).
//   k_oc            OcOptimizer.Update (Optimization/OcOptimizer.cs:12-175): one persistent cooperative kernel.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>
#include <cooperative_groups.h>
#include <cuda_pipeline.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "internal.h"
#include "libm_pow.h"

namespace mycel {

constexpr int kBlock = 8192;  // PcgSolver.BlockSize

// ---------------------------------------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ double lane_sum(double a0, double a1, double a2, double a3) {
  return (a0 + a1) + (a2 + a3);  // Vector256<double>.Sum: Sum(lower) + Sum(upper) on .NET 8+
}

// Math.Pow on the path (FemOperator.cs:100,133; SensitivityAnalysis.cs:93-95): the host C library's pow,
// restated with its rounding sequence (libm_pow.h), so E_e and dE/drho carry the reference's bits for every
// exponent.
__device__ __forceinline__ double path_pow(double x, double y) { return libm_pow::pow(x, y); }

__device__ __forceinline__ int local_index(int ox, int oy, int oz) {
  // Hex8 local node order (Hex8Element.cs:8-16): (0,0,0),(1,0,0),(1,1,0),(0,1,0), then the same at z=1
  int base = oy ? (ox ? 2 : 3) : (ox ? 1 : 0);
  return base + 4 * oz;
}

// dynamic shared memory above 48 KB, allowed once per kernel and device
template <auto K>
static void allow_smem(int device, size_t bytes) {
  static std::atomic<uint64_t> done[4];
  if (device < 0 || device >= 256) device = 255;
  const uint64_t bit = 1ull << (device & 63);
  if (done[device >> 6].load(std::memory_order_acquire) & bit) return;
  cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  done[device >> 6].fetch_or(bit, std::memory_order_release);
}

__device__ __forceinline__ double ld_volatile(const double* p) { return *(const volatile double*)p; }

// Parity-class node mapping: blockIdx.y = class (px | py<<1 | pz<<2); nodes of one class have the same
// parity in i, j, k, so the colour order of their incident elements is the same for the whole warp.
struct ClassNode {
  int i, j, k, px, py, pz;
  bool valid;
};
__device__ __forceinline__ ClassNode class_node(const GridDims& g, int cls, int64_t t) {
  ClassNode c;
  c.px = cls & 1; c.py = (cls >> 1) & 1; c.pz = (cls >> 2) & 1;
  int cx = (g.nx1 - c.px + 1) >> 1, cy = (g.ny1 - c.py + 1) >> 1, cz = (g.nz1 - c.pz + 1) >> 1;
  int64_t tot = (int64_t)cx * cy * cz;
  c.valid = t < tot;
  if (!c.valid) { c.i = c.j = c.k = 0; return c; }
  int a = (int)(t % cx);
  int64_t rest = t / cx;
  int b = (int)(rest % cy);
  int cc = (int)(rest / cy);
  c.i = c.px + 2 * a; c.j = c.py + 2 * b; c.k = c.pz + 2 * cc;
  return c;
}

inline dim3 class_grid(const GridDims& g, int threads) {
  int cx = (g.nx1 + 1) >> 1, cy = (g.ny1 + 1) >> 1, cz = (g.nz1 + 1) >> 1;
  int64_t tot = (int64_t)cx * cy * cz;
  return dim3((unsigned)((tot + threads - 1) / threads), 8, 1);
}

// ---------------------------------------------------------------------------------------------------------
// problem set-up: active nodes, constrained mask (FeModel.cs:80-183)
// ---------------------------------------------------------------------------------------------------------
__global__ void k_node_flags(GridDims g, const uint8_t* __restrict__ dom, uint8_t* __restrict__ nf) {
  int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= g.nn) return;
  int i = (int)(n % g.nx1);
  int64_t r = n / g.nx1;
  int j = (int)(r % g.ny1), k = (int)(r / g.ny1);
  bool act = false;
  for (int dz = -1; dz <= 0; ++dz)
    for (int dy = -1; dy <= 0; ++dy)
      for (int dx = -1; dx <= 0; ++dx) {
        int ie = i + dx, je = j + dy, ke = k + dz;
        if (ie >= 0 && ie < g.nx && je >= 0 && je < g.ny && ke >= 0 && ke < g.nz)
          act |= dom[ie + (int64_t)g.nx * (je + (int64_t)g.ny * ke)] != 0;
      }
  nf[n] = act ? NF_ACTIVE : (uint8_t)(NF_CX | NF_CY | NF_CZ);
}

__global__ void k_fixed_flags(GridDims g, const int32_t* __restrict__ fixed, int32_t nfix, uint8_t* nf) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nfix) return;
  int32_t d = fixed[t];
  int64_t node = d / 3;
  int c = d % 3;
  // several threads may touch one node byte: use a 32-bit atomicOr on the containing word
  unsigned int* w = (unsigned int*)((uintptr_t)(nf + node) & ~(uintptr_t)3);
  int sh = (int)(((uintptr_t)(nf + node) & 3) * 8);
  atomicOr(w, (unsigned int)(1u << c) << sh);
}

// count unique fixed DOFs on active nodes (FeModel.ActiveFixedDofCount, :165-183)
__global__ void k_count_active_fixed(GridDims g, const uint8_t* __restrict__ nf, const uint8_t* __restrict__ fixmask,
                                     int32_t* count) {
  int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int v = 0;
  if (d < g.nd) v = (fixmask[d] != 0) && (nf[d / 3] & NF_ACTIVE);
  v = __syncthreads_count(v);
  if (threadIdx.x == 0 && v) atomicAdd(count, v);
}

__global__ void k_mark_fixed(const int32_t* __restrict__ fixed, int32_t nfix, uint8_t* fixmask) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nfix) fixmask[fixed[t]] = 1;
}

void launch_setup_nodes(mycel_problem* p, const int32_t* d_fixed, int32_t n_fixed, int32_t* d_count) {
  const GridDims& g = p->g;
  cudaStream_t s = p->ctx->stream;
  k_node_flags<<<(unsigned)((g.nn + 255) / 256), 256, 0, s>>>(g, p->d_domain, p->d_nflags);
  p->ctx->launches++;
  if (n_fixed > 0) {
    k_fixed_flags<<<(n_fixed + 255) / 256, 256, 0, s>>>(g, d_fixed, n_fixed, p->d_nflags);
    p->ctx->launches++;
    // reuse tmp0 as a byte mask of fixed DOFs
    uint8_t* fixmask = (uint8_t*)p->d_tmp0;
    cudaMemsetAsync(fixmask, 0, (size_t)g.nd, s);
    k_mark_fixed<<<(n_fixed + 255) / 256, 256, 0, s>>>(d_fixed, n_fixed, fixmask);
    k_count_active_fixed<<<(unsigned)((g.nd + 255) / 256), 256, 0, s>>>(g, p->d_nflags, fixmask, d_count);
    p->ctx->launches += 2;
  }
}

// ---------------------------------------------------------------------------------------------------------
// E_e = Emin + rho^p (E0 - Emin)   (FemOperator.cs:100, :133)
// ---------------------------------------------------------------------------------------------------------
__global__ void k_update_E(int64_t na, const int32_t* __restrict__ active, const double* __restrict__ rho,
                           double emin, double e0, double penal, double* __restrict__ E, float* __restrict__ Ef) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= na) return;
  int32_t e = active[t];
  double v = emin + path_pow(rho[e], penal) * (e0 - emin);
  E[e] = v;
  if (Ef) Ef[e] = (float)v;
}

void launch_update_E(mycel_problem* p, const double* d_rho_box, double penal) {
  p->e_version++;
  if (p->n_active == 0) return;
  k_update_E<<<(unsigned)((p->n_active + 255) / 256), 256, 0, p->ctx->stream>>>(
      p->n_active, p->d_active, d_rho_box, p->emin, p->e0, penal, p->d_E, p->d_Ef);
  p->ctx->launches++;
}

// DiagA[dof] = sum over colours of E_e * DiagKe[k]; constrained -> 1; invD = |d| > 1e-30 ? 1/d : 1
struct Diag24 { double v[24]; };
__global__ void __launch_bounds__(256) k_diag(GridDims g, const __grid_constant__ Diag24 dk, const double* __restrict__ E,
                                              const uint8_t* __restrict__ dom, const uint8_t* __restrict__ nf,
                                              double* __restrict__ diag, double* __restrict__ invd,
                                              float* __restrict__ invdf) {
  ClassNode cn = class_node(g, blockIdx.y, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
  if (!cn.valid) return;
  double d0 = 0.0, d1 = 0.0, d2 = 0.0;
#pragma unroll 1
  for (int col = 0; col < 8; ++col) {
    int ox = (col & 1) ^ cn.px, oy = ((col >> 1) & 1) ^ cn.py, oz = ((col >> 2) & 1) ^ cn.pz;
    int ie = cn.i - ox, je = cn.j - oy, ke = cn.k - oz;
    if (ie < 0 || ie >= g.nx || je < 0 || je >= g.ny || ke < 0 || ke >= g.nz) continue;
    int64_t e = ie + (int64_t)g.nx * (je + (int64_t)g.ny * ke);
    if (!dom[e]) continue;
    double ee = E[e];
    int a = local_index(ox, oy, oz);
    d0 = d0 + ee * dk.v[3 * a];
    d1 = d1 + ee * dk.v[3 * a + 1];
    d2 = d2 + ee * dk.v[3 * a + 2];
  }
  int64_t n = cn.i + (int64_t)g.nx1 * (cn.j + (int64_t)g.ny1 * cn.k);
  uint8_t f = nf[n];
  double dd[3] = {d0, d1, d2};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double d = (f & (1 << c)) ? 1.0 : dd[c];
    double iv = fabs(d) > 1e-30 ? 1.0 / d : 1.0;
    diag[3 * n + c] = d;
    invd[3 * n + c] = iv;
    if (invdf) invdf[pidx(g, cn.i, cn.j + (int64_t)g.ny1 * cn.k, c)] = (float)iv;
  }
}

void launch_diag(mycel_problem* p) {
  Diag24 dk;
  for (int i = 0; i < 24; ++i) dk.v[i] = p->diag_ke[i];
  k_diag<<<class_grid(p->g, 256), 256, 0, p->ctx->stream>>>(p->g, dk, p->d_E, p->d_domain, p->d_nflags, p->d_diag,
                                                            p->d_invd, p->d_invdf);
  p->ctx->launches++;
}

// ---------------------------------------------------------------------------------------------------------
// y = K x (projected: y = x on constrained DOFs, ApplyA with xIsAlreadyProjected)
// Bound by the FP64 pipe: 1,344 separately rounded operations per node (8 elements x (24 scalings + 3 rows of
// 47), 24 adds). A CTA takes kMvNodes consecutive nodes of one node plane, in node order over rows (no lane is
// lost to a tile edge), stages their neighbourhood in the planes k-1, k, k+1 in shared memory with 16-byte
// asynchronous copies, all in flight at once, and each thread forms its node's eight contributions with
// compile-time element positions, so that the KE entries are constant-bank operands and nothing but 24 shared
// loads and the arithmetic is left per element; the contributions are kept and added in the colour order of the
// node's parity (selects for x and y, a uniform branch for z). A lane chain is finished before the next is begun,
// which keeps the live registers low.
// FUSE: x = z + beta p_old (or z at a start), formed in shared memory; the owned nodes' values go to p_new, so the
// iteration needs no pass of its own for p.
// Against the z-marching 64 x 4 tiles this replaces (per-node runtime KE rows), p update included: 30x10x4 elements
// 29.9 -> 7.6 us, 96x48x24 51.3 -> 22.6 us, 192x96x96 446 (without p) -> 263 us. What is left over the FP64 pipe's
// 10 and 133 us are issue slots: a constant load for each KE entry and the selects of the colour order.
// ---------------------------------------------------------------------------------------------------------
constexpr int kMvNodes = 128;

// Staged ranges of a plane, in doubles: one contiguous range of the CTA's nodes and the rows before and after
// (row pitch nx1), or, for rows longer than the CTA's span, three (one per node row). A range starts at the even
// global index at or below its first entry (16-byte copies).
struct MvStage {
  int pitch;    // node positions between neighbouring rows
  int nseg;     // ranges per plane
  int seglen;   // doubles of a range
  int segstep;  // doubles between ranges in shared memory (even)
};
__host__ __device__ inline MvStage mv_stage(int nx1) {
  MvStage m;
  const bool rows3 = nx1 > kMvNodes + 2;
  m.pitch = rows3 ? kMvNodes + 2 : nx1;
  m.nseg = rows3 ? 3 : 1;
  m.seglen = 3 * (rows3 ? kMvNodes + 2 : kMvNodes + 2 + 2 * nx1);
  m.segstep = (m.seglen + 3) & ~1;
  return m;
}
inline size_t mv_smem(int nx1, bool fuse) {
  const MvStage m = mv_stage(nx1);
  return sizeof(double) * 3 * (size_t)m.nseg * m.segstep * (fuse ? 2 : 1);
}

template <int FUSE>
__global__ void __launch_bounds__(kMvNodes, 4) k_matvec64(GridDims g, const __grid_constant__ KeD ke,
                                                          const double* x, const double* pold,
                                                          double* __restrict__ pnew, double* __restrict__ y,
                                                          const double* __restrict__ E, const uint8_t* __restrict__ dom,
                                                          const uint8_t* __restrict__ nf, int projected,
                                                          const PcgState* st, unsigned chunks) {
  extern __shared__ __align__(16) double xs[];  // [plane k-1, k, k+1][range][position][component]; FUSE: then p_old's
  const int tid = threadIdx.x;
  const int k = (int)(blockIdx.x / chunks);
  const int np = g.nx1 * g.ny1;  // nodes of a plane (all DOF indices fit in 31 bits)
  const int n0 = (int)(blockIdx.x - (unsigned)k * chunks) * kMvNodes;
  const MvStage m = mv_stage(g.nx1);
  const int half = 3 * m.nseg * m.segstep;
  const int nl = n0 + tid, n = nl < np ? nl : np - 1;
  const int j = n / g.nx1, i = n - j * g.nx1;
  const bool mine = nl < np;
  // the node's elements (i-1+sx, j-1+sy, k-1+sz): E and whether they contribute
  double ee[8];
  unsigned act = 0;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int ex = i - 1 + (v & 1), ey = j - 1 + ((v >> 1) & 1), ez = k - 1 + (v >> 2);
    const bool in = mine && ex >= 0 && ex < g.nx && ey >= 0 && ey < g.ny && ez >= 0 && ez < g.nz;
    const int64_t e = ex + (int64_t)g.nx * (ey + (int64_t)g.ny * ez);
    if (in && dom[e]) act |= 1u << v;
    ee[v] = in ? E[e] : 0.0;
  }
  dep_begin();
  const int status = st ? st->status : PCG_RUNNING;
  const double beta = FUSE ? st->beta : 0.0;
  const bool first = FUSE ? st->first != 0 : false;
  const int64_t top = (g.nd + 1) & ~int64_t(1);  // vectors are allocated in multiples of 16 bytes
  // first entry of range sgm of plane pl in the global vector (may lie before it)
  auto range = [&](int pl, int sgm) -> int64_t {
    return (int64_t)3 * np * (k - 1 + pl) + 3 * (n0 - 1 + (m.nseg == 3 ? (sgm - 1) * g.nx1 : -g.nx1));
  };
  int off[3][3];  // staged position of the CTA's first node in row dy of plane pl
#pragma unroll
  for (int pl = 0; pl < 3; ++pl)
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
      const int sgm = m.nseg == 3 ? dy : 0;
      off[pl][dy] = (pl * m.nseg + sgm) * m.segstep + (int)(range(pl, sgm) & 1) + (m.nseg == 3 ? 0 : 3 * dy * m.pitch);
    }
  for (int pl = 0; pl < 3; ++pl) {
    if (k - 1 + pl < 0 || k - 1 + pl >= g.nz1) continue;  // read by no contributing element
    for (int sgm = 0; sgm < m.nseg; ++sgm) {
      const int64_t f0 = range(pl, sgm), a0 = f0 & ~int64_t(1);
      double* dst = xs + (pl * m.nseg + sgm) * m.segstep;
      const int n2 = (int)((f0 - a0 + m.seglen + 1) >> 1);
      for (int q = tid; q < n2; q += kMvNodes) {
        const int64_t f = a0 + 2 * q;
        if (f < 0 || f >= top) continue;
        __pipeline_memcpy_async(dst + 2 * q, x + f, 16);
        if (FUSE) __pipeline_memcpy_async(dst + half + 2 * q, pold + f, 16);
      }
    }
  }
  __pipeline_commit();
  __pipeline_wait_prior(0);
  __syncthreads();
  if (status != PCG_RUNNING) return;
  if (FUSE && !first) {
    double2 *z2 = reinterpret_cast<double2*>(xs), *q2 = reinterpret_cast<double2*>(xs + half);
    for (int q = tid; q < half / 2; q += kMvNodes) {
      const double2 zv = z2[q], pv = q2[q];
      z2[q] = make_double2(zv.x + beta * pv.x, zv.y + beta * pv.y);
    }
    __syncthreads();
  }
  double wl[4][3], wu[4][3];  // the elements below and above the node plane: [colour order][component]
  const bool io = i & 1, jo = j & 1;
  const double* xt = xs + 3 * (tid + 1);
#pragma unroll 1  // half the code: the unrolled body waits for instructions (4 % slower on 192x96x96)
  for (int sz = 0; sz < 2; ++sz) {
    const double* kz = ke.v + (1 - sz) * (4 * 3 * 24);  // KE rows of the node's local position in these elements
    const unsigned on4 = act >> (4 * sz);
    double e4[4];
    int o[2][3];
#pragma unroll
    for (int q = 0; q < 4; ++q) e4[q] = sz ? ee[4 + q] : ee[q];
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
      o[0][dy] = sz ? off[1][dy] : off[0][dy];
      o[1][dy] = sz ? off[2][dy] : off[1][dy];
    }
    double v[2][2][3];
#pragma unroll
    for (int sy = 0; sy < 2; ++sy)
#pragma unroll
      for (int sx = 0; sx < 2; ++sx) {
        const int el = sx + 2 * sy;
        const bool on = on4 >> el & 1;
        if (!__any_sync(0xffffffffu, on)) {
#pragma unroll
          for (int c = 0; c < 3; ++c) v[sy][sx][c] = 0.0;
          continue;
        }
        const int a = (1 - sy) ? ((1 - sx) ? 2 : 3) : ((1 - sx) ? 1 : 0);
        double s01[3], s[3], s23[3];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
          for (int t = 0; t < 6; ++t) {
            const int col = q + 4 * t, b = col / 3, cb = col % 3;
            const int bx = (b == 1 || b == 2 || b == 5 || b == 6) ? 1 : 0;
            const int by = (b == 2 || b == 3 || b == 6 || b == 7) ? 1 : 0;
            const int bz = b >= 4 ? 1 : 0;
            const double ue = xt[o[bz][sy + by] + 3 * (sx - 1 + bx) + cb] * e4[el];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const double pr = kz[(3 * a + c) * 24 + col] * ue;
              s[c] = t == 0 ? pr : s[c] + pr;
            }
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) {  // Vector256.Sum: (l0 + l1) + (l2 + l3)
            if (q == 0) s01[c] = s[c];
            else if (q == 1) s01[c] = s01[c] + s[c];
            else if (q == 2) s23[c] = s[c];
            else s23[c] = s23[c] + s[c];
          }
        }
        // an element that does not contribute adds +0, which leaves the running sum (never -0) as it is
#pragma unroll
        for (int c = 0; c < 3; ++c) v[sy][sx][c] = on ? s01[c] + s23[c] : 0.0;
      }
    // colour order: even element row first (sy = 0 when j is odd), in it the even element first
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double a0 = jo ? v[0][0][c] : v[1][0][c], a1 = jo ? v[0][1][c] : v[1][1][c];
      const double b0 = jo ? v[1][0][c] : v[0][0][c], b1 = jo ? v[1][1][c] : v[0][1][c];
      const double t0 = io ? a0 : a1, t1 = io ? a1 : a0, t2 = io ? b0 : b1, t3 = io ? b1 : b0;
      if (sz == 0) wl[0][c] = t0, wl[1][c] = t1, wl[2][c] = t2, wl[3][c] = t3;
      else wu[0][c] = t0, wu[1][c] = t1, wu[2][c] = t2, wu[3][c] = t3;
    }
  }
  if (!mine) return;
  double acc[3] = {0.0, 0.0, 0.0};
  if (k & 1) {  // the plane below has even elements
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[c] = acc[c] + (q < 4 ? wl : wu)[q & 3][c];
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[c] = acc[c] + (q < 4 ? wu : wl)[q & 3][c];
  }
  const int64_t nn = n + (int64_t)np * k;
  const uint8_t f = projected ? nf[nn] : 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double xv = xt[off[1][1] + c];
    y[3 * nn + c] = (f & (1 << c)) ? xv : acc[c];
    if (FUSE) pnew[3 * nn + c] = xv;
  }
}

template <int FUSE>
static void launch_mv(mycel_problem* p, const double* x, const double* pold, double* pnew, double* y, int projected,
                      const PcgState* st) {
  const GridDims& g = p->g;
  const unsigned chunks = (unsigned)(((int64_t)g.nx1 * g.ny1 + kMvNodes - 1) / kMvNodes);
  allow_smem<k_matvec64<FUSE>>(p->ctx->device, std::max(mv_smem(kMvNodes + 2, FUSE != 0), mv_smem(kMvNodes + 3, FUSE != 0)));
  // in the iteration an early dependent; E and the domain, which its first loads read, are older than the solve
  launch_dep(FUSE != 0 && dep_early(p), k_matvec64<FUSE>, chunks * (unsigned)g.nz1, kMvNodes,
             mv_smem(g.nx1, FUSE != 0), p->ctx->stream, g, p->ke, x, pold, pnew, y, p->d_E, p->d_domain, p->d_nflags,
             projected, st, chunks);
  p->ctx->launches++;
}

void launch_matvec64(mycel_problem* p, const double* x, double* y, int projected) {
  launch_mv<0>(p, x, nullptr, nullptr, y, projected, nullptr);
}

void launch_pcg_matvec(mycel_problem* p, int it) {
  launch_mv<1>(p, p->d_z, it & 1 ? p->d_p : p->d_p2, it & 1 ? p->d_p2 : p->d_p, p->d_ap, 1, p->d_state);
}

// ---------------------------------------------------------------------------------------------------------
// exact block/lane reductions
// ---------------------------------------------------------------------------------------------------------
// One CTA per 8192-block: producer warps form the products chunk by chunk and stage them in shared memory, a row
// per lane chain; lanes 0-3 of a warp run the sequential chains of a set.
// What bounds it is the chain: 2,048 dependent additions of 8.1 cycles (8.5 us at 1.965 GHz). Everything else is
// kept out of its way: a ring of kRing chunks is handed over by named barriers (no CTA-wide barrier stops a chain
// for a producer's loads), the producers' accesses are contiguous over a warp (their traffic delays the chain's
// loads: at a 32-byte stride the fused update's chain took 13.8 cycles an addition, now 11.7), and one group of
// producers keeps ahead of the chain (two, or all chunks resident, were slower). 96x48x24 elements (44 blocks):
// the direction's dot 22.0 -> 15.0 us, the fused update 30.8 -> 16.5 us; one block (30x10x4): 15.1 -> 9.2 and
// 22.5 -> 10.1 us; 192x96x96 (666 blocks, bound by memory): 39 and 74 us.
constexpr int kCh = 768;                         // elements per chunk
constexpr int kRing = 4;                         // chunks in shared memory
constexpr int kRow = kCh / 4 + 4;                // doubles per staged lane row (no bank conflicts)
constexpr int kProd = kCh / 4;                   // producer threads, two pairs of elements each
constexpr int chain_threads(int sets) { return 32 * sets + kProd; }
static_assert(2 * kRing < 15 && kProd % 32 == 0 && kRow % 8 == 4, "barrier ids 1 .. 2 kRing, 15 hands a set over");

template <int SETS>
__device__ __forceinline__ void nb_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(32 * SETS + kProd) : "memory");
}
template <int SETS>
__device__ __forceinline__ void nb_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(32 * SETS + kProd) : "memory");
}

// acc + row[0] + row[1] + ... + row[m - 1], in that order (m <= kProd). A whole row is unrolled, so that the loads
// run ahead of the additions (8.8 cycles an addition; loops over batches of 16 or 32 took 9.8 to 10.7).
__device__ __forceinline__ double chain_row(double acc, const double* row, int m) {
  const double2* r2 = reinterpret_cast<const double2*>(row);
  if (m == kProd) {
#pragma unroll
    for (int q = 0; q < kProd / 2; ++q) {
      const double2 v = r2[q];
      acc = acc + v.x;
      acc = acc + v.y;
    }
    return acc;
  }
  int q = 0;
  for (; q + 32 <= m; q += 32) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const double2 v = r2[q / 2 + k];
      acc = acc + v.x;
      acc = acc + v.y;
    }
  }
  for (; q < m; ++q) acc = acc + row[q];
  return acc;
}

// The chains of one block over np pairs of elements (np even), SETS chain sets. A producer thread takes the pairs h
// and h + kProd of a chunk (a warp's accesses are contiguous): load(q, h) fetches pair h as the thread's q-th,
// store(q, h, put) gives its products to put(set, second, value). Pair h's entries belong to lanes 2 (h & 1) and
// 2 (h & 1) + 1, column h >> 1. The caller has loaded the first chunk's pairs (first_pair) before it looks at the
// solve's status. Returns lane l's chain of set w in lane l of warp w.
template <int SETS>
__device__ __forceinline__ int first_pair() {
  return (int)threadIdx.x - 32 * SETS;
}

template <int SETS, class Load, class Store>
__device__ __forceinline__ double block_chains(int np, double (*buf)[SETS][4][kRow], Load&& load, Store&& store) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int nch = (np + 2 * kProd - 1) / (2 * kProd);
  double acc = 0.0;
  if (tid >= 32 * SETS) {
    const int pt = tid - 32 * SETS;
    for (int t = 0; t < nch; ++t) {
      if (t >= kRing) nb_sync<SETS>(1 + kRing + t % kRing);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = pt + q * kProd, h = 2 * kProd * t + c;
        if (h < np) store(q, h, [&](int set, int second, double v) { buf[t % kRing][set][2 * (c & 1) + second][c >> 1] = v; });
      }
      nb_arrive<SETS>(1 + t % kRing);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int h = 2 * kProd * (t + 1) + pt + q * kProd;
        if (h < np) load(q, h);
      }
    }
  } else {
    const int set = tid >> 5;
    for (int t = 0; t < nch; ++t) {
      nb_sync<SETS>(1 + t % kRing);
      if (lane < 4)
        acc = chain_row(acc, buf[t % kRing][set][lane], min(kProd, (np >> 1) - t * kProd));
      __syncwarp();
      if (t + kRing < nch) nb_arrive<SETS>(1 + kRing + t % kRing);
    }
  }
  return acc;
}

// The block partials' final sums, by warp 0 of the last CTA to arrive: lane 0 publishes the CTA's partials (s1
// only when SETS is 2) and counts it in; the last one's warp adds part[0], part[1], ... in block order (its lanes
// load 32 partials at once, shuffles keep the order). True in the last CTA's warp 0, whose lanes all get the sums.
// One block needs none of it.
template <int SETS>
__device__ __forceinline__ bool sum_blocks(double* part, unsigned* counter, double& s0, double& s1) {
  const unsigned nb = gridDim.x, lane = threadIdx.x & 31;
  if (nb == 1) {
    s0 = 0.0 + s0;
    s1 = 0.0 + s1;
    return true;
  }
  unsigned prev = 0;
  if (lane == 0) {
    part[blockIdx.x] = s0;
    if (SETS == 2) part[nb + blockIdx.x] = s1;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(counter) : "memory");
  }
  if (__shfl_sync(0xffffffffu, prev, 0) != nb - 1) return false;
  __threadfence();
  s0 = s1 = 0.0;
  double v0 = lane < nb ? ld_volatile(part + lane) : 0.0;
  double v1 = SETS == 2 && lane < nb ? ld_volatile(part + nb + lane) : 0.0;
  for (unsigned base = 0; base < nb; base += 32) {
    const unsigned nx = base + 32 + lane;  // the next 32 are on their way while these are added
    const double w0 = nx < nb ? ld_volatile(part + nx) : 0.0;
    const double w1 = SETS == 2 && nx < nb ? ld_volatile(part + nb + nx) : 0.0;
    const unsigned cnt = min(32u, nb - base);
#pragma unroll 8
    for (unsigned q = 0; q < cnt; ++q) {
      s0 = s0 + __shfl_sync(0xffffffffu, v0, q);
      if (SETS == 2) s1 = s1 + __shfl_sync(0xffffffffu, v1, q);
    }
    v0 = w0;
    v1 = w1;
  }
  return true;
}

// Phases of the single-chain dot kernel.
enum DotPhase : int { PH_PAP = 0, PH_INIT_RR = 1 };

__global__ void __launch_bounds__(chain_threads(1), 4) k_dot_exact(const double* a, const double* b,
                                                             int64_t n, double* part, PcgState* st, int phase) {
  __shared__ __align__(16) double buf[kRing][1][4][kRow];
  dep_begin();
  const int64_t start = (int64_t)blockIdx.x * kBlock;
  const int cnt = (int)min((int64_t)kBlock, n - start);
  const int vc4 = cnt & ~3;
  const int tid = threadIdx.x, lane = tid & 31;
  const double2 *a2 = reinterpret_cast<const double2*>(a + start), *b2 = reinterpret_cast<const double2*>(b + start);
  double2 av[2], bv[2];
  double tv = 0.0;  // the block's last n mod 4 entries' products (lanes 0-2 of warp 0), added after the chains
  if (tid < cnt - vc4) tv = a[start + vc4 + tid] * b[start + vc4 + tid];
  const double rho0 = st->rho0, bnorm = st->bnorm, tol = st->tol;
  const int iter = st->iter;
  auto load = [&](int q, int h) {
    av[q] = a2[h];
    bv[q] = b2[h];
  };
  const int status = st->status, np = vc4 >> 1, h0 = first_pair<1>();
  if (h0 >= 0 && h0 < np) load(0, h0);
  if (h0 >= 0 && h0 + kProd < np) load(1, h0 + kProd);
  if (status != PCG_RUNNING) return;
  const double acc = block_chains<1>(np, buf, load, [&](int q, int, auto&& put) {
    put(0, 0, av[q].x * bv[q].x);
    put(0, 1, av[q].y * bv[q].y);
  });
  if (tid >= 32) return;
  const double l0 = __shfl_sync(0xffffffffu, acc, 0), l1 = __shfl_sync(0xffffffffu, acc, 1);
  const double l2 = __shfl_sync(0xffffffffu, acc, 2), l3 = __shfl_sync(0xffffffffu, acc, 3);
  double sum = lane_sum(l0, l1, l2, l3), none = 0.0;
  for (int q = 0; q < cnt - vc4; ++q) sum = sum + __shfl_sync(0xffffffffu, tv, q);
  if (!sum_blocks<1>(part, &st->counter, sum, none) || lane != 0) return;
  st->counter = 0;
  if (phase == PH_PAP) {
    st->iter = iter + 1;
    st->first = 0;
    double pap = sum;
    st->pap = pap;
    if (!(pap > 1e-30) || !isfinite(pap)) {
      st->last_bad = pap;
      st->status = PCG_BREAK_CURVATURE;
      return;
    }
    double alpha = rho0 / pap;
    if (!isfinite(alpha) || alpha <= 0.0) {
      st->last_bad = alpha;
      st->status = PCG_BREAK_ALPHA;
      return;
    }
    st->alpha = alpha;
  } else {  // PH_INIT_RR: rNormSq for a non-zero warm start (PcgSolver.cs:176-197)
    st->rn2 = sum;
    double rel = sqrt(sum) / bnorm;
    st->rel = rel;
    st->prev = rel;
    if (rel <= tol) st->status = PCG_INIT_CONVERGED;
  }
}

// Fused x/r update with ||r||^2 and z = r*invD with r.z. INIT: only the z part (rho0; the first direction is z).
template <int INIT>
__global__ void __launch_bounds__(chain_threads(2), 3) k_xr_exact(double* __restrict__ x, double* __restrict__ r,
                                                            double* __restrict__ z, const double* p,
                                                            const double* ap,
                                                            const double* __restrict__ invd, int64_t n, double* part,
                                                            PcgState* st) {
  extern __shared__ __align__(16) double xr_buf[];
  auto buf = reinterpret_cast<double (*)[2][4][kRow]>(xr_buf);  // sets: r.r (not used at a start), r.z
  __shared__ double rz_sum;
  dep_begin();
  const int64_t start = (int64_t)blockIdx.x * kBlock;
  const int cnt = (int)min((int64_t)kBlock, n - start);
  const int vc4 = cnt & ~3;
  const int tid = threadIdx.x, lane = tid & 31;
  const int status = st->status;
  const double alpha = st->alpha;
  double2 *x2 = reinterpret_cast<double2*>(x + start), *r2 = reinterpret_cast<double2*>(r + start),
          *z2 = reinterpret_cast<double2*>(z + start);
  const double2 *p2 = reinterpret_cast<const double2*>(p + start), *q2 = reinterpret_cast<const double2*>(ap + start),
                *d2 = reinterpret_cast<const double2*>(invd + start);
  double2 xv[2], rv[2], pv[2], qv[2], dv[2];
  // the block's last n mod 4 entries, by lanes 0-2 of warp 0 (their terms are added after the chains)
  const int64_t tj = start + vc4 + tid;
  const bool tail = tid < cnt - vc4;
  double tr = 0.0, tx = 0.0, tp = 0.0, tap = 0.0, td = 0.0;
  if (tail) {
    tr = r[tj];
    td = invd[tj];
    if (!INIT) tx = x[tj], tp = p[tj], tap = ap[tj];
  }
  const double rho0 = st->rho0, bnorm = st->bnorm, tol = st->tol, prev = st->prev;
  const int iter = st->iter, max_iter = st->max_iter, stag = st->stag;
  auto load = [&](int q, int h) {
    rv[q] = r2[h];
    dv[q] = d2[h];
    if (!INIT) {
      qv[q] = q2[h];
      pv[q] = p2[h];
      xv[q] = x2[h];
    }
  };
  const int np = vc4 >> 1, h0 = first_pair<2>();
  if (h0 >= 0 && h0 < np) load(0, h0);
  if (h0 >= 0 && h0 + kProd < np) load(1, h0 + kProd);
  if (status != PCG_RUNNING) return;
  const double acc = block_chains<2>(np, buf, load, [&](int q, int h, auto&& put) {
    double2 rn = rv[q];
    if (!INIT) {
      x2[h] = make_double2(xv[q].x + alpha * pv[q].x, xv[q].y + alpha * pv[q].y);
      rn = make_double2(rv[q].x - alpha * qv[q].x, rv[q].y - alpha * qv[q].y);
      r2[h] = rn;
    }
    const double2 zn = make_double2(rn.x * dv[q].x, rn.y * dv[q].y);
    z2[h] = zn;
    put(0, 0, rn.x * rn.x);
    put(0, 1, rn.y * rn.y);
    put(1, 0, rn.x * zn.x);
    put(1, 1, rn.y * zn.y);
  });
  if (tid >= 64) return;
  const double l0 = __shfl_sync(0xffffffffu, acc, 0), l1 = __shfl_sync(0xffffffffu, acc, 1);
  const double l2 = __shfl_sync(0xffffffffu, acc, 2), l3 = __shfl_sync(0xffffffffu, acc, 3);
  double rn2 = lane_sum(l0, l1, l2, l3);  // warp 0: r.r; warp 1: r.z, handed over
  if (tid == 32) rz_sum = rn2;
  asm volatile("bar.sync 15, 64;" ::: "memory");
  if (tid >= 32) return;
  double rho1 = rz_sum, trr = 0.0, trz = 0.0;
  if (tail) {
    if (!INIT) {
      x[tj] = tx + alpha * tp;
      tr = tr - alpha * tap;
      r[tj] = tr;
      trr = tr * tr;
    }
    const double tz = tr * td;
    z[tj] = tz;
    trz = tr * tz;
  }
  for (int q = 0; q < cnt - vc4; ++q) {
    rn2 = rn2 + __shfl_sync(0xffffffffu, trr, q);
    rho1 = rho1 + __shfl_sync(0xffffffffu, trz, q);
  }
  if (!sum_blocks<2>(part, &st->counter, rn2, rho1) || lane != 0) return;
  st->counter = 0;
  if (INIT) {
    st->rho0 = rho1;
    st->first = 1;
    if (max_iter <= 0) st->status = PCG_MAXITER;
    return;
  }
  st->rn2 = rn2;
  double rel = sqrt(rn2) / bnorm;
  st->rel = rel;
  if (rel <= tol) {
    st->status = PCG_CONVERGED;
    return;
  }
  if (fabs(rel - prev) < 1e-15 * rel) {
    st->stag = stag + 1;
    if (stag + 1 > 50) {
      st->status = PCG_STAGNATED;
      return;
    }
  } else {
    st->stag = 0;
  }
  st->prev = rel;
  double beta = rho1 / rho0;
  if (!isfinite(beta) || beta < 0.0) {
    st->last_bad = beta;
    st->status = PCG_BREAK_BETA;
    return;
  }
  st->beta = beta;
  st->rho0 = rho1;
  if (iter >= max_iter) st->status = PCG_MAXITER;
}

static void launch_dot(mycel_problem* p, const double* a, const double* b, int phase) {
  launch_dep(dep_early(p), k_dot_exact, (unsigned)num_blocks8192(p->g.nd), chain_threads(1), 0, p->ctx->stream, a, b,
             p->g.nd, p->d_part, p->d_state, phase);
  p->ctx->launches++;
}

template <int INIT>
static void launch_xr(mycel_problem* p, const double* dir) {
  constexpr size_t smem = sizeof(double) * kRing * 2 * 4 * kRow;
  allow_smem<k_xr_exact<INIT>>(p->ctx->device, smem);
  launch_dep(dep_early(p), k_xr_exact<INIT>, (unsigned)num_blocks8192(p->g.nd), chain_threads(2), smem,
             p->ctx->stream, p->d_x, p->d_r, p->d_z, dir, p->d_ap, p->d_invd, p->g.nd, p->d_part, p->d_state);
  p->ctx->launches++;
}

// x projection (PcgSolver.cs:113-125) and "has non-zero x" flag
__global__ void k_project_x(int64_t nd, const uint8_t* __restrict__ nf, double* x, int* flag) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int nz = 0;
  if (i < nd) {
    if (nf[i / 3] & (1 << (i % 3))) x[i] = 0.0;
    else nz = x[i] != 0.0;
  }
  if (__syncthreads_or(nz) && threadIdx.x == 0) atomicOr(flag, 1);
}

// ||P b||^2: the reference adds b_i^2 over unconstrained i in index order; zero terms leave the running sum
// unchanged, so the sum over the ascending list of non-zero P b entries is the same number.
__global__ void k_bnorm_list(const double* __restrict__ b, const int32_t* __restrict__ idx, int32_t cnt,
                             PcgState* st) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double s = 0.0;
  constexpr int kB = 16;  // loads of 16 entries issued before they are added, in list order
  for (int32_t q0 = 0; q0 < cnt; q0 += kB) {
    double v[kB];
#pragma unroll
    for (int k = 0; k < kB; ++k) v[k] = q0 + k < cnt ? b[idx[q0 + k]] : 0.0;
#pragma unroll
    for (int k = 0; k < kB; ++k)
      if (q0 + k < cnt) s = s + v[k] * v[k];
  }
  st->bn2 = s;
  st->bnorm = sqrt(s);
}

void launch_project_x(mycel_problem* p, double* x, int* d_flag) {
  k_project_x<<<(unsigned)((p->g.nd + 255) / 256), 256, 0, p->ctx->stream>>>(p->g.nd, p->d_nflags, x, d_flag);
  p->ctx->launches++;
}

void launch_pcg_bnorm(mycel_problem* p) {
  k_bnorm_list<<<1, 32, 0, p->ctx->stream>>>(p->d_b, p->d_bnz, p->n_bnz, p->d_state);
  p->ctx->launches++;
}

// r = P(b - A x) or P b (PcgSolver.cs:176-192)
__global__ void k_init_r(int64_t nd, const uint8_t* __restrict__ nf, const double* __restrict__ b,
                         const double* __restrict__ ap, double* __restrict__ r, int nonzero) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nd) return;
  bool con = nf[i / 3] & (1 << (i % 3));
  r[i] = con ? 0.0 : (nonzero ? (b[i] - ap[i]) : b[i]);
}

void launch_pcg_init_r(mycel_problem* p, int nonzero) {
  k_init_r<<<(unsigned)((p->g.nd + 255) / 256), 256, 0, p->ctx->stream>>>(p->g.nd, p->d_nflags, p->d_b, p->d_ap,
                                                                         p->d_r, nonzero);
  p->ctx->launches++;
}

void launch_pcg_dot_rr(mycel_problem* p) {
  launch_dot(p, p->d_r, p->d_r, PH_INIT_RR);
}

void launch_pcg_init_z(mycel_problem* p) { launch_xr<1>(p, nullptr); }

// PCG iteration `it` (PcgSolver.cs:235-357): p = z + beta p and Ap = A p (the direction alternates between two
// buffers, d_p in even iterations); pAp, alpha; x, r, ||r||; z, rho1, beta.
void launch_pcg_iteration(mycel_problem* p, int it, bool skip_matvec) {
  const double* dir = it & 1 ? p->d_p2 : p->d_p;
  if (!skip_matvec) launch_pcg_matvec(p, it);
  launch_dot(p, dir, p->d_ap, PH_PAP);
  launch_xr<0>(p, dir);
}

// ---------------------------------------------------------------------------------------------------------
// compliance C = F.u (sequential over non-zero F in index order), max |u| over active nodes, reactions
// ---------------------------------------------------------------------------------------------------------
__global__ void k_compliance(const double* __restrict__ F, const double* __restrict__ u,
                             const int32_t* __restrict__ idx, int32_t cnt, double* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double c = 0.0;
  constexpr int kB = 16;  // loads of 16 terms issued before they are added, in list order
  for (int32_t q0 = 0; q0 < cnt; q0 += kB) {
    double fv[kB], uv[kB];
#pragma unroll
    for (int k = 0; k < kB; ++k) {
      const int32_t j = q0 + k < cnt ? idx[q0 + k] : 0;
      fv[k] = q0 + k < cnt ? F[j] : 0.0;
      uv[k] = q0 + k < cnt ? u[j] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kB; ++k)
      if (q0 + k < cnt) c = c + fv[k] * uv[k];
  }
  *out = c;
}

void launch_compliance(mycel_problem* p, const double* u, double* d_out) {
  launch_compliance(p, p->d_F, p->d_fnz, p->n_fnz, u, d_out);
}

void launch_compliance(mycel_problem* p, const double* F, const int32_t* fnz, int32_t n_fnz, const double* u,
                       double* d_out) {
  k_compliance<<<1, 32, 0, p->ctx->stream>>>(F, u, fnz, n_fnz, d_out);
  p->ctx->launches++;
}

__device__ __forceinline__ unsigned long long dbl_key(double v) {
  // non-negative doubles order like their bit patterns
  return (unsigned long long)__double_as_longlong(v);
}

__global__ void k_max_disp(GridDims g, const uint8_t* __restrict__ nf, const double* __restrict__ u,
                           unsigned long long* out) {
  double m = 0.0;
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < g.nn; n += (int64_t)gridDim.x * blockDim.x) {
    if (!(nf[n] & NF_ACTIVE)) continue;
    double ux = u[3 * n], uy = u[3 * n + 1], uz = u[3 * n + 2];
    double s = ux * ux + uy * uy + uz * uz;
    if (s > m) m = s;
  }
  for (int o = 16; o > 0; o >>= 1) {
    double v = __shfl_down_sync(0xffffffffu, m, o);
    if (v > m) m = v;
  }
  if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(out, dbl_key(m));
}

__global__ void k_sqrt_inplace(unsigned long long* v) {
  double d = __longlong_as_double((long long)*v);
  *(double*)v = sqrt(d);
}

void launch_max_disp(mycel_problem* p, const double* u, double* d_out) { launch_max_disp(p, &u, 1, 0, d_out); }

// largest |u| over the active nodes of m displacement vectors, u[k] at us[k] + k * stride
void launch_max_disp(mycel_problem* p, const double* const* us, int m, int64_t stride, double* d_out) {
  cudaMemsetAsync(d_out, 0, sizeof(double), p->ctx->stream);
  int blocks = std::max(1, std::min<int>((int)((p->g.nn + 255) / 256), p->ctx->num_sms * 8));
  for (int k = 0; k < m; ++k)
    k_max_disp<<<blocks, 256, 0, p->ctx->stream>>>(p->g, p->d_nflags, stride ? us[0] + k * stride : us[k],
                                                   (unsigned long long*)d_out);
  k_sqrt_inplace<<<1, 1, 0, p->ctx->stream>>>((unsigned long long*)d_out);
  p->ctx->launches += 1 + m;
}

__global__ void k_reactions(const double* __restrict__ ku, double* out, const int32_t* __restrict__ fixed, int32_t nf) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nf) out[fixed[t]] = ku[fixed[t]];
}

void launch_reactions(mycel_problem* p, const double* ku, double* out, const int32_t* d_fixed, int32_t n_fixed) {
  cudaMemsetAsync(out, 0, sizeof(double) * p->g.nd, p->ctx->stream);
  if (n_fixed > 0) {
    k_reactions<<<(n_fixed + 255) / 256, 256, 0, p->ctx->stream>>>(ku, out, d_fixed, n_fixed);
    p->ctx->launches++;
  }
}

// Element von Mises at the centroid (StaticAnalysis.cs:144-216)
struct VmConst {
  double bc[144];
  double d[36];
  double invh;
};
__global__ void k_von_mises(GridDims g, const __grid_constant__ VmConst vc, const double* __restrict__ u, const double* __restrict__ E,
                            const uint8_t* __restrict__ dom, double* __restrict__ vm) {
  int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= g.ne) return;
  if (!dom[e]) {
    vm[e] = 0.0;
    return;
  }
  int ix = (int)(e % g.nx);
  int64_t r = e / g.nx;
  int iy = (int)(r % g.ny), iz = (int)(r / g.ny);
  const int64_t sy = g.nx1, sz = (int64_t)g.nx1 * g.ny1;
  int64_t n0 = ix + sy * iy + sz * iz;
  const int64_t off[8] = {0, 1, 1 + sy, sy, sz, sz + 1, sz + 1 + sy, sz + sy};
  double ue[24];
  for (int b = 0; b < 8; ++b)
    for (int c = 0; c < 3; ++c) ue[3 * b + c] = u[3 * (n0 + off[b]) + c];
  double eps[6], sig[6];
  for (int q = 0; q < 6; ++q) {
    double s = 0.0;
    for (int k = 0; k < 24; ++k) s = s + vc.bc[q * 24 + k] * ue[k];
    eps[q] = s * vc.invh;
  }
  double ee = E[e];
  for (int q = 0; q < 6; ++q) {
    double s = 0.0;
    for (int k = 0; k < 6; ++k) s = s + vc.d[q * 6 + k] * eps[k];
    sig[q] = s * ee;
  }
  double d1 = sig[0] - sig[1], d2 = sig[1] - sig[2], d3 = sig[2] - sig[0];
  vm[e] = sqrt(0.5 * (d1 * d1 + d2 * d2 + d3 * d3) + 3.0 * (sig[3] * sig[3] + sig[4] * sig[4] + sig[5] * sig[5]));
}

void launch_von_mises(mycel_problem* p, const double* u, double* vm) {
  VmConst vc;
  // Hex8Element.BaseBc = EvaluateB(0,0,0,h=1) (Hex8Element.cs:71, :183-215)
  static const double xi[8] = {-1, 1, 1, -1, -1, 1, 1, -1}, eta[8] = {-1, -1, 1, 1, -1, -1, 1, 1},
                      zeta[8] = {-1, -1, -1, -1, 1, 1, 1, 1};
  for (int i = 0; i < 144; ++i) vc.bc[i] = 0.0;
  for (int a = 0; a < 8; ++a) {
    double dx = (0.25 * 1.0) * xi[a] * (1.0 + eta[a] * 0.0) * (1.0 + zeta[a] * 0.0);
    double dy = (0.25 * 1.0) * eta[a] * (1.0 + xi[a] * 0.0) * (1.0 + zeta[a] * 0.0);
    double dz = (0.25 * 1.0) * zeta[a] * (1.0 + xi[a] * 0.0) * (1.0 + eta[a] * 0.0);
    vc.bc[0 * 24 + 3 * a] = dx; vc.bc[1 * 24 + 3 * a + 1] = dy; vc.bc[2 * 24 + 3 * a + 2] = dz;
    vc.bc[3 * 24 + 3 * a + 1] = dz; vc.bc[3 * 24 + 3 * a + 2] = dy;
    vc.bc[4 * 24 + 3 * a] = dz; vc.bc[4 * 24 + 3 * a + 2] = dx;
    vc.bc[5 * 24 + 3 * a] = dy; vc.bc[5 * 24 + 3 * a + 1] = dx;
  }
  double nu = p->nu;
  double factor = 1.0 / ((1.0 + nu) * (1.0 - 2.0 * nu));
  double c1 = factor * (1.0 - nu), c2 = factor * nu, c3 = 1.0 / (2.0 * (1.0 + nu));
  for (int i = 0; i < 36; ++i) vc.d[i] = 0.0;
  vc.d[0] = c1; vc.d[1] = c2; vc.d[2] = c2; vc.d[6] = c2; vc.d[7] = c1; vc.d[8] = c2;
  vc.d[12] = c2; vc.d[13] = c2; vc.d[14] = c1; vc.d[21] = c3; vc.d[28] = c3; vc.d[35] = c3;
  vc.invh = 1.0 / (double)p->h;
  k_von_mises<<<(unsigned)((p->g.ne + 255) / 256), 256, 0, p->ctx->stream>>>(p->g, vc, u, p->d_E, p->d_domain, vm);
  p->ctx->launches++;
}

// StaticAnalysis.AverageElementToNode (Fem/StaticAnalysis.cs:222-268): per node, the mean of the scalars of the
// active elements meeting there, 0 where none does. A node gathers its (up to 8) elements in increasing element
// index, the order in which the reference's element loop adds to the node's sum, so the sums are bit-identical.
__global__ void k_avg_e2n(GridDims g, const double* __restrict__ es, const uint8_t* __restrict__ dom,
                          double* __restrict__ out) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= g.nn) return;
  const int i = (int)(n % g.nx1), j = (int)((n / g.nx1) % g.ny1), k = (int)(n / ((int64_t)g.nx1 * g.ny1));
  double sum = 0.0;
  int cnt = 0;
  for (int ez = k - 1; ez <= k; ++ez)
    for (int ey = j - 1; ey <= j; ++ey)
      for (int ex = i - 1; ex <= i; ++ex) {
        if (ex < 0 || ey < 0 || ez < 0 || ex >= g.nx || ey >= g.ny || ez >= g.nz) continue;
        const int64_t e = ex + (int64_t)g.nx * (ey + (int64_t)g.ny * ez);
        if (!dom[e]) continue;
        sum = sum + es[e];
        cnt++;
      }
  out[n] = cnt > 0 ? sum / (double)cnt : 0.0;
}

void launch_average_e2n(mycel_problem* p, const double* es, double* out) {
  k_avg_e2n<<<(unsigned)((p->g.nn + 255) / 256), 256, 0, p->ctx->stream>>>(p->g, es, p->d_domain, out);
  p->ctx->launches++;
}

// active <-> box index maps
__global__ void k_scatter_active(int64_t na, const int32_t* __restrict__ act, const double* __restrict__ src,
                                 double* __restrict__ dst) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < na) dst[act[t]] = src[t];
}
__global__ void k_gather_active(int64_t na, const int32_t* __restrict__ act, const double* __restrict__ src,
                                double* __restrict__ dst) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < na) dst[t] = src[act[t]];
}
__global__ void k_fill(int64_t n, double* p, double v) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < n) p[t] = v;
}

void launch_scatter_active(mycel_problem* p, const double* src_active, double* dst_box, double fill) {
  k_fill<<<(unsigned)((p->g.ne + 255) / 256), 256, 0, p->ctx->stream>>>(p->g.ne, dst_box, fill);
  p->ctx->launches++;
  if (p->n_active == 0) return;
  k_scatter_active<<<(unsigned)((p->n_active + 255) / 256), 256, 0, p->ctx->stream>>>(p->n_active, p->d_active,
                                                                                      src_active, dst_box);
  p->ctx->launches++;
}

void launch_gather_active(mycel_problem* p, const double* src_box, double* dst_active) {
  if (p->n_active == 0) return;
  k_gather_active<<<(unsigned)((p->n_active + 255) / 256), 256, 0, p->ctx->stream>>>(p->n_active, p->d_active,
                                                                                     src_box, dst_active);
  p->ctx->launches++;
}

// ---------------------------------------------------------------------------------------------------------
// Density filter as a stencil (DensityFilter.cs:61-198)
// ---------------------------------------------------------------------------------------------------------
// invHs per active element: hs accumulated over included neighbours in loop order.
__global__ void k_filter_invhs(GridDims g, const uint8_t* __restrict__ dom, const int4* __restrict__ off,
                               const double* __restrict__ w, int noff, double* __restrict__ invhs) {
  int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= g.ne || !dom[e]) return;
  int ex = (int)(e % g.nx);
  int64_t r = e / g.nx;
  int ey = (int)(r % g.ny), ez = (int)(r / g.ny);
  double hs = 0.0;
  for (int q = 0; q < noff; ++q) {
    int4 o = off[q];
    int jx = ex + o.x, jy = ey + o.y, jz = ez + o.z;
    if (jx < 0 || jx >= g.nx || jy < 0 || jy >= g.ny || jz < 0 || jz >= g.nz) continue;
    if (!dom[jx + (int64_t)g.nx * (jy + (int64_t)g.ny * jz)]) continue;
    hs = hs + w[q];
  }
  invhs[e] = hs > 0.0 ? 1.0 / hs : 1.0;
}

// forward: out_r = sum_j (w_rj * invHs_r) * in_j, j in loop order.
// adjoint: out_i = sum_r (w_ri * invHs_r) * in_r, r ascending (the adjoint CSR rows are filled in forward-row
//          order, DensityFilter.cs:172-185); with in = 1 this is S_i (:188-198).
template <int ADJ>
__global__ void k_filter_apply(GridDims g, const uint8_t* __restrict__ dom, const int4* __restrict__ off,
                               const double* __restrict__ w, int noff, const double* __restrict__ invhs,
                               const double* __restrict__ in, double* __restrict__ out, int ones) {
  int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= g.ne || !dom[e]) return;
  int ex = (int)(e % g.nx);
  int64_t r = e / g.nx;
  int ey = (int)(r % g.ny), ez = (int)(r / g.ny);
  double s = 0.0;
  const double ih = invhs[e];
  for (int q = 0; q < noff; ++q) {
    int4 o = off[q];
    int jx = ex + o.x, jy = ey + o.y, jz = ez + o.z;
    if (jx < 0 || jx >= g.nx || jy < 0 || jy >= g.ny || jz < 0 || jz >= g.nz) continue;
    int64_t j = jx + (int64_t)g.nx * (jy + (int64_t)g.ny * jz);
    if (!dom[j]) continue;
    if (ADJ) {
      double wt = w[q] * invhs[j];
      s = s + (ones ? wt : wt * in[j]);
    } else {
      s = s + (w[q] * ih) * in[j];
    }
  }
  out[e] = s;
}

// The forward filter as a shared-memory stencil: a CTA stages a 32 x 8 x 2 element tile with an rc-element halo
// (the input and the element flags; outside the grid or inactive: flag 0) and the offset list as index steps,
// then each thread forms its elements' sums from shared memory in the reference's neighbour order with the same
// operations, so the results are those of k_filter_apply<0> bit for bit (206 -> 147 us on the 192x96x96
// bridge). The adjoint stays per element: staged with 1/Hs its tile needs 74 KB, and at the occupancy that
// leaves it ran slower (237 against 201 us).
constexpr int kFtX = 32, kFtY = 8, kFtZ = 2;

__host__ __device__ inline size_t filter_tile_smem(int rc, int noff) {
  const size_t nt = (size_t)(kFtX + 2 * rc) * (kFtY + 2 * rc) * (kFtZ + 2 * rc);
  size_t b = nt * 8;
  b = (b + 15) & ~(size_t)15;
  b += (size_t)noff * 8 + (size_t)noff * 4 + nt;
  return b;
}

__global__ void __launch_bounds__(256) k_filter_tile(GridDims g, int rc, const uint8_t* __restrict__ dom,
                                                     const int4* __restrict__ off, const double* __restrict__ w,
                                                     int noff, const double* __restrict__ invhs,
                                                     const double* __restrict__ in, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char ftile[];
  const int PX = kFtX + 2 * rc, PY = kFtY + 2 * rc, PZ = kFtZ + 2 * rc, nt = PX * PY * PZ;
  double* sv = reinterpret_cast<double*>(ftile);
  size_t ob = (size_t)nt * 8;
  ob = (ob + 15) & ~(size_t)15;
  double* sw = reinterpret_cast<double*>(ftile + ob);
  int* so = reinterpret_cast<int*>(sw + noff);  // offsets as shared-memory index steps
  uint8_t* sd = reinterpret_cast<uint8_t*>(so + noff);
  const int tid = threadIdx.x;
  const int x0 = blockIdx.x * kFtX - rc, y0 = blockIdx.y * kFtY - rc, z0 = blockIdx.z * kFtZ - rc;
  for (int i = tid; i < nt; i += blockDim.x) {
    const int gx = x0 + i % PX, gy = y0 + (i / PX) % PY, gz = z0 + i / (PX * PY);
    uint8_t d = 0;
    double v = 0.0;
    if (gx >= 0 && gx < g.nx && gy >= 0 && gy < g.ny && gz >= 0 && gz < g.nz) {
      const int64_t j = gx + (int64_t)g.nx * (gy + (int64_t)g.ny * gz);
      d = dom[j];
      if (d) v = in[j];
    }
    sd[i] = d;
    sv[i] = v;
  }
  for (int q = tid; q < noff; q += blockDim.x) {
    const int4 o = off[q];
    so[q] = o.x + PX * (o.y + PY * o.z);
    sw[q] = w[q];
  }
  __syncthreads();
  const int tx = tid % kFtX, ty = tid / kFtX;
  for (int tz = 0; tz < kFtZ; ++tz) {
    const int ex = blockIdx.x * kFtX + tx, ey = blockIdx.y * kFtY + ty, ez = blockIdx.z * kFtZ + tz;
    if (ex >= g.nx || ey >= g.ny || ez >= g.nz) continue;
    const int li = (tx + rc) + PX * ((ty + rc) + PY * (tz + rc));
    if (!sd[li]) continue;
    const int64_t e = ex + (int64_t)g.nx * (ey + (int64_t)g.ny * ez);
    double s = 0.0;
    const double ih = invhs[e];
#pragma unroll 4
    for (int q = 0; q < noff; ++q) {
      const int lj = li + so[q];
      if (!sd[lj]) continue;
      s = s + (sw[q] * ih) * sv[lj];
    }
    out[e] = s;
  }
}

// largest shared-memory tile a CTA may use; beyond it (large filter radii) the per-element kernel runs
constexpr size_t kFilterTileMax = 200 * 1024;

static bool filter_tiled(mycel_filter* f) {
  static std::once_flag once;
  static bool ok = false;
  std::call_once(once, [] {
    ok = cudaFuncSetAttribute(k_filter_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFilterTileMax) ==
         cudaSuccess;
    cudaGetLastError();
  });
  return ok && filter_tile_smem(f->rc, f->n_off) <= kFilterTileMax;
}

static dim3 filter_tile_grid(const GridDims& g) {
  return dim3((unsigned)((g.nx + kFtX - 1) / kFtX), (unsigned)((g.ny + kFtY - 1) / kFtY),
              (unsigned)((g.nz + kFtZ - 1) / kFtZ));
}

int filter_setup(mycel_filter* f) {
  mycel_problem* p = f->p;
  double rmin = f->rmin;
  int rc = (int)ceil(rmin);
  double rsq = rmin * rmin;
  std::vector<int4> offs;
  std::vector<double> ws;
  for (int dz = -rc; dz <= rc; ++dz)
    for (int dy = -rc; dy <= rc; ++dy)
      for (int dx = -rc; dx <= rc; ++dx) {
        int ds = dz * dz + dy * dy + dx * dx;
        if (!((double)ds < rsq)) continue;
        double dist = sqrt((double)ds);
        if (!(dist < rmin)) continue;
        offs.push_back(make_int4(dx, dy, dz, 0));
        ws.push_back(rmin - dist);
      }
  f->n_off = (int)offs.size();
  f->rc = rc;
  cudaStream_t s = p->ctx->stream;
  if (cudaMallocAsync(&f->d_off, sizeof(int4) * offs.size(), s) != cudaSuccess) return MYCEL_E_OOM;
  if (cudaMallocAsync(&f->d_w, sizeof(double) * ws.size(), s) != cudaSuccess) return MYCEL_E_OOM;
  if (cudaMallocAsync(&f->d_invhs, sizeof(double) * p->g.ne, s) != cudaSuccess) return MYCEL_E_OOM;
  if (cudaMallocAsync(&f->d_s, sizeof(double) * p->g.ne, s) != cudaSuccess) return MYCEL_E_OOM;
  p->device_bytes += (int64_t)(sizeof(int4) * offs.size() + sizeof(double) * ws.size() + 16 * p->g.ne);
  cudaMemcpyAsync(f->d_off, offs.data(), sizeof(int4) * offs.size(), cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(f->d_w, ws.data(), sizeof(double) * ws.size(), cudaMemcpyHostToDevice, s);
  cudaMemsetAsync(f->d_invhs, 0, sizeof(double) * p->g.ne, s);
  cudaMemsetAsync(f->d_s, 0, sizeof(double) * p->g.ne, s);
  unsigned nb = (unsigned)((p->g.ne + 127) / 128);
  k_filter_invhs<<<nb, 128, 0, s>>>(p->g, p->d_domain, f->d_off, f->d_w, f->n_off, f->d_invhs);
  k_filter_apply<1><<<nb, 128, 0, s>>>(p->g, p->d_domain, f->d_off, f->d_w, f->n_off, f->d_invhs, nullptr, f->d_s, 1);
  p->ctx->launches += 2;
  cudaError_t le = cudaGetLastError();
  cudaError_t se = cudaStreamSynchronize(s);  // host vectors above must outlive the copies
  if (le != cudaSuccess || se != cudaSuccess) {
    set_error(p->ctx, MYCEL_E_DEVICE, std::string("filter set-up: ") +
                                          cudaGetErrorString(le != cudaSuccess ? le : se));
    return MYCEL_E_DEVICE;
  }
  return MYCEL_OK;
}

void launch_filter_fwd(mycel_filter* f, const double* in_box, double* out_box) {
  mycel_problem* p = f->p;
  if (filter_tiled(f))
    k_filter_tile<<<filter_tile_grid(p->g), 256, filter_tile_smem(f->rc, f->n_off), p->ctx->stream>>>(
        p->g, f->rc, p->d_domain, f->d_off, f->d_w, f->n_off, f->d_invhs, in_box, out_box);
  else
    k_filter_apply<0><<<(unsigned)((p->g.ne + 127) / 128), 128, 0, p->ctx->stream>>>(
        p->g, p->d_domain, f->d_off, f->d_w, f->n_off, f->d_invhs, in_box, out_box, 0);
  p->ctx->launches++;
}

void launch_filter_adj(mycel_filter* f, const double* in_box, double* out_box) {
  mycel_problem* p = f->p;
  k_filter_apply<1><<<(unsigned)((p->g.ne + 127) / 128), 128, 0, p->ctx->stream>>>(
      p->g, p->d_domain, f->d_off, f->d_w, f->n_off, f->d_invhs, in_box, out_box, 0);
  p->ctx->launches++;
}

// ---------------------------------------------------------------------------------------------------------
// compliance sensitivities dc/drhoBar_e = -(p rho^(p-1) dE) * ue^T KE ue   (SensitivityAnalysis.cs:98-144)
// ---------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_sens(GridDims g, const __grid_constant__ KeD ke, const double* __restrict__ u,
                                              const double* __restrict__ rho, const uint8_t* __restrict__ dom,
                                              double penal, double dE, double* __restrict__ dc, int accumulate) {
  int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= g.ne || !dom[e]) return;
  int ix = (int)(e % g.nx);
  int64_t r = e / g.nx;
  int iy = (int)(r % g.ny), iz = (int)(r / g.ny);
  const int64_t sy = g.nx1, sz = (int64_t)g.nx1 * g.ny1;
  int64_t n0 = ix + sy * iy + sz * iz;
  const int64_t off[8] = {0, 1, 1 + sy, sy, sz, sz + 1, sz + 1 + sy, sz + sy};
  double ue[24];
#pragma unroll
  for (int b = 0; b < 8; ++b)
#pragma unroll
    for (int c = 0; c < 3; ++c) ue[3 * b + c] = __ldg(u + 3 * (n0 + off[b]) + c);
  double se = 0.0;
#pragma unroll
  for (int rr = 0; rr < 24; ++rr) {
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 24; ++c) s = s + ke.v[rr * 24 + c] * ue[c];
    se = se + ue[rr] * s;
  }
  double dEdr = penal * path_pow(rho[e], penal - 1.0) * dE;
  const double v = -dEdr * se;
  dc[e] = accumulate ? dc[e] + v : v;  // load cases apart: summed over the cases in case order
}

void launch_sens(mycel_problem* p, const double* u, const double* rho_box, double penal, double* dc_box,
                 bool accumulate) {
  k_sens<<<(unsigned)((p->g.ne + 127) / 128), 128, 0, p->ctx->stream>>>(p->g, p->ke, u, rho_box, p->d_domain, penal,
                                                                        p->e0 - p->emin, dc_box, accumulate ? 1 : 0);
  p->ctx->launches++;
}

// ---------------------------------------------------------------------------------------------------------
// HeavisideProjection (Optimization/HeavisideProjection.cs:12-37), an option of TopologyOptimizer.Run
// (:192-199, :279-290): the reference's expression order, every operation rounded once (this unit is built
// without contraction); Math.Clamp lets NaN through and Math.Max propagates it, as here. tanh is CUDA's, which
// can differ from the C library's in the last bit.
// ---------------------------------------------------------------------------------------------------------
__global__ void k_heaviside(int64_t n, const int32_t* __restrict__ idx, const double* __restrict__ rt,
                            const double* __restrict__ dcb, double* __restrict__ out, double beta, double eta,
                            int mode) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t e = idx ? (int64_t)idx[t] : t;
  const double den = tanh(beta * eta) + tanh(beta * (1.0 - eta));
  const double inv = 1.0 / den;
  if (mode == 0) {
    const double tbe = tanh(beta * eta);
    const double v = (tbe + tanh(beta * (rt[e] - eta))) * inv;
    out[e] = v < 0.0 ? 0.0 : (v > 1.0 ? 1.0 : v);  // Math.Clamp(v, 0, 1)
    return;
  }
  const double th = tanh(beta * (rt[e] - eta));
  double d = beta * (1.0 - th * th) * inv;
  d = isnan(d) ? d : (d > 1e-12 ? d : 1e-12);  // Math.Max(d, 1e-12)
  out[e] = mode == 1 ? dcb[e] * d : d;
}

void launch_heaviside(mycel_ctx* ctx, int64_t n, const int32_t* idx, const double* rt, const double* dcb,
                      double* out, double beta, double eta, int mode) {
  if (n <= 0) return;
  k_heaviside<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(n, idx, rt, dcb, out, beta, eta, mode);
  ctx->launches++;
}

// Math.Pow over arrays, evaluated by the kernels' own path_pow (out[i] = x[i]^y[i], or x[i]^y[0] when y_len
// is 1): lets a host check the device's bits against its C library's pow.
__global__ void k_pow(int64_t n, const double* __restrict__ x, const double* __restrict__ y, int y_scalar,
                      double* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = path_pow(x[i], y[y_scalar ? 0 : i]);
}

// ---------------------------------------------------------------------------------------------------------
// OC update: persistent cooperative kernel with a bounded grid barrier
// ---------------------------------------------------------------------------------------------------------
// The barrier counts arrivals without end (launch_oc clears the word): its k-th use waits for k * gridDim.x of
// them, so a waiter sees the last arrival itself and no second word is needed. Only thread 0's own stores (and what
// it has observed of its CTA's by __syncthreads) are released: the callers publish partial sums only.
// Every wait gives up after OcArgs::max_polls polls (about 1 s by default, longer for large n, see launch_oc; all
// but the first 64 sleep 64 ns) and sets the error flag, so a grid that cannot meet ends with MYCEL_E_TIMEOUT.
struct GridBar {
  unsigned int* bar;  // bar[0]: arrivals
  int* err;
  long long max_polls;
  unsigned int extra;  // arrivals waited for beyond the grid (0; 1 only to test the time-out path)
  unsigned int target = 0;
};
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// arrival and wait by one thread of the CTA; false once any CTA has given up
__device__ __forceinline__ bool grid_meet(GridBar& g) {
  unsigned int old;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(g.bar) : "memory");
  const unsigned int want = g.target + g.extra;
  if (old + 1 != want) {
    long long polls = 0;
    while (ld_acquire(g.bar) < want) {
      if (++polls > g.max_polls || ((polls & 15) == 0 && *(volatile int*)g.err)) {
        atomicExch(g.err, 1);
        return false;
      }
      if (polls > 64) __nanosleep(64);
    }
  }
  return *(volatile int*)g.err == 0;
}
__device__ bool grid_sync_bounded(GridBar& g) {
  g.target += gridDim.x;
  bool ok = true;
  __syncthreads();
  if (threadIdx.x == 0) ok = grid_meet(g);
  return __syncthreads_and(ok ? 1 : 0) != 0;
}

__device__ __forceinline__ double clampd(double v, double lo, double hi) {
  if (v < lo) return lo;
  if (v > hi) return hi;
  return v;
}
__device__ __forceinline__ double maxd(double a, double b) {
  if (isnan(a) || isnan(b)) return __longlong_as_double(0x7ff8000000000000ll);
  return a > b ? a : b;
}
__device__ __forceinline__ double mind(double a, double b) {
  if (isnan(a) || isnan(b)) return __longlong_as_double(0x7ff8000000000000ll);
  return a < b ? a : b;
}

// volume term of element i for multiplier lam (OcOptimizer.EvaluateVolume :134-175) and the new density
__device__ __forceinline__ double oc_new_rho(double r, double dc, double si, bool pas, double lam, double move,
                                             double rmin) {
  if (pas) return 1.0;
  double lo = maxd(rmin, r - move), hi = mind(1.0, r + move);
  double nd = -dc;
  if (nd <= 0.0 || si <= 0.0) return lo;
  double b = nd / (lam * si);
  return clampd(r * sqrt(b), lo, hi);
}

// CTA sums of two values (lanes by a fixed shuffle tree, then the warps in order): bits as of one sum after the
// other. Thread 0 has the first, thread 1 the second.
__device__ __forceinline__ double block_sum2(double v0, double v1, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v0 = v0 + __shfl_down_sync(0xffffffffu, v0, o);
    v1 = v1 + __shfl_down_sync(0xffffffffu, v1, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) {
    sh[w] = v0;
    sh[8 + w] = v1;
  }
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 2) {
#pragma unroll
    for (int k = 0; k < 8; ++k) t = t + sh[8 * threadIdx.x + k];
  }
  return t;
}

struct OcArgs {
  int64_t n;
  const int32_t* idx;
  const double* rho;
  const double* dc;
  const double* s;
  const uint8_t* pas;
  double* rho_new;
  const double* rho_phys;
  const double* rho_grey;
  double* scratch;  // oc_scratch_doubles(gridDim.x) doubles, layout below
  unsigned int* bar;
  int* err;
  OcOut* out;
  long long max_polls;    // polls of each wait before it gives up
  unsigned int extra;     // arrivals a barrier waits for beyond the grid (0; 1 only to test the time-out path)
};
// scratch layout (grid = gridDim.x): [0, 4 grid) two alternating pairs of per-block partial sums (value, sum of
// magnitudes) of the volume trials; [4 grid, 7 grid) per-block max change, volume and grey sums;
// [7 grid, 7 grid + 4) two alternating broadcast cells of sequential sums; the barrier words (4 doubles); then
// [7 grid + 8, 11 grid + 8) the chunks of a sequential sum: totals, binades, steps from an even and an odd sum.

// Grid-wide deterministic sums of two per-thread values; every thread of every block gets the same totals.
// Latency is all there is to it: both values go through one reduction, one warp carries the partials to and from
// memory, and its loads of the other blocks' partials are issued together. Lane l takes blocks l, l + 32, ... in
// order, then a fixed shuffle tree (the same order in every block, so every block gets the same bits).
__device__ __forceinline__ bool grid_total2(double m0, double m1, const OcArgs& a, GridBar& g, int slot, double* sh,
                                            double* t0, double* t1) {
  const double b = block_sum2(m0, m1, sh);
  double* part = a.scratch + (size_t)slot * 2 * gridDim.x;
  const unsigned n = gridDim.x;
  g.target += n;
  bool ok = true;
  if (threadIdx.x < 32) {
    if (threadIdx.x < 2) part[threadIdx.x * n + blockIdx.x] = b;
    __syncwarp();
    if (threadIdx.x == 0) ok = grid_meet(g);
    __syncwarp();
    double s0 = 0.0, s1 = 0.0;
    for (unsigned k0 = threadIdx.x; k0 < n; k0 += 32 * 10) {
      double p0[10], p1[10];
#pragma unroll
      for (int j = 0; j < 10; ++j) {
        const unsigned k = k0 + 32 * j;
        p0[j] = k < n ? ld_volatile(part + k) : 0.0;
        p1[j] = k < n ? ld_volatile(part + n + k) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 10; ++j)
        if (k0 + 32 * j < n) {
          s0 = s0 + p0[j];
          s1 = s1 + p1[j];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s0 = s0 + __shfl_xor_sync(0xffffffffu, s0, o);
      s1 = s1 + __shfl_xor_sync(0xffffffffu, s1, o);
    }
    if (threadIdx.x == 0) {
      sh[16] = s0;
      sh[17] = s1;
    }
  }
  ok = __syncthreads_and(ok ? 1 : 0) != 0;
  *t0 = sh[16];
  *t1 = sh[17];
  return ok;
}

// ---- sums in element order, in parallel ------------------------------------------------------------------
// The reference adds n terms one after the other. While the running sum stays in one binade [2^e, 2^(e+1)) it is
// an integer M of units u = 2^(e-52), and adding a term t >= 0 rounds to M + round(t / u): the integer nearest to
// t / u, whatever M is, except that a tie goes to the even sum and so depends on M's last bit. A run of terms is
// therefore a pair of integers, the increments from an even and from an odd M; pairs compose (associatively), so
// threads, warps and blocks can each take a run and the sum comes out with the bits of the sequential one. What a
// run may not do is leave the binade: then (and for terms that are negative or not finite) its terms are added one
// by one. The binade a chunk of terms begins in is guessed from an ordinary parallel sum of the chunks before it;
// the guess is checked against the sum itself, so a wrong one costs time only. With n terms of like size the sum
// crosses about log2 n binades, most of them in the first chunk.
struct SumStep {
  long long even, odd;  // increments (units of the binade) from an even and from an odd sum; kStepOut: leaves it
};
constexpr long long kStepOut = 1ll << 54;
__device__ __forceinline__ SumStep step_then(SumStep f, SumStep g) {
  SumStep r;
  r.even = min(f.even + ((f.even & 1) ? g.odd : g.even), kStepOut);
  r.odd = min(f.odd + ((f.odd & 1) ? g.even : g.odd), kStepOut);
  return r;
}
__device__ __forceinline__ SumStep step_of(double t, double inv_u) {
  const double q = t * inv_u;  // a power of two: exact (or far below one half)
  SumStep r;
  if (t >= 0.0 && q < 0x1p53) {
    const long long k = __double2ll_rn(q);  // nearest, ties to even: the increment of an even sum
    r.even = k;
    r.odd = fabs(q - (double)k) == 0.5 ? (long long)(q + q) - k : k;  // a tie: the other neighbour
  } else {
    r.even = r.odd = kStepOut;
  }
  return r;
}
__device__ __forceinline__ SumStep warp_steps(SumStep v) {  // lane 0: the lanes' steps in lane order
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    SumStep w;
    w.even = __shfl_down_sync(0xffffffffu, v.even, o);
    w.odd = __shfl_down_sync(0xffffffffu, v.odd, o);
    v = step_then(v, w);
  }
  return v;
}
// biased exponent of a sum that can take steps, or 0 (zero, negative, not finite, or so large or small that the
// units or their reciprocal leave the normal range)
__device__ __forceinline__ int sum_binade(double acc) {
  const int hi = (int)((unsigned long long)__double_as_longlong(acc) >> 52);
  return hi >= 100 && hi <= 1900 ? hi : 0;
}
__device__ __forceinline__ double binade_inv_u(int b) { return __longlong_as_double((long long)(2098 - b) << 52); }
// acc after a run's step taken in binade b; false (acc unchanged) if the sum is not in b or the run leaves it
__device__ __forceinline__ bool take_step(double& acc, int b, long long even, long long odd) {
  const long long bits = __double_as_longlong(acc);
  if (b == 0 || (int)((unsigned long long)bits >> 52) != b) return false;
  const long long m = (bits & 0xfffffffffffffll) | (1ll << 52);
  const long long m2 = m + ((m & 1) ? odd : even);
  if (m2 >= (1ll << 53)) return false;
  acc = __longlong_as_double(((long long)b << 52) | (m2 & 0xfffffffffffffll));
  return true;
}

enum OcSum : int { OC_SUM_S, OC_SUM_VOLUME, OC_SUM_PHYS, OC_SUM_GREY };
__device__ __forceinline__ double oc_seq_term(const OcArgs& a, const OcParams& prm, int kind, double lam, int64_t i) {
  const int64_t e = a.idx ? (int64_t)a.idx[i] : i;
  if (kind == OC_SUM_PHYS) return a.rho_phys[e];
  if (kind == OC_SUM_GREY) {
    const double rb = a.rho_grey[e];
    return rb * (1.0 - rb);
  }
  const double si = a.s[e];
  if (kind == OC_SUM_S) return si;
  return si * ((a.pas && a.pas[e]) ? 1.0 : oc_new_rho(a.rho[e], a.dc[e], si, false, lam, prm.move, prm.rho_min));
}

constexpr int kSeqTile = 1024, kSeqPiece = 128;  // terms of a CTA's tile; of a warp's piece of it
struct SeqSmem {
  double term[kSeqTile];
  SumStep piece[8];
  SumStep chunk[256];
  int binade[256];
  double acc;
  int next;
};
// acc + terms [i0, i1) in order, by one CTA (acc in sm.acc): a tile of terms at a time, each warp the step of one
// piece in the sum's present binade; thread 0 takes the steps in order and adds the terms of a piece that leaves
// the binade one by one, after which the pieces behind it are stepped again in the new one.
__device__ __forceinline__ void seq_range(const OcArgs& a, const OcParams& prm, int kind, double lam, int64_t i0,
                                          int64_t i1, SeqSmem& sm) {
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  for (int64_t base = i0; base < i1; base += kSeqTile) {
    const int cnt = (int)min((int64_t)kSeqTile, i1 - base);
    const int np = (cnt + kSeqPiece - 1) / kSeqPiece;
    for (int k = tid; k < np * kSeqPiece; k += 256)
      sm.term[k] = k < cnt ? oc_seq_term(a, prm, kind, lam, base + k) : 0.0;  // a running sum + 0 is itself
    __syncthreads();
    for (int lo = 0; lo < np;) {
      const int b = sum_binade(sm.acc);
      if (b && w >= lo && w < np) {
        const double iu = binade_inv_u(b);
        const double* t = sm.term + w * kSeqPiece + 4 * l;
        SumStep v = step_then(step_then(step_of(t[0], iu), step_of(t[1], iu)),
                              step_then(step_of(t[2], iu), step_of(t[3], iu)));
        v = warp_steps(v);
        if (l == 0) sm.piece[w] = v;
      }
      __syncthreads();
      if (tid == 0) {
        double acc = sm.acc;
        int k = lo;
        while (k < np && take_step(acc, b, sm.piece[k].even, sm.piece[k].odd)) ++k;
        if (k < np) {
          const double* t = sm.term + k * kSeqPiece;
#pragma unroll 16
          for (int j = 0; j < kSeqPiece; ++j) acc = acc + t[j];
          ++k;
        }
        sm.acc = acc;
        sm.next = k;
      }
      __syncthreads();
      lo = sm.next;
    }
  }
}

// Sum of a kind of term over i = 0 .. n-1 in that order (the reference's sequential loops); every thread gets it.
// Short sums: block 0 alone. Else the blocks take one chunk each: a plain sum (for the guess of the binade the
// next chunks begin in), then the chunk's step in the guessed binade; block 0 takes the steps in order and walks
// through the chunks whose step does not hold.
__device__ __noinline__ double sequential_sum(const OcArgs& a, const OcParams& prm, int kind, double lam, int cell,
                                              GridBar& g, double* sh, SeqSmem& sm, bool* ok) {
  const int tid = threadIdx.x;
  const unsigned nb = gridDim.x;
  double* c = a.scratch + (size_t)7 * nb + 2 * cell;
  double* tot = a.scratch + (size_t)7 * nb + 8;
  long long* bin = (long long*)(tot + nb);
  long long* even = (long long*)(tot + 2 * (size_t)nb);
  long long* odd = (long long*)(tot + 3 * (size_t)nb);
  const bool split = a.n > 2 * kSeqTile;
  const int64_t len = max((int64_t)256, (a.n + nb - 1) / nb);
  const int nchunk = (int)((a.n + len - 1) / len);
  *ok = true;
  if (split) {
    const int64_t i0 = min(a.n, (int64_t)blockIdx.x * len), i1 = min(a.n, i0 + len);
    double v = 0.0;
    for (int64_t i = i0 + tid; i < i1; i += 256) v = v + oc_seq_term(a, prm, kind, lam, i);
    const double bs = block_sum2(v, 0.0, sh);
    if (tid == 0) tot[blockIdx.x] = bs;
    if (!grid_sync_bounded(g)) {
      *ok = false;
      return 0.0;
    }
    double before = 0.0;
    for (unsigned k = tid; k < blockIdx.x; k += 256) before = before + ld_volatile(tot + k);
    before = block_sum2(before, 0.0, sh);
    if (tid == 0) sm.acc = before;
    __syncthreads();
    const int b = sum_binade(sm.acc);
    const double iu = binade_inv_u(b);
    // thread t: a run of consecutive terms, so that lanes and warps compose in term order
    const int64_t run = (i1 - i0 + 255) / 256;
    const int64_t r0 = min(i1, i0 + tid * run), r1 = min(i1, r0 + run);
    SumStep st{0, 0};
    if (b)
      for (int64_t i = r0; i < r1; ++i) st = step_then(st, step_of(oc_seq_term(a, prm, kind, lam, i), iu));
    st = warp_steps(st);
    if ((tid & 31) == 0) sm.piece[tid >> 5] = st;
    __syncthreads();
    if (tid == 0) {
      st = sm.piece[0];
      for (int k = 1; k < 8; ++k) st = step_then(st, sm.piece[k]);
      bin[blockIdx.x] = b;
      even[blockIdx.x] = st.even;
      odd[blockIdx.x] = st.odd;
    }
    if (!grid_sync_bounded(g)) {
      *ok = false;
      return 0.0;
    }
  }
  if (blockIdx.x == 0) {
    if (tid == 0) sm.acc = 0.0;
    __syncthreads();
    if (!split) {
      seq_range(a, prm, kind, lam, 0, a.n, sm);
    } else {
      for (int k0 = 0; k0 < nchunk;) {
        const int k = k0 + tid, kn = min(256, nchunk - k0);
        if (tid < kn) {
          sm.binade[tid] = (int)*(volatile long long*)(bin + k);
          sm.chunk[tid].even = *(volatile long long*)(even + k);
          sm.chunk[tid].odd = *(volatile long long*)(odd + k);
        }
        __syncthreads();
        if (tid == 0) {
          double acc = sm.acc;
          int j = 0;
          while (j < kn && take_step(acc, sm.binade[j], sm.chunk[j].even, sm.chunk[j].odd)) ++j;
          sm.acc = acc;
          sm.next = j;
        }
        __syncthreads();
        const int j = sm.next;
        k0 += j;
        __syncthreads();  // sm.next is read before seq_range writes it
        if (j < kn) {
          seq_range(a, prm, kind, lam, k0 * len, min(a.n, (k0 + 1) * len), sm);
          ++k0;
        }
      }
    }
    if (tid == 0) *(volatile double*)c = sm.acc;
  }
  if (!grid_sync_bounded(g)) {
    *ok = false;
    return 0.0;
  }
  return ld_volatile(c);
}

// A volume V(lambda) of the bisection: the grid's tree sum, with an error bound against any other order of the
// same terms, or (exact) the sum in the reference's element order.
struct OcVol {
  double v, bound;
  bool exact;
};

// What bounds it: a trial's terms are one divide and one square root per element, a few microseconds at most; below
// about a million elements the trials (30 to 50 a call) are bound by the latency of the grid's sum and barrier. So a
// thread keeps its elements in registers when 8 per thread hold them, and the sum and the barrier are one step
// (grid_total2).
// Measured on B200, a whole call: 221,184 elements deciding on sums in element order 5.81 ms -> 0.56 ms (those sums
// were added by one warp, 13 ns a term); 121,635 elements on the grid's sums 227 us -> 152 us.
__global__ void __launch_bounds__(256) k_oc(const __grid_constant__ OcArgs a, const __grid_constant__ OcParams prm) {
  __shared__ double sh[32];
  __shared__ SeqSmem sm;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  bool ok = true;
  int slot = 0, cell = 0;
  GridBar gb{a.bar, a.err, a.max_polls, a.extra};
  auto element = [&](int64_t i) -> int64_t { return a.idx ? (int64_t)a.idx[i] : i; };
  auto seq = [&](int kind, double lam) -> double {
    cell ^= 1;
    return sequential_sum(a, prm, kind, lam, cell, gb, sh, sm, &ok);
  };
  // tree depth of a grid total: the per-thread chain, the warp and block steps, the lane-strided block partials
  const double depth = (double)((a.n + stride - 1) / stride) + 5.0 + 8.0 + (double)((gridDim.x + 31) / 32) + 5.0;
  // the thread's elements t0, t0 + stride, ... summed in that order; the loads of 8 of them are issued before
  // their terms are added, so the index -> data load chains overlap; with at most 8 they are loaded once
  constexpr int kB = 8;
  double si[kB], rr[kB], dd[kB];
  unsigned pp = 0;
  auto load = [&](int64_t base) {
    pp = 0;
#pragma unroll
    for (int k = 0; k < kB; ++k) {
      const int64_t i = base + k * stride;
      const int64_t e = i < a.n ? element(i) : 0;
      if (i < a.n && a.pas && a.pas[e]) pp |= 1u << k;
      si[k] = i < a.n ? a.s[e] : 0.0;
      rr[k] = i < a.n ? a.rho[e] : 0.0;
      dd[k] = i < a.n ? a.dc[e] : 0.0;
    }
  };
  const bool held = a.n <= kB * stride;
  if (held) load(t0);
  auto volume = [&](double lam) -> OcVol {
    double v = 0.0, va = 0.0;
    for (int64_t base = t0; base < a.n; base += kB * stride) {
      if (!held) load(base);
#pragma unroll
      for (int k = 0; k < kB; ++k)
        if (base + k * stride < a.n) {
          const double t =
              si[k] * (((pp >> k) & 1) ? 1.0 : oc_new_rho(rr[k], dd[k], si[k], false, lam, prm.move, prm.rho_min));
          v = v + t;
          va = va + fabs(t);
        }
    }
    double tv = 0.0, ta = 0.0;
    if (!grid_total2(v, va, a, gb, slot, sh, &tv, &ta)) ok = false;
    slot ^= 1;
    OcVol r;
    r.v = tv;
    // |tree - exact| <= gamma_depth sum|t| and |sequential - exact| <= gamma_(n-1) sum|t|, gamma_k = k u / (1 - k u);
    // doubled for the rounding of the computed sum of magnitudes and of the bound itself
    r.bound = 2.0 * ((double)a.n + depth) * 0x1p-53 * ta * 1.0000001;
    r.exact = false;
    return r;
  };
  // the volume at lam in the reference's order, when a decision needs it
  auto make_exact = [&](OcVol& x, double lam) {
    if (x.exact) return;
    x.v = seq(OC_SUM_VOLUME, lam);
    x.bound = 0.0;
    x.exact = true;
  };
  // total S (OcOptimizer.cs:28-33): sequential in element order, or the value the caller has cached
  double ts;
  if (prm.total_s >= 0.0) {
    ts = prm.total_s;
  } else if (prm.exact) {
    ts = seq(OC_SUM_S, 0.0);
  } else {
    double sv = 0.0;
    for (int64_t i = t0; i < a.n; i += stride) sv = sv + a.s[element(i)];
    double t1 = 0.0;
    if (!grid_total2(sv, 0.0, a, gb, slot, sh, &ts, &t1)) ok = false;
    slot ^= 1;
  }
  if (!ok) return;
  const double tv = prm.f * ts;
  // the comparisons of the reference (v < target, v > target, relErr <= tolerance) taken on the tree sum unless
  // it is within its error bound of the threshold; then on the sequential sum (exact mode)
  auto less_than_target = [&](OcVol& x, double lam) -> bool {
    if (prm.exact && !x.exact && fabs(x.v - tv) <= x.bound) make_exact(x, lam);
    return x.v < tv;
  };
  auto greater_than_target = [&](OcVol& x, double lam) -> bool {
    if (prm.exact && !x.exact && fabs(x.v - tv) <= x.bound) make_exact(x, lam);
    return x.v > tv;
  };
  const double denom = maxd(tv, 1e-12);
  auto within_tolerance = [&](OcVol& x, double lam) -> bool {
    if (prm.exact && !x.exact) {
      const double d = fabs(x.v - tv), lim = prm.vol_tol * denom;
      if (fabs(d - lim) <= x.bound + 0x1p-50 * (d + lim)) make_exact(x, lam);
    }
    return fabs(x.v - tv) / denom <= prm.vol_tol;
  };
  const double lg = prm.lambda_guess;
  bool gok = lg > 0.0 && !isinf(lg) && !isnan(lg);
  double l1 = gok ? lg * 0.5 : 1e-12;
  double l2 = gok ? lg * 2.0 : 1e12;
  if (l1 <= 1e-50) l1 = 1e-12;
  if (l2 <= l1) l2 = l1 * 10.0;
  int trials = 0;
  OcVol v1 = volume(l1);
  OcVol v2 = volume(l2);
  trials += 2;
  if (!ok) return;
  int ex = 0;
  while (less_than_target(v1, l1) && l1 > 1e-50 && ex++ < 50) {
    if (!ok) return;
    l2 = l1;
    v2 = v1;
    l1 *= 0.1;
    v1 = volume(l1);
    ++trials;
    if (!ok) return;
  }
  if (!ok) return;
  ex = 0;
  while (greater_than_target(v2, l2) && l2 < 1e50 && ex++ < 50) {
    if (!ok) return;
    l1 = l2;
    v1 = v2;
    l2 *= 10.0;
    v2 = volume(l2);
    ++trials;
    if (!ok) return;
  }
  if (!ok) return;
  double lm = sqrt(l1 * l2);
  for (int st = 0; st < prm.max_bisect; ++st) {
    lm = sqrt(l1 * l2);
    OcVol vm = volume(lm);
    ++trials;
    if (!ok) return;
    const bool done = within_tolerance(vm, lm);
    if (!ok) return;
    if (done) break;
    const bool high = greater_than_target(vm, lm);
    if (!ok) return;
    if (high) l1 = lm;
    else l2 = lm;
    if (fabs(l2 - l1) <= 1e-15 * lm) break;
  }
  // final densities and the iteration metrics (TopologyOptimizer.cs:323-338)
  double mc = 0.0, vs = 0.0, gs = 0.0;
  for (int64_t i = t0; i < a.n; i += stride) {
    int64_t e = element(i);
    bool pas = a.pas && a.pas[e];
    double r = a.rho[e];
    double nr = oc_new_rho(r, a.dc[e], a.s[e], pas, lm, prm.move, prm.rho_min);
    a.rho_new[e] = nr;
    double d = fabs(nr - r);
    if (d > mc) mc = d;
    if (a.rho_phys && !prm.exact) {
      vs = vs + a.rho_phys[e];
      double rb = a.rho_grey[e];
      gs = gs + rb * (1.0 - rb);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    double v = __shfl_down_sync(0xffffffffu, mc, o);
    if (v > mc) mc = v;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mc;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k)
      if (sh[k] > mc) mc = sh[k];
  }
  double* part = a.scratch + (size_t)4 * gridDim.x;
  const double bsum = block_sum2(vs, gs, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = mc;
  if (threadIdx.x < 2) part[(1 + threadIdx.x) * gridDim.x + blockIdx.x] = bsum;
  if (!grid_sync_bounded(gb)) return;
  // exact mode: the volume and grey sums in the reference's element order (:328-335)
  double svol = 0.0, sgrey = 0.0;
  if (prm.exact && a.rho_phys) {
    svol = seq(OC_SUM_PHYS, 0.0);
    if (!ok) return;
    sgrey = seq(OC_SUM_GREY, 0.0);
    if (!ok) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    double m = 0.0, v = 0.0, gg = 0.0;
    for (unsigned k = 0; k < gridDim.x; ++k) {
      double q = ld_volatile(part + k);
      if (q > m) m = q;
      v = v + ld_volatile(part + gridDim.x + k);
      gg = gg + ld_volatile(part + 2 * gridDim.x + k);
    }
    a.out->lambda = lm;
    a.out->max_change = m;
    a.out->vol_sum = prm.exact ? svol : v;
    a.out->grey_sum = prm.exact ? sgrey : gg;
    a.out->total_s = ts;
    a.out->err = 0;
    a.out->trials = trials;
  }
}

int oc_blocks_per_sm(int* out) {
  int b = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_oc, 256, 0);
  if (e != cudaSuccess) return MYCEL_E_DEVICE;
  *out = std::max(1, std::min(b, 2));
  return MYCEL_OK;
}

int launch_oc(mycel_ctx* ctx, int64_t n, const int32_t* d_index, const double* rho, const double* dc, const double* s,
              const uint8_t* passive, double* rho_new, const double* rho_phys_for_metrics,
              const double* rho_tilde_for_grey, const OcParams& prm, double* d_scratch, size_t scratch_doubles,
              OcOut* d_out) {
  const int grid = ctx->oc_grid;  // fixed when the context was created
  if (grid < 1 || oc_scratch_doubles(grid) > scratch_doubles) return MYCEL_E_ARG;
  unsigned int* bar = (unsigned int*)(d_scratch + 7 * (size_t)grid + 4);
  int* err = (int*)(bar + 4);
  if (cudaMemsetAsync(bar, 0, 8 * sizeof(unsigned int), ctx->stream) != cudaSuccess) return MYCEL_E_DEVICE;
  // each wait: about 1 s of polling, plus room for the sequential sums of the exact mode (at worst, when no step of
  // one holds, block 0 adds all terms one by one at about 10 ns each)
  long long polls = ctx->oc_wait_polls > 0 ? ctx->oc_wait_polls : (1ll << 24) + 4 * (long long)n;
  OcArgs a{n, d_index, rho, dc, s, passive, rho_new, rho_phys_for_metrics,
           rho_tilde_for_grey ? rho_tilde_for_grey : rho_phys_for_metrics, d_scratch, bar, err, d_out,
           polls, ctx->oc_wait_unreachable ? 1u : 0u};
  OcParams pp = prm;
  void* args[] = {&a, &pp};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_oc, dim3(grid), dim3(256), args, 0, ctx->stream);
  ctx->launches++;
  if (e != cudaSuccess) return MYCEL_E_DEVICE;
  return MYCEL_OK;
}

// ---------------------------------------------------------------------------------------------------------
// OC update without device allocation.
// Some callers cannot allocate device memory at the time they run the OC step: a host whose device memory is
// reserved in full by another allocator in the same process (a caching allocator or a fixed pool), or a loop
// that must not pay the device-wide synchronisation a cudaMalloc/cudaFree pair can cost. This entry point
// takes the caller's device buffers and keeps the OC kernel's scratch (block partials, barrier words, result)
// in the file-scope array below, which every GPU that loads the library holds until the process exits.
// ---------------------------------------------------------------------------------------------------------
constexpr int kOcNoAllocMaxBlocks = 1024;                                // persistent OC blocks it can serve
constexpr int kOcNoAllocScratch = 12 * kOcNoAllocMaxBlocks + 8;          // partials, barrier words, chunk steps
constexpr int kOcNoAllocOut = (int)((sizeof(OcOut) + sizeof(double) - 1) / sizeof(double));
static __device__ __align__(256) double g_oc_noalloc[kOcNoAllocScratch + kOcNoAllocOut];  // 98.4 KB

namespace {
std::mutex g_oc_noalloc_mu;
void* g_oc_noalloc_addr[128] = {};  // device address of g_oc_noalloc, per device, filled on first use
}  // namespace

}  // namespace mycel

extern "C" int32_t mycel_oc_update_noalloc(mycel_ctx* ctx, int32_t n, const double* rho, const double* dc,
                                           const double* s, const uint8_t* passive, double* rho_new,
                                           double target_volume_fraction, double move_limit, double rho_min,
                                           double lambda_guess, int32_t max_bisection_steps,
                                           double volume_tolerance, double* lambda_out) {
  using namespace mycel;
  if (!ctx) return set_error(nullptr, MYCEL_E_ARG, "NULL context");
  if (n < 0 || (n > 0 && (!rho || !dc || !s || !rho_new)) || !lambda_out)
    return set_error(ctx, MYCEL_E_ARG, "All spans must have length >= rho.Length.");
  if (ctx->device < 0 || ctx->device >= 128) return set_error(ctx, MYCEL_E_ARG, "device index out of range");
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return set_error(ctx, MYCEL_E_DEVICE, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
  // set-up, once per device, with that device current: the host-side name of the array is not a device
  // address, so the kernel gets the address the runtime reports for this device
  void* base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_oc_noalloc_mu);
    if (!g_oc_noalloc_addr[ctx->device]) {
      e = cudaGetSymbolAddress(&g_oc_noalloc_addr[ctx->device], g_oc_noalloc);
      if (e != cudaSuccess) {
        g_oc_noalloc_addr[ctx->device] = nullptr;
        return set_error(ctx, MYCEL_E_DEVICE, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      }
    }
    base = g_oc_noalloc_addr[ctx->device];
  }
  const int grid = ctx->oc_grid;  // the grid launch_oc uses, fixed when the context was created
  if (oc_scratch_doubles(grid) > (size_t)kOcNoAllocScratch)
    return set_error(ctx, MYCEL_E_ARG, "OC without allocation: this device needs " + std::to_string(grid) +
                                           " persistent blocks, the static scratch holds " +
                                           std::to_string(kOcNoAllocMaxBlocks));
  double* scratch = static_cast<double*>(base);
  OcOut* out = reinterpret_cast<OcOut*>(scratch + kOcNoAllocScratch);
  // the array keeps the previous call's contents: clear the result (launch_oc clears the barrier words)
  e = cudaMemsetAsync(out, 0, sizeof(OcOut), ctx->stream);
  if (e != cudaSuccess) return set_error(ctx, MYCEL_E_DEVICE, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
  OcParams prm{target_volume_fraction, move_limit, rho_min, lambda_guess, volume_tolerance, max_bisection_steps, 0};
  if (launch_oc(ctx, n, nullptr, rho, dc, s, passive, rho_new, nullptr, nullptr, prm, scratch, kOcNoAllocScratch,
                out))
    return set_error(ctx, MYCEL_E_DEVICE, std::string("OC kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
  OcOut* h = reinterpret_cast<OcOut*>(ctx->pinned);
  e = cudaMemcpyAsync(h, out, sizeof(OcOut), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return set_error(ctx, MYCEL_E_DEVICE, std::string("OC kernel: ") + cudaGetErrorString(e));
  if (h->trials == 0) return set_error(ctx, MYCEL_E_TIMEOUT, "OC grid barrier timed out");
  *lambda_out = h->lambda;
  return MYCEL_OK;
}

extern "C" int32_t mycel_pow(mycel_ctx* ctx, int64_t n, const double* x, const double* y, int64_t y_len,
                             double* out) {
  using namespace mycel;
  if (!ctx) return set_error(nullptr, MYCEL_E_ARG, "NULL context");
  if (n < 0 || (n > 0 && (!x || !y || !out)) || (n > 0 && y_len != 1 && y_len != n))
    return set_error(ctx, MYCEL_E_ARG, "pow: x and out need n values, y 1 or n");
  if (n == 0) return MYCEL_OK;
  MYCEL_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  double *dx = nullptr, *dy = nullptr, *dout = nullptr;
  MYCEL_CUDA(ctx, cudaMallocAsync((void**)&dx, sizeof(double) * n, st));
  MYCEL_CUDA(ctx, cudaMallocAsync((void**)&dy, sizeof(double) * y_len, st));
  MYCEL_CUDA(ctx, cudaMallocAsync((void**)&dout, sizeof(double) * n, st));
  cudaError_t e = cudaMemcpyAsync(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dy, y, sizeof(double) * y_len, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)ctx->num_sms * 8);
    k_pow<<<blocks, 256, 0, st>>>(n, dx, dy, y_len == 1 ? 1 : 0, dout);
    ctx->launches++;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, dout, sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(dx, st);
  cudaFreeAsync(dy, st);
  cudaFreeAsync(dout, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return set_error(ctx, MYCEL_E_DEVICE, std::string("pow: ") + cudaGetErrorString(e));
  return MYCEL_OK;
}

// HeavisideProjection.Project / Derivative over host arrays (kernel-level entry points).
static int32_t heaviside_entry(mycel_ctx* ctx, int64_t n, const double* rt, double* out, double beta, double eta,
                               int mode) {
  using namespace mycel;
  if (!ctx) return set_error(nullptr, MYCEL_E_ARG, "NULL context");
  if (n < 0 || (n > 0 && (!rt || !out))) return set_error(ctx, MYCEL_E_ARG, "NULL argument");
  if (n == 0) return MYCEL_OK;
  MYCEL_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  double *din = nullptr, *dout = nullptr;
  MYCEL_CUDA(ctx, cudaMallocAsync((void**)&din, sizeof(double) * n, st));
  MYCEL_CUDA(ctx, cudaMallocAsync((void**)&dout, sizeof(double) * n, st));
  cudaError_t e = cudaMemcpyAsync(din, rt, sizeof(double) * n, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    launch_heaviside(ctx, n, nullptr, din, nullptr, dout, beta, eta, mode);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, dout, sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(din, st);
  cudaFreeAsync(dout, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return set_error(ctx, MYCEL_E_DEVICE, std::string("Heaviside: ") + cudaGetErrorString(e));
  return MYCEL_OK;
}

extern "C" int32_t mycel_heaviside_project(mycel_ctx* ctx, int64_t n, const double* rho_tilde, double* rho_bar,
                                           double beta, double eta) {
  return heaviside_entry(ctx, n, rho_tilde, rho_bar, beta, eta, 0);
}

extern "C" int32_t mycel_heaviside_derivative(mycel_ctx* ctx, int64_t n, const double* rho_tilde, double* deriv,
                                              double beta, double eta) {
  return heaviside_entry(ctx, n, rho_tilde, deriv, beta, eta, 2);
}
