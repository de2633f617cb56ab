// The iterations of one warp with the whole state of a pair on chip.
//
// iterate_split_kernel reads and writes u, p, D, rho_c and the warped gradient through memory in
// every iteration. Where a level's volume fits into the registers and shared memory of the GPU,
// none of that traffic is needed: resident_kernel gives every CTA one box of a pair's volume and
// runs all iterations of a warp (tvl13d.py:213-253) in one launch, p and the per-voxel constants
// in registers, u and q = D p in shared memory. Only the faces of u and q cross CTAs.
//
// Per iteration and CTA:
//   halo of u   the six faces of the neighbouring boxes' u arrive (below); barrier;
//   dual        p_new = proj(p + sigma D grad u) of the own voxels, q = D p_new to shared memory,
//               q_x / q_y / q_z of the box's faces published to the neighbours;
//   halo of q   the neighbours' faces arrive; barrier;
//   primal      u_new = prox(u - tau adjoint(q)) in place, faces of u published.
// No dual is recomputed on a halo (the march kernels recompute 20-30%), and a thread owns NP
// pairs of x-adjacent voxels (packed FP32 arithmetic) stacked along z, so the z neighbours of u
// are mostly its own registers.
//
// Exchange: one 16-byte word per face voxel, {three components, tag}, written and polled with
// single 128-bit relaxed accesses, so a word's data and its tag arrive together and no fence or
// flag is needed. Each box has one incoming word per face voxel for u and one for q. A word is
// overwritten only after it was read: a box publishes q(t+1) to a neighbour after consuming that
// neighbour's u(t), which the neighbour published after consuming q(t); u likewise. Tags count
// iterations from 1; the reader clears its words when the launch ends, so every launch starts
// from tag 0. Polling is bounded (ResidentArgs::wait_us); a box that gives up raises the abort
// word, which ends its neighbours' waits and the plan's later launches.
//
// CLUSTER: a volume of at most 16 boxes runs in one thread-block cluster instead. The faces are then
// stored asynchronously into the halo cells of the neighbours' shared memory and counted by an
// mbarrier there, one per field, which replaces words, tags and polling through L2 (every box has read
// its halo before it sends what lets a neighbour write again: the same order as above). No box of
// another pair is waited for, so the launch is not cooperative. An exchange takes about 0.55 us instead of 1.25
// (0.75 with a cluster barrier per exchange, whose release waits until the stores have arrived):
// 20^3 2.8 -> 2.0 us per iteration (16 boxes of 10x10x5), 9x11x12 2.7 -> 1.5, 18x21x24 2.85 -> 2.45
// (1.8, 1.25 and 2.2 with EARLY and two word slots, below; f32 1.7, 1.13 and 2.06). From about
// 200 voxel pairs per box on, the boxes' arithmetic is worth more than that (24^3: 2.6 us on 144 SMs),
// and the choice in plan_resident sees it.
//
// Measured on one B200 (us per iteration; before: one launch per iteration, march along z):
//   f16-flow32 80^3 10.5 (20.4), 48^3 3.2 (14.4), 40^3 2.85 (10.3), 20^3 1.8 (8.2);
//   f32 80^3 13.8 (20.5), 48^3 3.15 (12.3), 20^3 1.7 (10.3); 12 pairs of 40^3 f16-flow32 16.1 (26.7).
// Small boxes are bound by the two exchanges (about 2.5 us: publish, poll, barriers). 80^3 is
// bound by the latency of 12 warps of 168 registers (about 8,000 cycles of dual, 5,800 of primal)
// and by the words' L2 traffic (3.6 MB per exchange each way). Its f32 form keeps p alone (90
// registers of 168, 350 bytes spilled) and reads D (12 MB) and rho_c, gw (8 MB) from L2 in every
// iteration; reading D one pair ahead took 15.5 us (12 more registers), 8 pairs by 256 threads 21.5.
//
// Boundaries (MIRROR with power-of-two 0.5/h only, see resident_ok in svs_solver.cu): central
// differences vanish on a face and the adjoint sees q = 0 there, so with u mirrored into the cell
// outside the volume (u[-1] = u[1], u[n] = u[n-2]) and q's normal component zeroed on the face,
// every voxel runs the interior stencil; 0.5/h being a power of two, the products are exact and
// the difference is exactly zero. The arithmetic per voxel is that of iterate_split_kernel
// (dual_row, primal_step, primal_apply, the same fused operations), so the results agree bitwise.
#pragma once

#include "svs_iterate.cuh"

namespace svs {

// A launch: up to kResSlots boxes of up to kResSlots pairs, as a kernel parameter (constant memory,
// so that everything derived from it stays in uniform registers). Pair i's boxes are a
// gx x gy x gz grid of bx x by x bz boxes (the last of an axis may reach past the volume), blocks
// first .. first + gx gy gz - 1, x fastest; its neighbours are therefore at fixed distances.
constexpr int kResSlots = 160;
struct ResPair {
  int desc, first;
  unsigned char gx, gy, gz, pad0;
  unsigned char bx, by, bz, pad1;
};
struct ResLaunch {
  ResPair pair[kResSlots];
  unsigned char of[kResSlots];  // pair of each block
  int cluster;                  // CLUSTER shapes: blocks per cluster (a pair each), else 0
};

struct ResidentArgs {
  const float* sig;  // [iters] sigma and tau of each iteration
  const float* tau;
  float wm, wtv;     // weight_matching (factor = tau * wm), weight_tv
  int src, dst;      // ping-pong copies read at the start and written at the end
  int iters;
  unsigned wait_us;  // bound of a wait for a neighbour
  int words;         // exchange words per box and field
  int mute;          // MUTE: block that keeps its faces to itself (test hook of the waits), else -1
  uint4* xbuf;       // [boxes][u, q][words]
  int* abort;        // raised when a wait gave up
};

// Compiled shapes: NP voxel pairs per thread, up to NT threads; CU floats per component of u (with
// its halo planes, rows and columns) and CQ of each of q_x (halo columns), q_y (halo rows) and
// q_z (halo planes); up to NE face voxels per thread. KEEP_D, KEEP_R: the tensor, and rho_c and
// the warped gradient, stay in registers; else they are read again in every iteration, D where it
// is used, the others before the wait for q's halo. ROLL: the primal keeps q_z of two planes from pair
// to pair instead of reading each plane twice. Taken where p alone is held (f32 80^3 14.7 -> 13.8 us
// per iteration); with D held too it takes registers that are not there (f16-flow32 80^3 10.6 -> 10.8).
// EARLY: the part of the primal that needs no q, the step of the shrinkage, is computed between publishing q's
// faces and waiting for the neighbours' (35x41x47 f16-flow32 3.43 -> 3.27 us, 40^3 3.37 -> 3.2, 20^3 2.0 -> 1.83). The
// 5-pair shape is short of registers for it (10.6 -> 11.0, f32 13.8 -> 15.7).
// MUTE: the form with the test hook of the waits (ResidentArgs::mute), apart because its one comparison
// cost the cluster form 2% by other registers (f32 9x11x12 1.132 -> 1.158 us).
template <int NP_, int NT_, int CU_, int CQ_, int NE_, bool KEEP_D_, bool KEEP_R_, bool CLUSTER_ = false, bool MUTE_ = false>
struct ResShape {
  static constexpr int NP = NP_, NT = NT_, CU = CU_, CQ = CQ_, NE = NE_;
  static constexpr bool CLUSTER = CLUSTER_, EARLY = NP <= 2, MUTE = MUTE_;
  using WithMute = ResShape<NP_, NT_, CU_, CQ_, NE_, KEEP_D_, KEEP_R_, CLUSTER_, true>;
  static constexpr bool KEEP_D = KEEP_D_, KEEP_R = KEEP_R_, ROLL = !KEEP_D;
  // the register file holds 16,384 registers per scheduler, a quarter of the warps each
  static constexpr int WARPS = (NT + 31) / 32, MAXREG = 16384 / ((WARPS + 3) / 4 * 32) / 8 * 8;
  static constexpr int REGS = MAXREG > 255 ? 255 : MAXREG;
  static constexpr int BAR = (3 * CU + 9 * CQ) * 4;      // CLUSTER: two mbarriers behind the arrays
  static constexpr int SMEM = BAR + (CLUSTER ? 16 : 0);
  static_assert(SMEM <= 227 * 1024, "fits one CTA per SM");
  static_assert(CU % 2 == 0 && CQ % 2 == 0, "8-byte aligned components");
  static_assert(CU < 65536 && 7 * CQ < 65536, "cells are 16-bit");
};

// The state of a voxel pair in registers, as stored: float2, or two 16-bit values in one word.
template <typename SP> struct Held;
template <> struct Held<float> {
  using T = float2;
  static __device__ __forceinline__ void pin(float2&) {}
  static __device__ __forceinline__ float2 get(float2 v) { return v; }
  static __device__ __forceinline__ float2 put(float2 v) { return v; }
};
template <> struct Held<__half> {
  using T = __half2;
  static __device__ __forceinline__ void pin(__half2& v) { asm volatile("" : "+r"(reinterpret_cast<unsigned&>(v))); }
  static __device__ __forceinline__ float2 get(__half2 v) { return __half22float2(v); }
  static __device__ __forceinline__ __half2 put(float2 v) { return __floats2half2_rn(v.x, v.y); }
};
template <> struct Held<__nv_bfloat16> {
  using T = __nv_bfloat162;
  static __device__ __forceinline__ void pin(__nv_bfloat162& v) { asm volatile("" : "+r"(reinterpret_cast<unsigned&>(v))); }
  static __device__ __forceinline__ float2 get(__nv_bfloat162 v) { return __bfloat1622float2(v); }
  static __device__ __forceinline__ __nv_bfloat162 put(float2 v) { return __floats2bfloat162_rn(v.x, v.y); }
};
// u rounded to its storage type (the value the next iteration reads)
template <typename SU> __device__ __forceinline__ float2 as_stored(float2 v) { return Held<SU>::get(Held<SU>::put(v)); }

// Single 128-bit accesses at GPU scope: {a, b, c, tag}.
__device__ __forceinline__ void word_publish(uint4* p, float a, float b, float c, unsigned tag) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\t"
      "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 t, {lo, hi};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(tag)
      : "memory");
}
// ...read only if `on` (zeros otherwise: a word that is already here is not asked for again)
__device__ __forceinline__ uint4 word_poll(const uint4* p, unsigned on) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\tmov.b64 lo, 0;\n\tmov.b64 hi, 0;\n\tmov.b128 t, {lo, hi};\n\t"
      "@q ld.relaxed.gpu.global.b128 t, [%4];\n\tmov.b128 {lo, hi}, t;\n\t"
      "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p), "r"(on)
      : "memory");
  return v;
}
// Shared memory of another CTA of the cluster...
__device__ __forceinline__ unsigned peer_address(const void* p, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
// ...stored to asynchronously; the bytes are counted by an mbarrier of that CTA
__device__ __forceinline__ void peer_store(unsigned p, float v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(p), "f"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
  asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool bar_done(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 q, [%1], %2;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
// Every thread of the cluster that has not returned; what was written before can be read after.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return vadd(a, make_float2(-b.x, -b.y)); }

template <typename SU, typename SP, typename C>
__global__ void __launch_bounds__(C::NT) __maxnreg__(C::REGS)
resident_kernel(const __grid_constant__ ResLaunch L, const Desc* __restrict__ descs, const ResidentArgs a,
                int* __restrict__ status) {
  constexpr int NP = C::NP;
  using H = Held<SP>;
  using HT = typename H::T;
  extern __shared__ __align__(16) float sm[];
  float* const su = sm;
  float* const sqx = sm + 3 * C::CU;
  float* const sqy = sqx + 3 * C::CQ;
  float* const sqz = sqy + 3 * C::CQ;

  const ResPair& B = L.pair[L.of[blockIdx.x]];
  const Desc& d = descs[B.desc];
  // a stopped pair (the flag is the same in every box of the pair), or an earlier launch gave up
  if constexpr (C::CLUSTER) {
    if (d.stop && *d.stop) return;
    if (blockIdx.x - B.first >= B.gx * B.gy * B.gz) return;  // no box for this block of the cluster
  } else {
    if (__syncthreads_or((d.stop && *d.stop) || *reinterpret_cast<volatile int*>(a.abort))) return;
  }
  const int bx = __shfl_sync(~0u, (int)B.bx, 0), by = __shfl_sync(~0u, (int)B.by, 0), bz = __shfl_sync(~0u, (int)B.bz, 0);
  const int box = blockIdx.x - B.first;
  const int gz_ = box / (B.gx * B.gy), gy_ = (box - gz_ * B.gx * B.gy) / B.gx, gx_ = box - (gz_ * B.gy + gy_) * B.gx;
  const int x0 = gx_ * bx, y0 = gy_ * by, z0 = gz_ * bz;
  const int rx = d.nx - x0, ry = d.ny - y0, rz = d.nz - z0;  // voxels from the box's origin to the volume's end
  const int bid = blockIdx.x, ny_step = B.gx, nz_step = B.gx * B.gy;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int PU = (by + 2) * bx, PX = by * bx;      // plane strides of u and q_y, of q_x and q_z
  const int UXLO = (bz + 2) * PU, UXHI = UXLO + bz * by;  // halo columns, one cell per (z, y)
  const int QXLO = bz * PX, QXHI = QXLO + bz * by;
  const int nface = 2 * (bz * by + bz * bx + by * bx);
  const int fy0 = 2 * bz * by, fz0 = fy0 + 2 * bz * bx;  // first y face word, first z face word
  const int cs = (int)d.cs;
  const int gplane = d.pitch * d.ny;
  const SU* u_src = reinterpret_cast<const SU*>(d.u[a.src]);

  for (int i = tid; i < C::SMEM / 4; i += nt) sm[i] = 0.f;
  __syncthreads();

  // ---- this thread's face voxels (word tid + i nt of each field): across a face with a neighbour,
  // the own cell to publish and the halo cell to fill; on a face of the volume, the cell outside
  // that mirrors u (filled from two cells further in) and the own cell whose q is zero
  const int S = a.words;
  unsigned ucell[C::NE], qcell[C::NE];  // halo | own << 16 (u's from 0, q's from sqx)
  int word[C::NE];                      // word to publish to (u), -1: volume face, -2: none
  unsigned peer[C::CLUSTER ? C::NE : 1];  // CLUSTER: u of the neighbouring box (halo: its cells)
#pragma unroll
  for (int i = 0; i < C::NE; ++i) {
    const int e = tid + i * nt;
    word[i] = -2;
    ucell[i] = qcell[i] = 0;
    if (e >= nface) continue;
    int f, k, x = 0, y = 0, z = 0;
    if (e < fy0) {
      f = e >= bz * by;
      k = e - f * bz * by;
      z = k / by;
      y = k - z * by;
    } else if (e < fz0) {
      f = 2 + (e - fy0 >= bz * bx);
      k = e - fy0 - (f - 2) * bz * bx;
      z = k / bx;
      x = k - z * bx;
    } else {
      f = 4 + (e - fz0 >= by * bx);
      k = e - fz0 - (f - 4) * by * bx;
      y = k / bx;
      x = k - y * bx;
    }
    if (x >= rx || y >= ry || z >= rz) continue;
    const int ax = f >> 1, hi = f & 1;
    const int n = ax == 0 ? bx : ax == 1 ? by : bz, r = ax == 0 ? rx : ax == 1 ? ry : rz;
    const int org = ax == 0 ? x0 : ax == 1 ? y0 : z0, step = ax == 0 ? 1 : ax == 1 ? ny_step : nz_step;
    const bool nb = hi ? r > n : org > 0;
    const int m = min(n, r);  // the box's extent along the axis
    auto at = [&](int v) {    // u cell at coordinate v along the axis (-1 and the box's end: halo)
      const int cx = ax == 0 ? v : x, cy = ax == 1 ? v : y, cz = ax == 2 ? v : z;
      if (cx < 0) return UXLO + cz * by + cy;
      if (cx == bx) return UXHI + cz * by + cy;
      return (cz + 1) * PU + (cy + 1) * bx + cx;
    };
    auto q_at = [&](int v) {  // cell of q's component normal to the face
      if (ax == 0) return v < 0 ? QXLO + k : v == bx ? QXHI + k : (z * by + y) * bx + v;
      if (ax == 1) return 3 * C::CQ + z * PU + (v + 1) * bx + x;
      return 6 * C::CQ + (v + 1) * PX + k;
    };
    const int outside = hi ? m : -1, edge = hi ? m - 1 : 0;
    if (nb) {
      const int first = ax == 0 ? 0 : ax == 1 ? fy0 : fz0, other = first + (hi ? 0 : (fy0 * (ax == 0) + (fz0 - fy0) * (ax == 1) + (nface - fz0) * (ax == 2)) / 2);
      word[i] = (bid + (hi ? step : -step)) * 2 * S + other + k;
      ucell[i] = at(outside) | at(edge) << 16;
      qcell[i] = q_at(outside) | q_at(edge) << 16;
      const int vx = ax == 0 ? outside : x, vy = ax == 1 ? outside : y, vz = ax == 2 ? outside : z;
      const int o = (z0 + vz) * gplane + (y0 + vy) * d.pitch + x0 + vx;
#pragma unroll
      for (int c = 0; c < 3; ++c) su[c * C::CU + at(outside)] = Store<SU>::ld(u_src + (long long)c * cs + o);
      if constexpr (C::CLUSTER) {
        peer[i] = peer_address(su, (unsigned)(box + (hi ? step : -step)));
        ucell[i] = at(hi ? -1 : n) | at(edge) << 16;
        qcell[i] = q_at(hi ? -1 : n) | q_at(edge) << 16;
      }
    } else {
      word[i] = -1;
      ucell[i] = at(outside) | at(hi ? m - 2 : 1) << 16;
      qcell[i] = q_at(edge) << 16;
    }
  }

  // ---- this thread's column: pairs (xl, xl+1) at (yl, zl0 .. zl0 + nj - 1)
  const int hx = bx >> 1, ncol = hx * by;
  const int zg = tid / ncol, col = tid - zg * ncol;
  const int yl = col / hx, xl = 2 * (col - yl * hx), zl0 = zg * NP;
  int nj = (xl < rx && yl < min(ry, by)) ? min(max(min(rz, bz) - zl0, 0), NP) : 0;
  int iu = ((zl0 + 1) * (by + 2) + yl + 1) * bx + xl;  // own cell of u; of q_y: - PU
  int iqx = (zl0 * by + yl) * bx + xl;                 // own cell of q_x; of q_z: + PX
  // cells left and right of the pair (halo columns at the box's ends) and their step along z; of
  // q_x: - dUQ at the ends
  const bool xlo = xl == 0, xhi = xl + 2 == bx;
  int aL = xlo ? UXLO + zl0 * by + yl : iu - 1, dL = xlo ? by : PU;
  int aR = xhi ? UXHI + zl0 * by + yl : iu + 2, dR = xhi ? by : PU;
  const int dUQ = UXLO - QXLO;
  int o0 = (z0 + zl0) * gplane + (y0 + yl) * d.pitch + x0 + xl;

  HT P[NP][9], D[C::KEEP_D ? NP : 1][6], R[NP][4];  // D not kept: one pair's
  auto load_D = [&](int j) {
    const int o = o0 + j * gplane;
#pragma unroll
    for (int c = 0; c < 6; ++c)
      D[C::KEEP_D ? j : 0][c] = __ldg(reinterpret_cast<const HT*>(reinterpret_cast<const SP*>(d.D) + (long long)c * cs + o));
  };
  auto load_R = [&](int j) {
    const int o = o0 + j * gplane;
    R[j][0] = __ldg(reinterpret_cast<const HT*>(reinterpret_cast<const SP*>(d.rc) + o));
#pragma unroll
    for (int c = 0; c < 3; ++c)
      R[j][1 + c] = __ldg(reinterpret_cast<const HT*>(reinterpret_cast<const SP*>(d.gw) + (long long)c * cs + o));
  };
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 9; ++c) P[j][c] = H::put(zero);
#pragma unroll
    for (int c = 0; c < 6; ++c) D[C::KEEP_D ? j : 0][c] = H::put(zero);
#pragma unroll
    for (int c = 0; c < 4; ++c) R[j][c] = H::put(zero);
    if (j < nj) {
      const int o = o0 + j * gplane;
      const bool two = xl + 1 < rx;
      auto take = [&](const void* base, int c) {
        HT v = *reinterpret_cast<const HT*>(reinterpret_cast<const SP*>(base) + (long long)c * cs + o);
        if (!two) v = H::put(make_float2(H::get(v).x, 0.f));
        return v;
      };
#pragma unroll
      for (int c = 0; c < 9; ++c) P[j][c] = take(d.p[a.src], c);
      if constexpr (C::KEEP_D) load_D(j);
      if constexpr (C::KEEP_R) load_R(j);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const SU* s = u_src + (long long)c * cs + o;
        su[c * C::CU + iu + j * PU] = Store<SU>::ld(s);
        if (two) su[c * C::CU + iu + j * PU + 1] = Store<SU>::ld(s + 1);
      }
    }
  }

  const float wtv2 = a.wtv * a.wtv;
  float2 step_len[C::EARLY ? NP : 1];  // EARLY: of the L1 shrinkage, computed while q's faces travel
  auto early_steps = [&](float factor) {
    if constexpr (C::EARLY) {
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        step_len[j] = make_float2(0.f, 0.f);
        if (j < nj) {
          float2 uo[3], g[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            uo[c] = *reinterpret_cast<const float2*>(su + c * C::CU + iu + j * PU);
            g[c] = H::get(R[j][1 + c]);
          }
          step_len[j] = primal_step(uo, factor, H::get(R[j][0]), g);
        }
      }
    }
  };

  auto pair_at = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
  const uint4* const in0 = a.xbuf + (long long)blockIdx.x * 2 * S;
  const uint64_t wait_ns = (uint64_t)a.wait_us * 1000ull;
  // faces of u (or of q) after every thread's part is in shared memory: published, or mirrored
  // (zeroed) at the volume's faces
  auto send = [&](bool q, unsigned tag) {
    float* s = q ? sqx : su;
    const int st = q ? C::CQ : C::CU;
    float v[C::NE][3];
#pragma unroll
    for (int i = 0; i < C::NE; ++i) {  // (a thread without a voxel here reads cell 0)
      const float* own = s + ((q ? qcell[i] : ucell[i]) >> 16);
      v[i][0] = own[0];
      v[i][1] = own[st];
      v[i][2] = own[2 * st];
    }
#pragma unroll
    for (int i = 0; i < C::NE; ++i) {
      if (word[i] >= 0) {
        if constexpr (C::CLUSTER) {
          const unsigned out = peer[i] + 4 * ((q ? 3 * C::CU : 0) + ((q ? qcell[i] : ucell[i]) & 0xffff));
#pragma unroll
          for (int c = 0; c < 3; ++c) peer_store(out + 4 * c * st, v[i][c], peer[i] + C::BAR + (q ? 8 : 0));
        } else {
          word_publish(a.xbuf + word[i] + (q ? S : 0), v[i][0], v[i][1], v[i][2], tag);
        }
      } else if (word[i] == -1) {
        float* out = s + (q ? qcell[i] >> 16 : ucell[i] & 0xffff);
        out[0] = q ? 0.f : v[i][0];
        out[st] = q ? 0.f : v[i][1];
        out[2 * st] = q ? 0.f : v[i][2];
      }
    }
  };
  // waits for the neighbours' words of one field and stores them; false: gave up
  auto receive = [&](bool q, unsigned tag) {
    const uint4* in = in0 + (q ? S : 0);
    float* s = q ? sqx : su;
    const int st = q ? C::CQ : C::CU;
    unsigned pending = 0;
#pragma unroll
    for (int i = 0; i < C::NE; ++i)
      if (word[i] >= 0) pending |= 1u << i;
    uint64_t t0 = 0;
    for (unsigned spin = 0; pending; ++spin) {
      uint4 w[C::NE];
#pragma unroll
      for (int i = 0; i < C::NE; ++i)
        w[i] = word_poll(in + tid + i * nt, pending & (1u << i));
#pragma unroll
      for (int i = 0; i < C::NE; ++i) {
        if (!(pending & (1u << i)) || w[i].w != tag) continue;
        float* out = s + ((q ? qcell[i] : ucell[i]) & 0xffff);
        out[0] = __uint_as_float(w[i].x);
        out[st] = __uint_as_float(w[i].y);
        out[2 * st] = __uint_as_float(w[i].z);
        pending &= ~(1u << i);
      }
      if (pending && (spin & 31) == 31) {
        if (*reinterpret_cast<volatile int*>(a.abort)) return false;
        const uint64_t now = global_ns();
        if (!t0) t0 = now;
        else if (now - t0 > wait_ns) {
          atomicExch(a.abort, 1);
          return false;
        }
      }
    }
    return true;
  };

  // CLUSTER: the neighbours' faces of one field have arrived (false: gave up). The phase is armed by
  // thread 0; bytes that came before that are already counted.
  const unsigned bars = (unsigned)__cvta_generic_to_shared(sm) + C::BAR;
  unsigned face_bytes = 0;
  if constexpr (C::CLUSTER) {
#pragma unroll
    for (int i = 0; i < C::NE; ++i) face_bytes += 12 * __syncthreads_count(word[i] >= 0);
    if (tid == 0) {
      bar_init(bars);
      bar_init(bars + 8);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  if constexpr (C::MUTE) {
    if (bid == a.mute) {
#pragma unroll
      for (int i = 0; i < C::NE; ++i)
        if (word[i] >= 0) word[i] = -2;
    }
  }
  auto arrived = [&](bool q, int it) {
    const unsigned bar = bars + (q ? 8 : 0);
    uint64_t t0 = 0;
    for (unsigned spin = 0; !bar_done(bar, it & 1); ++spin) {
      if ((spin & 31) != 31) continue;
      const uint64_t now = global_ns();
      if (!t0) t0 = now;
      else if (now - t0 > wait_ns) return false;
    }
    return true;
  };

  // u mirrored outside the volume for the first iteration
  __syncthreads();
#pragma unroll
  for (int i = 0; i < C::NE; ++i)
    if (word[i] == -1)
#pragma unroll
      for (int c = 0; c < 3; ++c) su[c * C::CU + (ucell[i] & 0xffff)] = su[c * C::CU + (ucell[i] >> 16)];
  __syncthreads();
  if constexpr (C::CLUSTER) cluster_barrier();  // every box's arrays are filled before a neighbour writes to them

  bool bad = false;
  float next_sigma = __ldg(a.sig), next_tau = __ldg(a.tau);
  for (int it = 0; it < a.iters; ++it) {
    // keeps what is derived from these from being computed once, before the loop, and held
    asm volatile("" : "+r"(iu), "+r"(iqx), "+r"(aL), "+r"(aR), "+r"(dL), "+r"(dR), "+r"(o0), "+r"(nj));
    if constexpr (C::KEEP_D) {
#pragma unroll
      for (int j = 0; j < NP; ++j)
#pragma unroll
        for (int c = 0; c < 6; ++c) H::pin(D[j][c]);
    }
    const float sigma = next_sigma, tau = next_tau;
    if (it + 1 < a.iters) {
      next_sigma = __ldg(a.sig + it + 1);
      next_tau = __ldg(a.tau + it + 1);
    }
    const float factor = __fmul_rn(tau, a.wm);  // opticalFlowOps.cu:440
    const float hsigma = 0.5f * sigma;
    // ---- dual
    if (nj > 0) {
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        if (j < nj) {
          const int i = iu + j * PU;
          if constexpr (!C::KEEP_D) load_D(j);
          // every read of u before the first write of q (the compiler cannot tell them apart)
          float2 e[3][3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float* s = su + c * C::CU;
            const float2 o = pair_at(s + i);
            e[c][0] = vsub(make_float2(o.y, s[aR + j * dR]), make_float2(s[aL + j * dL], o.x));
            e[c][1] = vsub(pair_at(s + i + bx), pair_at(s + i - bx));
            e[c][2] = vsub(pair_at(s + i + PU), pair_at(s + i - PU));
          }
          float2 Dk[6];
#pragma unroll
          for (int c = 0; c < 6; ++c) Dk[c] = H::get(D[C::KEEP_D ? j : 0][c]);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            float2 p0 = H::get(P[j][3 * c]), p1 = H::get(P[j][3 * c + 1]), p2 = H::get(P[j][3 * c + 2]);
            dual_row(Dk, e[c][0], e[c][1], e[c][2], p0, p1, p2, hsigma, a.wtv, wtv2);
            *reinterpret_cast<float2*>(sqx + c * C::CQ + iqx + j * PX) = dot3(Dk[0], Dk[1], Dk[2], p0, p1, p2);
            *reinterpret_cast<float2*>(sqy + c * C::CQ + i - PU) = dot3(Dk[1], Dk[3], Dk[4], p0, p1, p2);
            *reinterpret_cast<float2*>(sqz + c * C::CQ + iqx + PX + j * PX) = dot3(Dk[2], Dk[4], Dk[5], p0, p1, p2);
            P[j][3 * c] = H::put(p0);
            P[j][3 * c + 1] = H::put(p1);
            P[j][3 * c + 2] = H::put(p2);
          }
        }
      }
    }
    if constexpr (!C::KEEP_R) {
#pragma unroll
      for (int j = 0; j < NP; ++j)
        if (j < nj) load_R(j);
    }
    if constexpr (C::CLUSTER) {
      if (__syncthreads_or(bad)) {
        bad = true;
        break;
      }
      if (tid == 0) bar_expect(bars + 8, face_bytes);
      send(true, (unsigned)it + 1);
      early_steps(factor);
      __syncthreads();
      bad = !arrived(true, it);
    } else {
      __syncthreads();
      send(true, (unsigned)it + 1);
      early_steps(factor);
      bad = !receive(true, (unsigned)it + 1);
      if (__syncthreads_or(bad)) {
        bad = true;
        break;
      }
    }
    // ---- primal
    asm volatile("" : "+r"(iu), "+r"(iqx), "+r"(aL), "+r"(aR));
    float2 zm[3], zc[3];  // ROLL: q_z of the planes below and at the pair's
    if (C::ROLL && nj > 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        zm[c] = pair_at(sqz + c * C::CQ + iqx);
        zc[c] = pair_at(sqz + c * C::CQ + iqx + PX);
      }
    }
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      // (ROLL: planes past the box's last are computed, on cells inside the arrays, and not stored)
      if (C::ROLL ? nj > 0 : j < nj) {
        float2 uo[3], g[3], n[3], dv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          uo[c] = pair_at(su + c * C::CU + iu + j * PU);
          g[c] = H::get(R[j][1 + c]);
        }
        float2 t;
        if constexpr (C::EARLY) t = step_len[j];
        else t = primal_step(uo, factor, H::get(R[j][0]), g);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float* qx = sqx + c * C::CQ;
          const float* qy = sqy + c * C::CQ + iu - PU + j * PU;
          const float* qz = sqz + c * C::CQ + iqx + PX + j * PX;
          const float2 o = pair_at(qx + iqx + j * PX);
          const float2 dx = vsub(make_float2(qx[xlo ? aL - dUQ + j * by : iqx + j * PX - 1], o.x),
                                 make_float2(o.y, qx[xhi ? aR - dUQ + j * by : iqx + j * PX + 2]));
          const float2 dy = vsub(pair_at(qy - bx), pair_at(qy + bx));
          const float2 zp = pair_at(qz + PX);
          dv[c] = sum3(dx, dy, vsub(C::ROLL ? zm[c] : pair_at(qz - PX), zp));
          if constexpr (C::ROLL) {
            zm[c] = zc[c];
            zc[c] = zp;
          }
        }
        primal_apply(uo, dv, 0.5f * tau, t, g, n);
        // (the voxel beside the volume's last one, odd nx: a mirror cell, filled again below)
        if (!C::ROLL || j < nj)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            *reinterpret_cast<float2*>(su + c * C::CU + iu + j * PU) = as_stored<SU>(n[c]);
      }
    }
    if (it + 1 < a.iters) {
      if constexpr (C::CLUSTER) {
        if (__syncthreads_or(bad)) {
          bad = true;
          break;
        }
        if (tid == 0) bar_expect(bars, face_bytes);
        send(false, (unsigned)it + 1);
        __syncthreads();
        bad = !arrived(false, it);
      } else {
        __syncthreads();
        send(false, (unsigned)it + 1);
        bad = !receive(false, (unsigned)it + 1);
        if (__syncthreads_or(bad)) {
          bad = true;
          break;
        }
      }
    }
  }
  if constexpr (C::CLUSTER) bad = __syncthreads_or(bad);
  if (bad) {
    if (tid == 0) atomicOr(status, SVS_DEV_TIMEOUT);
    if constexpr (C::CLUSTER) {  // until no other block sends any more, and what it sent has landed
      cluster_barrier();
      for (const uint64_t t = global_ns(); global_ns() - t < 20000;) {}
    }
    return;
  }

  // ---- state back to memory, incoming words cleared for the next launch. The neighbours read
  // their first halos from copy `src` before they published what this box consumed, so the write
  // may go to the same copy.
  SU* u_dst = reinterpret_cast<SU*>(d.u[a.dst]);
  SP* p_dst = reinterpret_cast<SP*>(d.p[a.dst]);
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    if (j < nj) {
      const int o = o0 + j * gplane;
      const bool two = xl + 1 < rx;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float2 v = pair_at(su + c * C::CU + iu + j * PU);
        SU* s = u_dst + (long long)c * cs + o;
        Store<SU>::st(s, v.x);
        if (two) Store<SU>::st(s + 1, v.y);
      }
#pragma unroll
      for (int c = 0; c < 9; ++c) {
        SP* s = p_dst + (long long)c * cs + o;
        if (two) *reinterpret_cast<HT*>(s) = P[j][c];
        else Store<SP>::st(s, H::get(P[j][c]).x);
      }
    }
  }
  if constexpr (!C::CLUSTER) {
#pragma unroll
    for (int i = 0; i < C::NE; ++i) {
      if (word[i] < 0) continue;
      word_publish(const_cast<uint4*>(in0) + tid + i * nt, 0.f, 0.f, 0.f, 0u);
      word_publish(const_cast<uint4*>(in0) + S + tid + i * nt, 0.f, 0.f, 0.f, 0u);
    }
  }
}

// Compiled shapes, every storage mode (svs_resident.cu).
// (two face words per thread in the one-pair shapes: every exchange visits all of a thread's slots, and with
// four 35x41x47 took 3.25 us, 40^3 3.2, f32 9x11x12 in a cluster 1.43, against 3.05, 3.0 and 1.22)
using ResSmall = ResShape<1, 512, 1920, 1408, 2, true, true>;
using ResMid = ResShape<2, 512, 3456, 2688, 4, true, false>;
// (5 pairs by 384 threads: 6 by 320 took 13.4 us at 80^3 f16-flow32, 8 by 256 11.9-14, against 10.6;
// the register file is split by scheduler, so 13 to 16 warps would have 128 registers each)
template <typename SP> using ResLarge = ResShape<5, 384, 5408, 4480, 4, sizeof(SP) == 2, false>;
using ResCluster = ResShape<1, 512, 1920, 1408, 2, true, true, true>;
constexpr int kResShapes = 4, kResMaxWords = 2048;
constexpr int kResClusterBlocks = 16;  // of a cluster at most
// Host view of a shape: voxel pairs and threads, floats per component, face words per thread.
struct ResCaps {
  int np, nt, cu, cq, ne;
  bool cluster;
};
template <typename C> constexpr ResCaps res_caps() { return {C::NP, C::NT, C::CU, C::CQ, C::NE, C::CLUSTER}; }
constexpr ResCaps kResCaps[kResShapes] = {res_caps<ResSmall>(), res_caps<ResMid>(), res_caps<ResLarge<__half>>(),
                                           res_caps<ResCluster>()};

// op 0: set the kernel's attributes and return in *occ the CTAs one SM holds, or the clusters of
// kResClusterBlocks CTAs that the GPU holds (false: not usable); op 1: one launch of `grid` CTAs of `threads`
// threads on stream s, cooperative or in clusters of L->cluster. With a->mute set the launch takes the form
// with the hook (FP32 and f16-flow32 storage; false for the others).
bool resident_variant(int storage, int shape, int op, unsigned grid, unsigned threads, const ResLaunch* L,
                      const Desc* descs, const ResidentArgs* a, int* status, cudaStream_t s, int* occ);
bool resident_mute(int storage, int shape, int op, unsigned grid, unsigned threads, const ResLaunch* L, const Desc* descs,
                   const ResidentArgs* a, int* status, cudaStream_t s, int* occ);

// Attributes or launch of one instantiation (op as above).
template <typename SU, typename SP, typename C>
bool resident_run(int op, unsigned grid, unsigned threads, const ResLaunch* L, const Desc* descs, const ResidentArgs* a,
                  int* status, cudaStream_t s, int* occ) {
  const auto k = resident_kernel<SU, SP, C>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if constexpr (C::CLUSTER) {
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = op ? L->cluster : kResClusterBlocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  } else {
    // its CTAs wait for one another: a cooperative launch starts only a grid that fits the GPU at once
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
  }
  if (op == 0) {
    bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) == cudaSuccess;
    if constexpr (C::CLUSTER) {
      cfg.gridDim = dim3(kResClusterBlocks);
      cfg.blockDim = dim3(C::NT);
      ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
           cudaOccupancyMaxActiveClusters(occ, k, &cfg) == cudaSuccess;
    } else {
      ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, C::NT, C::SMEM) == cudaSuccess;
    }
    if (!ok) cudaGetLastError();
    return ok && *occ > 0;
  }
  return cudaLaunchKernelEx(&cfg, k, *L, descs, *a, status) == cudaSuccess;
}

}  // namespace svs
