// Tile kernels: one launch per time step, every row of a tile in parallel.
//
// The marching kernels (ds2d_fused.cuh, ds2d_pair.cuh, ds2d_tblock.cuh, ds2d_bwdbulk.cuh) walk a
// strip of columns row by row behind one or two barriers a row: about 1.3 us a row step, however
// few CTAs there are.  That is the right shape for batches that fill the chip several times over,
// and a serial chain of 100-200 us per launch for a batch that does not (one shot on 291x141 padded
// cells: 9 CTAs, 196 us a step, of which the 0.8 MB of state and the arithmetic would need about 1).
// Here a CTA owns TX x 32 output cells and all of its work is in flight at once:
//   load     the stencil inputs of the tile plus 8 cells on each side into shared memory;
//   stage 1  (velocities / reconstructed and adjoint stresses) of the tile plus 4 cells, written
//            to shared memory, the tile's own cells to global memory too;
//   stage 2  (stresses / velocities) of the tile.
// Two barriers in all.  A thread owns R consecutive rows of one column, so its x-taps come from a
// column of R + 7 shared loads per derivative instead of 8 R.  The redundant work (stage 1 on
// (TX + 8) x 40 cells for TX x 32) is paid from idle SMs; the state of such batches stays in L2.
// State ping-pongs between two buffers as in the marching kernels.
//
// Measured (B200, whole calls, against the marching kernels): forward of one 251x101 shot + 20 PML,
// 2000 steps: 391 -> 9.1 ms; RTM of 2 64x32 shots, 200 steps: 22 -> 1.25 ms; ELSRTM of 4 251x101
// shots, 500 steps: 536 -> 25 ms; CG-LSRTM of 8 96x48 shots: 245 -> 11 ms (7.8 with L^T on L's
// background).  What bounds a full grid is latency: registers hold an SM to 20-25 warps, which use
// 38-51 % of the issue slots, global loads first among the stalls.
//
// Launches of consecutive steps use programmatic dependent launch: a CTA fetches everything that
// no step writes (moduli, damping, image weights, trace indexes, residuals) before
// griddepcontrol.wait and the state after it, so that part of a step overlaps the previous one.
// The first launch behind other kernels is an ordinary one.
#pragma once
#include "ds2d_fused.cuh"
#include "ds2d_step.cuh"

namespace ds2d {

constexpr int kTileZ = 32;              // output columns of a tile
constexpr int kTileC1 = kTileZ + 8;     // stage-1 columns (tile + 4 on each side)
constexpr int kTileC0 = kTileZ + 16;    // input columns (tile + 8)
// Shape of a tile step: TX output rows, kG stage-1 row groups of R1 rows (40 kG threads), kG2 stage-2
// row groups of R2 rows (one warp each).
template <int kTX, int kG>
struct TileCfg {
  static constexpr int TX = kTX, G = kG, T = kTileC1 * kG, R1 = (kTX + 8) / kG;
  static_assert(R1 * kG == kTX + 8, "row groups cover the tile plus 8 rows");
  static constexpr int G2 = kTX <= T / 32 ? kTX : kTX / 2 <= T / 32 ? kTX / 2 : kTX / 4;
  static constexpr int R2 = kTX / G2;
  // Shared row pitch of the inputs: a multiple of 4 floats (16-byte copies) that puts the row
  // groups of neighbouring lanes 8 banks apart.
  static constexpr int P0 = R1 == 3 ? 56 : 52;
  static constexpr int N0 = (kTX + 16) * P0, N1 = (kTX + 8) * kTileC1;
  static constexpr int kLd = ((kTX + 16) * (kTileC0 / 4) + T - 1) / T;  // 16-byte copies per thread
  static constexpr size_t smem(int inputs, int mids) {
    return sizeof(float) * ((size_t)inputs * N0 + (size_t)mids * N1);
  }
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
// 16-byte copy global -> shared, zeros when !in.
__device__ __forceinline__ void cp_async16z(float *smem, const float *gmem, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}

// A product that is rounded before it is added: the update's two increments and the split parts are
// summed as rounded values, in every variant of a step and as in the PML ring kernels, so that a
// cell's bits do not depend on which class its tile belongs to (nor 16-bit strips on the path).
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }

// Tiles cover the updated cells [nop, n - nop) only.
template <int TX>
__device__ __forceinline__ int tile_x0() { return 4 + blockIdx.y * TX; }
__device__ __forceinline__ int tile_z0() { return 4 + blockIdx.x * kTileZ; }

// Class of a tile, a template parameter of the step functions so that the larger part of a grid runs
// without a test per cell: kTileInner = its whole input window lies in the interior, at least nop
// cells from the PML or random band (every cell is updated and imaged, none is a PML or strip
// cell); kTilePml = a PML context's other tiles; kTileEdge = a random-boundary context's.
constexpr int kTileEdge = 0, kTilePml = 1, kTileInner = 2;
template <int TX>
__device__ __forceinline__ bool tile_inner(const Dims &d, const ShotDev &sh) {
  const int e = d.pml + d.nop, x0 = tile_x0<TX>(), z0 = tile_z0();
  return x0 - 8 >= e && x0 + TX + 8 <= sh.nxp - e && z0 - 8 >= e && z0 + kTileZ + 8 <= d.nzp - e;
}

// Copies one field's input window (tile + 8) of the slot at `base` into dst.  Windows start on
// 16-byte boundaries (tile columns are multiples of 32, rows `ld` multiples of 32); rows and
// columns outside the padded grid are zeros.
template <class C, bool kIn = false>
__device__ __forceinline__ void tile_load(float *dst, const float *src, const Dims &d, int base,
                                          int x0, int z0) {
  for (int i = threadIdx.x; i < (C::TX + 16) * (kTileC0 / 4); i += C::T) {
    const int r = i / (kTileC0 / 4), c = (i - r * (kTileC0 / 4)) * 4;
    const int x = x0 - 8 + r, z = z0 - 8 + c;
    const bool in = kIn || (x >= 0 && x < d.nxp && z >= 0 && z < d.ld);
    cp_async16z(dst + r * C::P0 + c, src + (in ? base + x * d.ld + z : 0), in);
  }
}

// R derivatives along x of the cells p, p + pitch, ... (8 taps each): out[r] = sum c_i (f[+i] -
// f[1-i]) (kAhead) or sum c_i (f[i-1] - f[-i]).
template <int R, bool kAhead>
__device__ __forceinline__ void tile_dx(const float *p, int pitch, float (&out)[R]) {
  float w[R + 7];
#pragma unroll
  for (int j = 0; j < R + 7; j++) w[j] = p[(j - (kAhead ? 3 : 4)) * pitch];
#pragma unroll
  for (int r = 0; r < R; r++) out[r] = stencil4([&](int i) { return w[r + 3 + i] - w[r + 4 - i]; });
}
__device__ __forceinline__ float tile_dzp(const float *p) {
  return stencil4([&](int i) { return p[i] - p[1 - i]; });
}
__device__ __forceinline__ float tile_dzm(const float *p) {
  return stencil4([&](int i) { return p[i - 1] - p[-i]; });
}

// add_born_source (born.cu:351-405) of one cell from Dx- vx, Dz- vz, Dz+ vx, Dx+ vz.  The order of
// the fused multiply-adds is written out: it is the one k_fwd_ring and k_born round by, and the
// first-order set's images keep every bit of the source only if it does not vary between kernels.
struct BornSrc {
  float xx, zz, xz;
};
__device__ __forceinline__ BornSrc born_source(float lam, float mu, float dmp, float dms, float sa,
                                               float sb, float se, float sf, float rdx, float rdz) {
  const float l2m = lam + 2.0f * mu, m2 = 2.0f * mu;
  const float P = 2.0f * l2m * (-dmp);
  const float Q = 2.0f * __fmaf_rn(-m2, -dms, __fmul_rn(l2m, -dmp));
  BornSrc e;
  e.xx = __fmaf_rn(__fmul_rn(P, sa), rdx, __fmul_rn(__fmul_rn(Q, sb), rdz));
  e.zz = __fmaf_rn(__fmul_rn(P, sb), rdz, __fmul_rn(__fmul_rn(Q, sa), rdx));
  e.xz = __fmul_rn(m2 * (-dms), __fmaf_rn(sf, rdx, __fmul_rn(se, rdz)));
  return e;
}

// Whether the tile plus `m` cells holds PML cells.
template <int TX>
__device__ __forceinline__ bool tile_has_pml(const Dims &d, int x0, int z0, int m) {
  return x0 - m < d.pml || x0 + TX + m - 1 > d.nxp - d.pml || z0 - m < d.pml ||
         z0 + kTileZ + m - 1 > d.nzp - d.pml;
}

// PML factors of one cell: d1 = 1 - dt d / 2 and the rounded reciprocal of 1 + dt d / 2.
struct TileDamp {
  float d1, i2, d3, i4;
};
__device__ __forceinline__ TileDamp tile_damp(float dampx, float dampz, float dt) {
  const float ddx = dampx * dt * 0.5f, ddz = dampz * dt * 0.5f;
  return TileDamp{1.0f - ddx, __frcp_rn(1.0f + ddx), 1.0f - ddz, __frcp_rn(1.0f + ddz)};
}

// ---- forward step (modes of k_fwd_ring: 0 plain, 1 + Born source out, 2 overlay in and Born source
// out, 3 overlay in) ------------------------------------------------------------------------------
template <class C>
constexpr size_t fwd_tile_smem() { return C::smem(3, 2); }

template <int kCls, class C, int kMode>
__device__ __forceinline__ void fwd_tile(const FwdFusedArgs &a, int s, float *sm) {
  constexpr bool kPML = kCls == kTilePml, kIn = kCls == kTileInner;
  constexpr bool kOvIn = kMode >= 2, kBornOut = kMode == 1 || kMode == 2, kSrc = kMode < 2;
  constexpr int TX = C::TX, R1 = C::R1, R2 = C::R2, P0 = C::P0, N0 = C::N0;
  constexpr int kLd = C::kLd;
  float *const i_xx = sm, *const i_zz = sm + N0, *const i_xz = sm + 2 * N0;
  float *const v_x = sm + 3 * N0, *const v_z = v_x + C::N1;
  const int tid = threadIdx.x;
  const ShotDev sh = a.shots[s];
  const Dims d = slot_dims(a.d, sh);
  const int x0 = tile_x0<TX>(), z0 = tile_z0();
  if (x0 >= d.nxp - d.nop) return;  // beyond this slot's window, whole CTA
  const int base = (int)(d.slot * s), ld = d.ld;
  const float dtdx = d.dt / d.dx, dtdz = d.dt / d.dz;
  const bool tp = kPML && tile_has_pml<TX>(d, x0, z0, 4);
  // stage-1 cells: column z1, rows xs1 .. xs1 + R1 - 1; stage-2 cells: column z2, rows xs2 ...
  const int g1 = tid / kTileC1, c1 = tid - g1 * kTileC1, z1 = z0 - 4 + c1, xs1 = x0 - 4 + g1 * R1;
  const int g2 = tid >> 5, c2 = tid & 31, z2 = z0 + c2, xs2 = x0 + g2 * R2;
  const bool zu1 = z1 >= d.nop && z1 < d.nzp - d.nop;
  const bool zu2 = tid < 32 * C::G2 && (kIn || (z2 >= d.nop && z2 < d.nzp - d.nop));
  const bool zi2 = kIn || (z2 >= d.pml && z2 < d.nzp - d.pml);
  const int k1 = base + xs1 * ld + z1, k2 = base + xs2 * ld + z2;
  auto up1 = [&](int r) { return kIn || (zu1 && xs1 + r >= d.nop && xs1 + r < d.nxp - d.nop); };
  auto up2 = [&](int r) { return zu2 && (kIn || (xs2 + r >= d.nop && xs2 + r < d.nxp - d.nop)); };
  auto pm1 = [&](int r) { return tp && pml_cell(d, xs1 + r, z1); };
  auto pm2 = [&](int r) { return tp && pml_cell(d, xs2 + r, z2); };
  auto own1 = [&](int r) {
    const int x = xs1 + r;
    return x >= x0 && x < x0 + TX && c1 >= 4 && c1 < 4 + kTileZ;
  };
  // constants of the run
  float b_[R1], q1x[R1], q1z[R1], lam_[R2], mu_[R2], q2x[R2], q2z[R2], mp_[R2], ms_[R2];
  int tr[R1];
#pragma unroll
  for (int r = 0; r < R1; r++) {
    b_[r] = up1(r) ? __ldg(a.p.b + k1 + r * ld) : 0.f;
    q1x[r] = q1z[r] = 0.f;
    if (kPML && up1(r) && pm1(r)) {
      q1x[r] = __ldg(a.p.dampx + k1 + r * ld);
      q1z[r] = __ldg(a.p.dampz + k1 + r * ld);
    }
    tr[r] = -1;
    if (a.rec_on && z1 == sh.igz && up1(r) && own1(r))
      tr[r] = __ldg(a.rmap + (long long)s * d.nxp_max + xs1 + r);
  }
#pragma unroll
  for (int r = 0; r < R2; r++) {
    lam_[r] = up2(r) ? __ldg(a.p.lam + k2 + r * ld) : 0.f;
    mu_[r] = up2(r) ? __ldg(a.p.mu + k2 + r * ld) : 0.f;
    q2x[r] = q2z[r] = mp_[r] = ms_[r] = 0.f;
    if (kPML && up2(r) && pm2(r)) {
      q2x[r] = __ldg(a.p.dampx + k2 + r * ld);
      q2z[r] = __ldg(a.p.dampz + k2 + r * ld);
    }
    if (kBornOut && up2(r) && zi2 && (kIn || (xs2 + r >= d.pml && xs2 + r < d.nxp - d.pml))) {
      mp_[r] = __ldg(a.p.dmp + k2 + r * ld);
      ms_[r] = __ldg(a.p.dms + k2 + r * ld);
    }
  }
  const float sval = kSrc ? __ldg(a.wavelet + a.it) : 0.f;
  pdl_wait();
  // ---- state -------------------------------------------------------------------------------------
  tile_load<C, kIn>(i_xx, a.a.txx, d, base, x0, z0);
  tile_load<C, kIn>(i_zz, a.a.tzz, d, base, x0, z0);
  tile_load<C, kIn>(i_xz, a.a.txz, d, base, x0, z0);
  cp_async_commit();
  float4 ov[kOvIn ? kLd : 1][3];
  if (kOvIn) {
#pragma unroll
    for (int j = 0; j < kLd; j++) {
      const int i = tid + j * C::T, r = i / (kTileC0 / 4), c = (i - r * (kTileC0 / 4)) * 4;
      const int x = x0 - 8 + r, z = z0 - 8 + c;
      const bool in = r < TX + 16 && (kIn || (x >= 0 && x < d.nxp && z >= 0 && z < ld));
      const int k = in ? base + x * ld + z : 0;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      ov[j][0] = in ? *reinterpret_cast<const float4 *>(a.ovi_txx + k) : zero;
      ov[j][1] = in ? *reinterpret_cast<const float4 *>(a.ovi_tzz + k) : zero;
      ov[j][2] = in ? *reinterpret_cast<const float4 *>(a.ovi_txz + k) : zero;
    }
  }
  float s1[R1][4];  // vx, vz of a cell, or its four split parts in the PML
#pragma unroll
  for (int r = 0; r < R1; r++) {
    s1[r][0] = s1[r][1] = s1[r][2] = s1[r][3] = 0.f;
    if (!up1(r)) continue;
    const int k = k1 + r * ld;
    if (kPML && pm1(r)) {
      s1[r][0] = a.a.vx_x[k]; s1[r][1] = a.a.vx_z[k]; s1[r][2] = a.a.vz_x[k]; s1[r][3] = a.a.vz_z[k];
    } else {
      s1[r][0] = a.a.vx[k]; s1[r][1] = a.a.vz[k];
    }
  }
  float s2[R2][6];  // split stress parts of a PML cell; own stresses under an overlay
#pragma unroll
  for (int r = 0; r < R2; r++) {
#pragma unroll
    for (int j = 0; j < 6; j++) s2[r][j] = 0.f;
    if (!up2(r)) continue;
    const int k = k2 + r * ld;
    if (kPML && pm2(r)) {
      s2[r][0] = a.a.txx_x[k]; s2[r][1] = a.a.txx_z[k]; s2[r][2] = a.a.tzz_x[k];
      s2[r][3] = a.a.tzz_z[k]; s2[r][4] = a.a.txz_x[k]; s2[r][5] = a.a.txz_z[k];
    } else if (kOvIn || (kSrc && z2 == sh.isz && xs2 + r == sh.isx)) {
      s2[r][0] = a.a.txx[k]; s2[r][1] = a.a.tzz[k]; s2[r][2] = a.a.txz[k];
    }
  }
  pdl_launch();
  cp_async_wait<0>();
  if (kOvIn) {  // Born source of the previous set: a thread adds it to the chunks it copied
#pragma unroll
    for (int j = 0; j < kLd; j++) {
      const int i = tid + j * C::T, r = i / (kTileC0 / 4), c = (i - r * (kTileC0 / 4)) * 4;
      if (r >= TX + 16) continue;
#pragma unroll
      for (int f = 0; f < 3; f++) {
        float4 *p = reinterpret_cast<float4 *>(sm + f * N0 + r * P0 + c);
        float4 v = *p;
        v.x += ov[j][f].x; v.y += ov[j][f].y; v.z += ov[j][f].z; v.w += ov[j][f].w;
        *p = v;
      }
    }
  }
  if (kSrc) {  // explosive source (transient): the thread that copied the cell adds it
    const int r = sh.isx - (x0 - 8), c = sh.isz - (z0 - 8);
    if (r >= 0 && r < TX + 16 && c >= 0 && c < kTileC0 &&
        tid == (r * (kTileC0 / 4) + c / 4) % C::T) {
      i_xx[r * P0 + c] += sval;
      i_zz[r * P0 + c] += sval;
    }
  }
  __syncthreads();
  // ---- stage 1: velocities of the tile plus 4 cells ------------------------------------------------
  {
    const int o = (g1 * R1 + 4) * P0 + c1 + 4;
    float ax[R1], fx[R1];
    tile_dx<R1, true>(i_xx + o, P0, ax);
    tile_dx<R1, false>(i_xz + o, P0, fx);
#pragma unroll
    for (int r = 0; r < R1; r++) {
      float vxn = 0.f, vzn = 0.f;
      if (up1(r)) {
        const int k = k1 + r * ld;
        const float bz = tile_dzm(i_xz + o + r * P0);
        const float ez = tile_dzp(i_zz + o + r * P0);
        const float bb = b_[r];
        const float cbx = bb * dtdx, cbz = bb * dtdz;
        const float ux_x = mul(cbx, ax[r]), ux_z = mul(cbz, bz), uz_x = mul(cbx, fx[r]), uz_z = mul(cbz, ez);
        const bool own = own1(r);
        if (kPML && pm1(r)) {
          const TileDamp q = tile_damp(q1x[r], q1z[r], d.dt);
          const float vxx = mul(fmaf(q.d1, s1[r][0], ux_x), q.i2);
          const float vxz = mul(fmaf(q.d3, s1[r][1], ux_z), q.i4);
          const float vzx = mul(fmaf(q.d1, s1[r][2], uz_x), q.i2);
          const float vzz = mul(fmaf(q.d3, s1[r][3], uz_z), q.i4);
          if (own) {
            a.b.vx_x[k] = vxx; a.b.vx_z[k] = vxz; a.b.vz_x[k] = vzx; a.b.vz_z[k] = vzz;
          }
          vxn = vxx + vxz;
          vzn = vzx + vzz;
        } else {
          vxn = s1[r][0] + (ux_x + ux_z);
          vzn = s1[r][1] + (uz_x + uz_z);
        }
        if (own) {
          a.b.vx[k] = vxn;
          a.b.vz[k] = vzn;
          if (tr[r] >= 0) {
            const long long q = ((long long)s * d.max_ntr + tr[r]) * d.nt + a.it;
            a.rec_vz[q] = vzn;
            a.rec_vx[q] = vxn;
          }
        }
      }
      v_x[(g1 * R1 + r) * kTileC1 + c1] = vxn;
      v_z[(g1 * R1 + r) * kTileC1 + c1] = vzn;
    }
  }
  __syncthreads();
  // ---- stage 2: stresses of the tile ------------------------------------------------------------
  if (zu2) {
    const int o = (g2 * R2 + 4) * kTileC1 + c2 + 4, oi = (g2 * R2 + 8) * P0 + c2 + 8;
    float sa[R2], sf[R2];
    tile_dx<R2, false>(v_x + o, kTileC1, sa);
    tile_dx<R2, true>(v_z + o, kTileC1, sf);
#pragma unroll
    for (int r = 0; r < R2; r++) {
      if (!up2(r)) continue;
      const int k = k2 + r * ld, rs = xs2 + r;
      const float sb = tile_dzm(v_z + o + r * kTileC1);
      const float se = tile_dzp(v_x + o + r * kTileC1);
      const float lam = lam_[r], mu = mu_[r];
      const float l2m = lam + 2.0f * mu;
      const float xx_x = mul(l2m * dtdx, sa[r]), xx_z = mul(lam * dtdz, sb);
      const float zz_x = mul(lam * dtdx, sa[r]), zz_z = mul(l2m * dtdz, sb);
      const float xz_x = mul(dtdx * mu, sf[r]), xz_z = mul(dtdz * mu, se);
      if (kPML && pm2(r)) {
        const TileDamp q = tile_damp(q2x[r], q2z[r], d.dt);
        const float a1 = mul(fmaf(q.d1, s2[r][0], xx_x), q.i2);
        const float a2 = mul(fmaf(q.d3, s2[r][1], xx_z), q.i4);
        const float b1 = mul(fmaf(q.d1, s2[r][2], zz_x), q.i2);
        const float b2 = mul(fmaf(q.d3, s2[r][3], zz_z), q.i4);
        const float e1 = mul(fmaf(q.d1, s2[r][4], xz_x), q.i2);
        const float e2 = mul(fmaf(q.d3, s2[r][5], xz_z), q.i4);
        a.b.txx_x[k] = a1; a.b.txx_z[k] = a2;
        a.b.tzz_x[k] = b1; a.b.tzz_z[k] = b2;
        a.b.txz_x[k] = e1; a.b.txz_z[k] = e2;
        a.b.txx[k] = a1 + a2;
        a.b.tzz[k] = b1 + b2;
        a.b.txz[k] = e1 + e2;
      } else {
        float oxx = i_xx[oi + r * P0], ozz = i_zz[oi + r * P0], oxz = i_xz[oi + r * P0];
        if (kOvIn) {  // the inputs carry the overlay
          oxx = s2[r][0]; ozz = s2[r][1]; oxz = s2[r][2];
        } else if (kSrc && z2 == sh.isz && rs == sh.isx) {  // the injected cell: without the source
          oxx = s2[r][0]; ozz = s2[r][1];
        }
        a.b.txx[k] = oxx + (xx_x + xx_z);
        a.b.tzz[k] = ozz + (zz_x + zz_z);
        a.b.txz[k] = oxz + (xz_x + xz_z);
      }
      if (kBornOut && zi2 && (kIn || (rs >= d.pml && rs < d.nxp - d.pml))) {
        const BornSrc e = born_source(lam, mu, mp_[r], ms_[r], sa[r], sb, se, sf[r], 1.0f / d.dx, 1.0f / d.dz);
        a.ovo_txx[k] = e.xx;
        a.ovo_tzz[k] = e.zz;
        a.ovo_txz[k] = e.xz;
      }
    }
  }
}

// Strips of the state that a step reads (the state after step `it`): one warp per 32-element
// segment of a slot, spread over the CTAs of one grid slice.  Same values as k_strip_save.
__device__ __forceinline__ void tile_strips(const StripSaveArgs &a, int s) {
  const Dims d = slot_dims(a.d, a.shots[s]);
  const int lane = threadIdx.x & 31, nseg = (d.lb + 31) / 32;
  const int w0 = (blockIdx.y * gridDim.x + blockIdx.x) * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int nw = gridDim.x * gridDim.y * (blockDim.x / 32);
  pdl_wait();
  pdl_launch();
  for (int w = w0; w < 2 * nseg; w += nw) {
    const int comp = w >= nseg, seg = w - comp * nseg, bo = seg * 32 + lane;
    const bool valid = bo < d.lb;
    float v = 0.f;
    if (valid) {
      int ix, iz;
      band_cell(d, bo, ix, iz);
      v = (comp ? a.vz : a.vx)[d.slot * s + (long long)ix * d.ld + iz];
    }
    strip_put(a, d, s, comp, bo, v, valid);
  }
}

// One launch of a forward pass: up to three wavefield sets (grid slices of n shots each), set m
// one step behind set m - 1, whose Born source of the step before it reads; then the slices that
// save the strips of the states the sets read.  A set or strip slice with it < 0 has nothing to do.
struct FwdTileArgs {
  FwdFusedArgs set[3];
  StripSaveArgs st[2];
  int n, nset, nst;
};

// Forward tiles of 8 rows with a PML and one set serve the smallest batches, whose tiles are mostly
// PML: no separate code for inner tiles.  1000 steps: 0.047 M cells 4.93 -> 4.58 ms, 0.051 M 7.09 ->
// 6.93, 0.113 M 5.77 -> 5.70.  (With registers for 2 CTAs instead of 3 4.39, 6.79 and 7.67.)
template <bool kPML, class C, bool kBorn>
constexpr bool kSmall = kPML && !kBorn && C::TX == 8;

template <bool kPML, class C, bool kBorn>
__global__ void __launch_bounds__(C::T, C::TX == 8 ? 3 : C::TX == 16 ? 2 : 1) k_fwd_tile(const __grid_constant__ FwdTileArgs a) {
  extern __shared__ __align__(16) float tsm[];
  const int m = blockIdx.z / a.n, s = blockIdx.z - m * a.n;
  if (m >= a.nset) {
    const StripSaveArgs &st = a.st[m - a.nset];
    if (st.it >= 0) tile_strips(st, s);
    return;
  }
  if (a.set[m].it < 0) return;
  const FwdFusedArgs &f = a.set[m];
  constexpr int kRest = kPML ? kTilePml : kTileEdge;
  if (!kSmall<kPML, C, kBorn> && tile_inner<C::TX>(f.d, f.shots[s])) {
    if (!kBorn) fwd_tile<kTileInner, C, 0>(f, s, tsm);
    else if (m == 0) fwd_tile<kTileInner, C, 1>(f, s, tsm);
    else if (m == 1) fwd_tile<kTileInner, C, 2>(f, s, tsm);
    else fwd_tile<kTileInner, C, 3>(f, s, tsm);
  } else {
    if (!kBorn) fwd_tile<kRest, C, 0>(f, s, tsm);
    else if (m == 0) fwd_tile<kRest, C, 1>(f, s, tsm);
    else if (m == 1) fwd_tile<kRest, C, 2>(f, s, tsm);
    else fwd_tile<kRest, C, 3>(f, s, tsm);
  }
}

// band_offset with the left / right bands first.
__device__ __forceinline__ int band_offset_lr(const Dims &d, int ix, int iz) {
  const int N = d.nop, pml = d.pml;
  if (iz >= pml && iz < d.nzp - pml) {
    if (ix >= pml - N && ix < pml + N)
      return 4 * N * d.wnx + (ix - (pml - N)) * d.wnz + (iz - pml);
    if (ix >= d.nxp - pml - N && ix < d.nxp - pml + N)
      return 4 * N * d.wnx + 2 * N * d.wnz + (ix - (d.nxp - pml - N)) * d.wnz + (iz - pml);
  }
  return band_offset(d, ix, iz);
}

// ---- backward step (arithmetic of k_bwd_ring) --------------------------------------------------
// Loads one velocity field of a reconstructed set: in tiles that reach the strip band, element by
// element (strip value in the band, state elsewhere), otherwise by 16-byte copies.
// kAc: the acoustic L^T keeps the left / right band's element where two bands meet (the corners).
template <class C, bool kAc = false>
__device__ __forceinline__ void tile_load_strip(float *dst, const float *src, const Dims &d,
                                                int base, int s, int x0, int z0, const Strips &st,
                                                int it, int comp, bool band) {
  if (!band) {
    tile_load<C>(dst, src, d, base, x0, z0);
    return;
  }
  constexpr int kN = (C::TX + 16) * kTileC0, kL = (kN + C::T - 1) / C::T;
  float v[kL];
#pragma unroll
  for (int j = 0; j < kL; j++) {
    const int i = threadIdx.x + j * C::T, r = i / kTileC0, c = i - r * kTileC0;
    const int x = x0 - 8 + r, z = z0 - 8 + c;
    v[j] = 0.f;
    if (i < kN && x >= 0 && x < d.nxp && z >= 0 && z < d.nzp) {
      const int bo = kAc ? band_offset_lr(d, x, z) : band_offset(d, x, z);
      v[j] = bo >= 0 ? strip_get(st, d, s, it, comp, bo) : src[base + x * d.ld + z];
    }
  }
#pragma unroll
  for (int j = 0; j < kL; j++) {
    const int i = threadIdx.x + j * C::T, r = i / kTileC0, c = i - r * kTileC0;
    if (i < kN) dst[r * C::P0 + c] = v[j];
  }
}
// Whether the tile's input window reaches the strip band (4 cells on either side of the interior's
// edges).
template <int TX>
__device__ __forceinline__ bool tile_has_band(const Dims &d, int x0, int z0) {
  const int e = d.pml + d.nop;
  return x0 - 8 < e || x0 + TX + 8 > d.nxp - e || z0 - 8 < e || z0 + kTileZ + 8 > d.nzp - e;
}

template <class C>
constexpr size_t bwd_tile_smem() { return C::smem(4, 6); }

template <int kCls, class C>
__device__ __forceinline__ void bwd_tile(const BwdFusedArgs &a, int s, float *sm) {
  constexpr bool kPML = kCls == kTilePml, kIn = kCls == kTileInner;
  constexpr int TX = C::TX, R1 = C::R1, R2 = C::R2, P0 = C::P0, N0 = C::N0, N1 = C::N1;
  float *const i_bx = sm, *const i_bz = sm + N0, *const i_ax = sm + 2 * N0, *const i_az = sm + 3 * N0;
  float *const m0 = sm + 4 * N0;  // btxx, btzz, btxz, PL, M, PzLx of the tile plus 4 cells
  const int tid = threadIdx.x;
  const ShotDev sh = a.shots[s];
  const Dims d = slot_dims(a.d, sh);
  const int x0 = tile_x0<TX>(), z0 = tile_z0();
  if (x0 >= d.nxp - d.nop) return;
  const int base = (int)(d.slot * s), ld = d.ld, pml = d.pml;
  const float dtdx = d.dt / d.dx, dtdz = d.dt / d.dz;
  const float rdx = 1.0f / d.dx, rdz = 1.0f / d.dz;
  const bool tp = kPML && tile_has_pml<TX>(d, x0, z0, 4);
  const bool strips = kPML && a.strips_on, band = strips && tile_has_band<TX>(d, x0, z0);
  const int g1 = tid / kTileC1, c1 = tid - g1 * kTileC1, z1 = z0 - 4 + c1, xs1 = x0 - 4 + g1 * R1;
  const int g2 = tid >> 5, c2 = tid & 31, z2 = z0 + c2, xs2 = x0 + g2 * R2;
  const bool zin1 = z1 >= 0 && z1 < d.nzp, zin2 = tid < 32 * C::G2 && (kIn || z2 < d.nzp);
  const bool zi1 = kIn || (z1 >= pml && z1 < d.nzp - pml), zi2 = kIn || (z2 >= pml && z2 < d.nzp - pml);
  const bool zu1 = kIn || (z1 >= d.nop && z1 < d.nzp - d.nop), zu2 = kIn || (z2 >= d.nop && z2 < d.nzp - d.nop);
  const int k1 = base + xs1 * ld + z1, k2 = base + xs2 * ld + z2;
  auto in1 = [&](int r) { return kIn || (zin1 && xs1 + r >= 0 && xs1 + r < d.nxp); };
  auto in2 = [&](int r) { return zin2 && (kIn || xs2 + r < d.nxp); };
  auto xi = [&](int x) { return kIn || (x >= pml && x < d.nxp - pml); };
  auto xu = [&](int x) { return kIn || (x >= d.nop && x < d.nxp - d.nop); };
  auto pm1 = [&](int r) { return tp && pml_cell(d, xs1 + r, z1); };
  auto pm2 = [&](int r) { return tp && pml_cell(d, xs2 + r, z2); };
  auto own1 = [&](int r) {
    const int x = xs1 + r;
    return x >= x0 && x < x0 + TX && c1 >= 4 && c1 < 4 + kTileZ;
  };
  const int img_row = s * d.wnx_max;
  float *const img_pp = a.img, *const img_ps = a.img + a.img_plane, *const img_il = a.img + 2 * a.img_plane;
  // constants of the run, and the step's residuals
  float lam_[R1], mu_[R1], kp_[R1], ks_[R1], q1x[R1], q1z[R1], b_[R2], q2x[R2], q2z[R2];
#pragma unroll
  for (int r = 0; r < R1; r++) {
    const int k = k1 + r * ld;
    lam_[r] = in1(r) ? __ldg(a.p.lam + k) : 0.f;
    mu_[r] = in1(r) ? __ldg(a.p.mu + k) : 0.f;
    const bool im = own1(r) && zi1 && xi(xs1 + r);
    kp_[r] = im ? __ldg(a.p.kpp + k) : 0.f;
    ks_[r] = im ? __ldg(a.p.kps + k) : 0.f;
    q1x[r] = q1z[r] = 0.f;
    if (kPML && in1(r) && pm1(r)) {
      q1x[r] = __ldg(a.p.dampx + k);
      q1z[r] = __ldg(a.p.dampz + k);
    }
  }
#pragma unroll
  for (int r = 0; r < R2; r++) {
    const int k = k2 + r * ld;
    b_[r] = in2(r) ? __ldg(a.p.b + k) : 0.f;
    q2x[r] = q2z[r] = 0.f;
    if (kPML && in2(r) && pm2(r)) {
      q2x[r] = __ldg(a.p.dampx + k);
      q2z[r] = __ldg(a.p.dampz + k);
    }
  }
  const int rc = sh.igz - (z0 - 8);  // the receiver row's input column
  const bool has_rec = rc >= 0 && rc < kTileC0;
  float rz = 0.f, rx = 0.f;
  if (has_rec && tid < TX + 16) {
    const int x = x0 - 8 + tid;
    const int tr = x >= 0 && x < d.nxp ? __ldg(a.rmap + (long long)s * d.nxp_max + x) : -1;
    if (tr >= 0) {
      const long long q = ((long long)s * d.max_ntr + tr) * d.nt + a.it;
      rz = __ldg(a.res_vz + q);
      rx = __ldg(a.res_vx + q);
    }
  }
  pdl_wait();
  // ---- state -------------------------------------------------------------------------------------
  tile_load<C, kIn>(i_ax, a.aa.vx, d, base, x0, z0);
  tile_load<C, kIn>(i_az, a.aa.vz, d, base, x0, z0);
  tile_load_strip<C>(i_bx, a.ra.vx, d, base, s, x0, z0, a.st, a.it, 0, band);
  tile_load_strip<C>(i_bz, a.ra.vz, d, base, s, x0, z0, a.st, a.it, 1, band);
  cp_async_commit();
  float s1[R1][9];  // btxx btzz btxz atxx atzz atxz (or its two split parts), images pp, ps
#pragma unroll
  for (int r = 0; r < R1; r++) {
#pragma unroll
    for (int j = 0; j < 9; j++) s1[r][j] = 0.f;
    if (!in1(r)) continue;
    const int k = k1 + r * ld;
    s1[r][0] = a.ra.txx[k]; s1[r][1] = a.ra.tzz[k]; s1[r][2] = a.ra.txz[k];
    s1[r][3] = a.aa.txx[k]; s1[r][4] = a.aa.tzz[k];
    if (kPML && pm1(r)) {
      s1[r][5] = a.aa.txz_x[k];
      s1[r][6] = a.aa.txz_z[k];
    } else {
      s1[r][5] = a.aa.txz[k];
    }
    if (own1(r) && zi1 && xi(xs1 + r)) {
      const int o = (img_row + xs1 + r - pml) * d.ild + z1;
      s1[r][7] = img_pp[o];
      s1[r][8] = img_ps[o];
    }
  }
  float s2[R2][7];  // adjoint split parts, or own avx, avz at the receivers; own bvx, bvz; image
#pragma unroll
  for (int r = 0; r < R2; r++) {
#pragma unroll
    for (int j = 0; j < 7; j++) s2[r][j] = 0.f;
    if (!in2(r)) continue;
    const int k = k2 + r * ld, x = xs2 + r;
    if (kPML && pm2(r)) {
      s2[r][0] = a.aa.vx_x[k]; s2[r][1] = a.aa.vx_z[k]; s2[r][2] = a.aa.vz_x[k]; s2[r][3] = a.aa.vz_z[k];
    } else if (z2 == sh.igz) {
      s2[r][0] = a.aa.vx[k]; s2[r][1] = a.aa.vz[k];
    }
    if (zi2 && xi(x)) {
      if (band) {
        s2[r][4] = a.ra.vx[k];
        s2[r][5] = a.ra.vz[k];
      }
      s2[r][6] = img_il[(img_row + x - pml) * d.ild + z2];
    }
  }
  pdl_launch();
  cp_async_wait<0>();
  __syncthreads();
  if (has_rec) {  // receiver-side injection (transient)
    if (tid < TX + 16) {
      i_az[tid * P0 + rc] += rz;
      i_ax[tid * P0 + rc] += rx;
    }
    __syncthreads();
  }
  // ---- stage 1: stresses of the tile plus 4 cells, images ------------------------------------------
  {
    const int o = (g1 * R1 + 4) * P0 + c1 + 4;
    float bsa[R1], bsf[R1], asa[R1], asf[R1];
    tile_dx<R1, false>(i_bx + o, P0, bsa);
    tile_dx<R1, true>(i_bz + o, P0, bsf);
    tile_dx<R1, false>(i_ax + o, P0, asa);
    tile_dx<R1, true>(i_az + o, P0, asf);
#pragma unroll
    for (int r = 0; r < R1; r++) {
      float btxx = s1[r][0], btzz = s1[r][1], btxz = s1[r][2], PL = 0.f, M = 0.f, PzLx = 0.f;
      if (in1(r)) {
        const int k = k1 + r * ld, x = xs1 + r;
        const bool own = own1(r), inter = zi1 && xi(x);
        const float lam = lam_[r], mu = mu_[r], l2m = lam + 2.0f * mu;
        float gx_vx = 0.f, gz_vz = 0.f, gz_vx = 0.f, gx_vz = 0.f;
        if (inter) {
          const float sa = bsa[r], sf = bsf[r];
          const float sb = tile_dzm(i_bz + o + r * P0);
          const float se = tile_dzp(i_bx + o + r * P0);
          const float dir = -1.0f;
          btxx = btxx + (dir * l2m * dtdx * sa + dir * lam * dtdz * sb);
          btzz = btzz + (dir * lam * dtdx * sa + dir * l2m * dtdz * sb);
          btxz = btxz + (dir * mu * dtdx * sf + dir * mu * dtdz * se);
          gx_vx = sa * rdx;
          gz_vz = sb * rdz;
          gz_vx = se * rdz;
          gx_vz = sf * rdx;
          if (own) {
            a.rb.txx[k] = btxx;
            a.rb.tzz[k] = btzz;
            a.rb.txz[k] = btxz;
          }
        }
        float atxx = 0.f, atzz = 0.f, atxz = 0.f;
        if (zu1 && xu(x)) {
          const float sa = asa[r], sf = asf[r];
          const float sb = tile_dzm(i_az + o + r * P0);
          const float se = tile_dzp(i_ax + o + r * P0);
          const float xx = -dtdx * sa, zz = -dtdz * sb, xz_x = -dtdx * sf, xz_z = -dtdz * se;
          const float oxx = s1[r][3], ozz = s1[r][4];
          if (kPML && pm1(r)) {
            const TileDamp q = tile_damp(q1x[r], q1z[r], d.dt);
            atxx = fmaf(q.d1, oxx, xx) * q.i2;
            atzz = fmaf(q.d3, ozz, zz) * q.i4;
            const float e1 = fmaf(q.d1, s1[r][5], xz_x) * q.i2;
            const float e2 = fmaf(q.d3, s1[r][6], xz_z) * q.i4;
            if (own) {
              a.ab.txz_x[k] = e1;
              a.ab.txz_z[k] = e2;
            }
            atxz = e1 + e2;
          } else {
            atxx = oxx + xx;
            atzz = ozz + zz;
            atxz = s1[r][5] + (xz_x + xz_z);
          }
          if (own) {
            a.ab.txx[k] = atxx;
            a.ab.tzz[k] = atzz;
            a.ab.txz[k] = atxz;
          }
        }
        PL = l2m * atxx + lam * atzz;
        M = mu * atxz;
        PzLx = l2m * atzz + lam * atxx;
        if (own && inter) {
          const int oi = (img_row + x - pml) * d.ild + z1;
          const float lamda_grad = (gx_vx + gz_vz) * (atxx + atzz);
          const float miu_grad = -2.0f * (gx_vx * atzz + gz_vz * atxx) + (gz_vx + gx_vz) * atxz;
          img_pp[oi] = s1[r][7] + kp_[r] * lamda_grad;
          img_ps[oi] = s1[r][8] + ks_[r] * miu_grad;
        }
      }
      const int q = (g1 * R1 + r) * kTileC1 + c1;
      m0[q] = btxx;
      m0[N1 + q] = btzz;
      m0[2 * N1 + q] = btxz;
      m0[3 * N1 + q] = PL;
      m0[4 * N1 + q] = M;
      m0[5 * N1 + q] = PzLx;
    }
  }
  __syncthreads();
  // ---- stage 2: velocities of the tile ------------------------------------------------------------
  if (zin2) {
    const int o = (g2 * R2 + 4) * kTileC1 + c2 + 4, oi = (g2 * R2 + 8) * P0 + c2 + 8;
    float ax[R2], fx[R2], tx[R2], sx[R2];
    tile_dx<R2, true>(m0 + o, kTileC1, ax);
    tile_dx<R2, false>(m0 + 2 * N1 + o, kTileC1, fx);
    tile_dx<R2, true>(m0 + 3 * N1 + o, kTileC1, tx);
    tile_dx<R2, false>(m0 + 4 * N1 + o, kTileC1, sx);
#pragma unroll
    for (int r = 0; r < R2; r++) {
      if (!in2(r)) continue;
      const int k = k2 + r * ld, x = xs2 + r;
      const float cbx = b_[r] * dtdx, cbz = b_[r] * dtdz;
      if (zi2 && xi(x)) {
        const float bz = tile_dzm(m0 + 2 * N1 + o + r * kTileC1);
        const float ez = tile_dzp(m0 + N1 + o + r * kTileC1);
        float ovx = i_bx[oi + r * P0], ovz = i_bz[oi + r * P0];
        if (band) {  // own state, not the strip
          ovx = s2[r][4];
          ovz = s2[r][5];
        }
        const float vx = ovx + (-cbx * ax[r] + -cbz * bz);
        const float vz = ovz + (-cbx * fx[r] + -cbz * ez);
        a.rb.vx[k] = vx;
        a.rb.vz[k] = vz;
        img_il[(img_row + x - pml) * d.ild + z2] = s2[r][6] + (vx * vx + vz * vz);
      }
      if (zu2 && xu(x)) {
        const float t_xz = tile_dzm(m0 + 4 * N1 + o + r * kTileC1);
        const float s_z = tile_dzp(m0 + 5 * N1 + o + r * kTileC1);
        const float ux_x = -cbx * tx[r], ux_z = -cbz * t_xz;
        const float uz_x = -cbx * sx[r], uz_z = -cbz * s_z;
        float vx, vz;
        if (kPML && pm2(r)) {
          const TileDamp q = tile_damp(q2x[r], q2z[r], d.dt);
          const float vxx = fmaf(q.d1, s2[r][0], ux_x) * q.i2;
          const float vxz = fmaf(q.d3, s2[r][1], ux_z) * q.i4;
          const float vzx = fmaf(q.d1, s2[r][2], uz_x) * q.i2;
          const float vzz = fmaf(q.d3, s2[r][3], uz_z) * q.i4;
          a.ab.vx_x[k] = vxx; a.ab.vx_z[k] = vxz; a.ab.vz_x[k] = vzx; a.ab.vz_z[k] = vzz;
          vx = vxx + vxz;
          vz = vzx + vzz;
        } else {
          float ovx = i_ax[oi + r * P0], ovz = i_az[oi + r * P0];
          if (z2 == sh.igz) {  // receiver row: the state without the residual
            ovx = s2[r][0];
            ovz = s2[r][1];
          }
          vx = ovx + (ux_x + ux_z);
          vz = ovz + (uz_x + uz_z);
        }
        a.ab.vx[k] = vx;
        a.ab.vz[k] = vz;
      }
    }
  }
}

// ---- reverse step of the first-order scattered set (arithmetic of k_bwd_scat_ring and k_born) -----
// The Born source of the background's reconstructed velocities is formed here from those
// velocities instead of being written and read back.
template <class C>
constexpr size_t scat_tile_smem() { return C::smem(4, 3); }

template <int kCls, class C>
__device__ __forceinline__ void scat_tile(const BwdScatArgs &a, const float *fvx, const float *fvz,
                                          int s, float *sm) {
  constexpr bool kPML = kCls == kTilePml, kIn = kCls == kTileInner;
  constexpr int TX = C::TX, R1 = C::R1, R2 = C::R2, P0 = C::P0, N0 = C::N0, N1 = C::N1;
  float *const i_bx = sm, *const i_bz = sm + N0, *const i_fx = sm + 2 * N0, *const i_fz = sm + 3 * N0;
  float *const m0 = sm + 4 * N0;  // btxx, btzz, btxz plus the Born source
  const int tid = threadIdx.x;
  const Dims d = slot_dims(a.d, a.shots[s]);
  const int x0 = tile_x0<TX>(), z0 = tile_z0();
  if (x0 >= d.nxp - d.nop) return;
  const int base = (int)(d.slot * s), ld = d.ld, pml = d.pml;
  const float dtdx = d.dt / d.dx, dtdz = d.dt / d.dz;
  const float rdx = 1.0f / d.dx, rdz = 1.0f / d.dz;
  const bool band = kPML && a.strips_on && tile_has_band<TX>(d, x0, z0);
  const int g1 = tid / kTileC1, c1 = tid - g1 * kTileC1, z1 = z0 - 4 + c1, xs1 = x0 - 4 + g1 * R1;
  const int g2 = tid >> 5, c2 = tid & 31, z2 = z0 + c2, xs2 = x0 + g2 * R2;
  const bool zin1 = z1 >= 0 && z1 < d.nzp, zi1 = kIn || (z1 >= pml && z1 < d.nzp - pml);
  const bool zi2 = tid < 32 * C::G2 && (kIn || (z2 >= pml && z2 < d.nzp - pml));
  const int k1 = base + xs1 * ld + z1, k2 = base + xs2 * ld + z2;
  auto in1 = [&](int r) { return kIn || (zin1 && xs1 + r >= 0 && xs1 + r < d.nxp); };
  auto xi = [&](int x) { return kIn || (x >= pml && x < d.nxp - pml); };
  auto own1 = [&](int r) {
    const int x = xs1 + r;
    return x >= x0 && x < x0 + TX && c1 >= 4 && c1 < 4 + kTileZ;
  };
  const int img_row = s * d.wnx_max;
  float *const img_b = a.img + 3 * a.img_plane, *const img_bs = a.img + 4 * a.img_plane;
  float lam_[R1], mu_[R1], mp_[R1], ms_[R1], kp_[R1], ks_[R1], b_[R2];
#pragma unroll
  for (int r = 0; r < R1; r++) {
    const int k = k1 + r * ld;
    const bool in = zi1 && xi(xs1 + r), im = in && own1(r);
    lam_[r] = in ? __ldg(a.p.lam + k) : 0.f;
    mu_[r] = in ? __ldg(a.p.mu + k) : 0.f;
    mp_[r] = in ? __ldg(a.p.dmp + k) : 0.f;
    ms_[r] = in ? __ldg(a.p.dms + k) : 0.f;
    kp_[r] = im ? __ldg(a.p.kpp + k) : 0.f;
    ks_[r] = im ? __ldg(a.p.kps + k) : 0.f;
  }
#pragma unroll
  for (int r = 0; r < R2; r++) b_[r] = zi2 && xi(xs2 + r) ? __ldg(a.p.b + k2 + r * ld) : 0.f;
  pdl_wait();
  tile_load<C, kIn>(i_fx, fvx, d, base, x0, z0);
  tile_load<C, kIn>(i_fz, fvz, d, base, x0, z0);
  tile_load_strip<C>(i_bx, a.ra.vx, d, base, s, x0, z0, a.st, a.it, 0, band);
  tile_load_strip<C>(i_bz, a.ra.vz, d, base, s, x0, z0, a.st, a.it, 1, band);
  cp_async_commit();
  float s1[R1][8];  // btxx btzz btxz | atxx atzz atxz, images of own interior cells
#pragma unroll
  for (int r = 0; r < R1; r++) {
#pragma unroll
    for (int j = 0; j < 8; j++) s1[r][j] = 0.f;
    if (!in1(r)) continue;
    const int k = k1 + r * ld;
    s1[r][0] = a.ra.txx[k]; s1[r][1] = a.ra.tzz[k]; s1[r][2] = a.ra.txz[k];
    if (own1(r) && zi1 && xi(xs1 + r)) {
      s1[r][3] = a.atxx[k]; s1[r][4] = a.atzz[k]; s1[r][5] = a.atxz[k];
      const int o = (img_row + xs1 + r - pml) * d.ild + z1;
      s1[r][6] = img_b[o];
      s1[r][7] = img_bs[o];
    }
  }
  float s2[R2][2];
#pragma unroll
  for (int r = 0; r < R2; r++) {
    s2[r][0] = s2[r][1] = 0.f;
    if (band && zi2 && xi(xs2 + r)) {
      s2[r][0] = a.ra.vx[k2 + r * ld];
      s2[r][1] = a.ra.vz[k2 + r * ld];
    }
  }
  pdl_launch();
  cp_async_wait<0>();
  __syncthreads();
  {
    const int o = (g1 * R1 + 4) * P0 + c1 + 4;
    float bsa[R1], bsf[R1], fsa[R1], fsf[R1];
    tile_dx<R1, false>(i_bx + o, P0, bsa);
    tile_dx<R1, true>(i_bz + o, P0, bsf);
    tile_dx<R1, false>(i_fx + o, P0, fsa);
    tile_dx<R1, true>(i_fz + o, P0, fsf);
#pragma unroll
    for (int r = 0; r < R1; r++) {
      float pxx = s1[r][0], pzz = s1[r][1], pxz = s1[r][2];
      const int k = k1 + r * ld, x = xs1 + r;
      if (zi1 && xi(x)) {
        const float sa = bsa[r], sf = bsf[r];
        const float sb = tile_dzm(i_bz + o + r * P0);
        const float se = tile_dzp(i_bx + o + r * P0);
        const float lam = lam_[r], mu = mu_[r];
        const float l2m = lam + 2.0f * mu;
        const float dir = -1.0f;
        const float btxx = pxx + (dir * l2m * dtdx * sa + dir * lam * dtdz * sb);
        const float btzz = pzz + (dir * lam * dtdx * sa + dir * l2m * dtdz * sb);
        const float btxz = pxz + (dir * mu * dtdx * sf + dir * mu * dtdz * se);
        if (own1(r)) {
          a.rb.txx[k] = btxx;
          a.rb.tzz[k] = btzz;
          a.rb.txz[k] = btxz;
          const float gx_vx = sa * rdx, gz_vz = sb * rdz, gz_vx = se * rdz, gx_vz = sf * rdx;
          const float atxx = s1[r][3], atzz = s1[r][4], atxz = s1[r][5];
          const float lamda_grad = (gx_vx + gz_vz) * (atxx + atzz);
          const float miu_grad = -2.0f * (gx_vx * atzz + gz_vz * atxx) + (gz_vx + gx_vz) * atxz;
          const int oi = (img_row + x - pml) * d.ild + z1;
          img_b[oi] = s1[r][6] + kp_[r] * lamda_grad;
          img_bs[oi] = s1[r][7] + ks_[r] * miu_grad;
        }
        // Born source of the background's velocities; rounded adds, as when it goes through memory
        const BornSrc e = born_source(lam, mu, mp_[r], ms_[r], fsa[r], tile_dzm(i_fz + o + r * P0),
                                      tile_dzp(i_fx + o + r * P0), fsf[r], rdx, rdz);
        pxx = __fadd_rn(btxx, e.xx);
        pzz = __fadd_rn(btzz, e.zz);
        pxz = __fadd_rn(btxz, e.xz);
      }
      const int q = (g1 * R1 + r) * kTileC1 + c1;
      m0[q] = pxx;
      m0[N1 + q] = pzz;
      m0[2 * N1 + q] = pxz;
    }
  }
  __syncthreads();
  if (zi2) {
    const int o = (g2 * R2 + 4) * kTileC1 + c2 + 4, oi = (g2 * R2 + 8) * P0 + c2 + 8;
    float ax[R2], fx[R2];
    tile_dx<R2, true>(m0 + o, kTileC1, ax);
    tile_dx<R2, false>(m0 + 2 * N1 + o, kTileC1, fx);
#pragma unroll
    for (int r = 0; r < R2; r++) {
      const int k = k2 + r * ld;
      if (!xi(xs2 + r)) continue;
      const float cbx = b_[r] * dtdx, cbz = b_[r] * dtdz;
      const float bz = tile_dzm(m0 + 2 * N1 + o + r * kTileC1);
      const float ez = tile_dzp(m0 + N1 + o + r * kTileC1);
      float ovx = i_bx[oi + r * P0], ovz = i_bz[oi + r * P0];
      if (band) {  // own state, not the strip
        ovx = s2[r][0];
        ovz = s2[r][1];
      }
      a.rb.vx[k] = ovx + (-cbx * ax[r] + -cbz * bz);
      a.rb.vz[k] = ovz + (-cbx * fx[r] + -cbz * ez);
    }
  }
}

// One launch of a backward pass: the backward step of every shot (b.it >= 0) and, in a second grid
// slice, the scattered set's reverse step of the step before (sc.it >= 0), whose background
// velocities and adjoint stresses are this launch's inputs.
struct BwdTileArgs {
  BwdFusedArgs b;
  BwdScatArgs sc;
  const float *fvx, *fvz;
  int n;
};
// Register budget: 64 (3 CTAs an SM of 8 rows, 2 of 16) except for the PML step alone at 8 rows: the
// occupancy gains more than a few spilled values cost.
template <bool kPML, class C, bool kScat>
__global__ void __launch_bounds__(C::T, C::TX == 8 ? (!kPML || kScat ? 3 : 2) : C::TX == 16 ? 2 : 1) k_bwd_tile(const __grid_constant__ BwdTileArgs a) {
  extern __shared__ __align__(16) float tsm[];
  const int m = blockIdx.z / a.n, s = blockIdx.z - m * a.n;
  constexpr int kRest = kPML ? kTilePml : kTileEdge;
  if (m == 0) {
    if (a.b.it < 0) return;
    if (tile_inner<C::TX>(a.b.d, a.b.shots[s])) bwd_tile<kTileInner, C>(a.b, s, tsm);
    else bwd_tile<kRest, C>(a.b, s, tsm);
  } else if (kScat && a.sc.it >= 0) {
    if (tile_inner<C::TX>(a.sc.d, a.sc.shots[s])) scat_tile<kTileInner, C>(a.sc, a.fvx, a.fvz, s, tsm);
    else scat_tile<kRest, C>(a.sc, a.fvx, a.fvz, s, tsm);
  }
}

// ---- acoustic Born pair -------------------------------------------------------------------------
// The arithmetic of the half-step kernels (k_ac_vel, k_ac_str, k_ac_born, k_ac_adj_v, k_ac_adj_s),
// random band and PML, forward and reverse, on the same tiles.

// a dx + b dz with the fused multiply-add written out, in the order that the kernel the same step
// otherwise runs on rounds by (k_ac_pair / k_ac_rev_pair without a PML, the half steps with one), so
// a batch gives the same bits on either and 16-bit strips quantise the same values.
template <bool kPML>
__device__ __forceinline__ float ac_sum(float a, float dx, float b, float dz) {
  return kPML ? __fmaf_rn(a, dx, __fmul_rn(b, dz)) : __fmaf_rn(b, dz, __fmul_rn(a, dx));
}

struct AcTileArgs {
  Dims d;
  const ShotDev *shots;
  const float *vx, *vz, *s, *sx, *sz;  // state at t-1 (sx, sz: split stress of the PML cells)
  float *vx_n, *vz_n, *s_n, *sx_n, *sz_n;
  const float *b, *lam, *m, *dampx, *dampz;
  const float *e_in;   // scattered set: Born source of the same step (overlay on s)
  float *e_out;        // background: Born source of its new velocities, or null
  const float *wavelet;
  int it;              // < 0: nothing to do
  const int *rmap;
  float *rec_vz, *rec_vx;  // scattered set: records
};
template <class C>
constexpr size_t ac_tile_smem() { return C::smem(1, 2); }

template <int kCls, class C, bool kScat, bool kCtxPml>
__device__ __forceinline__ void ac_tile(const AcTileArgs &a, int s, float *sm) {
  constexpr bool kPML = kCls == kTilePml, kIn = kCls == kTileInner;
  constexpr int TX = C::TX, R1 = C::R1, R2 = C::R2, P0 = C::P0, N0 = C::N0;
  constexpr int kLd = C::kLd;
  float *const i_s = sm, *const v_x = sm + N0, *const v_z = v_x + C::N1;
  const int tid = threadIdx.x;
  const ShotDev sh = a.shots[s];
  const Dims d = slot_dims(a.d, sh);
  const int x0 = tile_x0<TX>(), z0 = tile_z0();
  if (x0 >= d.nxp - d.nop) return;
  const int base = (int)(d.slot * s), ld = d.ld;
  const float cx = d.dt / d.dx, cz = d.dt / d.dz;
  const bool tp = kPML && tile_has_pml<TX>(d, x0, z0, 4);
  const int g1 = tid / kTileC1, c1 = tid - g1 * kTileC1, z1 = z0 - 4 + c1, xs1 = x0 - 4 + g1 * R1;
  const int g2 = tid >> 5, c2 = tid & 31, z2 = z0 + c2, xs2 = x0 + g2 * R2;
  const bool zu1 = z1 >= d.nop && z1 < d.nzp - d.nop;
  const bool zu2 = tid < 32 * C::G2 && (kIn || (z2 >= d.nop && z2 < d.nzp - d.nop));
  const bool zi2 = kIn || (z2 >= d.pml && z2 < d.nzp - d.pml);
  const int k1 = base + xs1 * ld + z1, k2 = base + xs2 * ld + z2;
  auto up1 = [&](int r) { return kIn || (zu1 && xs1 + r >= d.nop && xs1 + r < d.nxp - d.nop); };
  auto up2 = [&](int r) { return zu2 && (kIn || (xs2 + r >= d.nop && xs2 + r < d.nxp - d.nop)); };
  auto pm1 = [&](int r) { return tp && pml_cell(d, xs1 + r, z1); };
  auto pm2 = [&](int r) { return tp && pml_cell(d, xs2 + r, z2); };
  auto own1 = [&](int r) {
    const int x = xs1 + r;
    return x >= x0 && x < x0 + TX && c1 >= 4 && c1 < 4 + kTileZ;
  };
  float b_[R1], q1x[R1], q1z[R1], lam_[R2], q2x[R2], q2z[R2], m_[R2];
  int tr[R1];
#pragma unroll
  for (int r = 0; r < R1; r++) {
    b_[r] = up1(r) ? __ldg(a.b + k1 + r * ld) : 0.f;
    q1x[r] = q1z[r] = 0.f;
    if (kPML && up1(r) && pm1(r)) {
      q1x[r] = __ldg(a.dampx + k1 + r * ld);
      q1z[r] = __ldg(a.dampz + k1 + r * ld);
    }
    tr[r] = -1;
    if (kScat && z1 == sh.igz && up1(r) && own1(r))
      tr[r] = __ldg(a.rmap + (long long)s * d.nxp_max + xs1 + r);
  }
#pragma unroll
  for (int r = 0; r < R2; r++) {
    lam_[r] = up2(r) ? __ldg(a.lam + k2 + r * ld) : 0.f;
    q2x[r] = q2z[r] = 0.f;
    if (kPML && up2(r) && pm2(r)) {
      q2x[r] = __ldg(a.dampx + k2 + r * ld);
      q2z[r] = __ldg(a.dampz + k2 + r * ld);
    }
    m_[r] = 0.f;
    if (!kScat && a.e_out && up2(r) && zi2 && (kIn || (xs2 + r >= d.pml && xs2 + r < d.nxp - d.pml)))
      m_[r] = __ldg(a.m + k2 + r * ld);
  }
  const float sval = kScat ? 0.f : __ldg(a.wavelet + a.it);
  pdl_wait();
  tile_load<C, kIn>(i_s, a.s, d, base, x0, z0);
  cp_async_commit();
  float4 ov[kScat ? kLd : 1];
  if (kScat) {
#pragma unroll
    for (int j = 0; j < kLd; j++) {
      const int i = tid + j * C::T, r = i / (kTileC0 / 4), c = (i - r * (kTileC0 / 4)) * 4;
      const int x = x0 - 8 + r, z = z0 - 8 + c;
      const bool in = r < TX + 16 && (kIn || (x >= 0 && x < d.nxp && z >= 0 && z < ld));
      ov[j] = in ? *reinterpret_cast<const float4 *>(a.e_in + base + x * ld + z)
                 : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  float s1[R1][2], s2[R2][2];
#pragma unroll
  for (int r = 0; r < R1; r++) {
    s1[r][0] = up1(r) ? a.vx[k1 + r * ld] : 0.f;
    s1[r][1] = up1(r) ? a.vz[k1 + r * ld] : 0.f;
  }
#pragma unroll
  for (int r = 0; r < R2; r++) {
    s2[r][0] = s2[r][1] = 0.f;
    if (!up2(r)) continue;
    if (kPML && pm2(r)) {
      s2[r][0] = a.sx[k2 + r * ld];
      s2[r][1] = a.sz[k2 + r * ld];
    } else {
      s2[r][0] = a.s[k2 + r * ld];
    }
  }
  pdl_launch();
  cp_async_wait<0>();
  if (kScat) {
#pragma unroll
    for (int j = 0; j < kLd; j++) {
      const int i = tid + j * C::T, r = i / (kTileC0 / 4), c = (i - r * (kTileC0 / 4)) * 4;
      if (r >= TX + 16) continue;
      float4 *p = reinterpret_cast<float4 *>(i_s + r * P0 + c);
      float4 v = *p;
      v.x += ov[j].x; v.y += ov[j].y; v.z += ov[j].z; v.w += ov[j].w;
      *p = v;
    }
  } else {
    const int r = sh.isx - (x0 - 8), c = sh.isz - (z0 - 8);
    if (r >= 0 && r < TX + 16 && c >= 0 && c < kTileC0 &&
        tid == (r * (kTileC0 / 4) + c / 4) % C::T)
      i_s[r * P0 + c] += sval;
  }
  __syncthreads();
  {
    const int o = (g1 * R1 + 4) * P0 + c1 + 4;
    float ax[R1];
    tile_dx<R1, true>(i_s + o, P0, ax);
#pragma unroll
    for (int r = 0; r < R1; r++) {
      float vx = 0.f, vz = 0.f;
      if (up1(r)) {
        const float az = tile_dzp(i_s + o + r * P0), bb = b_[r];
        if (kPML && pm1(r)) {
          const TileDamp q = tile_damp(q1x[r], q1z[r], d.dt);
          vx = fmaf(q.d1, s1[r][0], bb * cx * ax[r]) * q.i2;
          vz = fmaf(q.d3, s1[r][1], bb * cz * az) * q.i4;
        } else {
          vx = s1[r][0] + (bb * cx) * ax[r];
          vz = s1[r][1] + (bb * cz) * az;
        }
        if (own1(r)) {
          a.vx_n[k1 + r * ld] = vx;
          a.vz_n[k1 + r * ld] = vz;
          if (tr[r] >= 0) {
            const long long q = ((long long)s * d.max_ntr + tr[r]) * d.nt + a.it;
            a.rec_vz[q] = vz;
            a.rec_vx[q] = vx;
          }
        }
      }
      v_x[(g1 * R1 + r) * kTileC1 + c1] = vx;
      v_z[(g1 * R1 + r) * kTileC1 + c1] = vz;
    }
  }
  __syncthreads();
  if (zu2) {
    const int o = (g2 * R2 + 4) * kTileC1 + c2 + 4;
    float dx[R2];
    tile_dx<R2, false>(v_x + o, kTileC1, dx);
#pragma unroll
    for (int r = 0; r < R2; r++) {
      if (!up2(r)) continue;
      const int k = k2 + r * ld;
      const float dz = tile_dzm(v_z + o + r * kTileC1), lam = lam_[r];
      if (kPML && pm2(r)) {
        const TileDamp q = tile_damp(q2x[r], q2z[r], d.dt);
        const float nx = fmaf(q.d1, s2[r][0], lam * cx * dx[r]) * q.i2;
        const float nz = fmaf(q.d3, s2[r][1], lam * cz * dz) * q.i4;
        a.sx_n[k] = nx;
        a.sz_n[k] = nz;
        a.s_n[k] = nx + nz;
      } else {
        a.s_n[k] = fmaf(lam, ac_sum<kCtxPml>(cx, dx[r], cz, dz), s2[r][0]);
      }
      if (!kScat && a.e_out && zi2 && (kIn || (xs2 + r >= d.pml && xs2 + r < d.nxp - d.pml)))
        a.e_out[k] = -2.0f * lam * m_[r] * ac_sum<kCtxPml>(1.0f / d.dx, dx[r], 1.0f / d.dz, dz);
    }
  }
}

// One launch of a forward pass: the background's step, the scattered set's step before it (grid
// slice n .. 2n) and, in the slice behind the sets, the strips of the background state it reads.
struct AcFwdTileArgs {
  AcTileArgs set[2];
  StripSaveArgs st;
  int n, nset;
};
template <bool kPML, class C>
__global__ void __launch_bounds__(C::T, 2) k_ac_tile(const __grid_constant__ AcFwdTileArgs a) {
  extern __shared__ __align__(16) float tsm[];
  const int m = blockIdx.z / a.n, s = blockIdx.z - m * a.n;
  if (m >= a.nset) {
    if (a.st.it >= 0) tile_strips(a.st, s);
  } else if (a.set[m].it >= 0) {
    constexpr int kRest = kPML ? kTilePml : kTileEdge;
    const AcTileArgs &f = a.set[m];
    if (tile_inner<C::TX>(f.d, f.shots[s])) {
      if (m == 0) ac_tile<kTileInner, C, false, kPML>(f, s, tsm);
      else ac_tile<kTileInner, C, true, kPML>(f, s, tsm);
    } else {
      if (m == 0) ac_tile<kRest, C, false, kPML>(f, s, tsm);
      else ac_tile<kRest, C, true, kPML>(f, s, tsm);
    }
  }
}

// Reverse step: the adjoint pair, the gradient with the background's velocities of the step, and the
// background one step back (with a PML: on the interior, its velocities in the strip band taken from
// the strips).
struct AcRevTileArgs {
  Dims d;
  const ShotDev *shots;
  const float *yx, *yz, *ys, *ysx, *ysz;  // adjoint state
  float *yx_n, *yz_n, *ys_n, *ysx_n, *ysz_n;
  const float *vx, *vz, *s;               // background
  float *vx_n, *vz_n, *s_n;
  const float *b, *lam, *dampx, *dampz, *wavelet;
  float *grad;
  int it;
  const int *rmap;
  const float *res_vz, *res_vx;
  Strips st;
};
template <class C>
constexpr size_t ac_rev_tile_smem() { return C::smem(4, 4); }

template <int kCls, class C, bool kCtxPml>
__device__ __forceinline__ void ac_rev_tile(const AcRevTileArgs &a, float *tsm) {
  constexpr bool kPML = kCls == kTilePml, kIn = kCls == kTileInner;
  constexpr int TX = C::TX, R1 = C::R1, R2 = C::R2, P0 = C::P0, N0 = C::N0, N1 = C::N1;
  constexpr int kLd = C::kLd;
  float *const i_vx = tsm, *const i_vz = tsm + N0, *const i_wx = tsm + 2 * N0;
  float *const m0 = tsm + 4 * N0;  // ux, uz, background stress + source, gradient factor
  const int tid = threadIdx.x, s = blockIdx.z;
  const ShotDev sh = a.shots[s];
  const Dims d = slot_dims(a.d, sh);
  const int x0 = tile_x0<TX>(), z0 = tile_z0();
  if (x0 >= d.nxp - d.nop) return;
  const int base = (int)(d.slot * s), ld = d.ld, pml = d.pml;
  const float cx = d.dt / d.dx, cz = d.dt / d.dz;
  const bool tp = kPML && tile_has_pml<TX>(d, x0, z0, 8);  // the adjoint's split stress is read
  const bool band = kPML && tile_has_band<TX>(d, x0, z0);
  float *const i_wz = kPML && tp ? tsm + 3 * N0 : i_wx;  // x and z parts differ in the PML only
  const int g1 = tid / kTileC1, c1 = tid - g1 * kTileC1, z1 = z0 - 4 + c1, xs1 = x0 - 4 + g1 * R1;
  const int g2 = tid >> 5, c2 = tid & 31, z2 = z0 + c2, xs2 = x0 + g2 * R2;
  const bool zu1 = z1 >= d.nop && z1 < d.nzp - d.nop, zi1 = kIn || (z1 >= pml && z1 < d.nzp - pml);
  const bool zu2 = tid < 32 * C::G2 && (kIn || (z2 >= d.nop && z2 < d.nzp - d.nop));
  const bool zi2 = kIn || (z2 >= pml && z2 < d.nzp - pml);
  const int k1 = base + xs1 * ld + z1, k2 = base + xs2 * ld + z2;
  auto xi = [&](int x) { return kIn || (x >= pml && x < d.nxp - pml); };
  auto in1 = [&](int r) { return kIn || (z1 >= 0 && z1 < d.nzp && xs1 + r >= 0 && xs1 + r < d.nxp); };
  auto up1 = [&](int r) { return kIn || (zu1 && xs1 + r >= d.nop && xs1 + r < d.nxp - d.nop); };
  auto up2 = [&](int r) { return zu2 && (kIn || (xs2 + r >= d.nop && xs2 + r < d.nxp - d.nop)); };
  // cells where the background is rebuilt
  auto rb1 = [&](int r) { return kCtxPml ? zi1 && xi(xs1 + r) : up1(r); };
  auto rb2 = [&](int r) { return kCtxPml ? zu2 && zi2 && xi(xs2 + r) : up2(r); };
  auto pm1 = [&](int r) { return tp && pml_cell(d, xs1 + r, z1); };
  auto pm2 = [&](int r) { return tp && pml_cell(d, xs2 + r, z2); };
  auto own1 = [&](int r) {
    const int x = xs1 + r;
    return x >= x0 && x < x0 + TX && c1 >= 4 && c1 < 4 + kTileZ;
  };
  float b1[R1], lam1[R1], q1x[R1], q1z[R1], rz[R1], rx[R1], b2[R2], q2x[R2], q2z[R2];
#pragma unroll
  for (int r = 0; r < R1; r++) {
    const int k = k1 + r * ld;
    b1[r] = up1(r) ? __ldg(a.b + k) : 0.f;
    lam1[r] = up1(r) ? __ldg(a.lam + k) : 0.f;
    q1x[r] = q1z[r] = rz[r] = rx[r] = 0.f;
    if (kPML && up1(r) && pm1(r)) {
      q1x[r] = __ldg(a.dampx + k);
      q1z[r] = __ldg(a.dampz + k);
    }
    if (z1 == sh.igz && up1(r)) {
      const int tr = __ldg(a.rmap + (long long)s * d.nxp_max + xs1 + r);
      if (tr >= 0) {
        const long long q = ((long long)s * d.max_ntr + tr) * d.nt + a.it;
        rz[r] = __ldg(a.res_vz + q);
        rx[r] = __ldg(a.res_vx + q);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R2; r++) {
    const int k = k2 + r * ld;
    b2[r] = rb2(r) ? __ldg(a.b + k) : 0.f;
    q2x[r] = q2z[r] = 0.f;
    if (kPML && up2(r) && pm2(r)) {
      q2x[r] = __ldg(a.dampx + k);
      q2z[r] = __ldg(a.dampz + k);
    }
  }
  float4 lw[kLd];  // lam on the input chunks (outside the PML)
#pragma unroll
  for (int j = 0; j < kLd; j++) {
    const int i = tid + j * C::T, r = i / (kTileC0 / 4), c = (i - r * (kTileC0 / 4)) * 4;
    const int x = x0 - 8 + r, z = z0 - 8 + c;
    const bool in = r < TX + 16 && (kIn || (x >= 0 && x < d.nxp && z >= 0 && z < ld));
    lw[j] = in ? __ldg(reinterpret_cast<const float4 *>(a.lam + base + x * ld + z))
               : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float sval = __ldg(a.wavelet + a.it);
  pdl_wait();
  tile_load_strip<C, true>(i_vx, a.vx, d, base, s, x0, z0, a.st, a.it, 0, band);
  tile_load_strip<C, true>(i_vz, a.vz, d, base, s, x0, z0, a.st, a.it, 1, band);
  cp_async_commit();
#pragma unroll
  for (int j = 0; j < kLd; j++) {
    const int i = tid + j * C::T, r = i / (kTileC0 / 4), c = (i - r * (kTileC0 / 4)) * 4;
    const int x = x0 - 8 + r, z = z0 - 8 + c;
    if (r >= TX + 16) continue;
    const bool in = kIn || (x >= 0 && x < d.nxp && z >= 0 && z < ld);
    const int k = in ? base + x * ld + z : base;
    const float4 y = in ? *reinterpret_cast<const float4 *>(a.ys + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 wx = make_float4(lw[j].x * y.x, lw[j].y * y.y, lw[j].z * y.z, lw[j].w * y.w), wz = wx;
    if (kPML && tp) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        if (!in || !pml_cell(d, x, z + e)) continue;
        const TileDamp q = tile_damp(__ldg(a.dampx + k + e), __ldg(a.dampz + k + e), d.dt);
        const float lam = (&lw[j].x)[e];
        (&wx.x)[e] = lam * a.ysx[k + e] * q.i2;
        (&wz.x)[e] = lam * a.ysz[k + e] * q.i4;
      }
      *reinterpret_cast<float4 *>(i_wz + r * P0 + c) = wz;
    }
    *reinterpret_cast<float4 *>(i_wx + r * P0 + c) = wx;
  }
  float s1[R1][3], s2[R2][3];
#pragma unroll
  for (int r = 0; r < R1; r++) {
    const int k = k1 + r * ld;
    s1[r][0] = up1(r) ? a.yx[k] : 0.f;
    s1[r][1] = up1(r) ? a.yz[k] : 0.f;
    s1[r][2] = in1(r) ? a.s[k] : 0.f;
  }
#pragma unroll
  for (int r = 0; r < R2; r++) {
    const int k = k2 + r * ld;
    s2[r][0] = s2[r][1] = s2[r][2] = 0.f;
    if (!up2(r)) continue;
    if (kPML && pm2(r)) {
      s2[r][0] = a.ysx[k];
      s2[r][1] = a.ysz[k];
    } else {
      s2[r][0] = a.ys[k];
    }
    if (zi2 && xi(xs2 + r)) s2[r][2] = a.grad[(s * d.wnx_max + xs2 + r - pml) * d.ild + z2];
  }
  pdl_launch();
  cp_async_wait<0>();
  __syncthreads();
  {
    const int o = (g1 * R1 + 4) * P0 + c1 + 4;
    float tx[R1], dx[R1];
    tile_dx<R1, true>(i_wx + o, P0, tx);
    tile_dx<R1, false>(i_vx + o, P0, dx);
#pragma unroll
    for (int r = 0; r < R1; r++) {
      const int k = k1 + r * ld, q = (g1 * R1 + r) * kTileC1 + c1;
      float ux = 0.f, uz = 0.f, sn = s1[r][2], f = 0.f;
      if (up1(r)) {
        const float tz = tile_dzp(i_wz + o + r * P0);
        float yx = s1[r][0], yz = s1[r][1];
        TileDamp p{1.f, 1.f, 1.f, 1.f};
        const bool pc = kPML && pm1(r);
        if (pc) {
          p = tile_damp(q1x[r], q1z[r], d.dt);
          yx *= p.d1 * p.i2;
          yz *= p.d3 * p.i4;
        }
        if (z1 == sh.igz) {  // transpose of the recording
          yz += rz[r];
          yx += rx[r];
        }
        yx = yx - cx * tx[r];
        yz = yz - cz * tz;
        ux = b1[r] * cx * yx;
        uz = b1[r] * cz * yz;
        if (pc) {
          ux *= p.i2;
          uz *= p.i4;
        }
        if (own1(r)) {
          a.yx_n[k] = yx;
          a.yz_n[k] = yz;
        }
      }
      if (rb1(r)) {
        const float dz = tile_dzm(i_vz + o + r * P0);
        sn = fmaf(-lam1[r], ac_sum<kCtxPml>(cx, dx[r], cz, dz), sn);
        f = -2.0f * lam1[r] * ac_sum<kCtxPml>(1.0f / d.dx, dx[r], 1.0f / d.dz, dz);
        if (own1(r)) a.s_n[k] = sn;
      }
      if (z1 == sh.isz && xs1 + r == sh.isx) sn += sval;
      m0[q] = ux;
      m0[N1 + q] = uz;
      m0[2 * N1 + q] = sn;
      m0[3 * N1 + q] = f;
    }
  }
  __syncthreads();
  if (zu2) {
    const int o = (g2 * R2 + 4) * kTileC1 + c2 + 4, oi = (g2 * R2 + 8) * P0 + c2 + 8;
    float gx[R2], ax[R2];
    tile_dx<R2, false>(m0 + o, kTileC1, gx);
    tile_dx<R2, true>(m0 + 2 * N1 + o, kTileC1, ax);
#pragma unroll
    for (int r = 0; r < R2; r++) {
      if (!up2(r)) continue;
      const int k = k2 + r * ld;
      const float gz = tile_dzm(m0 + N1 + o + r * kTileC1);
      const float gs = -gx[r] - gz;
      if (kPML && pm2(r)) {
        const TileDamp p = tile_damp(q2x[r], q2z[r], d.dt);
        a.ysx_n[k] = fmaf(p.d1 * p.i2, s2[r][0], gs);
        a.ysz_n[k] = fmaf(p.d3 * p.i4, s2[r][1], gs);
      } else {
        a.ys_n[k] = s2[r][0] + gs;
      }
      if (zi2 && xi(xs2 + r))
        a.grad[(s * d.wnx_max + xs2 + r - pml) * d.ild + z2] =
            s2[r][2] + m0[3 * N1 + o + r * kTileC1] * gs;
      if (rb2(r)) {
        const float az = tile_dzp(m0 + 2 * N1 + o + r * kTileC1), bb = b2[r];
        a.vx_n[k] = i_vx[oi + r * P0] + -1.0f * (bb * cx) * ax[r];
        a.vz_n[k] = i_vz[oi + r * P0] + -1.0f * (bb * cz) * az;
      }
    }
  }
}

template <bool kPML, class C>
__global__ void __launch_bounds__(C::T, 2) k_ac_rev_tile(const __grid_constant__ AcRevTileArgs a) {
  extern __shared__ __align__(16) float tsm[];
  if (tile_inner<C::TX>(a.d, a.shots[blockIdx.z])) ac_rev_tile<kTileInner, C, kPML>(a, tsm);
  else ac_rev_tile<kPML ? kTilePml : kTileEdge, C, kPML>(a, tsm);
}

}  // namespace ds2d
