// One time step of the background and one of the scattered acoustic field in a single x-march
// (random boundary): the Born modelling L m.
//
// As two launches (k_ac_pair<0>, k_ac_pair<1>) the step moves 84 bytes per cell (b and lam read
// twice) and was bound by its issue slots, not by them (16 shots of 2001x601: 2 x 0.27 ms, 240
// instructions per cell and field, DRAM 40 %).  Here the scattered field runs one time step behind
// the background, so the two are independent within a launch, both at the same row, and take the
// same operators: every window entry, z-tap and stencil holds (background, scattered) in one
// 64-bit register and the packed FP32 instructions do both.  The Born source of the background's
// step goes through memory to the next launch (two buffers, because a CTA reads halo rows that its
// neighbour writes).  64 bytes per cell (68 with a density array).
//
// The march is k_bwd_bulk's: a CTA owns the columns [zs, zs + tz) (8 halo columns at inner edges)
// and xr rows, one bulk copy per field row into a ring of 4 slots, one barrier per row step that
// publishes the z-tap rows of two stages, out of two buffers:
//   V (row r-4)  v += b dt/d D+ S,  S = s + source (background), s + Born source (scattered)
//   S (row r-8)  s += lam (dt/dx D-x vx + dt/dz D-z vz), and the background's Born source
// The source enters S when its row enters the window, so window and z-taps both hold it; the
// stress rows of stage S are read again without it.  Sums are rounded as in k_ac_pair (dt/dx terms
// first, then one FMA), so the records agree bit for bit: scattered fields carry a one-ulp change
// of the background to 1e-4.
#pragma once
#include "ds2d_pair.cuh"

namespace ds2d {

struct AcDuoArgs {
  Dims d;
  const ShotDev *shots;
  const float *s[2], *vx[2], *vz[2];  // [0] background at step it, [1] scattered at step it - 1
  float *s_n[2], *vx_n[2], *vz_n[2];
  const float *b, *lam, *m;
  float bconst;       // Par::bconst
  const float *e_in;  // Born source of step it - 1
  float *e_out;       // Born source of step it
  const float *wavelet;
  int it, tz, xr;
  const int *rmap;
  float *rec_vz, *rec_vx;  // [slot][max_ntr][nt], written at it - 1
  int *err;
};

// s (2), e_in of row r; vx (2), vz (2), b of row r - 4; s (2), lam, m of row r - 8.
constexpr int kAcDuoFields = 12;
constexpr int kAcDuoD = 4;
__host__ __device__ constexpr size_t ac_duo_smem(int kT) {
  return sizeof(float) * (size_t)kAcDuoD * kAcDuoFields * kT + sizeof(pair_t) * 4 * kT +
         8 * kAcDuoD + sizeof(int) * 16;
}

template <int kT, int kMinB>
__global__ void __launch_bounds__(kT, kMinB) k_ac_duo(AcDuoArgs a) {
  constexpr int kD = kAcDuoD, NF = kAcDuoFields;
  extern __shared__ __align__(16) float ring[];  // [kD][NF][kT]
  pair_t *ztap = (pair_t *)(ring + (size_t)kD * NF * kT);  // [2 buffers][S, vz][kT]
  unsigned long long *bars = ztap + 4 * kT;
  int *s_tr = (int *)(bars + kD);  // receiver staging [16]
  const int sl = blockIdx.z, t = threadIdx.x, lane = t & 31;
  const Dims d = slot_dims(a.d, a.shots[sl]);
  const int zs = blockIdx.x * a.tz, ze = min(zs + a.tz, d.nzp);
  const int c0 = zs > 0 ? zs - 8 : 0;
  const int z = c0 + t;
  const int x0 = blockIdx.y * a.xr, x1 = min(x0 + a.xr, d.nxp);
  if (x0 >= d.nxp) return;  // beyond this slot's window (uneven batches), whole CTA
  if (__syncthreads_or(t == 0 && pair_err_raised(a.err))) return;  // whole CTA
  const int ld = d.ld, nop = d.nop, pml = d.pml;
  const long long fbase = d.slot * sl;
  const bool z_upd = z >= nop && z < d.nzp - nop;
  const bool c1 = z_upd && z >= zs - 4 && z < ze + 4;  // columns of stage V, of stage S
  const bool c2 = z_upd && z >= zs && z < ze;
  const bool z_int = z >= pml && z < d.nzp - pml;
  const ShotDev sh = a.shots[sl];
  const bool src_col = z == sh.isz, rec_col = c2 && z == sh.igz;
  const int *rmap = a.rmap + (long long)sl * d.nxp_max;
  const float cx = d.dt / d.dx, cz = d.dt / d.dz;
  const float rdx = 1.0f / d.dx, rdz = 1.0f / d.dz;

  // warp w, lane l owns ring field w + W l (W warps)
  const int my_f = (t >> 5) + (kT / 32) * lane;
  RingField fd{nullptr, 0, 0, d.nxp};
  {
    const float *src[NF] = {a.s[0], a.s[1], a.e_in, a.vx[0], a.vx[1], a.vz[0], a.vz[1],
                            a.bconst != 0.f ? nullptr : a.b, a.s[0], a.s[1], a.lam, a.m};
#pragma unroll
    for (int f = 0; f < NF; f++)
      if (my_f == f && src[f]) {
        fd.src = src[f] + fbase;
        fd.lag = f < 3 ? 0 : f < 8 ? 4 : 8;
      }
  }
  if (t == 0) {
    for (int k = 0; k < kD; k++) mbar_init(&bars[k], kT / 32);  // one arrival per warp
    mbar_fence_init();
  }
  __syncthreads();
  const int rs0 = x0 - 8;
  RowCopies rc;
  rc.init<kT>(fd, ring, my_f, rs0, ld, c0);
  const unsigned bar0 = smem_u32(bars);
  for (int j = 0; j < kD - 1; j++) rc.issue(j * NF * kT * 4, bar0 + 8 * j, ld, lane);

  pair_t w_S[8], w_vx[9], w_vz[5];
#pragma unroll
  for (int i = 0; i < 8; i++) w_S[i] = 0;
#pragma unroll
  for (int i = 0; i < 9; i++) w_vx[i] = 0;
#pragma unroll
  for (int i = 0; i < 5; i++) w_vz[i] = 0;

  RingCursor<kD> cur;
  bool ok = true, aborted = false;
#pragma unroll 2
  for (int r = rs0; r < x1 + 8; r++) {
    ok = mbar_wait(&bars[cur.slot], cur.phase);  // a wait that gives up ends the march below
    const float *S = ring + (size_t)cur.slot * NF * kT + t;
    if (rec_col && r + 4 < d.nxp && r + 4 >= 0)
      cp_async4((float *)&s_tr[(r + 4) & 15], (const float *)(rmap + r + 4));
    if (rec_col) cp_async_commit();
    float s0 = S[0];
    if (src_col && r == sh.isx) s0 += a.wavelet[a.it];  // FD2DGPU.cu:2039-2049
    push(w_S, pk(s0, S[kT] + S[2 * kT]));
    // z-tap rows: S of row r - 4, vz of row r - 8 (before this step's push: index 1)
    pair_t *const zS = ztap + (r & 1) * 2 * kT + t, *const zV = zS + kT;
    zS[0] = w_S[3];
    zV[0] = w_vz[1];
    if (__syncthreads_or(!ok)) {
      aborted = true;
      break;
    }
    {  // every thread is done with the previous slot
      const int ps = cur.slot == 0 ? kD - 1 : cur.slot - 1;
      rc.issue(ps * NF * kT * 4, bar0 + 8 * ps, ld, lane);
    }
    // ---- stage V: velocities of row rv = r - 4 ----------------------------------------------
    const int rv = r - 4;
    pair_t vx = 0, vz = 0;
    if (c1 && r >= x0 && rv >= nop && rv < d.nxp - nop) {
      const pair_t ax = stencil4x2([&](int i) { return sub2(w_S[3 + i], w_S[4 - i]); });
      const pair_t az =
          stencil4x2([&](int i) { return sub2(zS[i], i == 1 ? w_S[3] : zS[1 - i]); });
      const float bb = a.bconst != 0.f ? a.bconst : S[7 * kT];
      const float bx = bb * cx, bz = bb * cz;
      vx = fma2(pk(bx, bx), ax, pk(S[3 * kT], S[4 * kT]));
      vz = fma2(pk(bz, bz), az, pk(S[5 * kT], S[6 * kT]));
      if (c2 && rv >= x0 && rv < x1) {
        const long long k = fbase + (long long)rv * ld + z;
        const float2 ux = upk(vx), uz = upk(vz);
        a.vx_n[0][k] = ux.x;
        a.vx_n[1][k] = ux.y;
        a.vz_n[0][k] = uz.x;
        a.vz_n[1][k] = uz.y;
        if (rec_col) {
          const int tr = s_tr[rv & 15];
          if (tr >= 0) {
            const long long q = ((long long)sl * d.max_ntr + tr) * d.nt + a.it - 1;
            a.rec_vz[q] = uz.y;
            a.rec_vx[q] = ux.y;
          }
        }
      }
    }
    push(w_vx, vx);
    push(w_vz, vz);
    // ---- stage S: stress of row rs = r - 8 --------------------------------------------------
    const int rs = r - 8;
    if (c2 && rs >= x0 && rs < x1 && rs >= nop && rs < d.nxp - nop) {
      const pair_t dx = dxm_mid(w_vx);
      const pair_t dz =
          stencil4x2([&](int i) { return sub2(i == 1 ? w_vz[0] : zV[i - 1], zV[-i]); });
      const float lam = S[10 * kT];
      const float2 ns = upk(fma2(pk(lam, lam), fma2(pk(cz, cz), dz, mul2(pk(cx, cx), dx)),
                                 pk(S[8 * kT], S[9 * kT])));
      const long long k = fbase + (long long)rs * ld + z;
      a.s_n[0][k] = ns.x;
      a.s_n[1][k] = ns.y;
      if (z_int && rs >= pml && rs < d.nxp - pml)  // the band's cells stay zero
        a.e_out[k] =
            -2.0f * lam * S[11 * kT] * fmaf(rdz, upk(dz).x, __fmul_rn(rdx, upk(dx).x));
    }
    if (rec_col) cp_async_wait<7>();
    cur.advance();
  }
  pair_exit<kD>(bars, cur, aborted, ok, a.err);
  cp_async_wait<0>();
}

}  // namespace ds2d
