// sweep_mixed_row.cuh -- the mixed-precision sweep kernel: the rows of
// independent warps of sweep_fp64_row.cuh (same tasks, roles, rings and
// waits), with the two per-cell transforms as split 16-bit tensor-core
// products in FP32 accumulators, the face recurrence in FP32, and each
// octant's contribution to vo in FP32 (summed in FP64 by a second kernel).
//
// Same work as the reference's Sweeper_sweep_block_impl_global and
// Sweeper_sweep_cell (sweeper_kba_c_kernels.h:30-1383) under the host step
// loop of sweeper_kba_c.h:588-845.
//
// Numerics
//   T1  vs[angle]  = sum_m a_from_m[oct][m][angle] * vi[m]      (K = moments)
//   T2  vo[m]     += sum_a m_from_a[oct][a][m] * psi[a]          (K = angles)
//   Each operand is split into two 16-bit halves, x ~ hi + lo with
//   hi = rn16(x * 2^k), lo = rn16(x * 2^k - hi), where 2^k brings the largest
//   entry of the operand's row (or of the octant's matrix) to [2^14, 2^15);
//   the product keeps lo*hi + hi*lo + hi*hi and accumulates in FP32.  With
//   FP16 halves that is a 22-bit significand per operand (errors near FP32
//   rounding); with BF16 halves 16 bits.  vi carries one scale per 8 moments,
//   psi one per 16 angles, each with an accumulator of its own.
//   Quantities_solve (quantities_testing_kernels.h:337-447) runs in FP32 with
//   fused multiply-adds except its last step, psi = sm * cc + vs, which
//   carries the FP64 reciprocal 1 / (1 + octant) as an FP32 pair and the
//   product's and the sum's rounding errors (fma, TwoSum) to one final
//   rounding; faces are stored in FP32.
//
// Two cells of a row are the 16 rows of a warp-level product (8 columns =
// 2 groups x 4 unknowns each): the accumulator of the first product (row =
// column of the state, 8 angles per tile) is the A operand of the second as it
// stands, so psi never leaves registers.  Why warp-level products and not a
// CTA-wide 128-row MMA with accumulators in tensor memory: the sweep gives a
// warp two cells' worth of operands at a time, 36 products a pair, and the
// round trip through shared-memory operands, a commit, an mbarrier and a
// tensor-memory load per step, with all warps in lockstep, was what bounded
// that form (3 % tensor pipe).
//
// What bounds it: instruction issue (55 % of the slots with two warps per
// scheduler): about 430 warp instructions a cell, 190 of them the FP32 solve
// with its error terms, 18 products.  Measured, ms per sweep (conversion and
// partial sum included): 64^3 x 64 groups 63.0 (FP16) / 64.0 (BF16), the
// CTA-wide form 91.6 / 92.8; 64^3 x 16 15.7 / 23.4.  With 12 rows and 128
// registers no faster (16.5 where this one then took 16.6): the third warp
// gains what 32 rows in tiles of 12 lose.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sweep_fp64_row.cuh"

namespace msb {

// One (cell, group pair) of vi in the first transform's operand format: the
// cell's 8 rows (group g, unknown u: row 4 g + u), hi halves then lo halves,
// each 256 bytes ([moment chunk 8 m / 8][row][moment % 8], 2 bytes each), then
// the row scale 2^k1 of each (moment chunk, row) as one signed byte.
constexpr int kViBlock = 2 * 256 + 16;

enum MixFormat { MIX_F16 = 0, MIX_BF16 = 1 };

// ------------------------------------------------------- 16-bit splitting
template <int FMT>
struct Half16;
template <>
struct Half16<MIX_F16> {
  static __device__ __forceinline__ uint16_t rn(double x) { return __half_as_ushort(__double2half(x)); }
  static __device__ __forceinline__ float val(uint16_t h) { return __half2float(__ushort_as_half(h)); }
  static __device__ __forceinline__ uint32_t pack(float x, float y) {
    const __half2 t = __floats2half2_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&t);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t p) {
    return __half22float2(*reinterpret_cast<const __half2*>(&p));
  }
};
template <>
struct Half16<MIX_BF16> {
  static __device__ __forceinline__ uint16_t rn(double x) { return __bfloat16_as_ushort(__double2bfloat16(x)); }
  static __device__ __forceinline__ float val(uint16_t h) { return __bfloat162float(__ushort_as_bfloat16(h)); }
  static __device__ __forceinline__ uint32_t pack(float x, float y) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&t);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t p) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&p));
  }
};

// The scale 2^k that brings m (> 0) to [2^14, 2^15); k is clamped so that
// 2^k and 2^-k stay normal floats.  m = 0 gives k = 0.
__device__ __forceinline__ int split_scale_d(double m) {
  if (!(m > 0.0)) return 0;
  const int be = (int)((__double_as_longlong(m) >> 52) & 0x7ff);
  const int e = be == 0 ? -1021 : be - 1022;  // m in [2^(e-1), 2^e)
  return max(-120, min(120, 15 - e));
}
__device__ __forceinline__ int split_scale_f(float m) {
  if (!(m > 0.0f)) return 0;
  const int be = (__float_as_int(m) >> 23) & 0xff;
  const int e = be == 0 ? -125 : be - 126;
  return max(-120, min(120, 15 - e));
}
__device__ __forceinline__ float f_pow2(int k) { return __int_as_float((127 + k) << 23); }

__device__ __forceinline__ void mma_k8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0, Half16<MIX_F16>) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mma_k8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0, Half16<MIX_BF16>) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mma_k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1, Half16<MIX_F16>) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1, Half16<MIX_BF16>) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void lds4f(float (&v)[4], uint32_t p) {
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(p));
}
__device__ __forceinline__ void sts4f(uint32_t p, const float (&v)[4]) {
  asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
__device__ __forceinline__ void sts4f_p(uint32_t p, const float (&v)[4], bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %5, 0;\n @p st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n}" ::"r"(p), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ uint32_t lds1u(uint32_t p) {
  uint32_t a;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(a) : "r"(p));
  return a;
}
__device__ __forceinline__ int lds1s8(uint32_t p) {
  int a;
  asm volatile("ld.shared.s8 %0, [%1];" : "=r"(a) : "r"(p));
  return a;
}

// Sizes as in RowCfg (offsets in doubles); NT = 2 or 4 angle tiles.  A face
// entry is [tile pair][lane][2 tiles x 2 angles] floats.
template <int NM_, int FMT, int NT_>
struct MixRowCfg {
  static constexpr int NT = NT_, W = 4, R = 8;
  static constexpr int H = NM_ > 8 ? 2 : 1;   // moment chunks
  static constexpr int MT = (NM_ + 7) / 8;    // moment tiles of the second product
  static constexpr int S = NT / 2;            // 16-angle halves
  static constexpr int NTH = (R + 4) * 32;
  static constexpr int E = NT * 32;           // doubles per face entry
  static constexpr int D = 4;                 // input ring of a warp, in pairs of cells
  static constexpr int PAIR = 2 * kViBlock;   // bytes of a pair
  static constexpr int DY = 4;                // y faces between two rows
  static constexpr int NREC = 4;
  static constexpr int B1 = NT * H * 2 * 32, B2 = S * MT * 4 * 32;  // words: [t][h][hi, lo], [s][mt][b][hi, lo]
  static constexpr int MAT = (B1 + B2) / 2 + 2;                    // + the two matrix scales (doubles)
  static constexpr int SM_ZC = 0;
  static constexpr int SM_Y = SM_ZC + R * W * E;
  static constexpr int SM_X = SM_Y + R * DY * E;
  static constexpr int SM_BND = SM_X + R * E;
  static constexpr int SM_RING = SM_BND + R * E;
  static constexpr int SM_MAT = SM_RING + R * D * PAIR / 8;
  static constexpr int SM_BAR = SM_MAT + 2 * MAT;
  static constexpr int NBAR = 2 * R + 2 * R * DY;
  static constexpr int SM_REC = SM_BAR + NBAR;
  static constexpr int SM_CNT = SM_REC + NREC * 24;
  static constexpr int SM_END = SM_CNT + 16;
  static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)SM_END; }

  // The octant's matrices, split into scaled hi / lo halves, in fragment order.
  static __device__ __forceinline__ void load_matrices(double* mat, const Fp64Prob& Q, int oct, int lane) {
    using HF = Half16<FMT>;
    uint32_t* const m = reinterpret_cast<uint32_t*>(mat);
    const int q = lane >> 2, r = lane & 3;
    const size_t as = Q.a_stride ? (size_t)Q.a_stride : (size_t)Q.na;
    auto afm = [&](int ia, int im) {
      return ia < Q.na && im < NM_ ? __ldg(&Q.afm[ia + as * (im + (size_t)NM_ * oct)]) : 0.0;
    };
    auto mfa = [&](int ia, int im) {
      return ia < Q.na && im < NM_ ? __ldg(&Q.mfa[im + (size_t)NM_ * (ia + as * oct)]) : 0.0;
    };
    // twice through the entries: the largest, then the halves
    double m1 = 0.0, m2 = 0.0;
#pragma unroll 4
    for (int e = 0; e < NT * H * 2; ++e)
      m1 = fmax(m1, fabs(afm(8 * (e / (2 * H)) + q, 8 * ((e >> 1) % H) + 2 * r + (e & 1))));
#pragma unroll 4
    for (int e = 0; e < S * MT * 4; ++e)
      m2 = fmax(m2, fabs(mfa(16 * (e / (4 * MT)) + 8 * ((e >> 1) & 1) + 2 * r + (e & 1), 8 * ((e >> 2) % MT) + q)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
      m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    }
    const int kb1 = split_scale_d(m1), kb2 = split_scale_d(m2);
    const double s1 = d_pow2(kb1), s2 = d_pow2(kb2);
    auto split = [&](double x, double y, uint32_t* hi, uint32_t* lo) {
      const uint16_t xh = HF::rn(x), yh = HF::rn(y);
      const uint16_t xl = HF::rn(x - (double)HF::val(xh)), yl = HF::rn(y - (double)HF::val(yh));
      *hi = (uint32_t)xh | ((uint32_t)yh << 16);
      *lo = (uint32_t)xl | ((uint32_t)yl << 16);
    };
#pragma unroll 2
    for (int e = 0; e < NT * H; ++e) {
      const int ia = 8 * (e / H) + q, im = 8 * (e % H) + 2 * r;
      split(afm(ia, im) * s1, afm(ia, im + 1) * s1, &m[(2 * e) * 32 + lane], &m[(2 * e + 1) * 32 + lane]);
    }
#pragma unroll 2
    for (int e = 0; e < S * MT * 2; ++e) {  // (s, mt, b)
      const int ia = 16 * (e / (2 * MT)) + 8 * (e & 1) + 2 * r, im = 8 * ((e >> 1) % MT) + q;
      split(mfa(ia, im) * s2, mfa(ia + 1, im) * s2, &m[B1 + (2 * e) * 32 + lane], &m[B1 + (2 * e + 1) * 32 + lane]);
    }
    if (lane == 0) {
      m[B1 + B2] = (uint32_t)kb1;
      m[B1 + B2 + 1] = (uint32_t)kb2;
    }
  }
};

// One compute warp, as row_compute of the FP64 kernel; Q.vi is the converted
// vi (kViBlock bytes per (cell, group pair)), Q.vo the octants' FP32 partials
// (one state after another).
template <int NM_, int FMT, int NT, bool SPARE, class PP>
__device__ __forceinline__ void mix_row_compute(const PP& P, double* smem) {
  using C = MixRowCfg<NM_, FMT, NT>;
  using HF = Half16<FMT>;
  constexpr int E = C::E, W = C::W, D = C::D, DY = C::DY, R = C::R, H = C::H, MT = C::MT, S = C::S, PAIR = C::PAIR;
  const int lane = threadIdx.x & 31, warp = row_warp<SPARE>();
  const int q = lane >> 2, r = lane & 3;
  int* const cnt = reinterpret_cast<int*>(smem + C::SM_CNT);
  const uint32_t sb = smem_u32(smem);
  const uint32_t xfull = sb + 8 * (C::SM_BAR + warp), xempty = xfull + 8 * R;
  const uint32_t yfull = sb + 8 * (C::SM_BAR + 2 * R + warp * DY), yempty = yfull + 8 * R * DY;
  const uint32_t y_in_ring = sb + 8 * (C::SM_Y + warp * DY * E) + 16 * lane, y_out_ring = y_in_ring + 8 * DY * E;
  const uint32_t zc = sb + 8 * (C::SM_ZC + warp * W * E) + 16 * lane;
  const uint32_t xin = sb + 8 * (C::SM_X + warp * E) + 16 * lane, bnd = sb + 8 * (C::SM_BND + warp * E) + 16 * lane;
  const uint32_t ring = sb + 8 * C::SM_RING + warp * D * PAIR;
  float wz[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) wz[i] = 0.25f - 1.0f / (float)(1 << (2 * r + i));

  const int rw = P.pr.rw, row = warp % rw;
  uint32_t x_ph = 0;
  uint32_t yi = 0, yi_ph = 0, yo = 0, yo_ph = 1;  // y rings: positions and phases
  for (int k = 0;; ++k) {
    if (!row_wait_count(cnt + RC_POSTED, k + 1, cnt, P.sy, 64)) return;
    const RowRec& rec = reinterpret_cast<const RowRec*>(smem + C::SM_REC)[k % C::NREC];
    if (rec.stop) return;
    const int oct = rec.oct, flags = rec.flags, gp = rec.gp * (R / rw) + warp / rw;
    const Fp64Prob& Q = rec.q;
    const int w = rec.x1 - rec.x0, h = rec.y1 - rec.y0, nzr = rec.z1 - rec.z0;
    if (row >= h || gp >= Q.ngp) {
      __syncwarp();
      if (lane == 0) st_release_cta(cnt + RC_PLANES + warp, rec.plane0 + nzr);
      continue;
    }
    const bool y_feed = row > 0 || (flags & TF_Y_IN);
    const bool y_pass = row + 1 < h;
    const bool y_out = !y_pass && (flags & TF_Y_OUT);
    const bool x_in = (flags & TF_X_IN) != 0, z_in = (flags & TF_Z_IN) != 0;
    const bool x_out = (flags & TF_X_OUT) != 0, z_out = (flags & TF_Z_OUT) != 0;
    const int dx = (oct & 1) ? -1 : 1, dy = (oct & 2) ? -1 : 1, dz = (oct & 4) ? -1 : 1;
    const int ix0 = dx > 0 ? rec.x0 : rec.x1 - 1, iz0 = dz > 0 ? rec.z0 : rec.z1 - 1;
    const int iy = dy > 0 ? rec.y0 + row : rec.y1 - 1 - row;
    const int g_col = 2 * gp + (q >> 2);  // the lane's group
    const bool gval = g_col < Q.ne;
    const float so = (float)(1 + oct);
    const double so_rd = 1.0 / (double)(1 + oct);
    const float so_hi = __double2float_rn(so_rd), so_lo = __double2float_rn(so_rd - (double)so_hi);
    int sp0 = ix0 + 3 * iy + 7 * iz0 + 2 + Q.sp_off;  // log2 s_space of the row's first cell, mod 4
    // boundary flux without its space factor, which the coefficient cancels
    {
      const float face_k = gval ? (float)d_scale_energy(Q.ie_base + g_col) * (float)d_scale_unknown(q & 3) * so : 0.0f;
#pragma unroll
      for (int t2 = 0; t2 < S; ++t2) {
        float f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int ia = 16 * t2 + 8 * (i >> 1) + 2 * r + (i & 1), iag = Q.ia_base + ia;
          f[i] = ia < Q.na ? (float)((1 + iag) << (iag & 7)) * face_k : 0.0f;
        }
        sts4f(bnd + t2 * 512, f);
      }
    }
    uint32_t b1[NT][H][2], b2[S][MT][2][2];
    const uint32_t mat = sb + 8 * (C::SM_MAT + (k & 1) * C::MAT);
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int c = 0; c < H; ++c)
#pragma unroll
        for (int p = 0; p < 2; ++p) b1[t][c][p] = lds1u(mat + 4 * (((t * H + c) * 2 + p) * 32 + lane));
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int p = 0; p < 2; ++p)
            b2[s][mt][b][p] = lds1u(mat + 4 * (C::B1 + (((s * MT + mt) * 2 + b) * 2 + p) * 32 + lane));
    const int kb1 = (int)lds1u(mat + 4 * (C::B1 + C::B2)), kb2 = (int)lds1u(mat + 4 * (C::B1 + C::B2 + 1));
    const size_t slab = (size_t)NM_ * NU * Q.nx * Q.ny;
    float* vdst = reinterpret_cast<float*>(Q.vo) + slab * Q.ne * Q.nz * (size_t)oct +
                  (size_t)NM_ * NU * (ix0 + (size_t)Q.nx * iy) + slab * (size_t)g_col + slab * Q.ne * (size_t)iz0 +
                  NM_ * (q & 3) + 2 * r;
    const int vda = dx * NM_ * NU;
    const long long vdc = (long long)dz * slab * Q.ne - w * vda;

    // This warp's own copies, 16 bytes a lane: a pair of vi blocks (adjacent
    // in memory) D - 1 pairs ahead; the entering z faces of the row here.
    const int np = (w + 1) / 2;  // pairs per row
    const char* cpb = reinterpret_cast<const char*>(Q.vi) +
                      (((size_t)iz0 * Q.ngp + gp) * Q.ny * Q.nx + (size_t)iy * Q.nx + ix0) * kViBlock + 16 * lane;
    const long long cpc = (long long)dz * Q.ngp * Q.ny * Q.nx * kViBlock;
    int pa = 0, pleft = nzr * np;
    uint32_t pslot = 0;
    auto prefetch = [&]() {
      const bool on = pleft > 0;
      const int nc = min(2, w - pa), lo = dx > 0 ? pa : pa + nc - 1;
      const char* src = cpb + dx * lo * kViBlock;
      const uint32_t dst = ring + pslot * PAIR + 16 * lane;
      cp_async16_p(dst, src, on);
      cp_async16_p(dst + 512, src + 512, on && 32 + lane < 33 * nc);
      cp_async16_p(dst + 1024, src + 1024, on && 64 + lane < 33 * nc);
      cp_async_commit();
      --pleft;
      pa += 2;
      cpb += pa >= w ? cpc : 0;
      pa = pa >= w ? 0 : pa;
      pslot = pslot == D - 1 ? 0 : pslot + 1;
    };
    const size_t ent = (size_t)oct * Q.ngp + gp;
    if (z_in) {
      const double* f = Q.fxy + ((ent * Q.ny + iy) * Q.nx + ix0) * (size_t)E + 2 * lane;
      for (int a = 0; a < w; ++a, f += dx * E)
#pragma unroll
        for (int t2 = 0; t2 < S; ++t2) cp_async16_s(zc + a * (8 * E) + t2 * 512, f + t2 * 64);
    }
#pragma unroll
    for (int i = 0; i < D - 1; ++i) prefetch();

    // moments -> angles of a ring slot's pair, scaled: v[h][t][2 cell + i],
    // and the exponents of the two cells' rows
    auto transform1 = [&](float (&v)[H][NT][4], int (&k1)[2][H], uint32_t sl, int nc) {
      const uint32_t in0 = ring + sl * PAIR + (nc == 2 && dx < 0 ? kViBlock : 0);
      const uint32_t in1 = ring + sl * PAIR + (nc == 2 && dx > 0 ? kViBlock : 0);
#pragma unroll
      for (int c = 0; c < H; ++c) {
        const uint32_t o = c * 128 + q * 16 + r * 4;
        const uint32_t h0 = lds1u(in0 + o), h1 = lds1u(in1 + o), l0 = lds1u(in0 + 256 + o), l1 = lds1u(in1 + 256 + o);
        k1[0][c] = lds1s8(in0 + 512 + c * 8 + q);
        k1[1][c] = lds1s8(in1 + 512 + c * 8 + q);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          v[c][t][0] = v[c][t][1] = v[c][t][2] = v[c][t][3] = 0.0f;
          mma_k8(v[c][t], l0, l1, b1[t][c][0], HF());
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) mma_k8(v[c][t], h0, h1, b1[t][c][1], HF());
#pragma unroll
        for (int t = 0; t < NT; ++t) mma_k8(v[c][t], h0, h1, b1[t][c][0], HF());
      }
    };
    float v[H][NT][4];
    int k1[2][H];
    cp_async_wait<D - 2>();
    __syncwarp();
    transform1(v, k1, 0, min(2, w));

    uint32_t slot = 0;
    uint32_t zmask = z_in ? 3 : 0;  // 0: the z faces are the boundary flux
    const int ymask = y_feed ? 3 : 0;
    const bool vo_lane = gval && (NM_ >= 8 || r < 2);
    const bool arr = (lane == 0 && y_pass) || (lane == 1 && y_feed);
    for (int c = 0; c < nzr; ++c) {
      const bool last = c == nzr - 1;
      int sp = sp0;
      uint32_t xmask = 0;
      float fx[S][4];
      if (x_in) {
        xmask = 3;
        if (!__all_sync(0xffffffffu, bar_test(xfull, x_ph)) && !row_wait(xfull, x_ph, 0, 0, cnt, P.sy)) {
          cp_async_wait<0>();
          return;
        }
        x_ph ^= 1;
      }
#pragma unroll
      for (int t2 = 0; t2 < S; ++t2) lds4f(fx[t2], (x_in ? xin : bnd) + t2 * 512);
      if (x_in) {
        __syncwarp();
        if (lane == 0) bar_arrive(xempty);
      }
      for (int a = 0; a < w; a += 2) {
        const int nc = min(2, w - a);
        prefetch();
        cp_async_wait<D - 2>();  // this lane's copies for the next pair
        uint32_t ph[2][NT], pl[2][NT];  // psi of the two cells, split
        int k2[2][S];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (j == 1 && nc == 1) {
#pragma unroll
            for (int t = 0; t < NT; ++t) ph[1][t] = pl[1][t] = 0u;
#pragma unroll
            for (int s = 0; s < S; ++s) k2[1][s] = 0;
            break;
          }
          // ---- wait for the entering y face and for room for the leaving one
          const uint32_t yb = yfull + 8 * yi, eb = yempty + 8 * (DY + yo);
          if (!__all_sync(0xffffffffu, bar_test2(yb, yi_ph, y_feed, eb, yo_ph, y_pass)) &&
              !row_wait(y_feed ? yb : 0, yi_ph, y_pass ? eb : 0, yo_ph, cnt, P.sy)) {
            cp_async_wait<0>();
            return;
          }
          float fy[S][4], fz[S][4];
          const uint32_t za = zc + (a + j) * (8 * E);
          const uint32_t py = y_feed ? y_in_ring + yi * (8 * E) : bnd, pz = zmask ? za : bnd;
#pragma unroll
          for (int t2 = 0; t2 < S; ++t2) {
            lds4f(fy[t2], py + t2 * 512);
            lds4f(fz[t2], pz + t2 * 512);
          }
          // ---- Quantities_solve in FP32 (fused multiply-adds: fewer roundings)
          const float cxy = f_pow2(-1 - (int)((sp - 7 * dz) & zmask));
          const float cxz = f_pow2(-2 - ((sp - 3 * dy) & ymask));
          const float sx_r = f_pow2(-(int)((sp - dx) & xmask));
          const float cyz[2] = {__fmul_rn(wz[0], sx_r), __fmul_rn(wz[1], sx_r)};
          const float ccp = f_pow2(sp & 3);  // exact scalings of so_hi / so_lo
          const float cch = __fmul_rn(so_hi, ccp), ccl = __fmul_rn(so_lo, ccp);
          // vs = sum over the chunks of v * 2^-(k1 + kb1), each term in two
          // exact steps, the smaller factor first, so that no intermediate
          // leaves the FP32 range unless the term itself does
          float f1[H], f2[H];
#pragma unroll
          for (int ck = 0; ck < H; ++ck) {
            f1[ck] = f_pow2(min(-k1[j][ck], -kb1));
            f2[ck] = f_pow2(max(-k1[j][ck], -kb1));
          }
#pragma unroll
          for (int s = 0; s < S; ++s) {
            float psi[4], pmax = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int t = 2 * s + (i >> 1), ii = 2 * j + (i & 1);
              const float sab = __fmaf_rn(fz[s][i], cxy, __fmul_rn(fy[s][i], cxz));
              const float sm = __fmaf_rn(fx[s][i], cyz[i & 1], sab);
              float vs = __fmul_rn(__fmul_rn(v[0][t][ii], f1[0]), f2[0]);
              if constexpr (H == 2) vs = __fmaf_rn(__fmul_rn(v[H - 1][t][ii], f1[H - 1]), f2[H - 1], vs);
              // psi = sm * cc + vs rounded once to FP32, with cc the FP64
              // reciprocal of (1 + octant) as cch + ccl: the product's
              // rounding error (fma), the sum's (TwoSum) and the low part are
              // added back before the final rounding.  (With the FP32
              // reciprocal and a rounded product, the cancellation of the
              // large boundary fluxes in T2 amplified that rounding up to
              // 1e-4 relative in vo at na 64-128.)
              const float pp = __fmul_rn(sm, cch);
              const float plo = __fmaf_rn(sm, ccl, __fmaf_rn(sm, cch, -pp));
              const float s2 = __fadd_rn(pp, vs);
              const float bb = __fsub_rn(s2, pp);
              const float er = __fadd_rn(__fsub_rn(pp, __fsub_rn(s2, bb)), __fsub_rn(vs, bb));
              psi[i] = __fadd_rn(s2, __fadd_rn(er, plo));
              pmax = fmaxf(pmax, fabsf(psi[i]));
              fx[s][i] = __fmul_rn(psi[i], so);
            }
            // psi of these 16 angles -> scaled hi / lo (the row's largest, over its four lanes)
            pmax = fmaxf(pmax, __shfl_xor_sync(0xffffffffu, pmax, 1));
            pmax = fmaxf(pmax, __shfl_xor_sync(0xffffffffu, pmax, 2));
            k2[j][s] = split_scale_f(pmax);
            const float sc = f_pow2(k2[j][s]);
#pragma unroll
            for (int p = 0; p < 2; ++p) {
              const float x0 = __fmul_rn(psi[2 * p], sc), x1 = __fmul_rn(psi[2 * p + 1], sc);
              ph[j][2 * s + p] = HF::pack(x0, x1);
              const float2 hv = HF::unpack(ph[j][2 * s + p]);
              pl[j][2 * s + p] = HF::pack(__fsub_rn(x0, hv.x), __fsub_rn(x1, hv.y));
            }
          }
          // ---- leaving faces
#pragma unroll
          for (int t2 = 0; t2 < S; ++t2) {
            sts4f_p(y_out_ring + yo * (8 * E) + t2 * 512, fx[t2], y_pass);
            sts4f(za + t2 * 512, fx[t2]);
          }
          __syncwarp();
          bar_arrive_p(lane == 0 ? yfull + 8 * (DY + yo) : yempty + 8 * yi, arr);
          if (y_out || (last && z_out)) {
            const int ix = ix0 + dx * (a + j);
            double* const fo = Q.fxz + ((ent * Q.nz + (iz0 + dz * c)) * Q.nx + ix) * (size_t)E + 2 * lane;
            double* const fz2 = Q.fxy + ((ent * Q.ny + iy) * Q.nx + ix) * (size_t)E + 2 * lane;
#pragma unroll
            for (int t2 = 0; t2 < S; ++t2) {
              const float4 f4 = make_float4(fx[t2][0], fx[t2][1], fx[t2][2], fx[t2][3]);
              if (y_out) __stcg(reinterpret_cast<float4*>(fo + t2 * 64), f4);
              if (last && z_out) __stcg(reinterpret_cast<float4*>(fz2 + t2 * 64), f4);
            }
          }
          sp += dx;
          xmask = 3;
          if (y_feed) {
            yi = (yi + 1) % DY;
            yi_ph ^= yi == 0;
          }
          if (y_pass) {
            yo = (yo + 1) % DY;
            yo_ph ^= yo == 0;
          }
        }
        // ---- angles -> moments of this pair, moments -> angles of the next
        // (after the task's last pair: of a stale slot, unused)
        float d2[S][MT][4];
#pragma unroll
        for (int s = 0; s < S; ++s) {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            d2[s][mt][0] = d2[s][mt][1] = d2[s][mt][2] = d2[s][mt][3] = 0.0f;
            mma_k16(d2[s][mt], pl[0][2 * s], pl[1][2 * s], pl[0][2 * s + 1], pl[1][2 * s + 1], b2[s][mt][0][0],
                    b2[s][mt][1][0], HF());
          }
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
            mma_k16(d2[s][mt], ph[0][2 * s], ph[1][2 * s], ph[0][2 * s + 1], ph[1][2 * s + 1], b2[s][mt][0][1],
                    b2[s][mt][1][1], HF());
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
            mma_k16(d2[s][mt], ph[0][2 * s], ph[1][2 * s], ph[0][2 * s + 1], ph[1][2 * s + 1], b2[s][mt][0][0],
                    b2[s][mt][1][0], HF());
        }
        slot = slot == D - 1 ? 0 : slot + 1;
        __syncwarp();  // every lane's copies of the next pair
        transform1(v, k1, slot, a + 2 >= w ? min(2, w) : min(2, w - a - 2));
        // ---- this octant's partial of vo: each accumulator times 2^e with
        // e = -k2 - kb2 (|e| <= 240) in two exact power-of-two steps of e / 2
        // (an intermediate lies between the accumulator and the result), the
        // two halves' terms added with one rounding (fma)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (j < nc) {
            const int e0 = -k2[j][0] - kb2, e1 = S == 2 ? -k2[j][S - 1] - kb2 : 0;
            const float f0a = f_pow2(e0 / 2), f0b = f_pow2(e0 - e0 / 2);
            const float f1a = f_pow2(e1 / 2), f1b = f_pow2(e1 - e1 / 2);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
              float o[2];
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const float t1 = S == 2 ? __fmul_rn(__fmul_rn(d2[S - 1][mt][2 * j + i], f1a), f1b) : 0.0f;
                o[i] = __fmaf_rn(__fmul_rn(d2[0][mt][2 * j + i], f0a), f0b, t1);
              }
              if (vo_lane) *reinterpret_cast<float2*>(vdst + 8 * mt) = make_float2(o[0], o[1]);
            }
            vdst += vda;
          }
      }
      if (x_out) {
        double* const fo = Q.fyz + ((ent * Q.nz + (iz0 + dz * c)) * Q.ny + iy) * (size_t)E + 2 * lane;
#pragma unroll
        for (int t2 = 0; t2 < S; ++t2)
          __stcg(reinterpret_cast<float4*>(fo + t2 * 64), make_float4(fx[t2][0], fx[t2][1], fx[t2][2], fx[t2][3]));
      }
      sp0 += 7 * dz;
      zmask = 3;
      vdst += vdc;
      __syncwarp();
      if (lane == 0) st_release_cta(cnt + RC_PLANES + warp, rec.plane0 + c + 1);
    }
  }
}

template <int NM_, int FMT, int NT, bool SPARE>
__global__ void __launch_bounds__(384, 1) sweep_mixed_row_kernel(const Fp64Params P) {
  using C = MixRowCfg<NM_, FMT, NT>;
  extern __shared__ __align__(128) double smem[];
  if (threadIdx.x == 0) row_setup<C>(smem, true);
  __syncthreads();
  if ((threadIdx.x >> 5) >= C::R) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(80));
    row_producers<C, false>(P, 0, smem);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(208));
    mix_row_compute<NM_, FMT, NT, SPARE>(P, smem);
  }
}

// vi -> vi16, once per sweep, for the group pairs [gp0, gp1): thread t
// converts moment chunk `half` (moments 8 half .. 8 half + 7, zero padded) of
// row r8 = 4 g + u of the (t / 16)-th block of that range (cell (ix, iy, iz),
// group pair gp; group 2 gp + g, unknown u).  The chunk
// is scaled by 2^k1 so that its largest entry lies in [2^14, 2^15) (k1
// clamped to [-120, 120]), rounded to FP32 in FP64 and split into hi + lo
// 16-bit halves -- the operand every octant's first transform of that cell
// uses.  A group beyond ne (odd ne) and the chunks beyond NM are zeros.
template <int NM_, int FMT>
__global__ void __launch_bounds__(256) convert_vi16(const double* __restrict__ vi, unsigned char* __restrict__ out,
                                                    int nx, int ny, int nz, int ne, int ngp, int gp0, int gp1) {
  using H = Half16<FMT>;
  constexpr int NMC = NM_ < 8 ? NM_ : 8;  // moments of a chunk
  const int ngr = gp1 - gp0;  // the group pairs converted: [gp0, gp1)
  const long long nunit = (long long)nx * ny * nz * ngr * 16;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nunit;
       t += (long long)gridDim.x * blockDim.x) {
    const int r8 = (int)(t & 7), half = (int)((t >> 3) & 1);
    long long q = t >> 4;
    const int ix = (int)(q % nx);
    q /= nx;
    const int iy = (int)(q % ny);
    q /= ny;
    const int gp = gp0 + (int)(q % ngr), iz = (int)(q / ngr);
    const long long blk = (((long long)iz * ngp + gp) * ny + iy) * nx + ix;
    const int g = r8 >> 2, u = r8 & 3, ie = 2 * gp + g;
    int k1 = 0;
    uint32_t hi[4] = {0u, 0u, 0u, 0u}, lo[4] = {0u, 0u, 0u, 0u};
    if (ie < ne && 8 * half < NM_) {
      const double* src =
          vi + (size_t)NM_ * (u + (size_t)NU * (ix + (size_t)nx * (iy + (size_t)ny * (ie + (size_t)ne * iz)))) +
          8 * half;
      double v[NMC];
#pragma unroll
      for (int k = 0; k < NMC; ++k) v[k] = __ldcs(src + k);
      int emax = 0;  // largest biased exponent of the chunk
#pragma unroll
      for (int k = 0; k < NMC; ++k) emax = max(emax, (int)((__double_as_longlong(v[k]) >> 52) & 0x7ff));
      k1 = emax == 0 ? 0 : max(-120, min(120, 15 - (emax - 1022)));
      const double sc = d_pow2(k1);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float x0 = 2 * p < NMC ? __double2float_rn(v[2 * p < NMC ? 2 * p : 0] * sc) : 0.0f;
        const float x1 = 2 * p + 1 < NMC ? __double2float_rn(v[2 * p + 1 < NMC ? 2 * p + 1 : 0] * sc) : 0.0f;
        hi[p] = H::pack(x0, x1);
        const float2 hv = H::unpack(hi[p]);
        lo[p] = H::pack(__fsub_rn(x0, hv.x), __fsub_rn(x1, hv.y));
      }
    }
    unsigned char* b = out + (size_t)blk * kViBlock;
    const int o = half * 128 + r8 * 16;
    *reinterpret_cast<uint4*>(b + o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(b + 256 + o) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    reinterpret_cast<signed char*>(b + 512)[half * 8 + r8] = (signed char)k1;
  }
}

// vo = sum over the eight octants of their FP32 partials, in FP64 and in
// octant order (deterministic); with `accumulate` the sum is added to vo (the
// angle passes after the first of a larger na).  The elements summed are
// iz * zstride + off + [0, width) for iz in [0, nz): one contiguous run of
// groups per z-plane (the whole state: zstride = width, off = 0).  width,
// zstride and off are multiples of 4 (NM * NU elements per (cell, group)).
__global__ void __launch_bounds__(256) reduce_octant_partials(double* __restrict__ vo,
                                                              const float* __restrict__ part, size_t state,
                                                              int accumulate, size_t zstride, size_t off,
                                                              size_t width, int nz) {
  const size_t w4 = width / 4, n4 = w4 * (size_t)nz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
    size_t e4 = off / 4 + i;  // in units of 4 elements; one run when the groups are all of them
    if (zstride != width) {
      const size_t iz = i / w4;
      e4 = (iz * zstride + off) / 4 + (i - iz * w4);
    }
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (accumulate) {
      const double2* d = reinterpret_cast<const double2*>(vo) + 2 * e4;
      const double2 p0 = __ldcs(d), p1 = __ldcs(d + 1);
      a0 = p0.x;
      a1 = p0.y;
      a2 = p1.x;
      a3 = p1.y;
    }
#pragma unroll
    for (int o = 0; o < NOCTANT; ++o) {
      const float4 q = __ldcs(reinterpret_cast<const float4*>(part + state * o) + e4);
      a0 = __dadd_rn(a0, (double)q.x);
      a1 = __dadd_rn(a1, (double)q.y);
      a2 = __dadd_rn(a2, (double)q.z);
      a3 = __dadd_rn(a3, (double)q.w);
    }
    double2* d = reinterpret_cast<double2*>(vo) + 2 * e4;
    __stcs(d, make_double2(a0, a1));
    __stcs(d + 1, make_double2(a2, a3));
  }
}

}  // namespace msb
