// The row pass of the iteration from the state V = Y + U for row lengths whose
// transforms hand over in registers (ct_reg_edges: 64 to 2048, powers of two).
//
//   ROW_ITER, ROW_ITER_D  inverse row transform of the pair's spectrum rows,
//                         previous Y and U from V, over-relaxation, shrinkage,
//                         dual update, residual partial sums, new V, forward
//                         transform of Y - U (ROW_ITER_D: F holds the column
//                         pass's correction to Y - U only)
//   ROW_FIXUP             after a change of rho: forward transform of
//                         Y - U / rsf from V
//
// One transform group of g threads per row pair, groups synchronised by
// themselves (group_sync), CTAs of SC_ROWV_THREADS.  The pass is bound by
// latency and by the phases of its transforms (shared-memory exchange against
// arithmetic), so what counts is the number of row pairs in flight per SM and
// how few registers and bytes of shared memory a pair takes:
//  * one staging buffer per pair: the spectrum rows of the next pair land in
//    it during the forward transform, the pair's state rows during the inverse
//    one;
//  * the two rows of a pair are the two halves of packed FP32 instructions,
//    in the transforms and in the element-wise step alike;
//  * weights per element, the AMS map and the projections take a rolled loop
//    of their own, so that the common rows keep their registers.
// Measured per launch against row_kernel (256-thread CTAs in lock step, a
// staging buffer each for spectrum and state rows), ITER / FIXUP active:
// 2048 x 2048, 256 maps 4.99 -> 3.93 ms / 2.37 -> 1.9 ms (17.2 / 8.6 GB: 4.4
// TB/s; at 1965 MHz; 4.2 to 4.4 ms within a 100-iteration solve, where the power
// cap holds the clock at 1820 to 1890 MHz); 512 x 512, 100 maps 130 -> 101 us;
// 256 x 256, 64 maps 26 -> 18 us; 64 x 64, 32 maps 7.2 -> 4.7 us.
#pragma once

#include "sc_kernels.cuh"

// Shrinkage of both halves: sign(v) max(|v| - t, 0).
__device__ __forceinline__ f32x2 soft2(float2 v, float t0, float t1) {
  return pk2(copysignf(fmaxf(fabsf(v.x) - t0, 0.f), v.x),
             copysignf(fmaxf(fabsf(v.y) - t1, 0.f), v.y));
}

// PL: F in the paired layout (spec_re).
template <int MODE, int NW, bool PL>
__global__ void __launch_bounds__(SC_ROWV_THREADS, rowv_min_blocks(NW))
rowv_kernel(RowParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red_scratch[(SC_ROWV_THREADS / 32) * 5];
  pdl_enter();

  constexpr bool FIX = MODE == ROW_FIXUP;
  constexpr bool DL = MODE == ROW_ITER_D;
  constexpr int RM = row_radix(NW);
  constexpr int g = ct_threads(NW, RM);
  constexpr int BG = rowv_barrier(NW);
  constexpr int S = SC_ROWV_THREADS / g;
  constexpr int EM = NW / g;  // elements per thread
  constexpr int NP = ct_plan(NW, RM).np;
  constexpr int W = NW, Wf = NW / 2 + 1, Wp = (Wf + 3) & ~3;
  const int H = P.g.H;
  const int b = blockIdx.y;
  const int s = threadIdx.x / g;
  const int t = threadIdx.x - s * g;
  unsigned char* slot = smem_raw + (size_t)s * rowv_slot_bytes(NW);
  float2* z = reinterpret_cast<float2*>(slot);
  float2* fst = z + NW;                            // spectrum rows: 2 Wp
  float* vst = reinterpret_cast<float*>(fst);      // state rows: 2 W
  auto zs = [](int k) { return fft_slot<NW, RM, 1>(k); };

  const ImgState& st = P.st[b];
  if (st.done) return;
  float thr = 0.f, thr_prev;
  if constexpr (FIX) {
    if (st.rsf == 1.0 && !st.relay) return;
    thr_prev = (float)((double)P.lam[b] / st.rho_prev);
  } else {
    thr = (float)((double)P.lam[b] / st.rho);
    // no iteration yet: V = 0 and a zero threshold give Y = U = 0
    thr_prev = st.k == 0 ? 0.f : (float)((double)P.lam[b] / st.rho_prev);
  }
  const float uscale = (float)st.uscale;

  const int rows = P.g.M * H;  // rows per image
  const int npairs = (rows + 1) / 2;
  float2* Fi = P.F + (size_t)b * rows * Wp;
  const float* Vi = P.U + (size_t)b * rows * W;
  float* Vo = (P.Vo ? P.Vo : P.U) + (size_t)b * rows * W;
  const int32_t* mk = P.mask ? P.mask + (size_t)b * H * W : nullptr;
  const int pstride = gridDim.x * S;

  // threshold weights, AMS mask row and projections of image row r
  auto roww = [&](int r, bool ok) -> RowW {
    RowW o{P.l1_scalar, nullptr, nullptr, SC_NO_CUT, false};
    if (!ok) return o;
    const int m = r / H, h = r - m * H;
    if (P.l1_kind == 1) o.w = P.l1w[m];
    if (P.l1_kind == 2) o.wr = P.l1w + ((size_t)m * H + h) * W;
    if (mk && m == 0) o.mrow = mk + (size_t)h * W;
    o.nonneg = P.nonneg != 0;
    if (P.bnd_r > 0 && h >= P.bnd_r) o.kcut = 0;
    else if (P.bnd_c > 0 && P.bnd_c < W) o.kcut = P.bnd_c;
    return o;
  };
  auto issue_F = [&](int p) {
    if (p < npairs) {
      const int nch = (2 * p + 1 < rows ? 2 : 1) * (Wp / 2);
      const float2* src = Fi + (size_t)2 * p * Wp;
#pragma unroll
      for (int i = 0; i < (Wp + g - 1) / g; ++i) {
        const int q = t + i * g;
        if (q < nch) cp_async16(fst + 2 * q, src + 2 * q);
      }
    }
    cp_async_commit();
  };
  auto issue_V = [&](int p) {
    if (p < npairs) {
      const int nch = (2 * p + 1 < rows ? 2 : 1) * (W / 4);
      const float* src = Vi + (size_t)2 * p * W;
#pragma unroll
      for (int i = 0; i < (W / 2 + g - 1) / g; ++i) {
        const int q = t + i * g;
        if (q < nch) cp_async16(vst + 4 * q, src + 4 * q);
      }
    }
    cp_async_commit();
  };

  // PL: float indices of column t + g m and (EM - 1 - m for m) of its mirror
  // image W - (t + g m) = (g - t) + g (EM - 1 - m); with g a multiple of 32 the
  // column groups' order does not depend on m
  const int it = t, im = g - t;
  auto sre = [](int c, int m) -> int {
    return g % 32 == 0 ? spec_re(c) + 2 * g * m : spec_re(c + g * m);
  };
  auto sim = [](int c, int m) -> int {
    return g % 32 == 0 ? (spec_re(c) ^ 2) + 2 * g * m : spec_re(c + g * m) ^ 2;
  };

  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int p0 = blockIdx.x * S + s;
  if constexpr (FIX) issue_V(p0);
  else issue_F(p0);
  for (int pb = blockIdx.x * S; pb < npairs; pb += pstride) {
    const int p = pb + s;
    const bool valid = p < npairs;
    const int r0 = 2 * p;
    const bool has1 = valid && r0 + 1 < rows;
    float2 v[EM];
    if constexpr (!FIX) {
      cp_async_wait<0>();  // the spectrum rows
      group_sync<BG>();
      // v = conj(A + iB) of the Hermitian-extended rows A, B (the inverse
      // transform as conj(FFT(conj .))): element k below W / 2 from A[k],
      // B[k], above from their mirror images; the imaginary parts of bins 0
      // and W / 2 are ignored, as a C2R transform does
#pragma unroll
      for (int m = 0; m < EM; ++m) {
        const int k = t + g * m;
        const int kk = m < EM / 2 ? k : W - k;
        float2 A = make_float2(0.f, 0.f), B = A;
        if constexpr (PL) {
          const float* fs = reinterpret_cast<const float*>(fst);
          const int i = m < EM / 2 ? sre(it, m) : sre(im, EM - 1 - m);
          const int j = m < EM / 2 ? sim(it, m) : sim(im, EM - 1 - m);
          if (valid) A = make_float2(fs[i], fs[j]);
          if (has1) B = make_float2(fs[2 * Wp + i], fs[2 * Wp + j]);
        } else {
          if (valid) A = fst[kk];
          if (has1) B = fst[Wp + kk];
        }
        if ((m == 0 || m == EM / 2) && t == 0) A.y = B.y = 0.f;
        if (m < EM / 2) v[m] = up2(fma2(pk2(A), pk2(1.f, -1.f), pk2(-B.y, -B.x)));
        else v[m] = up2(fma2(pk2(B.y, B.x), pk2(1.f, -1.f), pk2(A)));
      }
      ct_first_from_regs<NW, RM, 1, BG, false, 1>(z, v, t);
      issue_V(p);  // the spectrum rows are consumed
      fft_ct_passes<NW, RM, g, 1, 1, NP - 1, BG, 1>(z, P.twW, t);
      cp_async_wait<0>();  // the state rows
      group_sync<BG>();
      ct_last_to_regs<NW, RM, 1, 1>(z, P.twW, v, t);
    } else {
      cp_async_wait<0>();
      group_sync<BG>();
    }
    if (valid) {
      const RowW w0 = roww(r0, true), w1 = roww(r0 + 1, has1);
      float* o0 = Vo + (size_t)r0 * W;
      if (has1 && w0.plain() && w1.plain()) {
        const float tq0 = thr_prev * w0.w, tq1 = thr_prev * w1.w;
        const f32x2 us = dup2(uscale);
        if constexpr (FIX) {
#pragma unroll
          for (int m = 0; m < EM; ++m) {
            const int k = t + g * m;
            const float2 sv = make_float2(vst[k], vst[W + k]);
            const f32x2 y = soft2(sv, tq0, tq1);
            v[m] = up2(sub2(y, mul2(sub2(pk2(sv), y), us)));
          }
        } else {
          const float tc0 = thr * w0.w, tc1 = thr * w1.w;
          const f32x2 a = dup2(P.relax), a1 = dup2(1.f - P.relax);
          f32x2 f[5];
#pragma unroll
          for (int i = 0; i < 5; ++i) f[i] = dup2(0.f);
#pragma unroll
          for (int m = 0; m < EM; ++m) {
            const int k = t + g * m;
            const float2 sv = make_float2(vst[k], vst[W + k]);
            const f32x2 yo = soft2(sv, tq0, tq1);
            const f32x2 uo = mul2(sub2(pk2(sv), yo), us);
            f32x2 x;
            // X = IFFT2(Z^ + conj(Df) SC / rho) = (Y - U) + the correction,
            // to which the column pass has applied 1 / (H W)
            if constexpr (DL) x = fma2(pk2(v[m]), pk2(1.f, -1.f), sub2(yo, uo));
            else x = mul2(pk2(v[m]), pk2(P.invN, -P.invN));
            // (a x, the larger product, is the fused one; see iter_elem)
            const f32x2 vn = add2(fma2(a, x, mul2(a1, yo)), uo);
            const float2 vv = up2(vn);
            const f32x2 y = soft2(vv, tc0, tc1);
            const f32x2 u = sub2(vn, y);
            o0[k] = vv.x;
            o0[W + k] = vv.y;
            const f32x2 dxy = sub2(x, y), dyy = sub2(yo, y);
            f[0] = fma2(x, x, f[0]);
            f[1] = fma2(y, y, f[1]);
            f[2] = fma2(u, u, f[2]);
            f[3] = fma2(dxy, dxy, f[3]);
            f[4] = fma2(dyy, dyy, f[4]);
            v[m] = up2(sub2(y, u));
          }
#pragma unroll
          for (int i = 0; i < 5; ++i) {
            const float2 h = up2(f[i]);
            acc[i] += (double)(h.x + h.y);
          }
        }
      } else {
        // full weights, the AMS map, projections, or a last row by itself
        IterC ic;
        ic.a = P.relax;
        ic.a1 = 1.f - P.relax;
        ic.relax = P.relax != 1.f;
        ic.uscale = uscale;
        ic.delta = DL;
        float f[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        // (a rolled loop over a copy: few rows come here, and unrolled it
        // would cost the common path registers)
        float2 lv[EM];
#pragma unroll
        for (int m = 0; m < EM; ++m) lv[m] = v[m];
#pragma unroll 1
        for (int m = 0; m < EM; ++m) {
          const int k = t + g * m;
          const float s0 = vst[k], s1 = has1 ? vst[W + k] : 0.f;
          float y0, y1 = 0.f;
          if constexpr (FIX) {
            y0 = shrink_y(s0, thr_prev, w0, k);
            y0 -= (s0 - y0) * uscale;
            if (has1) {
              y1 = shrink_y(s1, thr_prev, w1, k);
              y1 -= (s1 - y1) * uscale;
            }
          } else {
            const float xn = DL ? 1.f : P.invN;
            y0 = iter_elem<true, false, DL ? 1 : 0>(lv[m].x * xn, s0, 0.f, w0, k, thr, thr_prev,
                                                    ic, f, o0 + k, nullptr);
            if (has1)
              y1 = iter_elem<true, false, DL ? 1 : 0>(-lv[m].y * xn, s1, 0.f, w1, k, thr,
                                                      thr_prev, ic, f, o0 + W + k, nullptr);
          }
          lv[m] = make_float2(y0, y1);
        }
#pragma unroll
        for (int m = 0; m < EM; ++m) v[m] = lv[m];
#pragma unroll
        for (int i = 0; i < 5; ++i) acc[i] += (double)f[i];
      }
    } else {
#pragma unroll
      for (int m = 0; m < EM; ++m) v[m] = make_float2(0.f, 0.f);
    }
    ct_first_from_regs<NW, RM, 1, BG, true, 1>(z, v, t);
    // the state rows are consumed: the next pair's rows land during this
    // pair's forward transform
    if constexpr (FIX) issue_V(p + pstride);
    else issue_F(p + pstride);
    fft_ct_passes<NW, RM, g, 1, 1, NP, BG, 1>(z, P.twW, t);
    if (valid) {
      // A = (Z_k + conj Z_-k) / 2,  B = (Z_k - conj Z_-k) / 2i
      float2* fa = Fi + (size_t)r0 * Wp;
#pragma unroll
      for (int m = 0; m <= EM / 2; ++m) {
        const int k = t + g * m;
        if (m < EM / 2 || t == 0) {
          const f32x2 Zk = pk2(z[zs(k)]), Zm = pk2(z[zs(k == 0 ? 0 : W - k)]);
          const f32x2 h = dup2(0.5f);
          const float2 a = up2(mul2(fma2(Zm, pk2(1.f, -1.f), Zk), h));
          const float2 bb = up2(mul2(swap2(fma2(Zm, pk2(-1.f, 1.f), Zk)), pk2(0.5f, -0.5f)));
          if constexpr (PL) {
            float* fs = reinterpret_cast<float*>(fa);
            const int i = sre(it, m), j = sim(it, m);
            fs[i] = a.x;
            fs[j] = a.y;
            if (has1) {
              fs[2 * Wp + i] = bb.x;
              fs[2 * Wp + j] = bb.y;
            }
          } else {
            fa[k] = a;
            if (has1) fa[Wp + k] = bb;
          }
        }
      }
    }
    // (the next pair's first barrier comes before z is written again)
  }
  cp_async_wait<0>();
  if constexpr (FIX) return;
  block_sum<5>(acc, red_scratch);
  if (threadIdx.x == 0) {
    double* out = P.partials + ((size_t)b * P.nblk + blockIdx.x) * 5;
#pragma unroll
    for (int i = 0; i < 5; ++i) out[i] = acc[i];
  }
}

// ------------------------------------------------------ any row length --
// One pass of a runtime plan in packed instructions, every twiddle from the table
// (as products of table entries the error of X after 30 iterations at 3 x 320 x
// 480 was 1.65e-6 instead of 1.17e-6, at the same speed; out of line: see
// fft_pass).
template <int R, int BG>
__device__ __forceinline__ void rt_pass_r(float2* z, int n, int Ns, const float2* __restrict__ tw,
                                          int t, int g) {
  constexpr int MAXB = (16 + R - 1) / R;
  const int B = n / R, step = n / (Ns * R);
  const unsigned mN = div_magic(Ns);
  float2 v[MAXB][R];
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int j = t + i * g;
    if (j < B) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[i][q] = z[j + q * B];
      if (Ns > 1) {
        const int ks = (j - div_by(j, mN) * Ns) * step;
#pragma unroll
        for (int q = 1; q < R; ++q) v[i][q] = p_mul(v[i][q], __ldg(&tw[q * ks]));
      }
      pdft_r<R>(v[i]);
    }
  }
  group_sync<BG>();
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int j = t + i * g;
    if (j < B) {
      const int k = j - div_by(j, mN) * Ns, base = (j - k) * R + k;
#pragma unroll
      for (int q = 0; q < R; ++q) z[base + q * Ns] = v[i][q];
    }
  }
  group_sync<BG>();
}
template <int BG>
__device__ __noinline__ void rt_pass(float2* z, int n, int R, int Ns,
                                     const float2* __restrict__ tw, int t, int g) {
  switch (R) {
    case 2: rt_pass_r<2, BG>(z, n, Ns, tw, t, g); break;
    case 3: rt_pass_r<3, BG>(z, n, Ns, tw, t, g); break;
    case 4: rt_pass_r<4, BG>(z, n, Ns, tw, t, g); break;
    case 5: rt_pass_r<5, BG>(z, n, Ns, tw, t, g); break;
    case 8: rt_pass_r<8, BG>(z, n, Ns, tw, t, g); break;
    default: generic_pass<16, BG>(z, n, R, Ns, 1, tw, t, g); break;
  }
}
template <int BG>
__device__ __forceinline__ void rt_fft(float2* z, const FftPlan& pl, const float2* __restrict__ tw,
                                       int t, int g) {
  int Ns = 1;
  for (int p = 0; p < pl.npass; ++p) {
    rt_pass<BG>(z, pl.n, pl.radix[p], Ns, tw, t, g);
    Ns *= pl.radix[p];
  }
}

// The row pass from the state V at any other row length (ROW_ITER, ROW_FIXUP):
// the same single staging buffer, groups of BG threads (P.gsz; 0: the whole CTA
// of 256) and passes of a runtime plan whose odd radices come first (the first
// pass's stores then have an odd stride, without bank conflicts).  Measured per
// launch against row_kernel's runtime plan, ITER / FIXUP: 3 x 320 x 480, 36
// maps, non-negative 343 / 99 -> 254 / 74 us; 475 x 315, 48 maps 208 / 84 -> 176
// / 71 us (4 / 5 / 6 / 8 CTAs per SM: 198 / 176 / 192 / 198 us); bound by the
// passes' shared-memory exchanges and the registers saved around their calls.
template <int MODE, int BG>
__global__ void __launch_bounds__(BG ? SC_ROWV_THREADS : 256, BG ? 5 : 2)
rowg_kernel(RowParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red_scratch[8 * 5];
  pdl_enter();

  constexpr bool FIX = MODE == ROW_FIXUP;
  constexpr int g = BG ? BG : 256;
  const int W = P.g.W, Wf = P.g.Wf, Wp = P.g.Wp, H = P.g.H;
  const int S = blockDim.x / g;
  const int b = blockIdx.y;
  const int s = threadIdx.x / g;
  const int t = threadIdx.x - s * g;
  float2* z = reinterpret_cast<float2*>(smem_raw + (size_t)s * rowg_slot_bytes(W, Wp));
  float2* fst = z + ((W + 1) & ~1);            // spectrum rows: 2 Wp
  float* vst = reinterpret_cast<float*>(fst);  // state rows: 2 W

  const ImgState& st = P.st[b];
  if (st.done) return;
  float thr = 0.f, thr_prev;
  if constexpr (FIX) {
    if (st.rsf == 1.0 && !st.relay) return;
    thr_prev = (float)((double)P.lam[b] / st.rho_prev);
  } else {
    thr = (float)((double)P.lam[b] / st.rho);
    thr_prev = st.k == 0 ? 0.f : (float)((double)P.lam[b] / st.rho_prev);
  }
  const float uscale = (float)st.uscale;
  const bool paired = P.paired != 0, delta = P.delta != 0;

  const int rows = P.g.M * H;  // rows per image
  const int npairs = (rows + 1) / 2;
  float2* Fi = P.F + (size_t)b * rows * Wp;
  const float* Vi = P.U + (size_t)b * rows * W;
  float* Vo = P.U + (size_t)b * rows * W;
  const int32_t* mk = P.mask ? P.mask + (size_t)b * H * W : nullptr;
  const int pstride = gridDim.x * S;
  const bool vec = (W & 3) == 0 || ((W & 1) == 0 && ((size_t)b * rows * W) % 4 == 0);

  auto roww = [&](int r, bool ok) -> RowW {
    RowW o{P.l1_scalar, nullptr, nullptr, SC_NO_CUT, false};
    if (!ok) return o;
    const int m = r / H, h = r - m * H;
    if (P.l1_kind == 1) o.w = P.l1w[m];
    if (P.l1_kind == 2) o.wr = P.l1w + ((size_t)m * H + h) * W;
    if (mk && m == 0) o.mrow = mk + (size_t)h * W;
    o.nonneg = P.nonneg != 0;
    if (P.bnd_r > 0 && h >= P.bnd_r) o.kcut = 0;
    else if (P.bnd_c > 0 && P.bnd_c < W) o.kcut = P.bnd_c;
    return o;
  };
  auto issue_F = [&](int p) {
    if (p < npairs) {
      const int nch = (2 * p + 1 < rows ? 2 : 1) * (Wp / 2);
      const float2* src = Fi + (size_t)2 * p * Wp;
      for (int q = t; q < nch; q += g) cp_async16(fst + 2 * q, src + 2 * q);
    }
    cp_async_commit();
  };
  auto issue_V = [&](int p) {
    if (p < npairs) {
      const int n = (2 * p + 1 < rows ? 2 : 1) * W;
      const float* src = Vi + (size_t)2 * p * W;
      if (vec && (n & 3) == 0) {
        for (int q = t; q < n / 4; q += g) cp_async16(vst + 4 * q, src + 4 * q);
      } else {
        for (int q = t; q < n; q += g) cp_async4(vst + q, src + q);
      }
    }
    cp_async_commit();
  };

  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  IterC ic;
  ic.a = P.relax;
  ic.a1 = 1.f - P.relax;
  ic.relax = P.relax != 1.f;
  ic.uscale = uscale;
  ic.delta = delta;
  const int p0 = blockIdx.x * S + s;
  if constexpr (FIX) issue_V(p0);
  else issue_F(p0);
  for (int pb = blockIdx.x * S; pb < npairs; pb += pstride) {
    const int p = pb + s;
    const bool valid = p < npairs;
    const int r0 = 2 * p;
    const bool has1 = valid && r0 + 1 < rows;
    cp_async_wait<0>();
    group_sync<BG>();
    if constexpr (!FIX) {
      if (valid)
        for (int k = t; k < W; k += g) z[k] = pack_inverse(fst, fst + Wp, has1, k, W, Wf, paired);
      group_sync<BG>();
      issue_V(p);  // the spectrum rows are consumed
      rt_fft<BG>(z, P.pw, P.twW, t, g);
      cp_async_wait<0>();  // the state rows
      group_sync<BG>();
    }
    if (valid) {
      const RowW w0 = roww(r0, true), w1 = roww(r0 + 1, has1);
      float* o0 = Vo + (size_t)r0 * W;
      const float xn = delta ? 1.f : P.invN;
      float f[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
      if (has1 && w0.plain() && w1.plain()) {
        const float tq0 = thr_prev * w0.w, tq1 = thr_prev * w1.w;
        const float tc0 = thr * w0.w, tc1 = thr * w1.w;
        const f32x2 us = dup2(uscale), a = dup2(P.relax), a1 = dup2(1.f - P.relax);
        const f32x2 xs = pk2(xn, -xn), dl = dup2(delta ? 1.f : 0.f);
        f32x2 f2[5];
#pragma unroll
        for (int i = 0; i < 5; ++i) f2[i] = dup2(0.f);
#pragma unroll 2
        for (int k = t; k < W; k += g) {
          const float2 sv = make_float2(vst[k], vst[W + k]);
          const f32x2 yo = soft2(sv, tq0, tq1);
          const f32x2 uo = mul2(sub2(pk2(sv), yo), us);
          if constexpr (FIX) {
            z[k] = up2(sub2(yo, uo));
          } else {
            const f32x2 x = fma2(pk2(z[k]), xs, mul2(dl, sub2(yo, uo)));
            // (a x, the larger product, is the fused one; see iter_elem)
            const f32x2 vn = add2(fma2(a, x, mul2(a1, yo)), uo);
            const float2 vv = up2(vn);
            const f32x2 y = soft2(vv, tc0, tc1);
            const f32x2 u = sub2(vn, y);
            o0[k] = vv.x;
            o0[W + k] = vv.y;
            const f32x2 dxy = sub2(x, y), dyy = sub2(yo, y);
            f2[0] = fma2(x, x, f2[0]);
            f2[1] = fma2(y, y, f2[1]);
            f2[2] = fma2(u, u, f2[2]);
            f2[3] = fma2(dxy, dxy, f2[3]);
            f2[4] = fma2(dyy, dyy, f2[4]);
            z[k] = up2(sub2(y, u));
          }
        }
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const float2 h = up2(f2[i]);
          f[i] = h.x + h.y;
        }
      } else {
        for (int k = t; k < W; k += g) {
          const float s0 = vst[k], s1 = has1 ? vst[W + k] : 0.f;
          float y0, y1 = 0.f;
          if constexpr (FIX) {
            y0 = shrink_y(s0, thr_prev, w0, k);
            y0 -= (s0 - y0) * uscale;
            if (has1) {
              y1 = shrink_y(s1, thr_prev, w1, k);
              y1 -= (s1 - y1) * uscale;
            }
          } else {
            const float2 zz = z[k];
            y0 = iter_elem<true, false>(zz.x * xn, s0, 0.f, w0, k, thr, thr_prev, ic, f, o0 + k,
                                        nullptr);
            if (has1)
              y1 = iter_elem<true, false>(-zz.y * xn, s1, 0.f, w1, k, thr, thr_prev, ic, f,
                                          o0 + W + k, nullptr);
          }
          z[k] = make_float2(y0, y1);
        }
      }
#pragma unroll
      for (int i = 0; i < 5; ++i) acc[i] += (double)f[i];
    }
    group_sync<BG>();
    // the state rows are consumed: the next pair's rows land during this
    // pair's forward transform
    if constexpr (FIX) issue_V(p + pstride);
    else issue_F(p + pstride);
    rt_fft<BG>(z, P.pw, P.twW, t, g);
    if (valid) {
      float2* fa = Fi + (size_t)r0 * Wp;
      for (int k = t; k < Wf; k += g) {
        const float2 Zk = z[k], Zm = z[k == 0 ? 0 : W - k];
        spec_put(fa, k, make_float2(0.5f * (Zk.x + Zm.x), 0.5f * (Zk.y - Zm.y)), paired);
        if (has1)
          spec_put(fa + Wp, k, make_float2(0.5f * (Zk.y + Zm.y), -0.5f * (Zk.x - Zm.x)), paired);
      }
    }
    // (FIX writes z before the next transform's first barrier)
    if constexpr (FIX) group_sync<BG>();
  }
  cp_async_wait<0>();
  if constexpr (FIX) return;
  block_sum<5>(acc, red_scratch);
  if (threadIdx.x == 0) {
    double* out = P.partials + ((size_t)b * P.nblk + blockIdx.x) * 5;
#pragma unroll
    for (int i = 0; i < 5; ++i) out[i] = acc[i];
  }
}
