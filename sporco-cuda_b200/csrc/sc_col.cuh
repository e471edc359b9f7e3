// The column pass of the problems whose filters have at most 16 rows: the
// column direction by direct convolution with the filter rows (plain and
// masked problems, and the gradient term with one non-negative weight).
//
// In the row-spectral domain (F = row spectra P_m of (Y - U)_m) filter m is
// E_m(t, kc), t < Kr (the row spectra of its rows), and its column spectrum is
// Df_m(kr) = sum_t E_m(t) w^(t kr).  Hence
//   sum_m Df_m Z^_m = FFTcol(a),   a(r) = sum_m sum_t E_m(t) P_m(r - t)
//   IFFTcol(conj(Df_m) SC)(r) = sum_t conj(E_m(t)) sc(r + t),  sc = IFFTcol(SC)
// (circular in r, unnormalised transforms): pass 1 accumulates a over the
// maps, one column transform pair per tile gives SC = S^ - cb and sc, and
// pass 2 writes every map's result.  The maps of a tile of four columns are
// shared by a cluster of CTAs.
//
// CONV_DELTA  plain problems, d = rho: pass 2 writes only the correction
//             sum_t conj(E_m(t)) sc(r + t) / (rho H W) (the row pass adds
//             Y - U) and reads no tile;
// CONV_FULL   the whole row spectra H P_m + sum_t conj(E_m(t)) sc(r + t) / rho
//             (masked problems);
// CONV_GRAD   d(kr, kc) = rho + mu w |G|^2 for every map (ColParams::two: for
//             all but map 0, whose d is rho):
//               IFFTcol(x^_m)(r) = IFFTcol(rho Z^_m / d)(r) + sum_t conj(E_m(t)) sc'(r + t),
//               sc' = IFFTcol(SC / d).
//             Along a column d = A - 2 B cos(theta) with B = mu w and
//             A = rho + B (2 + |G_col|^2), so 1 / d is the two-sided
//             exponential (q / B) / (1 - q^2) q^|n|, q = 2 B / (A + sqrt(A^2 -
//             4 B^2)) < 1: a first-order recursion up and one down the column,
//             circular, instead of two transforms per map.
//
// Measured per launch (before -> now): CONV_DELTA 2048 x 2048, 256 maps, 16
// taps 3.41 -> 2.99 ms (at 1965 MHz; 3.2 ms under the power cap of a long solve);
// 256 x 256, 64 maps, 8 taps 26.0 -> 17.7 us; 64 x 64, 32 maps 13.5 -> 7.5 us.
// CONV_FULL 512 x 512, 101 maps, 12 taps 115 -> 99 us.  CONV_GRAD 512 x 512, 100
// maps 209 (two transforms per map) -> 110 us; with the impulse map 384 x 512, 65
// maps, 8 taps 165 (COL_SOLVE_W) -> 68 us.  Without a compiled column length 3 x
// 320 x 480, 36 maps, 8 taps 266 (COL_SOLVE_P) -> 91 us.  Bound by the window
// loads' and the FMAs' latencies at 8 to 12 warps per SM (registers; FMA pipe 40
// to 60 % busy), DRAM a third busy.
//
// Each thread owns L consecutive rows of two adjacent columns and does both in
// packed FP32 instructions, in Gauss's three-multiply form (e = c + i d,
// P = a + i b: Re = c (a + b) - b (c + d), Im = c (a + b) + a (d - c), the
// three sums kept apart): three packed FMAs per two complex multiply-adds and
// one 16-byte shared-memory load per window row, where one column per thread
// took six FMAs and two loads.  (Plainly, with four packed FMAs, for columns of
// up to 128 rows, which are bound by latency: 64 x 64, 32 maps 7.5 us instead of
// 8.0; and at lengths without a compiled transform, where both are as fast.)
// Filters
// are padded with zero rows to KR = 8, 12 or 16 taps.
//
// F is in the paired layout (spec_re): a column pair's four values are its two
// real parts and its two imaginary parts, so that a 16-byte load gives the two
// register pairs that the packed FMAs take.  (From the interleaved layout the
// moves that form the pairs made pass 1 a third slower: 512 x 512, 12 taps
// 3.0 -> 1.9 thousand cycles per map, 2048 rows, 16 taps 8.3 -> 5.5.)  In every
// other group of eight pairs the imaginary parts come first; the kernel works
// on "first" and "second" parts throughout and takes the filter entries in the
// order that suits.
#pragma once

#include <type_traits>

#include "sc_kernels.cuh"

// Double precision: forward R-point DFTs in registers and the passes of a
// runtime plan (as stockham_pass and generic_pass of sc_fft.cuh).
__device__ __forceinline__ double2 d_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 d_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 d_mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a + s (-i) b
__device__ __forceinline__ double2 d_mi(double2 a, double s, double2 b) {
  return make_double2(a.x + s * b.y, a.y - s * b.x);
}
template <int R>
__device__ __forceinline__ void dft_d(double2* v) {
  if constexpr (R == 2) {
    const double2 a = v[0];
    v[0] = d_add(a, v[1]);
    v[1] = d_sub(a, v[1]);
  } else if constexpr (R == 3) {
    const double2 s = d_add(v[1], v[2]), e = d_sub(v[1], v[2]);
    const double2 m = make_double2(v[0].x - 0.5 * s.x, v[0].y - 0.5 * s.y);
    v[0] = d_add(v[0], s);
    v[1] = d_mi(m, 0.86602540378443864676, e);  // sin(2 pi / 3)
    v[2] = d_mi(m, -0.86602540378443864676, e);
  } else if constexpr (R == 4) {
    const double2 t0 = d_add(v[0], v[2]), t1 = d_sub(v[0], v[2]);
    const double2 t2 = d_add(v[1], v[3]), t3 = d_sub(v[1], v[3]);
    v[0] = d_add(t0, t2);
    v[2] = d_sub(t0, t2);
    v[1] = d_mi(t1, 1.0, t3);
    v[3] = d_mi(t1, -1.0, t3);
  } else if constexpr (R == 5) {
    // cos, sin of 2 pi / 5 and 4 pi / 5
    const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
    const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
    const double2 t1 = d_add(v[1], v[4]), e1 = d_sub(v[1], v[4]);
    const double2 t2 = d_add(v[2], v[3]), e2 = d_sub(v[2], v[3]);
    const double2 a = v[0];
    const double2 m1 = make_double2(a.x + c1 * t1.x + c2 * t2.x, a.y + c1 * t1.y + c2 * t2.y);
    const double2 m2 = make_double2(a.x + c2 * t1.x + c1 * t2.x, a.y + c2 * t1.y + c1 * t2.y);
    const double2 f1 = make_double2(s1 * e1.x + s2 * e2.x, s1 * e1.y + s2 * e2.y);
    const double2 f2 = make_double2(s2 * e1.x - s1 * e2.x, s2 * e1.y - s1 * e2.y);
    v[0] = d_add(a, d_add(t1, t2));
    v[1] = d_mi(m1, 1.0, f1);
    v[4] = d_mi(m1, -1.0, f1);
    v[2] = d_mi(m2, 1.0, f2);
    v[3] = d_mi(m2, -1.0, f2);
  } else {
    static_assert(R == 8);
    const double r = 0.70710678118654752440;  // cos(pi / 4)
    double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft_d<4>(e);
    dft_d<4>(o);
    const double2 o1 = make_double2(r * (o[1].x + o[1].y), r * (o[1].y - o[1].x));
    const double2 o3 = make_double2(r * (o[3].y - o[3].x), -r * (o[3].x + o[3].y));
    v[0] = d_add(e[0], o[0]);
    v[4] = d_sub(e[0], o[0]);
    v[1] = d_add(e[1], o1);
    v[5] = d_sub(e[1], o1);
    v[2] = d_mi(e[2], 1.0, o[2]);
    v[6] = d_mi(e[2], -1.0, o[2]);
    v[3] = d_add(e[3], o3);
    v[7] = d_sub(e[3], o3);
  }
}
template <int R>
__device__ __forceinline__ void pass_d(double2* data, int n, int Ns, int st,
                                       const double2* __restrict__ tw, int t, int g) {
  constexpr int MAXB = (16 + R - 1) / R;
  const int B = n / R, step = n / (Ns * R);
  double2 v[MAXB][R];
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int j = t + i * g;
    if (j < B) {
      const int k = j % Ns;
#pragma unroll
      for (int q = 0; q < R; ++q) v[i][q] = data[(j + q * B) * st];
      if (Ns > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[i][q] = d_mul(v[i][q], tw[q * k * step]);
      }
      dft_d<R>(v[i]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int j = t + i * g;
    if (j < B) {
      const int k = j % Ns, base = (j - k) * R + k;
#pragma unroll
      for (int q = 0; q < R; ++q) data[(base + q * Ns) * st] = v[i][q];
    }
  }
  __syncthreads();
}
// Any radix: every output formed directly.
static __device__ __noinline__ void generic_pass_d(double2* data, int n, int R, int Ns, int st,
                                                   const double2* __restrict__ tw, int t, int g) {
  const int B = n / R, step = n / (Ns * R);
  double2 out[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int o = t + i * g;
    if (o < n) {
      const int q = o / B, j = o - q * B;
      const int e1 = (j % Ns) * step + q * B;  // < n
      double2 acc = make_double2(0.0, 0.0);
      int e = 0;
      for (int s = 0; s < R; ++s) {
        const double2 x = data[(j + s * B) * st];
        const double2 w = tw[e];
        acc.x += x.x * w.x - x.y * w.y;
        acc.y += x.x * w.y + x.y * w.x;
        e += e1;
        if (e >= n) e -= n;
      }
      out[i] = acc;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int o = t + i * g;
    if (o < n) {
      const int q = o / B, j = o - q * B, k = j % Ns;
      data[((j - k) * R + k + q * Ns) * st] = out[i];
    }
  }
  __syncthreads();
}
static __device__ __noinline__ void pass_d_any(double2* data, int n, int R, int Ns, int st,
                                               const double2* __restrict__ tw, int t, int g) {
  switch (R) {
    case 2: pass_d<2>(data, n, Ns, st, tw, t, g); break;
    case 3: pass_d<3>(data, n, Ns, st, tw, t, g); break;
    case 4: pass_d<4>(data, n, Ns, st, tw, t, g); break;
    case 5: pass_d<5>(data, n, Ns, st, tw, t, g); break;
    case 8: pass_d<8>(data, n, Ns, st, tw, t, g); break;
    default: generic_pass_d(data, n, R, Ns, st, tw, t, g); break;
  }
}
// In-place forward DFT of data[0], data[st], ... (n <= 16 g elements).
__device__ __forceinline__ void fft_double(double2* data, const FftPlan& P, int st,
                                           const double2* __restrict__ tw, int t, int g) {
  int Ns = 1;
  for (int p = 0; p < P.npass; ++p) {
    pass_d_any(data, P.n, P.radix[p], Ns, st, tw, t, g);
    Ns *= P.radix[p];
  }
}

// 2 - 2 cos(theta) of a twiddle (cos, -sin), to a few roundings also where the
// cosine is close to 1.  (The recursions along the column and the 1 / d of SC
// have to be those of one d: with d from 2 - 2 cos in 32 bits the error of a
// column of 2048 rows was 3e-6 at mu w = 1e5 rho.)
__device__ __forceinline__ float two_minus_2cos(float2 w) {
  return w.x > 0.f ? __fdividef(2.f * w.y * w.y, 1.f + w.x) : 2.f - 2.f * w.x;
}

template <int KIND, int KR, int NH, int L>
__global__ void __launch_bounds__(conv_threads(NH, L), conv_min_blocks(KIND, NH, L, KR))
colc_kernel(ColParams P) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int T = 4;
  constexpr bool GRD = KIND == CONV_GRAD, DL = KIND == CONV_DELTA;
  constexpr int RMF = conv_radix(NH);
  const Geom& G = P.g;
  const int H = NH > 0 ? NH : G.H;
  const int Wf = G.Wf, Wp = G.Wp, M = G.M;
  const int NT = NH > 0 ? conv_threads(NH, L) : (int)blockDim.x;
  const int TL = (int)conv_tile_entries(H, L, KR);  // float2 entries of one tile
  constexpr int ES = KR * 8;  // float2 entries of one map's staged filter rows
  float2* A = reinterpret_cast<float2*>(smem_raw);  // pass 1 tile; cluster sum, spectrum, sc
  float2* Bt = A + TL;                              // tiles
  float2* Ct = Bt + TL;                             // tiles; partial sums
  float2* Es = Ct + TL;                             // [3][KR][2 column pairs][8 floats]
  float4* Cr = reinterpret_cast<float4*>(Es + 3 * ES);      // GRD: [2][2][NT] carries
  // GRD: the weights of blocks' ends ([NT]; [2][NT] with a short last block)
  constexpr int NW = NH > 0 ? 1 : 2;
  float2* Wt = reinterpret_cast<float2*>(Cr + (GRD ? 4 * NT : 0));
  float2* W4 = Wt + (GRD ? NW * NT : 0);  // GRD, two: map 0's tile

  const int b = blockIdx.z;
  const int rank = blockIdx.x;
  const int c0 = (P.tile0 + blockIdx.y) * T;
  const int tid = threadIdx.x;
  const int cp = tid & 1;   // column pair
  const int t = tid >> 1;   // row block
  const ImgState& st = P.st[b];
  if (st.done) return;  // uniform over the cluster (same image)
  const float rho = (float)st.rho;

  const int chunk = (M + P.G - 1) / P.G;
  const int m0 = rank * chunk;
  const int m1 = min(M, m0 + chunk);
  const size_t plane = (size_t)H * Wp;
  float2* Fi = P.F + (size_t)b * M * plane + c0;
  // rows of this thread: L, but for the last block of a column whose length is
  // not a multiple of L and the threads past the column
  const int r0 = NH > 0 ? t * L : min(t * L, H - 1);
  const int nr = NH > 0 ? L : max(0, min(L, H - t * L));
  const bool two = GRD && P.two != 0;
  const bool sw = (c0 >> 4) & 1;  // the imaginary parts come first in this tile

  // slot of tile row r: one pad row after every L, so that the 16-byte window
  // loads of consecutive threads fall into different banks
  auto slot = [&](int r) -> int { return L & 1 ? r : r + r / L; };
  // float4 index of row r0 + d of this thread's column pair; d is a
  // compile-time offset in (-KR, L + KR)
  constexpr int DB = (KR + L - 2) / L;  // blocks reached on either side
  int bbase[2 * DB + 1];
  if constexpr (NH > 0) {
#pragma unroll
    for (int dl = -DB; dl <= DB; ++dl) {
      int bi = t + dl;
      static_assert(DB <= NH / L, "one wrap reaches every block");
      bi = bi < 0 ? bi + NH / L : bi >= NH / L ? bi - NH / L : bi;
      bbase[dl + DB] = bi * (L + 1) * 2 + cp;
    }
  }
  auto at = [&](int d) -> int {
    if constexpr (NH > 0) {
      const int dl = d >= 0 ? d / L : -((-d + L - 1) / L);
      return bbase[dl + DB] + (d - dl * L) * 2;
    } else {
      int r = r0 + d;
      if (r < 0) r += H;
      if (r >= H) r -= H;
      return slot(r) * 2 + cp;
    }
  };
  auto issue_tile = [&](const float2* base, float2* dst) {
    for (int q = tid; q < 2 * H; q += NT) {
      const int r = q >> 1, h = q & 1;
      cp_async16(dst + slot(r) * T + 2 * h, base + (size_t)r * Wp + 2 * h);
    }
  };
  // filter rows of n maps from map m: per (row, column pair) 32 bytes
  auto issue_E = [&](int m, int n, float2* dst) {
    const float2* src = reinterpret_cast<const float2*>(P.E) + (size_t)m * KR * Wp * 2 + c0 * 2;
    for (int q = tid; q < n * KR * 4; q += NT) {
      const int r = q >> 2, h = q & 3;
      cp_async16(dst + q * 2, src + (size_t)r * Wp * 2 + h * 2);
    }
  };
  constexpr bool GA = conv_gauss(NH);
  f32x2 k1[L], k2[L], k3[L];
#pragma unroll
  for (int i = 0; i < L; ++i) k1[i] = k2[i] = k3[i] = dup2(0.f);
  // Entries of taps [T0, T0 + KB) of this thread's column pair, for e = c + i d
  // (conj: c - i d) times first and second parts (Re, Im), the other way round
  // in a tile with the imaginary parts first:
  //   Gauss:  c, and the factors of the second and the first parts,
  //           -(c + d) and d - c (conj: d - c and -(c + d)), so that
  //           first += c (f + s) + e2 s, second += c (f + s) + e1 f
  //   else:   c and e2 = -d (conj: d): first += c f + e2 s, second += c s - e2 f
  auto taps = [&](auto t0c, auto kbc, bool conj, const float2* e, f32x2* ec, f32x2* e2,
                  f32x2* e1) {
    constexpr int T0 = decltype(t0c)::value, KB = decltype(kbc)::value;
    const float sx = (conj != sw) ? 1.f : -1.f;
#pragma unroll
    for (int q = 0; q < KB; ++q) {
      const float2* u = e + ((T0 + q) * 2 + cp) * 4;
      ec[q] = pk2(u[0]);
      if constexpr (GA) {
        const int ox = (conj != sw) ? 2 : 1;  // entry of the second parts' factor
        e2[q] = mul2(pk2(u[ox]), dup2(sx));
        e1[q] = mul2(pk2(u[3 - ox]), dup2(-sx));
      } else {
        e2[q] = mul2(pk2(u[3]), dup2(sx));
      }
    }
  };
  // one window row (first parts a, second parts bb) into output i at tap tp
  auto mac = [&](int i, int tp, const f32x2* ec, const f32x2* e2, const f32x2* e1, f32x2 a,
                 f32x2 bb, f32x2 s) {
    if constexpr (GA) {
      k1[i] = fma2(ec[tp], s, k1[i]);
      k3[i] = fma2(e2[tp], bb, k3[i]);
      k2[i] = fma2(e1[tp], a, k2[i]);
    } else {
      k3[i] = fma2(ec[tp], a, k3[i]);
      k2[i] = fma2(ec[tp], bb, k2[i]);
      k3[i] = fma2(e2[tp], bb, k3[i]);
      k2[i] = fma2(e2[tp], s, k2[i]);  // s = -a
    }
  };
  auto wsum = [&](f32x2 a, f32x2 bb) -> f32x2 {
    if constexpr (GA) return add2(a, bb);
    const float2 v = up2(a);
    return pk2(-v.x, -v.y);
  };
  // (first, second) parts of row i
  auto result = [&](int i, float2& u, float2& v) {
    u = up2(GA ? add2(k1[i], k3[i]) : k3[i]);
    v = up2(GA ? add2(k1[i], k2[i]) : k2[i]);
  };
  // taps per sweep over the window: the entries of a sweep stay in registers
  constexpr int KB = conv_sweep(KR, L);
  constexpr int NS = KR / KB;

  // -------------------------------------------------------------- pass 1
  // The three tile buffers rotate: map m's tile is copied two maps ahead.
  // One barrier per map: after it, map m's tile is visible and every thread
  // is done with map m - 1's buffer, which then takes map m + 2.
  // At a length without a compiled transform every map's sum is formed by
  // itself and then added to the tile's, as the transform solve adds a map's
  // product, instead of in one long chain over maps and taps (3 x 320 x 480, 36
  // maps, 30 iterations: error of X 2.2e-6 -> 2.1e-6).
  constexpr bool BYMAP = NH == 0;
  f32x2 t2[BYMAP ? L : 1], t3[BYMAP ? L : 1];
#pragma unroll
  for (int i = 0; i < (BYMAP ? L : 1); ++i) t2[i] = t3[i] = dup2(0.f);
  auto add_map = [&]() {
    if constexpr (BYMAP) {
#pragma unroll
      for (int i = 0; i < L; ++i) {
        t2[i] = add2(t2[i], k2[i]);
        t3[i] = add2(t3[i], k3[i]);
        k2[i] = k3[i] = dup2(0.f);
      }
    }
  };
  auto store_sums = [&](float2* dst) {
    float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
    for (int i = 0; i < L; ++i) {
      if (NH > 0 || i < nr) {
        float2 re, im;
        result(i, re, im);
        if (sw) {
          const float2 x = re;
          re = im;
          im = x;
        }
        d4[at(i)] = make_float4(re.x, im.x, re.y, im.y);
      }
    }
  };
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (m0 + q < m1) {
      issue_tile(Fi + (size_t)(m0 + q) * plane, q ? Bt : A);
      issue_E(m0 + q, 1, Es + q * ES);
    }
    cp_async_commit();
  }
  {
    float2 *b0 = A, *b1 = Bt, *b2 = Ct;  // map m's tile, m + 1's, the free one
    int bi = 0;
    for (int m = m0; m < m1; ++m) {
      cp_async_wait<1>();  // map m (m + 1 may still be in flight)
      __syncthreads();
      const int bn = bi == 0 ? 2 : bi - 1;
      const bool more = m + 2 < m1;
      if (more) {
        if (NH == 0) issue_tile(Fi + (size_t)(m + 2) * plane, b2);
        issue_E(m + 2, 1, Es + bn * ES);
      }
      // map m + 2's tile: a 16-byte copy every few window rows (all at once
      // they would hold up the window loads behind them; 512 x 512: 3.0 -> 2.5
      // thousand cycles per map)
      const float2* cs = Fi + (size_t)(m + 2) * plane + (size_t)(tid >> 1) * Wp + 2 * (tid & 1);
      auto copy_chunk = [&](int c) {
        const int r = (tid >> 1) + c * (NT / 2);
        if (more) cp_async16(b2 + slot(r) * T + 2 * (tid & 1), cs + (size_t)c * (NT / 2) * Wp);
      };
      constexpr int R = NS * (L + KB - 1);  // window rows per map
      const float4* cur = reinterpret_cast<const float4*>(b0);
      const float2* ecur = Es + bi * ES;
      // window row j = P(r0 - (T0 + KB - 1) + j) meets output i at tap
      // T0 + KB - 1 + i - j, the last taps first
      auto sweep = [&](auto t0c) {
        constexpr int T0 = decltype(t0c)::value;
        f32x2 ec[KB], ep[KB], em[KB];
        taps(t0c, IntC<KB>{}, false, ecur, ec, ep, em);
#pragma unroll
        for (int j = 0; j < L + KB - 1; ++j) {
          if constexpr (NH > 0) {
            const int rr = (NS - 1 - T0 / KB) * (L + KB - 1) + j;
#pragma unroll
            for (int c = 0; c < L; ++c)
              if (c * R / L == rr) copy_chunk(c);
          }
          const float4 w = cur[at(j - (T0 + KB - 1))];
          const f32x2 a = pk2(w.x, w.y), bb = pk2(w.z, w.w);
          const f32x2 s = wsum(a, bb);
#pragma unroll
          for (int i = 0; i < L; ++i) {
            const int tp = KB - 1 + i - j;
            if (tp >= 0 && tp < KB) mac(i, tp, ec, ep, em, a, bb, s);
          }
        }
      };
      if constexpr (NS >= 4) sweep(IntC<3 * KB>{});
      if constexpr (NS >= 3) sweep(IntC<2 * KB>{});
      if constexpr (NS >= 2) sweep(IntC<KB>{});
      sweep(IntC<0>{});
      if (two && m == 0) {  // map 0 has a d of its own: its sum apart
        store_sums(W4);
#pragma unroll
        for (int i = 0; i < L; ++i) k1[i] = k2[i] = k3[i] = dup2(0.f);
      }
      add_map();
      cp_async_commit();
      float2* f = b0;
      b0 = b1;
      b1 = b2;
      b2 = f;
      bi = bi == 2 ? 0 : bi + 1;
    }
  }
  if constexpr (BYMAP) {
#pragma unroll
    for (int i = 0; i < L; ++i) {
      k2[i] = t2[i];
      k3[i] = t3[i];
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();

  // --------------------------------------------------- sum over the cluster
  // Ct holds this CTA's sums; A receives the whole sums.  The tile of S^ lands
  // in Ct afterwards and that of Psum in Bt, during the first transform.
  // At a length without a compiled transform (DBL) the whole sums, the tile's
  // transforms and SC are in double precision, in Z over A and Bt: in the
  // transform solve that stood there the errors of the maps' transforms average
  // out, here there is one transform per tile (error of X after 30 iterations
  // with single / double precision / the transform solve: 3 x 320 x 480, 36 maps
  // 2.1e-6 / 1.42e-6 / 1.44e-6; 317 x 203, 20 maps 3.2e-6 / 1.51e-6 / 1.81e-6).
  constexpr bool DBL = NH == 0;
  double2* Z = reinterpret_cast<double2*>(A);
  const int E = 2 * H;  // float4 entries
  auto s4 = [&](int e) -> int { return slot(e >> 1) * 2 + (e & 1); };
  for (int r = tid; !DBL && r < H; r += NT)
    cp_async16(reinterpret_cast<float4*>(Bt) + r, P.Psum + (size_t)r * Wp + c0);
  if (P.G > 1) {
    store_sums(Ct);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    // every CTA sums a slice of the tile over the cluster (in rank order, the
    // remote loads of eight ranks in flight at once) and stores it to all of
    // them: 2 tiles of remote traffic per CTA instead of G (every CTA summing
    // the whole tile took 14 thousand of 43 thousand cycles at 256 rows, G = 8)
    const int sl0 = (E + P.G - 1) / P.G;
    const int ee = min(E, (rank + 1) * sl0);
    for (int e = rank * sl0 + tid; e < ee; e += NT) {
      const int sl = s4(e);
      using V = std::conditional_t<DBL, double4, float4>;
      V v{0, 0, 0, 0};
      for (int rb = 0; rb < P.G; rb += 8) {
        float4 w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          w[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (rb + u < P.G)
            w[u] = reinterpret_cast<const float4*>(cluster.map_shared_rank(Ct, rb + u))[sl];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          v.x += w[u].x;
          v.y += w[u].y;
          v.z += w[u].z;
          v.w += w[u].w;
        }
      }
      for (int r = 0; r < P.G; ++r) {
        if constexpr (DBL) {
          double2* z = cluster.map_shared_rank(Z, r) + 2 * sl;
          z[0] = make_double2(v.x, v.y);
          z[1] = make_double2(v.z, v.w);
        } else {
          reinterpret_cast<float4*>(cluster.map_shared_rank(A, r))[sl] = v;
        }
      }
      if (two) {
        const float4 w = reinterpret_cast<const float4*>(cluster.map_shared_rank(W4, 0))[sl];
        for (int r = 1; r < P.G; ++r)
          reinterpret_cast<float4*>(cluster.map_shared_rank(W4, r))[sl] = w;
      }
    }
    cluster.sync();
  } else if constexpr (DBL) {
    store_sums(Ct);
    __syncthreads();
    for (int e = tid; e < 2 * E; e += NT) Z[e] = make_double2(Ct[e].x, Ct[e].y);
    __syncthreads();
  } else {
    store_sums(A);
    __syncthreads();
  }
  issue_tile(P.Sh + (size_t)b * plane + c0, Ct);
  cp_async_commit();

  // ------------------- SC = S^ - cb, sc = IFFTcol(SC) / rho (GRD: IFFTcol(SC / d))
  auto fft = [&](float2* tile) {
    if constexpr (NH > 0) {
      constexpr int gF = ct_threads(NH, RMF);
      constexpr int CR = conv_threads(NH, L) / gF;  // columns at once
      static_assert(CR * gF == conv_threads(NH, L) && (CR == 1 || CR == 2 || CR == 4),
                    "the CTA's threads cover whole columns");
#pragma unroll 1
      for (int h = 0; h < T; h += CR)
        fft_ct<NH, RMF, gF, T, 0, L, 2>(tile + h + tid % CR, P.twH, tid / CR);
    } else {
      if (tile == A) fft_double(Z + (tid & 3), P.ph, T, P.twHd, tid >> 2, NT >> 2);
      else fft_forward<16>(tile + (tid & 3), P.ph, T, P.twH, tid >> 2, NT >> 2);
    }
  };
  // gradient term: 1 / d at (kr, column c of the tile), B = mu w
  const float Bw = GRD ? P.mu * P.wgrd[two ? 1 : 0] : 0.f;
  const float irho = 1.f / rho;
  // conj(SC) / rho (DL: also times 1 / (H W), the row pass's normalisation of
  // its inverse transform)
  const float irho_s = DL ? (float)(1.0 / ((double)rho * H * G.W)) : irho;
  // |G|^2 of this thread's columns but for the column frequency (e & 1 is tid & 1
  // below)
  float dc[2] = {0.f, 0.f};
  if constexpr (GRD) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      dc[h] = two_minus_2cos(__ldg(&P.twW[min(c0 + 2 * cp + h, Wf - 1)]));
  }
  fft(A);
  if (two) fft(W4);
  cp_async_wait<0>();
  __syncthreads();
  for (int e = tid; e < E; e += NT) {
    const int kr = e >> 1, c = 2 * (e & 1);
    if constexpr (DBL) {  // the step below in double precision
      const float4 S = reinterpret_cast<const float4*>(Ct)[s4(e)];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double2 v = make_double2(0.0, 0.0);
        float2 v0 = make_float2(0.f, 0.f);
        const int kc = c0 + c + h;
        if (kc < Wf) {
          const double2 q = Z[2 * e + h];
          double2 q0 = make_double2(0.0, 0.0);
          double id = 1.0 / (double)rho, sd = 0.0;
          if (GRD)
            id = 1.0 / ((double)Bw * (2.0 - 2.0 * P.twHd[kr].x + dc[h]) + rho);
          if (two) {
            const float4 w = reinterpret_cast<const float4*>(W4)[s4(e)];
            q0 = h ? make_double2(w.z, w.w) : make_double2(w.x, w.y);
            sd = (double)P.Psum0[(size_t)kr * Wp + kc] / rho;
          }
          sd += (double)P.Psum[(size_t)kr * Wp + kc] * id;
          const double f = 1.0 / (1.0 + sd), ri = GRD ? rho * id : 1.0;
          const double x = ((double)(h ? S.z : S.x) - ri * q.x - q0.x) * f;
          const double y = ((double)(h ? S.w : S.y) - ri * q.y - q0.y) * f;
          const double sc = DL ? id / ((double)H * G.W) : id;
          v = make_double2(x * sc, -y * sc);
          v0 = make_float2((float)(x / rho), (float)(-y / rho));
        }
        Z[2 * e + h] = v;
        if (two) W4[2 * s4(e) + h] = v0;
      }
      continue;
    }
    float4* pa = reinterpret_cast<float4*>(A) + s4(e);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f), v0 = v;
    if (c0 + c < Wf) {
      const float4 q = *pa;  // sum_m Df_m Z^_m
      const float4 S = reinterpret_cast<const float4*>(Ct)[s4(e)];
      const float2 ps = reinterpret_cast<const float2*>(Bt)[e];
      // SC = S^ - cb with cb = (S^ Psum / d + rho q / d) / (1 + Psum / d),
      // computed as SC = (S^ - rho q / d) / (1 + Psum / d): the same value
      // without subtracting cb, which is close to S^ when Psum >> d (many
      // maps), from S^ (that cancellation multiplied the rounding error of
      // SC by about 1 + Psum / d)
      if constexpr (GRD) {
        const float ghr = two_minus_2cos(__ldg(&P.twH[kr]));
        float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 p0 = make_float2(0.f, 0.f);
        if (two) {
          q0 = reinterpret_cast<const float4*>(W4)[s4(e)];
          p0 = *reinterpret_cast<const float2*>(P.Psum0 + (size_t)kr * Wp + c0 + c);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float id = 1.f / (Bw * (dc[h] + ghr) + rho);
          const float sd = (h ? ps.y : ps.x) * id + (h ? p0.y : p0.x) * irho;
          const float rid = rho * id;
          const float g1 = 1.f / (1.f + sd);
          const float x = ((h ? S.z : S.x) - rid * (h ? q.z : q.x) - (h ? q0.z : q0.x)) * g1;
          const float y = ((h ? S.w : S.y) - rid * (h ? q.w : q.y) - (h ? q0.w : q0.y)) * g1;
          (h ? v.z : v.x) = x * id;  // conj(SC) / d
          (h ? v.w : v.y) = -y * id;
          (h ? v0.z : v0.x) = x * irho;
          (h ? v0.w : v0.y) = -y * irho;
        }
      } else {
        const float f0 = irho_s / (1.f + ps.x * irho), f1 = irho_s / (1.f + ps.y * irho);
        v = make_float4((S.x - q.x) * f0, -(S.y - q.y) * f0, (S.z - q.z) * f1,
                        -(S.w - q.w) * f1);
      }
      if (c0 + c + 1 >= Wf) v.z = v.w = v0.z = v0.w = 0.f;
    }
    *pa = v;
    if (two) reinterpret_cast<float4*>(W4)[s4(e)] = v0;
  }
  __syncthreads();
  // pass 2's first map lands during the second transform
  auto issue_first = [&]() {
    if (!DL && m0 < m1) {
      issue_tile(Fi + (size_t)m0 * plane, Bt);
      issue_E(m0, 1, Es);
    }
    if (DL && m0 < m1) issue_E(m0, min(TL / ES, m1 - m0), Bt);
    cp_async_commit();
  };
  if (!DBL) issue_first();
  fft(A);
  if (two && rank == 0) fft(W4);
  // the window of pass 2 in the paired layout
  for (int e = tid; e < E; e += NT) {
    float4* pa = reinterpret_cast<float4*>(DBL ? Ct : A) + s4(e);
    float4 v;
    if constexpr (DBL) {
      const double2 z0 = Z[2 * e], z1 = Z[2 * e + 1];
      v = make_float4((float)z0.x, (float)z0.y, (float)z1.x, (float)z1.y);
    } else {
      v = *pa;
    }
    *pa = sw ? make_float4(-v.y, -v.w, v.x, v.z) : make_float4(v.x, v.z, -v.y, -v.w);
    if (two && rank == 0) {
      float4* pw = reinterpret_cast<float4*>(W4) + s4(e);
      const float4 w = *pw;
      *pw = sw ? make_float4(-w.y, -w.w, w.x, w.z) : make_float4(w.x, w.z, -w.y, -w.w);
    }
  }

  if constexpr (DBL) {  // the window is in Ct, A and Bt take the tiles
    __syncthreads();
    float2* w = A;
    A = Ct;
    Ct = Bt;
    Bt = w;
    issue_first();
  }

  // -------------------------------------------------------------- pass 2
  const bool ok0 = c0 + 2 * cp < Wf;
  float2* Fo = Fi + 2 * cp + (size_t)r0 * Wp;
  // (first, second) parts of L rows = (k1 + k3, k1 + k2) +=
  // sum_t conj(E_m(t)) w(r0 + i + t)
  auto conv2 = [&](const float4* win, const float2* ecur) {
    auto sweep = [&](auto t0c) {
      constexpr int T0 = decltype(t0c)::value;
      f32x2 ec[KB], ep[KB], em[KB];
      taps(t0c, IntC<KB>{}, true, ecur, ec, ep, em);
#pragma unroll
      for (int j = 0; j < L + KB - 1; ++j) {
        const float4 w = win[at(j + T0)];
        const f32x2 a = pk2(w.x, w.y), bb = pk2(w.z, w.w);
        const f32x2 s = wsum(a, bb);
#pragma unroll
        for (int i = 0; i < L; ++i) {
          const int tp = j - i;
          if (tp >= 0 && tp < KB) mac(i, tp, ec, ep, em, a, bb, s);
        }
      }
    };
    sweep(IntC<0>{});
    if constexpr (NS >= 2) sweep(IntC<KB>{});
    if constexpr (NS >= 3) sweep(IntC<2 * KB>{});
    if constexpr (NS >= 4) sweep(IntC<3 * KB>{});
  };
  auto write_map = [&](int m) {
    float2* d = Fo + (size_t)m * plane;
#pragma unroll
    for (int i = 0; i < L; ++i) {
      if (NH > 0 || i < nr) {
        float2 u, v;
        result(i, u, v);
        // (the row pass ignores the columns past the spectrum)
        if (ok0) *reinterpret_cast<float4*>(d + (size_t)i * Wp) = make_float4(u.x, u.y, v.x, v.y);
      }
    }
  };
  const float4* win = reinterpret_cast<const float4*>(A);
  if constexpr (DL) {
    // only filter rows are staged: as many maps at a time as fit in a tile
    const int per = TL / ES;
    int buf = 0;
    for (int mb = m0; mb < m1; mb += per, buf ^= 1) {
      cp_async_wait<0>();
      __syncthreads();  // also: the window is complete, the other buffer read
      const float2* eb = buf ? Ct : Bt;
      if (mb + per < m1) issue_E(mb + per, min(per, m1 - mb - per), buf ? Bt : Ct);
      cp_async_commit();
      const int n = min(per, m1 - mb);
      for (int mi = 0; mi < n; ++mi) {
#pragma unroll
        for (int i = 0; i < L; ++i) k1[i] = k2[i] = k3[i] = dup2(0.f);
        conv2(win, eb + mi * ES);
        write_map(mb + mi);
      }
    }
    return;
  }
  const float hs = (float)H;
  // the recursions of the gradient term, per column of the pair
  // (q as it is used, rounded to 32 bits, sets the gain, the blocks' weights and
  // the sum all the way around, each in 64 bits, so that a constant column comes
  // out as it should however close q is to 1.  In a 32-bit emulation the error of
  // a column with a mean is 1e-7 to 3e-7 at B up to 1e10 rho and 64 to 2048 rows;
  // with the gain of the unrounded q and 32-bit powers it was 3e-6 at 1e4 rho and
  // 2e-4 at 1e8 rho, with the weights alone in 32 bits up to 7e-6)
  f32x2 q2 = dup2(0.f), gain = q2, around = q2;
  int hops = 0;  // carries further away are below 2^-32 of their value
  if constexpr (GRD) {
    const int nb = (H + L - 1) / L;
    float qv[2], gv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double Bd = Bw;
      const double lo = (double)rho + Bd * dc[h];  // A - 2 B
      const double Ad = lo + 2.0 * Bd;
      qv[h] = fminf((float)(2.0 * Bd / (Ad + sqrt(lo * (lo + 4.0 * Bd)))), 0x1.fffffep-1f);
      const double q = qv[h];
      // H rho / (A - 2 B) (1 - q) / (1 + q): at d = A - 2 B the gain of both
      // recursions, 1 / (1 - q) + q / (1 - q), is 1 / d
      gv[h] = (float)((double)hs * rho * (1.0 - q) / (lo * (1.0 + q)));
    }
    q2 = pk2(qv[0], qv[1]);
    gain = pk2(gv[0], gv[1]);
    const float qm = fmaxf(qv[0], qv[1]);
    hops = qm > 0.f ? (int)fminf((float)nb, 1.f + ceilf(-32.f / (L * log2f(qm)))) : 0;
    auto powq = [&](int h, int n) {
      double r = 1.0, p = qv[h];
      for (; n > 0; n >>= 1, p *= p)
        if (n & 1) r *= p;
      return r;
    };
    // the weight of a block's end t blocks on, without the last, possibly short
    // block among them and with it
    if (t < hops) {
      Wt[tid] = make_float2((float)powq(0, L * t), (float)powq(1, L * t));
      if constexpr (NW > 1) {
        const int n = L * t - (nb * L - H);
        Wt[NT + tid] = make_float2((float)powq(0, n), (float)powq(1, n));
      }
    }
    if (hops >= nb) {  // 1 / (1 - q^H)
      around = pk2((float)(1.0 / (1.0 - powq(0, H))), (float)(1.0 / (1.0 - powq(1, H))));
    }
  }
  int it = 0;
  for (int m = m0; m < m1; ++m, ++it) {
    const float4* cur = reinterpret_cast<const float4*>((it & 1) ? Ct : Bt);
    const float2* ecur = Es + (it & 1) * ES;
    cp_async_wait<0>();  // the only copies in flight
    __syncthreads();
    if (m + 1 < m1) {
      issue_tile(Fi + (size_t)(m + 1) * plane, (it & 1) ? Bt : Ct);
      issue_E(m + 1, 1, Es + ((it + 1) & 1) * ES);
    }
    cp_async_commit();
    const bool plainm = !GRD || (two && m == 0);
    if (plainm) {
#pragma unroll
      for (int i = 0; i < L; ++i) {
        const float4 w = (NH > 0 || i < nr) ? cur[at(i)] : make_float4(0.f, 0.f, 0.f, 0.f);
        k1[i] = dup2(0.f);
        k3[i] = pk2(hs * w.x, hs * w.y);
        k2[i] = pk2(hs * w.z, hs * w.w);
      }
    }
    if constexpr (GRD) {
      // y = gain (f + g - x): f(r) = x(r) + q f(r - 1), g(r) = x(r) + q g(r + 1)
      // around the column.  Each thread runs its own rows from zero and
      // publishes where it ends; the recursions' values at its edges are sums
      // over the ends of the blocks before and after it.
      f32x2 fr[L], fi[L], gr[L], gi[L], pr = dup2(0.f), pi = pr;
      float4* cr = Cr + (it & 1) * 2 * NT;
      if (!plainm) {
#pragma unroll
        for (int i = 0; i < L; ++i) {
          const float4 w = (NH > 0 || i < nr) ? cur[at(i)] : make_float4(0.f, 0.f, 0.f, 0.f);
          gr[i] = pk2(w.x, w.y);
          gi[i] = pk2(w.z, w.w);
          // f - x = q f(r - 1) is kept
          fr[i] = i ? mul2(q2, pr) : dup2(0.f);
          fi[i] = i ? mul2(q2, pi) : dup2(0.f);
          pr = add2(gr[i], fr[i]);
          pi = add2(gi[i], fi[i]);
          if (i == L - 1 || (NH == 0 && i < nr)) {
            const float2 u = up2(pr), v = up2(pi);
            if (NH > 0 || i < nr) cr[tid] = make_float4(u.x, u.y, v.x, v.y);
          }
        }
        f32x2 br = gr[L - 1], bi = gi[L - 1];
        // g in place of x
#pragma unroll
        for (int i = L - 2; i >= 0; --i) {
          br = fma2(q2, br, gr[i]);
          bi = fma2(q2, bi, gi[i]);
          gr[i] = br;
          gi[i] = bi;
        }
        const float2 u = up2(br), v = up2(bi);
        cr[NT + tid] = make_float4(u.x, u.y, v.x, v.y);
      }
      __syncthreads();
      if (!plainm) {
        const int nb = (H + L - 1) / L;
        f32x2 sr = dup2(0.f), si = sr, ur = sr, ui = sr;
        int jf = t, jb = t;
        const int lf = t, lb = t < nb - 1 ? nb - 2 - t : nb;  // hops that reach the last block
        for (int k = 0; k < hops; ++k) {
          jf = jf == 0 ? nb - 1 : jf - 1;
          jb = jb >= nb - 1 ? 0 : jb + 1;
          const float4 f4 = cr[2 * jf + cp], g4 = cr[NT + 2 * jb + cp];
          // q^(rows in between)
          const f32x2 wf = pk2(Wt[(NW > 1 && k > lf ? NT : 0) + 2 * k + cp]);
          const f32x2 wb = NW > 1 ? pk2(Wt[(k > lb ? NT : 0) + 2 * k + cp]) : wf;
          sr = fma2(wf, pk2(f4.x, f4.y), sr);
          si = fma2(wf, pk2(f4.z, f4.w), si);
          ur = fma2(wb, pk2(g4.x, g4.y), ur);
          ui = fma2(wb, pk2(g4.z, g4.w), ui);
        }
        if (hops >= nb) {  // all the way around: 1 / (1 - q^H)
          sr = mul2(sr, around);
          si = mul2(si, around);
          ur = mul2(ur, around);
          ui = mul2(ui, around);
        }
#pragma unroll
        for (int i = 0; i < L; ++i) {
          sr = mul2(sr, q2);
          si = mul2(si, q2);
          fr[i] = add2(fr[i], sr);
          fi[i] = add2(fi[i], si);
        }
#pragma unroll
        for (int i = L - 1; i >= 0; --i) {
          if (NH > 0 || i < nr) {
            ur = mul2(ur, q2);
            ui = mul2(ui, q2);
          }
          k1[i] = dup2(0.f);
          k3[i] = mul2(gain, add2(fr[i], add2(gr[i], ur)));
          k2[i] = mul2(gain, add2(fi[i], add2(gi[i], ui)));
        }
      }
    }
    conv2(two && m == 0 ? reinterpret_cast<const float4*>(W4) : win, ecur);
    write_map(m);
  }
  cp_async_wait<0>();
}
