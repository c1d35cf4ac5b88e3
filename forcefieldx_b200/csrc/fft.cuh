// fft.cuh -- mesh convolution of axes with two factors among 1..10, 12, 15 and 16.
//
// A length N = F1 F2 line is transformed in two steps, each a DFT held in registers:
// step 1 takes the F1 elements j + r F2 (r < F1) of one j, step 2 the F2 results of one
// q < F1 with their twiddles exp(-+2 pi i q j / N), giving outputs q + F1 k.  A line so
// crosses shared memory once (the radix-4/2/3/5/7 Stockham passes it replaces crossed it
// three or four times, with run-time divisions in every index).  The forward transform of
// a z plane along x and y is one launch (k_fft_plane<S, false>), the transform along z,
// the influence function and the inverse along z one (k_fft_z), the inverse of the planes
// one (k_fft_plane<S, true>): three launches where the per-axis passes take five
// (Complex3DParallel.convolution, N/fft/Complex3DParallel.java:445, 775-1010).
//
// The meshes (0.06 to 14 MB) live in L2 and the launches are bound by latency: the round
// trip to L2, three block barriers and the launch itself.  A whole plane per CTA, so that
// the turn between the axes stays in its shared memory.  Spread over clusters of 2, 4 or 8
// CTAs per plane with the turn through distributed shared memory, the plane passes were no
// faster by themselves (64^3 FP32: 10.4 against 10.8 us) and cost the evaluation more where
// the pair field runs beside them (24,000 atoms FP64: 2,085-2,095 against 1,972 us), since
// a cluster starts only when all its CTAs find room at once.
//
// Measured per evaluation (host buffers, B200) against per-axis Stockham passes, the FP32
// 64 x 64 plane excepted, which had its own cluster pass: 648 atoms FP64 558 -> 436 us,
// 2,997 mixed 744 -> 559, 9,738 FP64 1,436 -> 1,221, 24,000 FP64 2,250 -> 2,138, 24,000
// mixed unchanged (device time 1,379 -> 1,344), 81,000 mixed 4,755 -> 4,215.
#pragma once

#include <utility>

#include "ffx_internal.cuh"

namespace ffx {

// Threads of a plane's CTA, and resident blocks its registers are held to: two of 512 threads
// in FP32, 64 registers, at which the narrow forward instance spills 156 bytes (the planes are
// read as FP64 values) and the wide instance would spill more, so that it has 384 threads and
// no bound.
template <typename S, bool WIDE> constexpr int fft_plane_threads() { return sizeof(S) == 8 ? 256 : WIDE ? 384 : 512; }
template <typename S, bool WIDE> constexpr int fft_plane_blocks() { return sizeof(S) == 8 || WIDE ? 0 : 2; }
constexpr int kFftZLines = 8;   // z lines per CTA: 64- or 128-byte runs of each z layer

// cos and sin of 2 pi k / n at compile time, by Taylor series on the first octant.
constexpr double kTwoPi = 6.283185307179586476925286766559;
__host__ __device__ constexpr double taylor_sin(double x) {
  double t = x, s = x;
  for (int j = 1; j < 14; j++) {
    t *= -x * x / ((2 * j) * (2 * j + 1));
    s += t;
  }
  return s;
}
__host__ __device__ constexpr double taylor_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int j = 1; j < 14; j++) {
    t *= -x * x / ((2 * j - 1) * (2 * j));
    s += t;
  }
  return s;
}
__host__ __device__ constexpr double cos_turn(int k, int n) {
  k %= n;
  if (2 * k > n) k = n - k;                                    // cos(-x) = cos x
  if (4 * k > n) return -cos_turn(n - 2 * k, 2 * n);           // cos(pi - x) = -cos x
  if (8 * k > n) return taylor_sin(kTwoPi * (n - 4 * k) / (4.0 * n));
  return taylor_cos(kTwoPi * k / n);
}
__host__ __device__ constexpr double sin_turn(int k, int n) {
  k %= n;
  if (2 * k > n) return -sin_turn(n - k, n);
  if (4 * k > n) return sin_turn(n - 2 * k, 2 * n);
  if (8 * k > n) return taylor_cos(kTwoPi * (n - 4 * k) / (4.0 * n));
  return taylor_sin(kTwoPi * k / n);
}

template <int... I, typename F>
__device__ __forceinline__ void unroll_seq(std::integer_sequence<int, I...>, F f) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void unroll(F f) {
  unroll_seq(std::make_integer_sequence<int, N>{}, f);
}

__host__ __device__ constexpr int dft_split(int r) {   // the first factor of a composite radix
  return r == 4 || r == 6 || r == 8 || r == 10 ? 2 : r == 9 || r == 12 || r == 15 ? 3 : r == 16 ? 4 : 1;
}

// DFT of R values in registers, natural order in and out, sign SG of the exponent.
template <int R, int SG, typename S>
__device__ __forceinline__ void dft(typename Vec2<S>::type *v) {
  using V = typename Vec2<S>::type;
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const V a = v[0], b = v[1];
    v[0] = mk2<S>(a.x + b.x, a.y + b.y);
    v[1] = mk2<S>(a.x - b.x, a.y - b.y);
  } else if constexpr (R == 4) {
    const V s02 = mk2<S>(v[0].x + v[2].x, v[0].y + v[2].y), d02 = mk2<S>(v[0].x - v[2].x, v[0].y - v[2].y);
    const V s13 = mk2<S>(v[1].x + v[3].x, v[1].y + v[3].y), d13 = mk2<S>(v[1].x - v[3].x, v[1].y - v[3].y);
    const V t = mk2<S>(SG > 0 ? -d13.y : d13.y, SG > 0 ? d13.x : -d13.x);   // SG i d13
    v[0] = mk2<S>(s02.x + s13.x, s02.y + s13.y);
    v[1] = mk2<S>(d02.x + t.x, d02.y + t.y);
    v[2] = mk2<S>(s02.x - s13.x, s02.y - s13.y);
    v[3] = mk2<S>(d02.x - t.x, d02.y - t.y);
  } else if constexpr (R == 3 || R == 5 || R == 7) {
    // Odd prime: sums and differences of the mirrored inputs share the real factors.
    constexpr int H = R / 2;
    V s[H], d[H];
#pragma unroll
    for (int j = 0; j < H; j++) {
      s[j] = mk2<S>(v[j + 1].x + v[R - 1 - j].x, v[j + 1].y + v[R - 1 - j].y);
      d[j] = mk2<S>(v[j + 1].x - v[R - 1 - j].x, v[j + 1].y - v[R - 1 - j].y);
    }
    const V v0 = v[0];
    V sum = v0;
#pragma unroll
    for (int j = 0; j < H; j++) sum = mk2<S>(sum.x + s[j].x, sum.y + s[j].y);
    v[0] = sum;
    unroll<H>([&](auto kk) {
      constexpr int k = decltype(kk)::value + 1;
      V e = v0, o = mk2<S>(S(0), S(0));
      unroll<H>([&](auto jj) {
        constexpr int j = decltype(jj)::value;
        constexpr S c = (S)cos_turn((j + 1) * k, R), z = (S)(SG * sin_turn((j + 1) * k, R));
        e = mk2<S>(e.x + c * s[j].x, e.y + c * s[j].y);
        o = mk2<S>(o.x + z * d[j].x, o.y + z * d[j].y);
      });
      v[k] = mk2<S>(e.x - o.y, e.y + o.x);
      v[R - k] = mk2<S>(e.x + o.y, e.y - o.x);
    });
  } else {
    // R = A B: B transforms of length A, twiddles, A transforms of length B.
    constexpr int A = dft_split(R), B = R / A;
    V w[R];
    unroll<B>([&](auto bb) {
      constexpr int b = decltype(bb)::value;
      V u[A];
#pragma unroll
      for (int a = 0; a < A; a++) u[a] = v[b + B * a];
      dft<A, SG, S>(u);
      unroll<A>([&](auto aa) {
        constexpr int a = decltype(aa)::value;
        constexpr S c = (S)cos_turn(a * b, R), z = (S)(SG * sin_turn(a * b, R));
        w[a * B + b] = (a * b == 0) ? u[a] : mk2<S>(u[a].x * c - u[a].y * z, u[a].x * z + u[a].y * c);
      });
    });
#pragma unroll
    for (int a = 0; a < A; a++) {
      dft<B, SG, S>(w + a * B);
#pragma unroll
      for (int b = 0; b < B; b++) v[a + A * b] = w[a * B + b];
    }
  }
}

// f(integral_constant R) for the run-time radix r.  WIDE: radices above 8 too (lengths
// whose larger factor exceeds 8 take this instance: it holds more registers).
template <bool WIDE, typename F>
__device__ __forceinline__ void with_radix(int r, F f) {
  switch (r) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    default:
      if constexpr (WIDE) {
        switch (r) {
          case 9: f(std::integral_constant<int, 9>{}); break;
          case 10: f(std::integral_constant<int, 10>{}); break;
          case 12: f(std::integral_constant<int, 12>{}); break;
          case 15: f(std::integral_constant<int, 15>{}); break;
          default: f(std::integral_constant<int, 16>{}); break;
        }
      }
  }
}

// t / n and t % n by a multiplication: exact while t n < 2^32 (t counts a block's items).
__device__ __forceinline__ int div_by(int t, FastDiv d) { return d.n == 1 ? t : (int)__umulhi((unsigned)t, d.m); }

// v[0 .. R) times the twiddles of step 2: exp(SG 2 pi i q r / N) from the table of
// exp(-2 pi i j / N).
template <int R, int SG, typename S>
__device__ __forceinline__ void twiddle(typename Vec2<S>::type *v, int q, const typename Vec2<S>::type *tw) {
#pragma unroll
  for (int r = 1; r < R; r++) {
    const auto w = tw[q * r];
    const S wy = SG > 0 ? -w.y : w.y;
    v[r] = mk2<S>(v[r].x * w.x - v[r].y * wy, v[r].x * wy + v[r].y * w.x);
  }
}

// Place of element e of a line in shared memory: F2-long runs at an odd stride, so that
// threads along q or along the lines (also at an odd stride) meet different banks.
__device__ __forceinline__ int run_stride(const FftLine &a) { return a.f2 | 1; }

// The (x, y) plane of one z layer.  Forward: the rows along x, then the columns along y; the
// input is the double accumulation mesh (real plane, then imaginary plane at src + ng),
// cleared behind the read so that the next spread starts from zero.  Inverse: the columns,
// then the rows, in place on `mesh`.  The lines of the first axis pass through a buffer of
// `chunk` of them; the second axis' lines, all of the plane, stay.
template <typename S, bool INV, bool WIDE>
__device__ __forceinline__ void k_fft_plane(VGrid vg, typename Vec2<S>::type *__restrict__ const &mesh,
                                            const FftPlan &pl, const typename Vec2<S>::type *__restrict__ const &tw_all,
                                            int const &tw_step, double *__restrict__ const &src, size_t const &ng,
                                            int *const &flags) {
  using V = typename Vec2<S>::type;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const FftLine &ax = pl.line[0], &ay = pl.line[1];
  const int nx = ax.n, ny = ay.n;
  const size_t plane = (size_t)vg.bid * nx * ny;
  const int sx = run_stride(ax), sy = run_stride(ay);
  const int RS = (ax.f1 * sx) | 1, CS = (ay.f1 * sy) | 1;   // row and column strides
  const int chunk = INV ? pl.col_chunk : pl.row_chunk;   // lines of the first axis at a time
  V *rows = reinterpret_cast<V *>(sm_raw), *cols = rows + (size_t)(INV ? ny : chunk) * RS;
  V *twx = cols + (size_t)(INV ? chunk : nx) * CS, *twy = twx + nx;
  for (int t = threadIdx.x; t < nx; t += blockDim.x) twx[t] = tw_all[t];
  for (int t = threadIdx.x; t < ny; t += blockDim.x) twy[t] = tw_all[tw_step + t];
  constexpr int SG = INV ? 1 : -1;
  for (int l0 = 0; l0 < (INV ? nx : ny); l0 += chunk) {
    const int nl = min(chunk, (INV ? nx : ny) - l0);
    if (l0) __syncthreads();
    if constexpr (!INV) {
      with_radix<WIDE>(ax.f1, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        for (int t = threadIdx.x; t < nl * ax.f2; t += blockDim.x) {
          const int l = div_by(t, ax.by_f2), j = t - l * ax.f2;
          const size_t g = plane + (size_t)(l0 + l) * nx + j;
          double re[R], im[R];
#pragma unroll
          for (int r = 0; r < R; r++) {
            re[r] = src[g + r * ax.f2];
            im[r] = src[ng + g + r * ax.f2];
          }
          V v[R];
          bool out = false;
#pragma unroll
          for (int r = 0; r < R; r++) {
            if constexpr (sizeof(S) == 4) out = out || quant_out(re[r]) || quant_out(im[r]);
            src[g + r * ax.f2] = 0.0;
            src[ng + g + r * ax.f2] = 0.0;
            v[r] = mk2<S>((S)re[r], (S)im[r]);
          }
          if (out) atomicOr(flags, FLAG_QUANT_RANGE);
          dft<R, SG, S>(v);
#pragma unroll
          for (int r = 0; r < R; r++) rows[l * RS + r * sx + j] = v[r];
        }
      });
    } else {
      with_radix<WIDE>(ay.f1, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        for (int t = threadIdx.x; t < chunk * ay.f2; t += blockDim.x) {
          const int j = div_by(t, pl.by_col_chunk), c = t - j * chunk;
          if (c >= nl) continue;
          const V *g = mesh + plane + (size_t)j * nx + l0 + c;
          V v[R];
#pragma unroll
          for (int r = 0; r < R; r++) v[r] = g[(size_t)r * ay.f2 * nx];
          dft<R, SG, S>(v);
#pragma unroll
          for (int r = 0; r < R; r++) cols[c * CS + r * sy + j] = v[r];
        }
      });
    }
    __syncthreads();
    // Step 2 of the first axis, its outputs placed for the second.
    if constexpr (!INV) {
      with_radix<WIDE>(ax.f2, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        for (int t = threadIdx.x; t < chunk * ax.f1; t += blockDim.x) {
          const int q = div_by(t, pl.by_row_chunk), l = t - q * chunk;
          if (l >= nl) continue;
          V v[R];
#pragma unroll
          for (int r = 0; r < R; r++) v[r] = rows[l * RS + q * sx + r];
          twiddle<R, SG, S>(v, q, twx);
          dft<R, SG, S>(v);
          const int yj = div_by(l0 + l, ay.by_f2);
          const int at = yj * sy + (l0 + l - yj * ay.f2);
#pragma unroll
          for (int r = 0; r < R; r++) cols[(q + r * ax.f1) * CS + at] = v[r];
        }
      });
    } else {
      with_radix<WIDE>(ay.f2, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        for (int t = threadIdx.x; t < chunk * ay.f1; t += blockDim.x) {
          const int q = div_by(t, pl.by_col_chunk), c = t - q * chunk;
          if (c >= nl) continue;
          V v[R];
#pragma unroll
          for (int r = 0; r < R; r++) v[r] = cols[c * CS + q * sy + r];
          twiddle<R, SG, S>(v, q, twy);
          dft<R, SG, S>(v);
          const int xj = div_by(l0 + c, ax.by_f2);
          const int at = xj * sx + (l0 + c - xj * ax.f2);
#pragma unroll
          for (int r = 0; r < R; r++) rows[(q + r * ay.f1) * RS + at] = v[r];
        }
      });
    }
  }
  __syncthreads();
  // The second axis: step 1 in place, step 2 to the mesh.
  if constexpr (!INV) {
    with_radix<WIDE>(ay.f1, [&](auto rr) {
      constexpr int R = decltype(rr)::value;
      for (int t = threadIdx.x; t < nx * ay.f2; t += blockDim.x) {
        const int j = div_by(t, ax.by_n), c = t - j * nx;
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = cols[c * CS + r * sy + j];
        dft<R, SG, S>(v);
#pragma unroll
        for (int r = 0; r < R; r++) cols[c * CS + r * sy + j] = v[r];
      }
    });
    __syncthreads();
    with_radix<WIDE>(ay.f2, [&](auto rr) {
      constexpr int R = decltype(rr)::value;
      for (int t = threadIdx.x; t < nx * ay.f1; t += blockDim.x) {
        const int q = div_by(t, ax.by_n), c = t - q * nx;
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = cols[c * CS + q * sy + r];
        twiddle<R, SG, S>(v, q, twy);
        dft<R, SG, S>(v);
        V *g = mesh + plane + (size_t)q * nx + c;
#pragma unroll
        for (int r = 0; r < R; r++) g[(size_t)r * ay.f1 * nx] = v[r];
      }
    });
  } else {
    with_radix<WIDE>(ax.f1, [&](auto rr) {
      constexpr int R = decltype(rr)::value;
      for (int t = threadIdx.x; t < ny * ax.f2; t += blockDim.x) {
        const int l = div_by(t, ax.by_f2), j = t - l * ax.f2;
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = rows[l * RS + r * sx + j];
        dft<R, SG, S>(v);
#pragma unroll
        for (int r = 0; r < R; r++) rows[l * RS + r * sx + j] = v[r];
      }
    });
    __syncthreads();
    with_radix<WIDE>(ax.f2, [&](auto rr) {
      constexpr int R = decltype(rr)::value;
      for (int t = threadIdx.x; t < ny * ax.f1; t += blockDim.x) {
        const int l = div_by(t, ax.by_f1), q = t - l * ax.f1;
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = rows[l * RS + q * sx + r];
        twiddle<R, SG, S>(v, q, twx);
        dft<R, SG, S>(v);
        V *g = mesh + plane + (size_t)l * nx + q;
#pragma unroll
        for (int r = 0; r < R; r++) g[r * ax.f1] = v[r];
      }
    });
  }
}

// Lines along z at kFftZLines consecutive (x, y): forward, times the influence function,
// inverse.  Step 2 of the forward transform leaves a thread exactly the inputs of step 1
// of the inverse with the factors exchanged (outputs q + F1 k, all k), so the product with
// the influence function happens in registers between the two.
template <typename S, bool WIDE>
__device__ __forceinline__ void k_fft_z(VGrid vg, typename Vec2<S>::type *__restrict__ const &mesh, const FftPlan &pl,
                                        const typename Vec2<S>::type *__restrict__ const &tw_all, int const &tw_step,
                                        const S *__restrict__ const &G) {
  using V = typename Vec2<S>::type;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  constexpr int L = kFftZLines;
  const FftLine &az = pl.line[2];
  const int nz = az.n, f1 = az.f1, f2 = az.f2;
  const size_t nxy = (size_t)pl.line[0].n * pl.line[1].n;
  V *a = reinterpret_cast<V *>(sm_raw), *b = a + (size_t)nz * L, *tw = b + (size_t)nz * L;
  for (int t = threadIdx.x; t < nz; t += blockDim.x) tw[t] = tw_all[2 * tw_step + t];
  const size_t p0 = (size_t)vg.bid * L;
  const int l = threadIdx.x & (L - 1), jt = threadIdx.x / L, js = blockDim.x / L;
  const bool live = p0 + l < nxy;
  V *line = mesh + p0 + l;
  if (live) {
    with_radix<WIDE>(f1, [&](auto rr) {
      constexpr int R = decltype(rr)::value;
      for (int j = jt; j < f2; j += js) {
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = line[(size_t)(j + r * f2) * nxy];
        dft<R, -1, S>(v);
#pragma unroll
        for (int r = 0; r < R; r++) a[(r * f2 + j) * L + l] = v[r];
      }
    });
  }
  __syncthreads();
  if (live) {
    with_radix<WIDE>(f2, [&](auto rr) {
      constexpr int R = decltype(rr)::value;
      for (int q = jt; q < f1; q += js) {
        S g[R];
#pragma unroll
        for (int r = 0; r < R; r++) g[r] = __ldg(G + (size_t)(q + r * f1) * nxy + p0 + l);
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = a[(q * f2 + r) * L + l];
        twiddle<R, -1, S>(v, q, tw);
        dft<R, -1, S>(v);
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = mk2<S>(v[r].x * g[r], v[r].y * g[r]);
        dft<R, 1, S>(v);
#pragma unroll
        for (int r = 0; r < R; r++) b[(r * f1 + q) * L + l] = v[r];
      }
    });
  }
  __syncthreads();
  if (live) {
    with_radix<WIDE>(f1, [&](auto rr) {
      constexpr int R = decltype(rr)::value;
      for (int q = jt; q < f2; q += js) {
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = b[(q * f1 + r) * L + l];
        twiddle<R, 1, S>(v, q, tw);
        dft<R, 1, S>(v);
#pragma unroll
        for (int r = 0; r < R; r++) line[(size_t)(q + r * f2) * nxy] = v[r];
      }
    });
  }
}

}  // namespace ffx
