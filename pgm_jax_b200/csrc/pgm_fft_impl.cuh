// pgm_fft_impl.cuh -- kernels and launchers of pgm_fft.cuh for one precision (included by one .cu each).
#pragma once
#include <type_traits>
#include <utility>

#include "pgm_fft.cuh"

namespace pgmfft {

// ------------------------------------------------------------------ transforms in registers
// cos and sin of 2 pi k / R at compile time (Taylor series on the first octant).
constexpr double PI2 = 6.28318530717958647692528676655900577;
constexpr double taylor(double x, bool sine) {
  double t = sine ? x : 1.0, s = t;
  for (int n = sine ? 2 : 1; n < 30; n += 2) {
    t *= -x * x / (n * (n + 1.0));
    s += t;
  }
  return s;
}
constexpr double cos_turn(int k, int R) {  // cos(2 pi k / R)
  k = ((k % R) + R) % R;
  if (2 * k > R) k = R - k;
  const bool neg = 4 * k > R;
  const int num = neg ? R - 2 * k : 2 * k;  // angle pi num / R in [0, pi / 2]
  const double c = 4 * num <= R ? taylor(PI2 * num / (2.0 * R), false) : taylor(PI2 * (R - 2 * num) / (4.0 * R), true);
  return neg ? -c : c;
}
constexpr double sin_turn(int k, int R) { return cos_turn(4 * k - R, 4 * R); }

template <typename F, int... I>
__device__ __forceinline__ void unroll_impl(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void unroll(F &&f) {
  unroll_impl(f, std::make_integer_sequence<int, N>{});
}

template <typename T>
__device__ __forceinline__ c2<T> cmul(c2<T> a, c2<T> b) {
  c2<T> r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}

// a exp(-2 pi i K / R), K and R compile-time.
template <typename T, int K, int R>
__device__ __forceinline__ c2<T> turn(c2<T> a) {
  c2<T> r;
  if constexpr (K % R == 0) {
    r = a;
  } else if constexpr (4 * K % R == 0) {
    constexpr int q = 4 * K / R % 4;
    if constexpr (q == 1) { r.x = a.y; r.y = -a.x; }
    else if constexpr (q == 2) { r.x = -a.x; r.y = -a.y; }
    else { r.x = -a.y; r.y = a.x; }
  } else {
    constexpr double c = cos_turn(K, R), s = sin_turn(K, R);
    r.x = a.x * T(c) + a.y * T(s);
    r.y = a.y * T(c) - a.x * T(s);
  }
  return r;
}

constexpr int split_of(int R) {  // the first factor of a composite register transform
  return R % 4 == 0 ? 4 : R % 5 == 0 ? 5 : R % 3 == 0 ? 3 : 2;
}

// Forward R-point transform of v in natural order: 2, 3, 4, 5 written out, others A x B of those.
template <typename T, int R>
__device__ __forceinline__ void dft(c2<T> (&v)[R]) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const c2<T> a = v[0], b = v[1];
    v[0].x = a.x + b.x; v[0].y = a.y + b.y;
    v[1].x = a.x - b.x; v[1].y = a.y - b.y;
  } else if constexpr (R == 3) {
    const T c = T(-0.5), s = T(sin_turn(1, 3));
    const T px = v[1].x + v[2].x, py = v[1].y + v[2].y, mx = v[1].x - v[2].x, my = v[1].y - v[2].y;
    const T ax = v[0].x + c * px, ay = v[0].y + c * py;
    v[0].x += px; v[0].y += py;
    v[1].x = ax + s * my; v[1].y = ay - s * mx;
    v[2].x = ax - s * my; v[2].y = ay + s * mx;
  } else if constexpr (R == 4) {
    const T ax = v[0].x + v[2].x, ay = v[0].y + v[2].y, bx = v[0].x - v[2].x, by = v[0].y - v[2].y;
    const T cx = v[1].x + v[3].x, cy = v[1].y + v[3].y, dx = v[1].x - v[3].x, dy = v[1].y - v[3].y;
    v[0].x = ax + cx; v[0].y = ay + cy;
    v[1].x = bx + dy; v[1].y = by - dx;
    v[2].x = ax - cx; v[2].y = ay - cy;
    v[3].x = bx - dy; v[3].y = by + dx;
  } else if constexpr (R == 5) {
    const T c1 = T(cos_turn(1, 5)), c2v = T(cos_turn(2, 5)), s1 = T(sin_turn(1, 5)), s2 = T(sin_turn(2, 5));
    const T ax = v[1].x + v[4].x, ay = v[1].y + v[4].y, bx = v[1].x - v[4].x, by = v[1].y - v[4].y;
    const T ex = v[2].x + v[3].x, ey = v[2].y + v[3].y, fx = v[2].x - v[3].x, fy = v[2].y - v[3].y;
    const T m1x = v[0].x + c1 * ax + c2v * ex, m1y = v[0].y + c1 * ay + c2v * ey;
    const T m2x = v[0].x + c2v * ax + c1 * ex, m2y = v[0].y + c2v * ay + c1 * ey;
    const T n1x = s1 * bx + s2 * fx, n1y = s1 * by + s2 * fy;
    const T n2x = s2 * bx - s1 * fx, n2y = s2 * by - s1 * fy;
    v[0].x += ax + ex; v[0].y += ay + ey;
    v[1].x = m1x + n1y; v[1].y = m1y - n1x;
    v[4].x = m1x - n1y; v[4].y = m1y + n1x;
    v[2].x = m2x + n2y; v[2].y = m2y - n2x;
    v[3].x = m2x - n2y; v[3].y = m2y + n2x;
  } else {
    constexpr int A = split_of(R), B = R / A;  // n = B a + b, k = ka + A kb
    c2<T> t[R];
    unroll<B>([&](auto bc) {
      constexpr int b = decltype(bc)::value;
      c2<T> u[A];
      unroll<A>([&](auto ac) { u[decltype(ac)::value] = v[B * decltype(ac)::value + b]; });
      dft<T, A>(u);
      unroll<A>([&](auto kc) {
        constexpr int ka = decltype(kc)::value;
        t[ka * B + b] = turn<T, b * ka, R>(u[ka]);
      });
    });
    unroll<A>([&](auto kc) {
      constexpr int ka = decltype(kc)::value;
      c2<T> u[B];
      unroll<B>([&](auto bc) { u[decltype(bc)::value] = t[ka * B + decltype(bc)::value]; });
      dft<T, B>(u);
      unroll<B>([&](auto bc) { v[ka + A * decltype(bc)::value] = u[decltype(bc)::value]; });
    });
  }
}

template <typename T>
__device__ __forceinline__ c2<T> swapped(c2<T> a) {
  c2<T> r;
  r.x = a.y; r.y = a.x;
  return r;
}

constexpr int n1_of(int N) {
  int d = 1;
  while (d * d < N || N % d != 0) ++d;
  return d;
}

// Step 1 of a line: the transform over n1 of the points n2 + N2 n1, times w_N^(n2 k1).
template <typename T, int N>
__device__ __forceinline__ void step1(c2<T> (&v)[n1_of(N)], int n2, const c2<T> *__restrict__ tw) {
  constexpr int N1 = n1_of(N);
  dft<T, N1>(v);
#pragma unroll
  for (int k = 1; k < N1; ++k) v[k] = cmul<T>(v[k], tw[n2 * k]);
}

template <int N>
constexpr int N1R = n1_of(N) > 18 ? 96 : 64;  // registers asked for (FP32)
// Blocks per SM that the compiler leaves registers for: FP32 64 a thread (k2, k3 passes), 80 (the convolution) or
// 96 (its energy form), 96 to 128 where N1 > 18, FP64 twice that.  Not every transform fits: 192 spills 76 bytes in the
// convolution, 128 180, 256 356 (136 in the k2 pass), most lengths below 144 none.
template <typename T>
constexpr int min_blocks(int threads, int regs32) {
  const int b = 65536 / (threads * (sizeof(T) == 4 ? regs32 : 2 * regs32));
  return b < 1 ? 1 : b > 16 ? 16 : b;
}

__device__ __forceinline__ bool pass_active(const CGSys *cg, int s, int act) {
  return act == 0 || (act == 1 && cg[s].active) || (act == 2 && cg[s].sweep2) || (act == 3 && cg[s].fallback);
}

__device__ __forceinline__ Tile tile_of(const Tiles &ts) {
  if (!ts.one) return ts.table[blockIdx.x];
  Tile t = ts.base;
  const int b = blockIdx.x;
  t.c0 = b * ts.c_step;
  t.rg += b * ts.r_step;
  t.cg += b * ts.g_step;
  if (ts.lines) t.n = min(t.n, (ts.lines - t.c0) / 2);
  t.q0 = min(ts.total, b * ts.share);
  t.q1 = min(ts.total, (b + 1) * ts.share);
  return t;
}

// ------------------------------------------------------------------ k3 passes
// Two real lines packed as one complex line (z = a + i b).  Threads of a pair are consecutive, so
// a pair's N2 loads of one n1 are contiguous; the shared line has an odd inner stride (N2 | 1) so that
// step 2's reads at stride N2 miss each other's banks.
template <typename T, int N>
struct XShape {
  static constexpr int N1 = n1_of(N), N2 = N / N1, NP = tile_width<T>(), S2 = N2 | 1, PS = N1 * S2, ZS = N + 1;
  static constexpr int ELEMS = NP * (PS > ZS ? PS : ZS), THREADS = NP * N1;
};

template <typename T, int N>
__global__ void __launch_bounds__(XShape<T, N>::THREADS, min_blocks<T>(XShape<T, N>::THREADS, N1R<N>)) k_x_fwd(Args<T> a, Tiles tiles, int act) {
  using X = XShape<T, N>;
  constexpr int N1 = X::N1, N2 = X::N2, Kh = N / 2 + 1;
  pgm::pdl_enter();
  __shared__ __align__(16) unsigned char raw[X::ELEMS * sizeof(c2<T>)];
  c2<T> *sh = reinterpret_cast<c2<T> *>(raw);
  const Tile t = tile_of(tiles);
  const int p = threadIdx.x / N1, r = threadIdx.x - p * N1;
  const bool on = p < t.n;
  c2<T> v[N1];  // loaded before the test of the system's flag
  if (on && r < N2) {
    const T *qa = a.Q + t.rg + (size_t)(t.c0 + 2 * p) * N + r, *qb = qa + N;
#pragma unroll
    for (int k = 0; k < N1; ++k) { v[k].x = qa[N2 * k]; v[k].y = qb[N2 * k]; }
  }
  if (!pass_active(a.cg, t.s, act)) return;
  if (on && r < N2) {
    step1<T, N>(v, r, a.tw + t.tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) sh[p * X::PS + k * X::S2 + r] = v[k];
  }
  __syncthreads();
  c2<T> u[N2];
#pragma unroll
  for (int k = 0; k < N2; ++k) u[k] = sh[p * X::PS + r * X::S2 + k];
  dft<T, N2>(u);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N2; ++k) sh[p * X::ZS + r + N1 * k] = u[k];
  __syncthreads();
  c2<T> *C = a.C + t.cg + (size_t)t.c0 * Kh;
  for (int w = threadIdx.x; w < t.n * Kh; w += X::THREADS) {
    const int l = w / Kh, m = w - l * Kh;
    const c2<T> Z = sh[l * X::ZS + m], W = sh[l * X::ZS + (m == 0 ? 0 : N - m)];
    c2<T> A, B;
    A.x = T(0.5) * (Z.x + W.x); A.y = T(0.5) * (Z.y - W.y);
    B.x = T(0.5) * (Z.y + W.y); B.y = T(-0.5) * (Z.x - W.x);  // (Z - conj W) / (2 i)
    C[(size_t)(2 * l) * Kh + m] = A;
    C[(size_t)(2 * l + 1) * Kh + m] = B;
  }
}

// Half complex -> real (unnormalised): the packed line's points straight from the two rows of C.
template <typename T, int N>
__device__ __forceinline__ c2<T> tangled(c2<T> A, c2<T> B, int mm, bool up) {
  if (mm == 0 || 2 * mm == N) { A.y = T(0); B.y = T(0); }
  if (up) { A.y = -A.y; B.y = -B.y; }
  c2<T> z;
  z.x = A.x - B.y; z.y = A.y + B.x;
  return z;
}

template <typename T, int N>
__global__ void __launch_bounds__(XShape<T, N>::THREADS, min_blocks<T>(XShape<T, N>::THREADS, N1R<N>)) k_x_inv(Args<T> a, Tiles tiles, int act) {
  using X = XShape<T, N>;
  constexpr int N1 = X::N1, N2 = X::N2, Kh = N / 2 + 1;
  pgm::pdl_enter();
  __shared__ __align__(16) unsigned char raw[X::ELEMS * sizeof(c2<T>)];
  c2<T> *sh = reinterpret_cast<c2<T> *>(raw);
  const Tile t = tile_of(tiles);
  if (!pass_active(a.cg, t.s, act)) return;
  const int p = threadIdx.x / N1, r = threadIdx.x - p * N1;
  const bool on = p < t.n;
  if (on && r < N2) {
    const c2<T> *ca = a.C + t.cg + (size_t)(t.c0 + 2 * p) * Kh, *cb = ca + Kh;
    c2<T> v[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      const int m = r + N2 * k;
      const bool up = m > N / 2;
      const int mm = up ? N - m : m;
      v[k] = swapped<T>(tangled<T, N>(ca[mm], cb[mm], mm, up));
    }
    step1<T, N>(v, r, a.tw + t.tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) sh[p * X::PS + k * X::S2 + r] = v[k];
  }
  __syncthreads();
  if (!on) return;
  c2<T> u[N2];
#pragma unroll
  for (int k = 0; k < N2; ++k) u[k] = sh[p * X::PS + r * X::S2 + k];
  dft<T, N2>(u);
  T *fa = a.Phi + t.rg + (size_t)(t.c0 + 2 * p) * N + r, *fb = fa + N;
#pragma unroll
  for (int k = 0; k < N2; ++k) { fa[N1 * k] = u[k].y; fb[N1 * k] = u[k].x; }
}

// ------------------------------------------------------------------ k2 pass (both directions)
// TC consecutive columns of the flattened (k1, m3) index; consecutive threads take consecutive
// columns, so global and shared accesses are contiguous.
template <typename T, int N>
struct YShape {
  static constexpr int N1 = n1_of(N), N2 = N / N1, TC = tile_width<T>(), THREADS = TC * N1;
};

template <typename T, int N>
__global__ void __launch_bounds__(YShape<T, N>::THREADS, min_blocks<T>(YShape<T, N>::THREADS, N1R<N>)) k_y(Args<T> a, Tiles tiles, int act, int sign) {
  using Y = YShape<T, N>;
  constexpr int N1 = Y::N1, N2 = Y::N2, TC = Y::TC;
  pgm::pdl_enter();
  __shared__ __align__(16) unsigned char raw[N * TC * sizeof(c2<T>)];
  c2<T> *sh = reinterpret_cast<c2<T> *>(raw);
  const Tile t = tile_of(tiles);
  const int r = threadIdx.x / TC, c = threadIdx.x - r * TC, col = t.c0 + c;
  const bool on = col < t.n;
  const int k1 = col / t.K3h, m3 = col - k1 * t.K3h;
  const size_t rs = t.K3h;
  c2<T> *C = a.C + t.cg + (size_t)k1 * N * rs + m3;
  c2<T> v[N1];  // loaded before the test of the system's flag
  if (on && r < N2)
#pragma unroll
    for (int k = 0; k < N1; ++k) v[k] = C[(r + N2 * k) * rs];
  if (!pass_active(a.cg, t.s, act)) return;
  if (on && r < N2) {
    if (sign > 0)
#pragma unroll
      for (int k = 0; k < N1; ++k) v[k] = swapped<T>(v[k]);
    step1<T, N>(v, r, a.tw + t.tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) sh[(k * N2 + r) * TC + c] = v[k];
  }
  if (sign < 0) {  // the k3 pass has consumed the real grid: clear this CTA's share for the next spread
    using V = pgm::v4<T>;
    V z;
    z.x = T(0); z.y = T(0); z.z = T(0); z.w = T(0);
    V *Q = reinterpret_cast<V *>(a.Q + t.rg);
    for (long long w = t.q0 / 4 + threadIdx.x; w < t.q1 / 4; w += Y::THREADS) Q[w] = z;
  }
  __syncthreads();
  if (!on) return;
  c2<T> u[N2];
#pragma unroll
  for (int k = 0; k < N2; ++k) u[k] = sh[(r * N2 + k) * TC + c];
  dft<T, N2>(u);
#pragma unroll
  for (int k = 0; k < N2; ++k) C[(r + N1 * k) * rs] = sign > 0 ? swapped<T>(u[k]) : u[k];
}

// ------------------------------------------------------------------ k1 pass with the convolution
// Columns c = k2 K3h + m3 (contiguous): forward along k1, times 2 G(m) (phi = dE/dQ = 2 K^3 irfft(G F[Q]),
// pme.py:370-376), inverse.  With ENERGY the reciprocal energy sum w3 G |F|^2 (pme.py:390-411) and
// the influence part of the virial are accumulated.
template <typename T, int N, bool ENERGY>
__global__ void __launch_bounds__(YShape<T, N>::THREADS, min_blocks<T>(YShape<T, N>::THREADS, N1R<N> + (ENERGY ? 32 : 16))) k_z(Args<T> a, Tiles tiles, int act) {
  using Y = YShape<T, N>;
  constexpr int N1 = Y::N1, N2 = Y::N2, TC = Y::TC;
  pgm::pdl_enter();
  __shared__ __align__(16) unsigned char raw[N * TC * sizeof(c2<T>)];
  c2<T> *sh = reinterpret_cast<c2<T> *>(raw);
  const Tile t = tile_of(tiles);
  const int r = threadIdx.x / TC, c = threadIdx.x - r * TC, col = t.c0 + c;
  const bool on = col < t.n;
  const size_t rs = t.n;
  c2<T> *C = a.C + t.cg + col;
  const T *G = a.Ginf + t.cg + col;
  const c2<T> *tw = a.tw + t.tw;
  c2<T> v[N1];
  T g[N2];
  if (on && r < N2)
#pragma unroll
    for (int k = 0; k < N1; ++k) v[k] = C[(r + N2 * k) * rs];
  if (!pass_active(a.cg, t.s, act)) return;  // after the loads
#pragma unroll
  for (int k = 0; k < N2; ++k) g[k] = on ? G[(r + N1 * k) * rs] : T(0);
  if (on && r < N2) {
    step1<T, N>(v, r, tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) sh[(k * N2 + r) * TC + c] = v[k];
  }
  __syncthreads();
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  if (on) {
    c2<T> u[N2];
#pragma unroll
    for (int k = 0; k < N2; ++k) u[k] = sh[(r * N2 + k) * TC + c];
    dft<T, N2>(u);
    if constexpr (ENERGY) {
      const BoxInfo &B = a.box[t.s];
      const int k2 = col / t.K3h, m3 = col - k2 * t.K3h;
      const double w3 = (m3 == 0 || 2 * m3 == t.K3) ? 1.0 : 2.0;
      const int m2 = 2 * k2 < t.K2 ? k2 : k2 - t.K2;
      const double pb = pgm::PI * pgm::PI / (a.beta * a.beta);
#pragma unroll
      for (int k = 0; k < N2; ++k) {
        if (g[k] == T(0)) continue;
        const int k1 = r + N1 * k, m1 = 2 * k1 < N ? k1 : k1 - N;
        const double e = w3 * double(g[k]) * (double(u[k].x) * double(u[k].x) + double(u[k].y) * double(u[k].y));
        double mv[3];
#pragma unroll
        for (int x = 0; x < 3; ++x) mv[x] = m1 * B.Hinv[x * 3 + 0] + m2 * B.Hinv[x * 3 + 1] + m3 * B.Hinv[x * 3 + 2];
        const double fac = 2.0 * (pb + 1.0 / (mv[0] * mv[0] + mv[1] * mv[1] + mv[2] * mv[2]));
        acc[0] += e;
        acc[1] += e * (fac * mv[0] * mv[0] - 1.0);
        acc[2] += e * (fac * mv[1] * mv[1] - 1.0);
        acc[3] += e * (fac * mv[2] * mv[2] - 1.0);
        acc[4] += e * fac * mv[0] * mv[1];
        acc[5] += e * fac * mv[0] * mv[2];
        acc[6] += e * fac * mv[1] * mv[2];
      }
    }
#pragma unroll
    for (int k = 0; k < N2; ++k) {
      const T g2 = T(2) * g[k];
      const c2<T> z = u[k];
      u[k].x = z.y * g2; u[k].y = z.x * g2;  // swapped: the inverse
    }
    dft<T, N2>(u);
    sh[(r * N2) * TC + c] = u[0];  // the slots this thread read
#pragma unroll
    for (int k = 1; k < N2; ++k) sh[(r * N2 + k) * TC + c] = cmul<T>(u[k], tw[r * k]);
  }
  __syncthreads();
  if (on && r < N2) {
#pragma unroll
    for (int k = 0; k < N1; ++k) v[k] = sh[(k * N2 + r) * TC + c];
    dft<T, N1>(v);
#pragma unroll
    for (int k = 0; k < N1; ++k) C[(r + N2 * k) * rs] = swapped<T>(v[k]);
  }
  if constexpr (ENERGY) {
    __shared__ double red[(Y::THREADS + 31) / 32][7];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int LAST = Y::THREADS % 32;  // threads of a last, partial warp (0: none)
    const unsigned mask = (LAST && warp == Y::THREADS / 32) ? (1u << LAST) - 1u : 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      double x = acc[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_down_sync(mask, x, o);
        x += (lane + o < 32 && ((mask >> (lane + o)) & 1u)) ? y : 0.0;
      }
      if (lane == 0) red[warp][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
      double x = 0;
      for (int w = 0; w < (Y::THREADS + 31) / 32; ++w) x += red[w][threadIdx.x];
      atomicAdd(&a.eacc[t.s].vinf[threadIdx.x], x);
    }
  }
}

// ------------------------------------------------------------------ plane passes (K2 = K3 = N)
// One CTA per k1 plane runs the k3 and the k2 pass in shared memory (two regions, A and B): one
// launch and one grid round trip instead of two, with three barriers.  The tasks of a phase (a line and
// a step's index) are spread over the CTA's threads; the k2 phases read the packed k3 lines' two
// halves directly.
template <int N>
struct PlaneShape {
  static constexpr int N1 = n1_of(N), N2 = N / N1, Kh = N / 2 + 1, NP = N / 2, S2 = N2 | 1, PS = N1 * S2, ZS = N + 1;
  static constexpr int REG_A = NP * PS > N * Kh ? NP * PS : N * Kh, REG_B = NP * ZS > N * Kh ? NP * ZS : N * Kh;
  static constexpr int TASKS = Kh * N1, ROUNDS = (TASKS + 639) / 640, THREADS = ((TASKS + ROUNDS - 1) / ROUNDS + 31) / 32 * 32;
};

template <typename T, int N>
__global__ void __launch_bounds__(PlaneShape<N>::THREADS) k_plane_fwd(Args<T> a, Tiles tiles, int act) {
  using S = PlaneShape<N>;
  constexpr int N1 = S::N1, N2 = S::N2, Kh = S::Kh, NP = S::NP;
  pgm::pdl_enter();
  extern __shared__ __align__(16) unsigned char raw[];
  c2<T> *A = reinterpret_cast<c2<T> *>(raw), *B = A + S::REG_A;
  const Tile t = tile_of(tiles);
  if (!pass_active(a.cg, t.s, act)) return;
  const c2<T> *tw = a.tw + t.tw;
  T *Q = a.Q + t.rg;
  for (int w = threadIdx.x; w < NP * N2; w += S::THREADS) {  // k3, step 1; Q is cleared for the next spread
    const int p = w / N2, r = w - p * N2;
    T *qa = Q + (size_t)(2 * p) * N + r, *qb = qa + N;
    c2<T> v[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) { v[k].x = qa[N2 * k]; v[k].y = qb[N2 * k]; }
    step1<T, N>(v, r, tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      A[p * S::PS + k * S::S2 + r] = v[k];
      qa[N2 * k] = T(0); qb[N2 * k] = T(0);
    }
  }
  __syncthreads();
  for (int w = threadIdx.x; w < NP * N1; w += S::THREADS) {  // k3, step 2
    const int p = w / N1, r = w - p * N1;
    c2<T> u[N2];
#pragma unroll
    for (int k = 0; k < N2; ++k) u[k] = A[p * S::PS + r * S::S2 + k];
    dft<T, N2>(u);
#pragma unroll
    for (int k = 0; k < N2; ++k) B[p * S::ZS + r + N1 * k] = u[k];
  }
  __syncthreads();
  for (int w = threadIdx.x; w < Kh * N2; w += S::THREADS) {  // k2, step 1, on the untangled rows
    const int r = w / Kh, m = w - r * Kh, mc = m == 0 ? 0 : N - m;
    c2<T> v[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      const int row = r + N2 * k;
      const c2<T> Z = B[(row >> 1) * S::ZS + m], W = B[(row >> 1) * S::ZS + mc];
      if (row & 1) { v[k].x = T(0.5) * (Z.y + W.y); v[k].y = T(-0.5) * (Z.x - W.x); }
      else { v[k].x = T(0.5) * (Z.x + W.x); v[k].y = T(0.5) * (Z.y - W.y); }
    }
    step1<T, N>(v, r, tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) A[(k * N2 + r) * Kh + m] = v[k];
  }
  __syncthreads();
  c2<T> *C = a.C + t.cg;
  for (int w = threadIdx.x; w < Kh * N1; w += S::THREADS) {  // k2, step 2
    const int r = w / Kh, m = w - r * Kh;
    c2<T> u[N2];
#pragma unroll
    for (int k = 0; k < N2; ++k) u[k] = A[(r * N2 + k) * Kh + m];
    dft<T, N2>(u);
#pragma unroll
    for (int k = 0; k < N2; ++k) C[(size_t)(r + N1 * k) * Kh + m] = u[k];
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(PlaneShape<N>::THREADS) k_plane_inv(Args<T> a, Tiles tiles, int act) {
  using S = PlaneShape<N>;
  constexpr int N1 = S::N1, N2 = S::N2, Kh = S::Kh, NP = S::NP;
  pgm::pdl_enter();
  extern __shared__ __align__(16) unsigned char raw[];
  c2<T> *A = reinterpret_cast<c2<T> *>(raw), *B = A + S::REG_A;
  const Tile t = tile_of(tiles);
  if (!pass_active(a.cg, t.s, act)) return;
  const c2<T> *tw = a.tw + t.tw;
  const c2<T> *C = a.C + t.cg;
  for (int w = threadIdx.x; w < Kh * N2; w += S::THREADS) {  // k2, step 1
    const int r = w / Kh, m = w - r * Kh;
    c2<T> v[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) v[k] = swapped<T>(C[(size_t)(r + N2 * k) * Kh + m]);
    step1<T, N>(v, r, tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) A[(k * N2 + r) * Kh + m] = v[k];
  }
  __syncthreads();
  for (int w = threadIdx.x; w < Kh * N1; w += S::THREADS) {  // k2, step 2: rows k2 of the half-complex plane
    const int r = w / Kh, m = w - r * Kh;
    c2<T> u[N2];
#pragma unroll
    for (int k = 0; k < N2; ++k) u[k] = A[(r * N2 + k) * Kh + m];
    dft<T, N2>(u);
#pragma unroll
    for (int k = 0; k < N2; ++k) B[(r + N1 * k) * Kh + m] = swapped<T>(u[k]);
  }
  __syncthreads();
  for (int w = threadIdx.x; w < NP * N2; w += S::THREADS) {  // k3, step 1, on pairs of rows
    const int p = w / N2, r = w - p * N2;
    c2<T> v[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      const int m = r + N2 * k;
      const bool up = m > N / 2;
      const int mm = up ? N - m : m;
      v[k] = swapped<T>(tangled<T, N>(B[(2 * p) * Kh + mm], B[(2 * p + 1) * Kh + mm], mm, up));
    }
    step1<T, N>(v, r, tw);
#pragma unroll
    for (int k = 0; k < N1; ++k) A[p * S::PS + k * S::S2 + r] = v[k];
  }
  __syncthreads();
  T *F = a.Phi + t.rg;
  for (int w = threadIdx.x; w < NP * N1; w += S::THREADS) {  // k3, step 2
    const int p = w / N1, r = w - p * N1;
    c2<T> u[N2];
#pragma unroll
    for (int k = 0; k < N2; ++k) u[k] = A[p * S::PS + r * S::S2 + k];
    dft<T, N2>(u);
    T *fa = F + (size_t)(2 * p) * N + r, *fb = fa + N;
#pragma unroll
    for (int k = 0; k < N2; ++k) { fa[N1 * k] = u[k].y; fb[N1 * k] = u[k].x; }
  }
}

// ------------------------------------------------------------------ launchers
// Every even mesh length 8 .. 256 with no prime factor above 5 (what pgm_create accepts).
using Lengths = std::integer_sequence<int, 8, 10, 12, 16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120,
                                      128, 144, 150, 160, 162, 180, 192, 200, 216, 240, 250, 256>;

template <typename F, int... L>
bool with_length_impl(int N, F &&f, std::integer_sequence<int, L...>) {
  bool hit = false;
  ((L == N ? (f(std::integral_constant<int, L>{}), hit = true) : false), ...);
  return hit;
}
template <typename F>
bool with_length(int N, F &&f) { return with_length_impl(N, f, Lengths{}); }

template <typename... KArgs, typename... Args_>
cudaError_t start(void (*k)(KArgs...), int grid, int block, size_t smem, cudaStream_t st, bool dependent, Args_... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

template <typename T, int N>
constexpr size_t plane_bytes() { return (size_t)(PlaneShape<N>::REG_A + PlaneShape<N>::REG_B) * sizeof(c2<T>); }

template <typename T>
bool supported(int N) { return with_length(N, [](auto) {}); }

template <typename T>
cudaError_t prepare(Pass p, int N) {
  cudaError_t e = cudaErrorInvalidValue;
  with_length(N, [&](auto Lc) {
    constexpr int L = decltype(Lc)::value;
    e = cudaSuccess;
    if constexpr (L <= PLANE_MAX) {
      const int bytes = (int)plane_bytes<T, L>();
      if (p == PLANE_FWD) e = cudaFuncSetAttribute(k_plane_fwd<T, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      else if (p == PLANE_INV) e = cudaFuncSetAttribute(k_plane_inv<T, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    }
  });
  return e;
}

template <typename T>
cudaError_t launch(Pass p, int N, const Args<T> &a, const Tiles &tiles, int ntiles, int act, int sign, cudaStream_t st, bool dependent) {
  cudaError_t e = cudaErrorInvalidValue;
  with_length(N, [&](auto Lc) {
    constexpr int L = decltype(Lc)::value;
    constexpr int XT = XShape<T, L>::THREADS, YT = YShape<T, L>::THREADS;
    switch (p) {
      case X_FWD: e = start(k_x_fwd<T, L>, ntiles, XT, 0, st, dependent, a, tiles, act); break;
      case X_INV: e = start(k_x_inv<T, L>, ntiles, XT, 0, st, dependent, a, tiles, act); break;
      case Y_PASS: e = start(k_y<T, L>, ntiles, YT, 0, st, dependent, a, tiles, act, sign); break;
      case Z_CONV: e = start(k_z<T, L, false>, ntiles, YT, 0, st, dependent, a, tiles, act); break;
      case Z_ENERGY: e = start(k_z<T, L, true>, ntiles, YT, 0, st, dependent, a, tiles, act); break;
      default:
        if constexpr (L <= PLANE_MAX) {
          constexpr int PT = PlaneShape<L>::THREADS;
          if (p == PLANE_FWD) e = start(k_plane_fwd<T, L>, ntiles, PT, plane_bytes<T, L>(), st, dependent, a, tiles, act);
          else e = start(k_plane_inv<T, L>, ntiles, PT, plane_bytes<T, L>(), st, dependent, a, tiles, act);
        }
    }
  });
  return e;
}

}  // namespace pgmfft
