// Row and column passes for grid sizes that are not powers of two.
//
// The reference accepts any even grid size (wigner_moyal_fftw_1d.py:55, 62;
// wigner_moyal_cuda_1d.py:63, 70).  The register-resident passes of
// wigner_passes.cu cover the powers of two in [128, 4096]; every other even
// size up to 4096 runs here.  One CTA owns CP row or column pairs of one
// instance (two real sequences packed into one complex transform each) and
// transforms them in shared memory with a mixed-radix Stockham FFT between two
// buffers, element i of pair c at slot i * CP + c plus one pad slot per 128
// bytes (the power-of-two strides of the first stages would hit one bank).
// The factors are 4s, then 2, 3, 5 and the remaining primes; neighbouring
// small ones run as one stage in registers (4 x 4, 5 x 5, 3 x 5, ...: half the
// shared-memory passes and barriers with the same twiddles and butterflies),
// 7, 11 and 13 in registers too, and a larger prime p as a direct transform
// over the sums and differences of mirrored inputs ((p-1)^2 multiply-adds
// instead of 4 p^2), spread over the CTA.  The spectral multiply handles bins k and
// N - k at once: their factors are conjugates, so one table read and one
// product pair serve two bins.
//
// Bound by shared-memory traffic and latency for smooth sizes, by the direct
// transform's multiply-adds for sizes with a large prime factor.  Against one
// pair per CTA, radix 4/2/3/5 stages only, every other prime as one thread's
// direct sum and unfused column half-steps: 8 x 600 x 1000 FP32, 10 steps,
// 3.93 -> 1.14 ms (1.13 with FP32 squares and weight spectra, which narrowed the
// observables); one 98 x 202 FP64 object, 10 steps, 42.7 -> 0.34 ms.
#include "fw_internal.h"
#include "wigner_tiles.cuh"

namespace fw {

constexpr int kGenThreads = 256;
constexpr int kGenMaxStages = 12;
// CTAs per SM the passes are compiled for, and the shared memory of one that
// lets as many be resident: the stages wait on shared memory and barriers, so FP32
// runs four CTAs of 64 registers (8 x 600 x 1000: 146 us a step with two, 118 with three,
// 106 with four; 8 x 300 x 900: 104, 81, 59), FP64, which would spill, two.
template <typename Rl> __host__ __device__ constexpr int gen_minb() { return sizeof(Rl) == 4 ? 4 : 2; }
constexpr size_t kGenSmem32 = (size_t)56 << 10, kGenSmem64 = (size_t)110 << 10;
// FP32 direct transforms of primes above this sum their terms in index order
// (gen_sequential) and keep the two potential half-steps on transform pairs of
// their own.  The rounding of such long FP32 sums is the same function of the
// data in every step, so it adds up: at P = 1198 (prime 599), 1150 points and
// 20 steps the other order alone moves the kinetic-energy sums by 6e-5 of the
// record, at primes up to 59 by less than 1e-5.  The line keeps results where they
// were; which order is nearer to 64 bits was not measured.  FP64 has no such limit.
constexpr int kGenSequentialAbove = 64;

// Stage s: radix ra * rb (rb = 1: one factor) on top of transforms of length
// ns = product of the earlier radices.
struct GenFactors {
  int n;
  int ra[kGenMaxStages], rb[kGenMaxStages], ns[kGenMaxStages];
  uint32_t mns[kGenMaxStages];  // multiplier of gen_div by ns
};

// t / d for t < 2^16, d <= 4096 (mul = ceil(2^32 / d); d = 1 has no multiplier)
inline uint32_t gen_mul(int d) { return d == 1 ? 0u : (uint32_t)((0x100000000ull + d - 1) / d); }
__device__ __forceinline__ int gen_div(int t, uint32_t mul) { return mul == 0 ? t : (int)__umulhi((uint32_t)t, mul); }

// wide: also the pairs whose 16 to 25 values per thread only FP32 holds in registers
GenFactors gen_factors(int N, bool wide) {
  int f[24], nf = 0, m = N;
  while (m % 4 == 0) { f[nf++] = 4; m /= 4; }
  for (int p = 2; m > 1; ++p)
    while (m % p == 0) { f[nf++] = p; m /= p; }
  GenFactors g{};
  int ns = 1;
  for (int i = 0; i < nf;) {
    const int a = f[i], b = i + 1 < nf ? f[i + 1] : 0;
    const bool pair = b != 0 && b <= 5 && a * b <= (wide ? 25 : 12);
    g.ra[g.n] = a;
    g.rb[g.n] = pair ? b : 1;
    g.ns[g.n] = ns;
    g.mns[g.n] = gen_mul(ns);
    ns *= a * g.rb[g.n];
    i += pair ? 2 : 1;
    ++g.n;
  }
  return g;
}

// Buffer slots of n elements x CP pairs, padded.
template <typename C> __host__ __device__ __forceinline__ int gen_slot(int s) {
  return s + (sizeof(C) == 16 ? s >> 3 : s >> 4);
}

// R-point transform in registers; for R = 7, 11, 13 cf[j] = exp(-2 pi i j / R), j <= (R-1)/2.
template <int R, int DIR, typename C> __device__ __forceinline__ void gen_dft(C* in, const C* cf) {
  using Rl = decltype(C::x);
  if constexpr (R == 2) {
    const C a = in[0], b = in[1];
    in[0] = cadd(a, b);
    in[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const C a0 = cadd(in[0], in[2]), a1 = csub(in[0], in[2]);
    const C b0 = cadd(in[1], in[3]), b1 = mul_i<DIR>(csub(in[1], in[3]));
    in[0] = cadd(a0, b0);
    in[1] = cadd(a1, b1);
    in[2] = csub(a0, b0);
    in[3] = csub(a1, b1);
  } else if constexpr (R == 3) {
    // exp(DIR 2 pi i / 3) = -1/2 + DIR i sqrt(3)/2
    const C s = cadd(in[1], in[2]), d = csub(in[1], in[2]);
    const C m = mk<C>(in[0].x - (Rl)0.5 * s.x, in[0].y - (Rl)0.5 * s.y);
    const C rot = mul_i<DIR>(cscale(d, (Rl)0.8660254037844386));
    in[0] = cadd(in[0], s);
    in[1] = cadd(m, rot);
    in[2] = csub(m, rot);
  } else if constexpr (R == 5) {
    // cos/sin of 2 pi/5 and 4 pi/5
    const Rl c1 = (Rl)0.30901699437494745, c2 = (Rl)-0.8090169943749475;
    const Rl s1 = (Rl)0.9510565162951535, s2 = (Rl)0.5877852522924731;
    const C t1 = cadd(in[1], in[4]), t2 = cadd(in[2], in[3]);
    const C t3 = csub(in[1], in[4]), t4 = csub(in[2], in[3]);
    const C a1 = mk<C>(in[0].x + c1 * t1.x + c2 * t2.x, in[0].y + c1 * t1.y + c2 * t2.y);
    const C a2 = mk<C>(in[0].x + c2 * t1.x + c1 * t2.x, in[0].y + c2 * t1.y + c1 * t2.y);
    const C b1 = mul_i<DIR>(mk<C>(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y));
    const C b2 = mul_i<DIR>(mk<C>(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y));
    in[0] = cadd(in[0], cadd(t1, t2));
    in[1] = cadd(a1, b1);
    in[4] = csub(a1, b1);
    in[2] = cadd(a2, b2);
    in[3] = csub(a2, b2);
  } else {
    constexpr int H = (R - 1) / 2;
    C s[H + 1], d[H + 1];
    C sum = in[0];
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      s[j] = cadd(in[j], in[R - j]);
      d[j] = csub(in[j], in[R - j]);
      sum = cadd(sum, s[j]);
    }
    const C x0 = in[0];
    in[0] = sum;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      C A = x0, B = mk<C>((Rl)0, (Rl)0);
#pragma unroll
      for (int j = 1; j <= H; ++j) {
        const int q = (j * k) % R, qq = q <= H ? q : R - q;
        A.x += s[j].x * cf[qq].x;
        A.y += s[j].y * cf[qq].x;
        const Rl w = q <= H ? cf[qq].y : -cf[qq].y;
        B.x += d[j].x * w;
        B.y += d[j].y * w;
      }
      const C iB = DIR < 0 ? mk<C>(-B.y, B.x) : mk<C>(B.y, -B.x);
      in[k] = cadd(A, iB);
      in[R - k] = csub(A, iB);
    }
  }
}

template <int DIR, typename C> __device__ __forceinline__ C gen_tw(const C* tw, int i) {
  const C w = tw[i];
  return DIR > 0 ? cconj(w) : w;
}

// One Stockham stage of radix R = RA * RB from x to y: butterfly t with
// k = t mod ns reads elements t + r N/R and writes (t / ns) ns R + k + s ns.
// RB > 1 is the radix-RA stage followed by the radix-RB stage (whose
// transforms have length ns RA), both in registers: sub-butterfly q of the
// first takes elements q, q + RB, ... and its output s feeds the second
// stage's butterfly s, with the twiddles of index k + s ns.
template <int RA, int RB, int DIR, typename C>
__device__ __forceinline__ void gen_stage_r(const C* x, C* y, int N, int ns, uint32_t mns, int lcp, const C* tw) {
  constexpr int R = RA * RB;
  constexpr int H = RA > 5 ? (RA - 1) / 2 : 0;
  C cf[H + 1];
#pragma unroll
  for (int j = 1; j <= H; ++j) cf[j] = tw[j * (N / RA)];
  const int nb = N / R, total = nb << lcp;
  const int ta = N / (ns * RA), tb = nb / ns;  // twiddle index steps of the two stages
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int c = idx & ((1 << lcp) - 1), t = idx >> lcp;
    const int blk = gen_div(t, mns), k = t - blk * ns;
    C v[RB][RA];
#pragma unroll
    for (int q = 0; q < RB; ++q)
#pragma unroll
      for (int r = 0; r < RA; ++r) v[q][r] = x[gen_slot<C>(((t + (q + r * RB) * nb) << lcp) + c)];
    if (ns > 1) {
#pragma unroll
      for (int r = 1; r < RA; ++r) {
        const C w = gen_tw<DIR>(tw, k * r * ta);
#pragma unroll
        for (int q = 0; q < RB; ++q) v[q][r] = cmul(v[q][r], w);
      }
    }
#pragma unroll
    for (int q = 0; q < RB; ++q) gen_dft<RA, DIR>(v[q], cf);
    const int o = blk * ns * R + k;
#pragma unroll
    for (int s = 0; s < RA; ++s) {
      C u[RB];
#pragma unroll
      for (int q = 0; q < RB; ++q) u[q] = q == 0 ? v[q][s] : cmul(v[q][s], gen_tw<DIR>(tw, (k + s * ns) * q * tb));
      if constexpr (RB > 1) gen_dft<RB, DIR>(u, cf);
#pragma unroll
      for (int q = 0; q < RB; ++q) y[gen_slot<C>(((o + (s + q * RA) * ns) << lcp) + c)] = u[q];
    }
  }
}

// A stage of large prime radix R (see above): first the sums and differences
// of mirrored inputs, in place in x, then outputs k and R - k into y from KT
// values of k and V butterflies per thread (register tile: a coefficient
// serves V butterflies, an input KT outputs).
template <int DIR, int KT, int V, typename C>
__device__ __forceinline__ void gen_direct(C* x, C* y, int N, int R, int ns, uint32_t mns, int lcp, const C* tw) {
  using Rl = decltype(C::x);
  const int nb = N / R, ncol = nb << lcp, h = (R - 1) / 2, ts = nb / ns;
  for (int idx = threadIdx.x; idx < ncol * h; idx += blockDim.x) {
    const int j = idx / ncol + 1, col = idx - (j - 1) * ncol, t = col >> lcp;
    const int k = t - gen_div(t, mns) * ns;
    C* pa = x + gen_slot<C>(col + j * ncol);
    C* pb = x + gen_slot<C>(col + (R - j) * ncol);
    C a = *pa, b = *pb;
    if (ns > 1) {
      a = cmul(a, gen_tw<DIR>(tw, k * j * ts));
      b = cmul(b, gen_tw<DIR>(tw, k * (R - j) * ts));
    }
    *pa = cadd(a, b);
    *pb = csub(a, b);
  }
  __syncthreads();
  const int nkg = (h + KT) / KT, ncg = (ncol + V - 1) / V;  // outputs k = 0 .. h
  for (int idx = threadIdx.x; idx < nkg * ncg; idx += blockDim.x) {
    const int kg = idx / ncg, cg = idx - kg * ncg;
    int col[V], ix[KT], sk[KT];
    C A[KT][V], B[KT][V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      col[v] = cg + v * ncg < ncol ? cg + v * ncg : cg;
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        A[q][v] = x[gen_slot<C>(col[v])];
        B[q][v] = mk<C>((Rl)0, (Rl)0);
      }
    }
#pragma unroll
    for (int q = 0; q < KT; ++q) {
      const int k = kg * KT + q;
      sk[q] = (k <= h ? k : 0) * nb;
      ix[q] = 0;
    }
#pragma unroll 2
    for (int j = 1; j <= h; ++j) {
      C w[KT];
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        ix[q] += sk[q];
        if (ix[q] >= N) ix[q] -= N;
        w[q] = tw[ix[q]];
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const C s = x[gen_slot<C>(col[v] + j * ncol)], d = x[gen_slot<C>(col[v] + (R - j) * ncol)];
#pragma unroll
        for (int q = 0; q < KT; ++q) {
          A[q][v].x += s.x * w[q].x;
          A[q][v].y += s.y * w[q].x;
          B[q][v].x += d.x * w[q].y;
          B[q][v].y += d.y * w[q].y;
        }
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (cg + v * ncg >= ncol) continue;
      const int t = col[v] >> lcp, c = col[v] & ((1 << lcp) - 1);
      const int blk = gen_div(t, mns), o = blk * ns * R + t - blk * ns;
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        const int k = kg * KT + q;
        if (k > h) continue;
        const C iB = DIR < 0 ? mk<C>(-B[q][v].y, B[q][v].x) : mk<C>(B[q][v].y, -B[q][v].x);
        y[gen_slot<C>(((o + k * ns) << lcp) + c)] = cadd(A[q][v], iB);
        if (k > 0) y[gen_slot<C>(((o + (R - k) * ns) << lcp) + c)] = csub(A[q][v], iB);
      }
    }
  }
}

// The same stage with every output's R terms summed in index order (4 R^2
// multiply-adds): the twiddles in place in x first, then KT outputs of V
// butterflies per thread.
template <int DIR, int KT, int V, typename C>
__device__ __forceinline__ void gen_sequential(C* x, C* y, int N, int R, int ns, uint32_t mns, int lcp, const C* tw) {
  using Rl = decltype(C::x);
  const int nb = N / R, ncol = nb << lcp, ts = nb / ns;
  if (ns > 1) {
    for (int idx = threadIdx.x + ncol; idx < ncol * R; idx += blockDim.x) {
      const int r = idx / ncol, t = (idx - r * ncol) >> lcp;
      C* pa = x + gen_slot<C>(idx);
      *pa = cmul(*pa, gen_tw<DIR>(tw, (t - gen_div(t, mns) * ns) * r * ts));
    }
    __syncthreads();
  }
  const int nkg = (R + KT - 1) / KT, ncg = (ncol + V - 1) / V;
  for (int idx = threadIdx.x; idx < nkg * ncg; idx += blockDim.x) {
    const int kg = idx / ncg, cg = idx - kg * ncg;
    int col[V], ix[KT], sk[KT];
    C acc[KT][V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      col[v] = cg + v * ncg < ncol ? cg + v * ncg : cg;
#pragma unroll
      for (int q = 0; q < KT; ++q) acc[q][v] = mk<C>((Rl)0, (Rl)0);
    }
#pragma unroll
    for (int q = 0; q < KT; ++q) {
      const int k = kg * KT + q;
      sk[q] = (k < R ? k : 0) * nb;
      ix[q] = 0;
    }
#pragma unroll 2
    for (int r = 0; r < R; ++r) {
      C w[KT];
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        w[q] = gen_tw<DIR>(tw, ix[q]);
        ix[q] += sk[q];
        if (ix[q] >= N) ix[q] -= N;
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const C u = x[gen_slot<C>(col[v] + r * ncol)];
#pragma unroll
        for (int q = 0; q < KT; ++q) acc[q][v] = cadd(acc[q][v], cmul(u, w[q]));
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (cg + v * ncg >= ncol) continue;
      const int t = col[v] >> lcp, c = col[v] & ((1 << lcp) - 1);
      const int blk = gen_div(t, mns), o = blk * ns * R + t - blk * ns;
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        const int k = kg * KT + q;
        if (k < R) y[gen_slot<C>(((o + k * ns) << lcp) + c)] = acc[q][v];
      }
    }
  }
}

// Forward (DIR < 0) or unnormalised inverse transform of z, natural order in
// and out; z2 is the other buffer (the two are exchanged stage by stage).
template <int DIR, typename C>
__device__ __forceinline__ void gen_fft(C*& z, C*& z2, int N, const GenFactors& g, int lcp, const C* tw) {
  for (int s = 0; s < g.n; ++s) {
    const int ns = g.ns[s], ra = g.ra[s];
    const uint32_t mns = g.mns[s];
#define GEN_R(A, B) case A * 32 + B: gen_stage_r<A, B, DIR, C>(z, z2, N, ns, mns, lcp, tw); break;
    switch (ra * 32 + g.rb[s]) {
      GEN_R(2, 1) GEN_R(3, 1) GEN_R(4, 1) GEN_R(5, 1) GEN_R(7, 1) GEN_R(11, 1) GEN_R(13, 1)
      GEN_R(4, 2) GEN_R(4, 3) GEN_R(2, 3) GEN_R(2, 5) GEN_R(3, 3)
      case 4 * 32 + 4: if constexpr (sizeof(C) == 8) gen_stage_r<4, 4, DIR, C>(z, z2, N, ns, mns, lcp, tw); break;
      case 4 * 32 + 5: if constexpr (sizeof(C) == 8) gen_stage_r<4, 5, DIR, C>(z, z2, N, ns, mns, lcp, tw); break;
      case 3 * 32 + 5: if constexpr (sizeof(C) == 8) gen_stage_r<3, 5, DIR, C>(z, z2, N, ns, mns, lcp, tw); break;
      case 5 * 32 + 5: if constexpr (sizeof(C) == 8) gen_stage_r<5, 5, DIR, C>(z, z2, N, ns, mns, lcp, tw); break;
      default: {
        // one output pair per thread while that keeps the CTA's threads busy, else the 4 x 2 register tile
        const int tasks = ((ra + 1) / 2) * ((N / ra) << lcp);
        if (sizeof(C) == 8 && ra > kGenSequentialAbove) {
          if constexpr (sizeof(C) == 8) {
            if (tasks <= 2 * (int)blockDim.x) gen_sequential<DIR, 1, 1, C>(z, z2, N, ra, ns, mns, lcp, tw);
            else gen_sequential<DIR, 4, 2, C>(z, z2, N, ra, ns, mns, lcp, tw);
          }
        } else if (tasks <= 4 * (int)blockDim.x) gen_direct<DIR, 1, 1, C>(z, z2, N, ra, ns, mns, lcp, tw);
        else gen_direct<DIR, 4, 2, C>(z, z2, N, ra, ns, mns, lcp, tw);
      }
    }
#undef GEN_R
    __syncthreads();
    C* t = z;
    z = z2;
    z2 = t;
  }
}

// Factors of bin kk <= N/2 of a pair: table entries at ta, tb (element
// offsets), times g[kk], real at kk = 0 and N/2.
template <typename Rl>
__device__ __forceinline__ void gen_factors_at(const void* tab, size_t ia, size_t ib, int real, const void* g, int kk,
                                               int N, cplx_t<Rl>& ea, cplx_t<Rl>& eb) {
  using C = cplx_t<Rl>;
  ea = tab_load<Rl>(tab, real, ia);
  eb = tab_load<Rl>(tab, real, ib);
  if (g != nullptr) {
    const C gk = __ldg(reinterpret_cast<const C*>(g) + kk);
    ea = cmul(ea, gk);
    eb = cmul(eb, gk);
  }
  ea = herm(ea, kk, N);
  eb = herm(eb, kk, N);
}

// Multiply both bins of every pair (k, N - k): mul(kk, c, A, Bi) turns
// A = Z_k + conj Z_(N-k) and Bi = Z_k - conj Z_(N-k) (twice the spectrum of the
// first sequence, 2i times that of the second) into their products X, Y; bin k
// becomes f (X + Y) and bin N - k becomes f conj(X - Y).
template <typename C, typename Mul>
__device__ __forceinline__ void gen_pair_mul(C* z, int N, int lcp, decltype(C::x) f, Mul mul) {
  const int total = (N / 2 + 1) << lcp;
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int c = idx & ((1 << lcp) - 1), k = idx >> lcp;
    const bool self = k == 0 || 2 * k == N;
    C* zk = z + gen_slot<C>(idx);
    C* zn = self ? zk : z + gen_slot<C>(((N - k) << lcp) + c);
    const C Zk = *zk, Zc = cconj(*zn);
    C X = cadd(Zk, Zc), Y = csub(Zk, Zc);
    mul(k, c, X, Y);
    *zk = cscale(cadd(X, Y), f);
    if (!self) *zn = cconj(cscale(csub(X, Y), f));
  }
  __syncthreads();
}

// Elements ld(i, c) of the CTA's pairs into z, or st(i, c, value) of each.
template <typename C, typename Ld> __device__ __forceinline__ void gen_fill(C* z, int N, int lcp, Ld ld) {
#pragma unroll 4
  for (int idx = threadIdx.x; idx < N << lcp; idx += blockDim.x)
    z[gen_slot<C>(idx)] = ld(idx >> lcp, idx & ((1 << lcp) - 1));
  __syncthreads();
}
template <typename C, typename St> __device__ __forceinline__ void gen_drain(const C* z, int N, int lcp, St st) {
#pragma unroll 4
  for (int idx = threadIdx.x; idx < N << lcp; idx += blockDim.x)
    st(idx >> lcp, idx & ((1 << lcp) - 1), z[gen_slot<C>(idx)]);
}

// Block-wide FP64 sums of NV values per thread, in thread 0.
template <int NV> __device__ __forceinline__ void gen_block_sum(double (&v)[NV], double (*red)[NV]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) red[w][q] = v[q];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double s = 0.0;
      for (int i = 0; i < nw; ++i) s += red[i][q];
      v[q] = s;
    }
}

template <typename Rl>
__global__ void __launch_bounds__(kGenThreads, gen_minb<Rl>()) gen_row_kernel(PassArgs a, GenFactors g, int lcp) {
  using C = cplx_t<Rl>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[34];
  const int N = a.X, b = blockIdx.y;
  C* tw = reinterpret_cast<C*>(smem_raw);
  C* z = tw + N;
  C* z2 = z + gen_slot<C>(N << lcp) + 1;
  dep_sync();
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = __ldg(reinterpret_cast<const C*>(a.tw) + i);
  const Rl s = (Rl)prev_scale(a, b, red, blockIdx.x == 0);
  __syncthreads();
  const int rp0 = blockIdx.x << lcp, np = a.P / 2;
  Rl* W = reinterpret_cast<Rl*>(a.W) + (size_t)b * a.w_bs;
  gen_fill(z, N, lcp, [&](int x, int c) {
    if (rp0 + c >= np) return mk<C>((Rl)0, (Rl)0);
    const Rl* w = W + (size_t)(2 * (rp0 + c)) * N + x;
    return mk<C>(__ldcg(w) * s, __ldcg(w + N) * s);
  });
  gen_fft<-1>(z, z2, N, g, lcp, tw);
  const size_t hs = N / 2 + 1;
  const char* tab = reinterpret_cast<const char*>(a.tab1) + (size_t)b * a.tab_bs * (a.tab_real ? sizeof(Rl) : sizeof(C));
  gen_pair_mul(z, N, lcp, (Rl)(a.out_scale * 0.5 / (double)N), [&](int kk, int c, C& X, C& Y) {
    if (rp0 + c >= np) return;
    C ea, eb;
    const size_t i = (size_t)(2 * (rp0 + c)) * hs + kk;
    gen_factors_at<Rl>(tab, i, i + hs, a.tab_real, a.g1, kk, N, ea, eb);
    X = cmul(X, ea);
    Y = cmul(Y, eb);
  });
  gen_fft<+1>(z, z2, N, g, lcp, tw);
  gen_drain(z, N, lcp, [&](int x, int c, C v) {
    if (rp0 + c >= np) return;
    Rl* w = W + (size_t)(2 * (rp0 + c)) * N + x;
    w[0] = v.x;
    w[N] = v.y;
  });
}

// Column pass (see PassArgs): one half-step, two around the real-space
// mid-point (mask, blend, observables), or (fuse_mid) two on one transform
// pair with the observables from the mid-point spectrum.
template <typename Rl>
__global__ void __launch_bounds__(kGenThreads, gen_minb<Rl>()) gen_col_kernel(PassArgs a, GenFactors g, int lcp) {
  using C = cplx_t<Rl>;
  using V2 = typename Vec2<Rl>::type;
  constexpr int NV = 2 + 2 * MAXO;  // sum, sum of squares, x-weights, p-weights
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[34];
  __shared__ double ored[kGenThreads / 32][NV];
  const int N = a.P, X = a.X, b = blockIdx.y;
  C* tw = reinterpret_cast<C*>(smem_raw);
  C* z = tw + N;
  C* z2 = z + gen_slot<C>(N << lcp) + 1;
  dep_sync();
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = __ldg(reinterpret_cast<const C*>(a.tw) + i);
  const Rl s = (Rl)prev_scale(a, b, red, blockIdx.x == 0);
  __syncthreads();
  const int x0 = blockIdx.x << (lcp + 1);  // first column of the tile
  Rl* W = reinterpret_cast<Rl*>(a.W) + (size_t)b * a.w_bs;
  const Rl* S0 = reinterpret_cast<const Rl*>(a.s0) + (a.s0 != nullptr ? (size_t)b * a.s0_bs : 0);
  const Rl bc = (Rl)a.blend_c;
  const size_t tb0 = (size_t)b * a.tab_bs;
  // X is even: a column pair is one vector wherever the instance starts on one
  auto vec = [](const Rl* base) { return (reinterpret_cast<uintptr_t>(base) & (sizeof(V2) - 1)) == 0; };
  auto pair_at = [&](const Rl* base, int p, int c) {
    const Rl* q = base + (size_t)p * X + x0 + 2 * c;
    if (!vec(base)) return mk<C>(q[0], q[1]);
    const V2 w = *reinterpret_cast<const V2*>(q);
    return mk<C>(w.x, w.y);
  };
  auto load = [&](int p, int c) {
    if (x0 + 2 * c >= X) return mk<C>((Rl)0, (Rl)0);
    C v = cscale(pair_at(W, p, c), s);
    if (a.blend_pre) {
      const C w0 = pair_at(S0, p, c);
      v = mk<C>(bc * v.x + w0.x, bc * v.y + w0.y);
    }
    return v;
  };
  const Rl os = (Rl)a.out_scale;
  auto store = [&](int p, int c, C v) {
    if (x0 + 2 * c >= X) return;
    Rl* q = W + (size_t)p * X + x0 + 2 * c;
    if (!vec(W)) {
      q[0] = v.x * os;
      q[1] = v.y * os;
      return;
    }
    V2 w;
    w.x = v.x * os;
    w.y = v.y * os;
    *reinterpret_cast<V2*>(q) = w;
  };
  auto factors = [&](const void* tab, const void* gv, int kk, int c, C& ea, C& eb) {
    const size_t i = tb0 + (size_t)kk * X + x0 + 2 * c;
    gen_factors_at<Rl>(tab, i, i + 1, a.tab_real, gv, kk, N, ea, eb);
  };
  const bool obs = a.part_out != nullptr;
  double acc[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) acc[q] = 0.0;
  // x-weighted sums of a column pair with sums ca, cb
  auto add_x = [&](int c, double ca, double cb) {
    const double* wx = a.wx + (size_t)b * a.wx_bs + x0 + 2 * c;
    acc[0] += ca + cb;
#pragma unroll
    for (int q = 0; q < MAXO; ++q)
      if (q < a.Mx) acc[2 + q] += ca * wx[(size_t)q * X] + cb * wx[(size_t)q * X + 1];
  };
  auto write_obs = [&] {
    gen_block_sum<NV>(acc, ored);
    if (threadIdx.x == 0) {
      double* rec = a.part_out + ((size_t)b * gridDim.x + blockIdx.x) * a.M;
      rec[0] = acc[0];
      rec[1] = acc[1];
#pragma unroll
      for (int q = 0; q < MAXO; ++q) {
        if (q < a.Mx) rec[2 + q] = acc[2 + q];
        if (q < a.Mp) rec[2 + a.Mx + q] = acc[2 + MAXO + q];
      }
    }
  };
  if (a.fuse_mid) {
    const double2* G = reinterpret_cast<const double2*>(a.wph) + (size_t)b * a.wph_bs;
    const bool same = a.tab1 == a.tab2 && a.g1 == a.g2;
    gen_fill(z, N, lcp, load);
    gen_fft<-1>(z, z2, N, g, lcp, tw);
    gen_pair_mul(z, N, lcp, (Rl)(0.5 / (double)N), [&](int kk, int c, C& A, C& Bi) {
      if (x0 + 2 * c >= X) return;
      C ea, eb;
      factors(a.tab1, a.g1, kk, c, ea, eb);
      A = cmul(A, ea);   // 2 x the spectra at the mid-point
      Bi = cmul(Bi, eb);
      if (obs) {
        const bool nyq = 2 * kk == N, self = kk == 0 || nyq;
        const double wgt = self ? 1.0 : 2.0;  // bins k and N - k
        const double ax = A.x, ay = A.y, bx = Bi.x, by = Bi.y;
        acc[1] += wgt * (ax * ax + ay * ay + bx * bx + by * by);
        if (kk == 0) add_x(c, 0.5 * ax, 0.5 * by);
        const double ux = wgt * (ax + by), uy = self ? 0.0 : wgt * (ay - bx);
#pragma unroll
        for (int q = 0; q < MAXO; ++q)
          if (q < a.Mp) {
            const double2 gk = __ldg(G + q * (N / 2) + (nyq ? 0 : kk));
            acc[2 + MAXO + q] += ux * (nyq ? gk.y : gk.x) + uy * gk.y;
          }
      }
      if (!same) factors(a.tab2, a.g2, kk, c, ea, eb);
      A = cmul(A, ea);
      Bi = cmul(Bi, eb);
    });
    if (obs) {
      acc[1] *= 0.25 / (double)N;
#pragma unroll
      for (int q = 0; q < MAXO; ++q) acc[2 + MAXO + q] *= 0.5 / (double)N;
      write_obs();
    }
    gen_fft<+1>(z, z2, N, g, lcp, tw);
    gen_drain(z, N, lcp, store);
    return;
  }
  const Rl f = (Rl)(0.5 / (double)N);
  const bool mid = a.bxp != nullptr || a.blend_post || obs || a.tab1 == nullptr;
  if (a.tab1 != nullptr) {
    gen_fill(z, N, lcp, load);
    gen_fft<-1>(z, z2, N, g, lcp, tw);
    gen_pair_mul(z, N, lcp, f, [&](int kk, int c, C& A, C& Bi) {
      if (x0 + 2 * c >= X) return;
      C ea, eb;
      factors(a.tab1, a.g1, kk, c, ea, eb);
      A = cmul(A, ea);
      Bi = cmul(Bi, eb);
    });
    gen_fft<+1>(z, z2, N, g, lcp, tw);
    if (!mid && a.tab2 == nullptr) {
      gen_drain(z, N, lcp, store);
      return;
    }
  }
  const Rl* Bm = reinterpret_cast<const Rl*>(a.bxp) + (a.bxp != nullptr ? (size_t)b * a.bxp_bs : 0);
  const double* wp = a.wp + (a.wp != nullptr ? (size_t)b * a.wp_bs : 0);
  if (mid) {
    // a thread keeps one column pair: blockDim is a multiple of CP
    const int c = threadIdx.x & ((1 << lcp) - 1);
    double ca = 0.0, cb = 0.0;
    if (x0 + 2 * c < X)
      for (int p = threadIdx.x >> lcp; p < N; p += blockDim.x >> lcp) {
        C v = a.tab1 != nullptr ? z[gen_slot<C>((p << lcp) + c)] : load(p, c);
        if (a.bxp != nullptr) {
          const C w = pair_at(Bm, p, c);
          v = mk<C>(v.x * w.x, v.y * w.y);
        }
        if (a.blend_post) {
          const C w0 = pair_at(S0, p, c);
          v = mk<C>(bc * v.x + w0.x, bc * v.y + w0.y);
        }
        if (obs) {
          const double wa = (double)v.x, wb = (double)v.y;
          ca += wa;
          cb += wb;
          acc[1] += wa * wa + wb * wb;
#pragma unroll
          for (int q = 0; q < MAXO; ++q)
            if (q < a.Mp) acc[2 + MAXO + q] += (wa + wb) * __ldg(wp + (size_t)q * N + p);
        }
        if (a.tab2 == nullptr) store(p, c, v);
        else z[gen_slot<C>((p << lcp) + c)] = v;
      }
    if (obs) {
      if (x0 + 2 * c < X) add_x(c, ca, cb);
      write_obs();
    }
    if (a.tab2 == nullptr) return;
    __syncthreads();
  }
  gen_fft<-1>(z, z2, N, g, lcp, tw);
  gen_pair_mul(z, N, lcp, f, [&](int kk, int c, C& A, C& Bi) {
    if (x0 + 2 * c >= X) return;
    C ea, eb;
    factors(a.tab2, a.g2, kk, c, ea, eb);
    A = cmul(A, ea);
    Bi = cmul(Bi, eb);
  });
  gen_fft<+1>(z, z2, N, g, lcp, tw);
  gen_drain(z, N, lcp, store);
}

// Spectra of the p-observable weights for the fused generic pass: block (q, b)
// transforms vector q of instance b in FP64, twiddles from sincospi of the exact
// ratio.  They stay FP64 whatever the state's precision, so that an FP32 pass
// weighs its spectra as exactly as it would its values: bins k < P/2 as
// out[b][q][k], the real value at P/2 in the imaginary part of bin 0, which is
// real too (the bytes of P complex FP32 entries a weight).
__global__ void __launch_bounds__(kGenThreads) gen_pweight_kernel(const double* wp, long long wp_bs, int P, double2* out,
                                                                  long long out_bs, GenFactors g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* tw = reinterpret_cast<double2*>(smem_raw);
  double2* z = tw + P;
  double2* z2 = z + gen_slot<double2>(P) + 1;
  const int q = blockIdx.x, b = blockIdx.y;
  dep_sync();
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    double sn, cs;
    sincospi(-2.0 * (double)i / (double)P, &sn, &cs);
    tw[i] = make_double2(cs, sn);
  }
  __syncthreads();
  const double* w = wp + (size_t)b * wp_bs + (size_t)q * P;
  gen_fill(z, P, 0, [&](int p, int) { return make_double2(w[p], 0.0); });
  gen_fft<-1>(z, z2, P, g, 0, tw);
  double2* o = out + (size_t)b * out_bs + (size_t)q * (P / 2);
  for (int k = threadIdx.x; k < P / 2; k += blockDim.x) {
    const double2 v = z[gen_slot<double2>(k)];
    o[k] = k > 0 ? v : make_double2(v.x, z[gen_slot<double2>(P / 2)].x);
  }
}

// ---------------------------------------------------------------------------
// Shared memory of one CTA: twiddles and two padded buffers.
template <typename C> static size_t gen_smem(int N, int lcp) {
  return sizeof(C) * ((size_t)N + 2 * (size_t)(gen_slot<C>(N << lcp) + 1));
}

// Pairs per CTA (as a power of two, the exponent): enough that a row of the
// tile fills the sectors it touches, as long as the CTAs of gen_minb fit an SM
// and the launch has two CTAs per SM (4 x 1000 x 1000 FP32: 101 us a step with
// two pairs and four CTAs, 112 with four pairs and two CTAs).
static int gen_lcp(int dtype, int N, int pairs, int batch) {
  auto smem = [&](int l) { return dtype == FW_F64 ? gen_smem<double2>(N, l) : gen_smem<float2>(N, l); };
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int l = dtype == FW_F64 ? 2 : 3;
  while (l > 0 && (smem(l) > (dtype == FW_F64 ? kGenSmem64 : kGenSmem32) ||
                   (long long)((pairs + (1 << l) - 1) >> l) * batch < 2LL * sms))
    --l;
  return l;
}

// Whether a column pass of length P may run both potential half-steps on one transform pair.
bool gen_fuses(int dtype, int P) {
  const GenFactors g = gen_factors(P, true);
  return dtype == FW_F64 || g.ra[g.n - 1] <= kGenSequentialAbove;
}

int gen_col_parts(int dtype, int P, int X, int batch) {
  const int l = gen_lcp(dtype, P, X / 2, batch);
  return (X / 2 + (1 << l) - 1) >> l;
}

template <typename Rl>
static cudaError_t gen_launch(const PassArgs& a, int dtype, bool row, cudaStream_t st, int* nparts) {
  const int N = row ? a.X : a.P, pairs = (row ? a.P : a.X) / 2;
  const GenFactors g = gen_factors(N, dtype == FW_F32);
  const int l = gen_lcp(dtype, N, pairs, a.batch);
  const size_t smem = gen_smem<cplx_t<Rl>>(N, l);
  // the attribute is the largest dynamic shared memory any launch of the
  // kernel may use (N up to 4096), not this launch's
  const size_t smem_max = gen_smem<cplx_t<Rl>>(4096, 0);
  const int tiles = (pairs + (1 << l) - 1) >> l;
  // about four elements per thread, a multiple of the warp (and of CP)
  int thr = ((N << l) / 4 + 31) / 32 * 32;
  if (thr < 128) thr = 128;
  if (thr > kGenThreads) thr = kGenThreads;
  if (row) {
    static PerDeviceOnce attr;
    cudaError_t e = set_smem_once(attr, gen_row_kernel<Rl>, smem_max);
    if (e != cudaSuccess) return e;
    return launch_dep(a.dep, gen_row_kernel<Rl>, dim3(tiles, a.batch), thr, smem, st, a, g, l);
  } else {
    static PerDeviceOnce attr;
    cudaError_t e = set_smem_once(attr, gen_col_kernel<Rl>, smem_max);
    if (e != cudaSuccess) return e;
    if (nparts) *nparts = tiles;
    return launch_dep(a.dep, gen_col_kernel<Rl>, dim3(tiles, a.batch), thr, smem, st, a, g, l);
  }
}

cudaError_t launch_generic_row(const PassArgs& a, int dtype, cudaStream_t st) {
  return dtype == FW_F32 ? gen_launch<float>(a, dtype, true, st, nullptr) : gen_launch<double>(a, dtype, true, st, nullptr);
}

cudaError_t launch_generic_col(const PassArgs& a, int dtype, cudaStream_t st, int* nparts) {
  return dtype == FW_F32 ? gen_launch<float>(a, dtype, false, st, nparts) : gen_launch<double>(a, dtype, false, st, nparts);
}

cudaError_t launch_generic_pweight(const double* wp, long long wp_bs, int Mp, int P, int nb, void* out,
                                   long long out_bs, int dep, cudaStream_t st) {
  const GenFactors g = gen_factors(P, false);
  static PerDeviceOnce attr;
  cudaError_t e = set_smem_once(attr, gen_pweight_kernel, gen_smem<double2>(4096, 0));
  if (e != cudaSuccess) return e;
  return launch_dep(dep, gen_pweight_kernel, dim3(Mp, nb), kGenThreads, gen_smem<double2>(P, 0), st, wp, wp_bs, P, out,
                    out_bs, g);
}

}  // namespace fw
