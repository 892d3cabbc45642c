// Closed-shell (T) on the GPU (RCCSD_TriplesCorrection, SCESS src/Quantum/CC/RCCSD_T.cpp:17-168).
//
// The virtuals are cut into blocks of nb.  For every block triple A >= B >= C
// the symmetrised connected triples W^{abc}_{ijk} (a in A, b in B, c in C) are
// accumulated in one buffer W[(a,b,c)][i,j,k] by 12 GEMMs: for each of the six
// simultaneous permutations of (ia),(jb),(kc) of Symmetrise (:78-106) the raw
//   w^{xyz}_{i'j'k'} = sum_f P(i',f,x,y) Q(f,j',k',z) - sum_m R(i',j',m,x) t2(m,k',y,z)
// of GetW (:62-68) is one (o nb^2) x (o^2 nb) x v GEMM plus one
// (o^2 nb) x (o nb^2) x o GEMM whose epilogue adds it to W at the permuted
// position, so no Symmetrise scratch copy exists.  An energy kernel then
// evaluates, per unique triple a >= b >= c of the block, V (GetV :70-75),
// Y = W + V, r3(Y), the denominators and the degeneracy (:135-157) and writes
// one partial energy per triple; a fixed-order reduction gives 2 * sum (:167).
//
// Both forms regroup the 12 products into three sets of four K segments, one grouped
// launch per block triple.  FP64 form: the slice GEMM (gemm_slice.h) writes three FP64
// buffers, kept within L2, that the energy kernel adds (12 DFMA GEMMs into one W where
// the sliced packs don't fit the device); FP64 energy arithmetic.  MIXED form: the
// epilogues of the tcgen05 GEMM add the groups into one FP32 W with L2 reductions, so
// that W (nb^3 o^3 floats, 55 MB at o = 20) stays in L2 between the launch and the energy
// kernel; the operands are packed once per call into FP16 hi/lo rows grouped
// by block.  The energy kernel reads W once, clears it for the next block
// triple and works in FP32 per element with denominators formed from the FP64
// orbital energies in double-float, compensated sums and FP64 per triple.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "gemm_slice.h"
#include "gemm_tc.h"
#include "launch.cuh"
#include "slice_math.cuh"
#include "triples.h"

namespace scess {

namespace {

__host__ __device__ inline int64_t triple_id(int64_t a, int64_t b, int64_t c) {
  return a * (a + 1) * (a + 2) / 6 + b * (b + 1) / 2 + c;
}

// x / y: fast FP32 division in the mixed form (2 ulp), IEEE division in FP64.
__device__ __forceinline__ double div_fast(double x, double y) { return x / y; }

// One CTA per local triple (a_l, b_l, c_l) of the block triple (A, B, C).
// Shared memory: Y (o^3) then Sbc, Sac, Sab (o^2 each) then t1 columns and the
// occupied orbital energies (o each), all in the arithmetic type CT.
template <typename WT, typename CT>
__global__ void __launch_bounds__(256) triples_energy_kernel(
    const WT *__restrict__ W, int64_t o, int64_t v, int64_t nb, int64_t A, int64_t Bk, int64_t C,
    const double *__restrict__ eps, const double *__restrict__ t1, const double *__restrict__ S,
    double *__restrict__ energies) {
  const int64_t al = blockIdx.x / (nb * nb), bl = (blockIdx.x / nb) % nb, cl = blockIdx.x % nb;
  const int64_t a = A * nb + al, b = Bk * nb + bl, c = C * nb + cl;
  if (a >= v || b >= v || c >= v || b > a || c > b) return;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  __shared__ double red[32];
  const int oo = (int)o, o2 = oo * oo, o3 = o2 * oo;
  // Y(i,j,k) at i + p1 j + p2 k with odd p1, p2: the six permuted reads of r3
  // walk consecutive i with strides 1, p1 or p2, all free of bank conflicts.
  const int p1 = oo | 1, p2 = (p1 * oo) | 1;
  CT *Y = reinterpret_cast<CT *>(sm_raw);
  CT *Sbc = Y + p2 * oo, *Sac = Sbc + o2, *Sab = Sac + o2;
  CT *ta = Sab + o2, *tb = ta + oo, *tc = tb + oo, *eo = tc + oo;
  const WT *Wt = W + ((al * nb + bl) * nb + cl) * (int64_t)o3;
  // S(i,j,a,b) = (ia|jb) at i + o j + o^2 (a + v b)
  for (int e = threadIdx.x; e < o2; e += blockDim.x) {
    Sbc[e] = (CT)S[e + o2 * (b + v * c)];
    Sac[e] = (CT)S[e + o2 * (a + v * c)];
    Sab[e] = (CT)S[e + o2 * (a + v * b)];
  }
  for (int i = threadIdx.x; i < oo; i += blockDim.x) {
    ta[i] = (CT)t1[i + o * a];
    tb[i] = (CT)t1[i + o * b];
    tc[i] = (CT)t1[i + o * c];
    eo[i] = (CT)eps[i];
  }
  __syncthreads();
  // element e = i + o j + o^2 k; thread t visits e = t, t + 256, ... with
  // incrementally maintained (i, j, k)
  const int di = 256 % oo, dj = (256 / oo) % oo, dk = 256 / o2;
  const int i0 = (int)threadIdx.x % oo, j0 = ((int)threadIdx.x / oo) % oo, k0 = (int)threadIdx.x / o2;
  {
    int i = i0, j = j0, k = k0;
    for (int e = threadIdx.x; e < o3; e += 256) {
      // V_ijk = t1_ia (jb|kc) + t1_jb (ia|kc) + t1_kc (ia|jb)   (GetV + Symmetrise)
      Y[i + p1 * j + p2 * k] =
          (CT)Wt[e] + ta[i] * Sbc[j + oo * k] + tb[j] * Sac[i + oo * k] + tc[k] * Sab[i + oo * j];
      i += di;
      int cj = 0;
      if (i >= oo) { i -= oo; cj = 1; }
      j += dj + cj;
      int ck = 0;
      if (j >= oo) { j -= oo; ck = 1; }
      k += dk + ck;
    }
  }
  __syncthreads();
  const CT evirt = (CT)(eps[o + a] + eps[o + b] + eps[o + c]);
  double acc = 0.0;
  CT part = 0;
  int cnt = 0;
  int i = i0, j = j0, k = k0;
  for (int e = threadIdx.x; e < o3; e += 256) {
    // r3(Y) = 4 Y_ijk + Y_kij + Y_jki - 2 Y_kji - 2 Y_ikj - 2 Y_jik               :152-154
    const CT r3 = (CT)4 * Y[i + p1 * j + p2 * k] + Y[k + p1 * i + p2 * j] +
                  Y[j + p1 * k + p2 * i] -
                  (CT)2 * (Y[k + p1 * j + p2 * i] + Y[i + p1 * k + p2 * j] + Y[j + p1 * i + p2 * k]);
    const CT d = ((eo[i] + eo[j]) + eo[k]) - evirt;                              // :155
    part += div_fast((CT)Wt[e] * r3, d);                                           // :156
    if (++cnt == 16) {
      acc += (double)part;
      part = 0;
      cnt = 0;
    }
    i += di;
    int cj = 0;
    if (i >= oo) { i -= oo; cj = 1; }
    j += dj + cj;
    int ck = 0;
    if (j >= oo) { j -= oo; ck = 1; }
    k += dk + ck;
  }
  acc += (double)part;
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) red[w] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) s += red[q];
    double deg = 1.0;                                                              // :135-139
    if (a == c) deg = 6.0;
    else if (a == b || b == c) deg = 2.0;
    energies[triple_id(a, b, c)] = s / deg;
  }
}

// FP32 copy of S(i, j, a, b) = (ia|jb) for the tensor-core energy kernel.
// out[r ld + c] = (float) x[r cols + c] for c < cols, 0 for cols <= c < ld.
__global__ void to_f32_rows_kernel(const double *__restrict__ x, int64_t rows, int64_t cols,
                                   int64_t ld, float *__restrict__ out) {
  const int64_t n = rows * ld;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / ld, c = e - r * ld;
    out[e] = c < cols ? (float)x[r * cols + c] : 0.0f;
  }
}

// Layout of the mixed form's W and of the FP32 copy of S its energy kernel reads: runs
// of o values of i are padded to op = o rounded up to a multiple of 4 floats, so that every
// quad of i values is aligned: W[((a_l nb + b_l) nb + c_l) o3p + i + op j + o2p k] with
// o2p = o op, o3p = o o2p; S as [(a + v b) o2p + i + op j].  The grouped GEMM's columns are
// padded the same way (o op of them), so that its groups add W in 16-byte reductions and
// the energy kernel reads it in 16-byte loads whatever o.  (With o = 13 unpadded the groups'
// reductions went through shared memory a float at a time: 97 us a launch at v = 117, 81 this way.)
__host__ __device__ inline int64_t pad4(int64_t n) { return (n + 3) & ~int64_t(3); }

// FP32 tables of the mixed energy kernel, built once per (T) call: every
// orbital energy as hi + lo (hi = the FP32 rounding of eps, lo = the FP32
// rounding of the remainder), t1 in FP32, and for every orbit (see orbit_table)
// its code, e_i + e_j + e_k as hi + lo and the weight of its six orderings.
__global__ void energy_tables_kernel(const double *__restrict__ eps, int64_t n,
                                     const double *__restrict__ t1, int64_t nt1,
                                     const uint32_t *__restrict__ codes, int64_t norbits,
                                     float2 *__restrict__ ehl, float *__restrict__ t1f,
                                     uint4 *__restrict__ orbits) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n + nt1 + norbits;
       e += (int64_t)gridDim.x * blockDim.x) {
    if (e < n) {
      const double x = eps[e];
      const float h = (float)x;
      ehl[e] = make_float2(h, (float)(x - (double)h));
    } else if (e < n + nt1) {
      t1f[e - n] = (float)t1[e - n];
    } else {
      const uint32_t code = codes[e - n - nt1];
      const double x = (eps[code & 255] + eps[(code >> 8) & 255]) + eps[(code >> 16) & 255];
      const float h = (float)x;
      const uint32_t m = code >> 24;
      const float mult = m == 0 ? 1.0f : (m == 1 ? 0.5f : (1.0f / 6.0f));
      orbits[e - n - nt1] = make_uint4(code, __float_as_uint(h), __float_as_uint((float)(x - (double)h)),
                                       __float_as_uint(mult));
    }
  }
}

// Double-float arithmetic in FP32: two_sum gives s + e == a + b exactly
// (Knuth's TwoSum, six FP32 operations, no branch).
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Orbits of (i, j, k) under the six orderings, i <= j <= k, for the energy
// kernel: entry = i | j << 8 | k << 16 | m << 24 with m = 0 (three distinct
// indices: the six orderings are six elements), 1 (two equal: each element
// counted twice), 2 (all equal: six times).
std::vector<uint32_t> orbit_table(int64_t o) {
  std::vector<uint32_t> t;
  for (int64_t k = 0; k < o; k++)
    for (int64_t j = 0; j <= k; j++)
      for (int64_t i = 0; i <= j; i++) {
        const uint32_t m = (i == k) ? 2u : ((i == j || j == k) ? 1u : 0u);
        t.push_back((uint32_t)i | (uint32_t)j << 8 | (uint32_t)k << 16 | m << 24);
      }
  return t;
}

// Energy of one block triple in the mixed form.  W^{abc}_{ijk} is the sum of
// the grouped launch's three products: NW = 3 buffers written by the groups
// (W_0[b,c][a], W_1[a,c][b], W_2[a,b][c], as laid out by their tables), or
// NW = 1 buffer the groups reduced into (W[a,b,c]), which this kernel clears
// after reading so that it starts at zero for the next block triple.  Each
// block is o^3 floats in (i, j, k) order, i + op j + o2p k.  One CTA per local
// triple (a_l, b_l, c_l).
//
// Pass 1: Y = W + V in shared memory, V_ijk = t1_ia (jb|kc) + t1_jb (ia|kc) +
// t1_kc (ia|jb) (GetV, RCCSD_T.cpp:70-75).  A thread owns four pairs (i, j) with
// consecutive i and some of the k; the loads of several k are issued before any is
// used, and what was read is cleared at once.
// Pass 2 (threads own orbits of (i, j, k)): r3 (:152-154) of an even ordering
// of the orbit is 3 Y + (S_e - 2 S_o), of an odd one 3 Y + (S_o - 2 S_e)
// (S_e, S_o: sums of Y over the even / odd orderings), and the denominator
// (:155) is the same for the whole orbit:
//   sum_orbit W r3(Y) / D = [sum_even W (3 Y + S_e - 2 S_o) + sum_odd W (3 Y + S_o - 2 S_e)] / D,
// one division per orbit instead of six; r3 is formed per ordering before it
// multiplies W (it is a small difference of similar Y values).  D needs no FP64
// arithmetic per orbit: energies are FP32 hi + lo pairs, e_i + e_j + e_k comes from
// the orbit table, and the difference is formed in double-float (two_sum) and rounded
// once.  The orbit sums are compensated (Kahan), the sums over the warp
// double-float, the CTA's FP64.
//
// The kernel is bound by instruction issue and shared-memory wavefronts (W comes from
// L2).  WS keeps (Y, W) pairs in shared memory: six 8-byte reads per orbit.  Where two
// such CTAs don't fit an SM (o >= 24) only Y is kept and W = Y - V recomputed from the
// (ia|jb) slices: 24 reads and 18 multiply-adds per orbit.  At o = 20 and 1728 triples:
// 45.5 us with V recomputed and the energies added per orbit, 38.3 this way.
constexpr int kEnergyMaxO = 32;
template <int NW, bool WS>
__global__ void __launch_bounds__(256, WS ? 4 : 3) triples_energy_orbit_kernel(
    float *__restrict__ W, int64_t o, int64_t v, int64_t nb, int64_t A, int64_t Bk, int64_t C,
    const float2 *__restrict__ ehl, const float *__restrict__ t1f, const float *__restrict__ S,
    const uint4 *__restrict__ orbits, int norbits, double *__restrict__ energies) {
  const int al = (int)(blockIdx.x / (nb * nb)), bl = (int)((blockIdx.x / nb) % nb),
            cl = (int)(blockIdx.x % nb);
  const int64_t a = A * nb + al, b = Bk * nb + bl, c = C * nb + cl;
  const int oo = (int)o, o2 = oo * oo;
  const int op = (int)pad4(oo), o2p = oo * op, o3p = oo * o2p;
  const int64_t nb3o3 = nb * nb * nb * (int64_t)o3p;
  float *W0;
  const float *W1 = nullptr, *W2 = nullptr;
  if (NW == 3) {
    W0 = W + ((bl * nb + cl) * nb + al) * (int64_t)o3p;
    W1 = W + nb3o3 + ((al * nb + cl) * nb + bl) * (int64_t)o3p;
    W2 = W + 2 * nb3o3 + ((al * nb + bl) * nb + cl) * (int64_t)o3p;
  } else {
    W0 = W + ((al * nb + bl) * nb + cl) * (int64_t)o3p;
  }
  // the next (T) launch may be scheduled once every CTA is here: it does not
  // touch W before this grid is complete
  if (threadIdx.x == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const bool unique = a < v && b < v && c < v && b <= a && c <= b;
  if (!unique) {
    // launched as a programmatic dependent of the grouped GEMM: W is complete
    // and visible only after this wait (no-op for an ordinary launch)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (NW == 1) {  // its block received the launch's sums all the same: clear it
      float4 *w4 = reinterpret_cast<float4 *>(W0);
      for (int e = threadIdx.x; e < o3p / 4; e += blockDim.x) w4[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }
  extern __shared__ __align__(16) unsigned char sm_raw[];
  __shared__ double red[8];
  __shared__ float s_ev[2];
  // tab[x] = (t1_xa, t1_xb, t1_xc); the (ia|jb) slices at x + ps y; Y or (Y, W) at
  // i + p1 j + p2 k.  Odd pitches keep reads along any one index free of bank conflicts
  // (the slices are read that way in pass 2 alone).
  constexpr int EL = WS ? 8 : 4;  // bytes of an element
  const int p1 = oo | 1, p2 = (p1 * oo) | 1, ps = WS ? op : p1, slice = WS ? o2p : p1 * oo;
  float4 *tab = reinterpret_cast<float4 *>(sm_raw);
  float *Sbc = reinterpret_cast<float *>(tab + oo), *Sac = Sbc + slice, *Sab = Sac + slice;
  float *Y = Sab + slice;
  if (!WS) Y = reinterpret_cast<float *>(sm_raw + ((reinterpret_cast<unsigned char *>(Y) - sm_raw + 7) & ~7));
  unsigned char *yb = reinterpret_cast<unsigned char *>(Y);
  const float *S_bc = S + (b + v * c) * o2p, *S_ac = S + (a + v * c) * o2p, *S_ab = S + (a + v * b) * o2p;
  if (WS) {
    for (int e = threadIdx.x; e < o2p / 4; e += blockDim.x) {
      reinterpret_cast<float4 *>(Sbc)[e] = reinterpret_cast<const float4 *>(S_bc)[e];
      reinterpret_cast<float4 *>(Sac)[e] = reinterpret_cast<const float4 *>(S_ac)[e];
      reinterpret_cast<float4 *>(Sab)[e] = reinterpret_cast<const float4 *>(S_ab)[e];
    }
  } else {
    for (int e = threadIdx.x; e < o2; e += blockDim.x) {
      const int x = e % oo, y = e / oo;
      Sbc[x + p1 * y] = S_bc[x + op * y];
      Sac[x + p1 * y] = S_ac[x + op * y];
      Sab[x + p1 * y] = S_ab[x + op * y];
    }
  }
  for (int i = threadIdx.x; i < oo; i += blockDim.x)
    tab[i] = make_float4(t1f[i + o * a], t1f[i + o * b], t1f[i + o * c], 0.f);
  if (threadIdx.x == 0) {  // e_a + e_b + e_c in double-float
    const float2 ea = ehl[o + a], eb = ehl[o + b], ec = ehl[o + c];
    float s1, e1, s2, e2;
    two_sum(ea.x, eb.x, s1, e1);
    two_sum(s1, ec.x, s2, e2);
    const float lo = (e1 + e2) + ((ea.y + eb.y) + ec.y);
    const float hi = s2 + lo;
    s_ev[0] = hi;
    s_ev[1] = lo - (hi - s2);
  }
  // the tables above come from the call's setup; W from the grouped GEMM just
  // before, complete after this wait
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // pass 1; the first loads go out before the barrier that publishes the tables
  constexpr int CH = 4;  // k loads of a thread in flight (more would spill)
  const int nu = o2p / 4, kgn = max(1, (int)blockDim.x / nu), units = nu * kgn;
  int t = threadIdx.x, i = 0, j = 0, k0 = 0;
  float4 r[CH];
  float *w = W0;
  auto begin = [&]() {
    k0 = t / nu;
    const int u = t - k0 * nu;
    j = u / (op / 4);
    i = 4 * u - j * op;
    w = W0 + 4 * u;
  };
  auto load = [&]() {
#pragma unroll
    for (int n = 0; n < CH; n++) {
      const int k = k0 + n * kgn;
      if (k < oo) {
        r[n] = *reinterpret_cast<const float4 *>(w + k * o2p);
        if (NW == 3) {
          const float4 x = *reinterpret_cast<const float4 *>(W1 + (w - W0) + k * o2p),
                       y = *reinterpret_cast<const float4 *>(W2 + (w - W0) + k * o2p);
          r[n] = make_float4(r[n].x + (x.x + y.x), r[n].y + (x.y + y.y), r[n].z + (x.z + y.z), r[n].w + (x.w + y.w));
        }
      }
    }
  };
  if (t < units) {
    begin();
    load();
  }
  __syncthreads();
  while (t < units) {
    // (values of i from o on are padding: read like the others, not stored)
    const float tbj = tab[j].y;
    float tai[4], sab[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      tai[q] = tab[i + q].x;
      sab[q] = Sab[i + q + ps * j];
    }
    unsigned char *y0 = yb + EL * (i + p1 * j);
#pragma unroll
    for (int n = 0; n < CH; n++) {
      const int k = k0 + n * kgn;
      if (k < oo) {
        const float bc = Sbc[j + ps * k], tck = tab[k].z;
        alignas(16) float ac[4];
        if (WS) {
          *reinterpret_cast<float4 *>(ac) = *reinterpret_cast<const float4 *>(Sac + i + ps * k);
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) ac[q] = Sac[i + q + ps * k];
        }
        const float wr[4] = {r[n].x, r[n].y, r[n].z, r[n].w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float y = wr[q] + (tai[q] * bc + tbj * ac[q] + tck * sab[q]);
          if (i + q < oo) {
            if (WS)
              *reinterpret_cast<float2 *>(y0 + EL * (p2 * k + q)) = make_float2(y, wr[q]);
            else
              *reinterpret_cast<float *>(y0 + EL * (p2 * k + q)) = y;
          }
        }
        // W is read: cleared for the next block triple's reductions
        if (NW == 1) *reinterpret_cast<float4 *>(w + k * o2p) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    k0 += CH * kgn;
    if (k0 >= oo) {
      t += blockDim.x;
      if (kgn > 1 || t >= units) break;
      begin();
    }
    load();
  }
  // (shared memory leaves the L1 cache little room: the orbit table comes from L2, an
  // entry ahead of its use)
  int q = threadIdx.x;
  uint4 next = q < norbits ? __ldg(orbits + q) : make_uint4(0, 0, 0, 0);
  __syncthreads();
  // pass 2: orbits
  const float evh = s_ev[0], evl = s_ev[1];
  const int s1 = EL * p1, s2 = EL * p2;
  float sum = 0.0f, comp = 0.0f;
  while (q < norbits) {
    const uint4 ob = next;
    q += blockDim.x;
    if (q < norbits) next = __ldg(orbits + q);
    const int i = ob.x & 255, j = (ob.x >> 8) & 255, k = (ob.x >> 16) & 255;
    const int bi = EL * i, bj = EL * j, bk = EL * k;
    const int pi = s1 * i, pj = s1 * j, pk = s1 * k, qi = s2 * i, qj = s2 * j, qk = s2 * k;
    // even orderings ijk, jki, kij; odd ikj, kji, jik
    float ye0, ye1, ye2, yo0, yo1, yo2, we0, we1, we2, wo0, wo1, wo2;
    if (WS) {
      auto at = [&](int off, float &y, float &w) {
        const float2 x = *reinterpret_cast<const float2 *>(yb + off);
        y = x.x;
        w = x.y;
      };
      at(bi + pj + qk, ye0, we0);
      at(bj + pk + qi, ye1, we1);
      at(bk + pi + qj, ye2, we2);
      at(bi + pk + qj, yo0, wo0);
      at(bk + pj + qi, yo1, wo1);
      at(bj + pi + qk, yo2, wo2);
    } else {
      auto at = [&](int off) { return *reinterpret_cast<const float *>(yb + off); };
      ye0 = at(bi + pj + qk), ye1 = at(bj + pk + qi), ye2 = at(bk + pi + qj);
      yo0 = at(bi + pk + qj), yo1 = at(bk + pj + qi), yo2 = at(bj + pi + qk);
      // V_xyz = t1_xa Sbc(y,z) + t1_yb Sac(x,z) + t1_zc Sab(x,y) over the orderings
      const float4 ti = tab[i], tj = tab[j], tk = tab[k];
      const int si = p1 * i, sj = p1 * j, sk = p1 * k;
      const float bc_jk = Sbc[j + sk], bc_kj = Sbc[k + sj], bc_ki = Sbc[k + si],
                  bc_ik = Sbc[i + sk], bc_ij = Sbc[i + sj], bc_ji = Sbc[j + si];
      const float ac_jk = Sac[j + sk], ac_kj = Sac[k + sj], ac_ki = Sac[k + si],
                  ac_ik = Sac[i + sk], ac_ij = Sac[i + sj], ac_ji = Sac[j + si];
      const float ab_jk = Sab[j + sk], ab_kj = Sab[k + sj], ab_ki = Sab[k + si],
                  ab_ik = Sab[i + sk], ab_ij = Sab[i + sj], ab_ji = Sab[j + si];
      we0 = ye0 - (ti.x * bc_jk + tj.y * ac_ik + tk.z * ab_ij);
      we1 = ye1 - (tj.x * bc_ki + tk.y * ac_ji + ti.z * ab_jk);
      we2 = ye2 - (tk.x * bc_ij + ti.y * ac_kj + tj.z * ab_ki);
      wo0 = yo0 - (ti.x * bc_kj + tk.y * ac_ij + tj.z * ab_ik);
      wo1 = yo1 - (tk.x * bc_ji + tj.y * ac_ki + ti.z * ab_kj);
      wo2 = yo2 - (tj.x * bc_ik + ti.y * ac_jk + tk.z * ab_ji);
    }
    const float Se = (ye0 + ye1) + ye2, So = (yo0 + yo1) + yo2;
    const float ce = Se - 2.0f * So, co = So - 2.0f * Se;                          // :152-154
    float num = we0 * fmaf(3.0f, ye0, ce);
    num = fmaf(we1, fmaf(3.0f, ye1, ce), num);
    num = fmaf(we2, fmaf(3.0f, ye2, ce), num);
    num = fmaf(wo0, fmaf(3.0f, yo0, co), num);
    num = fmaf(wo1, fmaf(3.0f, yo1, co), num);
    num = fmaf(wo2, fmaf(3.0f, yo2, co), num);
    // D = e_i + e_j + e_k - (e_a + e_b + e_c) in double-float, rounded once   :155
    float dh, de;
    two_sum(__uint_as_float(ob.y), -evh, dh, de);
    const float d = dh + (de + (__uint_as_float(ob.z) - evl));
    const float term = __fdividef(num * __uint_as_float(ob.w), d) - comp;          // :156
    const float t = sum + term;
    comp = (t - sum) - term;
    sum = t;
  }
  // warp sums in double-float, the CTA's in FP64
  float acc_hi = sum, acc_lo = -comp;
  for (int off = 16; off > 0; off >>= 1) {
    const float oh = __shfl_down_sync(0xffffffffu, acc_hi, off);
    const float ol = __shfl_down_sync(0xffffffffu, acc_lo, off);
    float h, e;
    two_sum(acc_hi, oh, h, e);
    acc_hi = h;
    acc_lo += e + ol;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = (double)acc_hi + (double)acc_lo;
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) total += red[q];
    // degeneracy of the virtual indices                                            :135-139
    if (a == c) total /= 6.0;
    else if (a == b || b == c) total *= 0.5;
    energies[triple_id(a, b, c)] = total;
  }
}

// FP64 form: one CTA per local triple (a_l, b_l, c_l) of the block triple.  W is
// read from the three group buffers of the sliced GEMM, problem-major with the
// GEMM rows contiguous:
//   W_g[y + nb z][s + o t][u + o x_l], (x, y, z) = (a, b, c), (b, a, c), (c, a, b),
// u the occupied partner of x and (s, t) the other two occupied indices in order;
// W = (W_0 + W_1) + W_2 is formed in shared memory.  Then as the mixed form: one
// thread per orbit of (i, j, k), six orderings sharing one denominator.  GB300
// issues about two FP64 lanes per cycle and SM, so this kernel is FP64-bound (about 70 % at o = 10): 18 FMAs
// for W + V of an orbit, 18 for r3 and its products, one division, and 12 adds for
// the sum of the buffers (10 FP64 operations per element; a thread per element with
// its own denominator took about 30).
__global__ void __launch_bounds__(256) triples_energy_orbit64_kernel(
    const double *__restrict__ W, int64_t o, int64_t v, int64_t nb, int64_t A, int64_t Bk, int64_t C,
    const double *__restrict__ eps, const double *__restrict__ t1, const double *__restrict__ S,
    const uint32_t *__restrict__ orbits, int norbits, double *__restrict__ energies) {
  const int n = (int)nb;
  const int al = blockIdx.x / (n * n), bl = (blockIdx.x / n) % n, cl = blockIdx.x % n;
  const int64_t a = A * nb + al, b = Bk * nb + bl, c = C * nb + cl;
  // the next block triple's GEMM may be placed: it waits for this grid before it writes W
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (a >= v || b >= v || c >= v || b > a || c > b) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const int oo = (int)o, o2 = oo * oo, o3 = o2 * oo;
  // W(i,j,k) at i + p1 j + p2 k and the slices at x + p1 y, p1 and p2 odd: reads along
  // any one index are free of bank conflicts
  const int p1 = oo | 1, p2 = (p1 * oo) | 1;
  double *Ws = reinterpret_cast<double *>(sm_raw);
  double *Sbc = Ws + p2 * oo, *Sac = Sbc + p1 * oo, *Sab = Sac + p1 * oo;
  double *ta = Sab + p1 * oo, *tb = ta + oo, *tc = tb + oo, *eo = tc + oo;
  const int64_t Mg = o * nb, prob = Mg * o2, grp = nb * nb * prob;
  const double *W0 = W + (bl + nb * cl) * prob + o * al, *W1 = W + grp + (al + nb * cl) * prob + o * bl,
               *W2 = W + 2 * grp + (al + nb * bl) * prob + o * cl;
  for (int e = threadIdx.x; e < o2; e += blockDim.x) {
    const int x = e % oo, y = e / oo;
    Sbc[x + p1 * y] = S[e + o2 * (b + v * c)];
    Sac[x + p1 * y] = S[e + o2 * (a + v * c)];
    Sab[x + p1 * y] = S[e + o2 * (a + v * b)];
  }
  for (int i = threadIdx.x; i < oo; i += blockDim.x) {
    ta[i] = t1[i + o * a];
    tb[i] = t1[i + o * b];
    tc[i] = t1[i + o * c];
    eo[i] = eps[i];
  }
  // S, t1 and eps come from the call's setup, W from the GEMM just before
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // Element e of a buffer: u = e % o, column e / o = s + o t.  W is summed in shared memory,
  // buffer after buffer; the next chunk's loads (the next buffer's too) go out before a
  // chunk is added.
  constexpr int kStage = 5;
  const int span = kStage * blockDim.x, nch = (o3 + span - 1) / span;
  double x[kStage], y[kStage];
  auto load = [&](int step, double *r) {
    const int g = step / nch;
    const double *Wg = g == 0 ? W0 : (g == 1 ? W1 : W2);
#pragma unroll
    for (int q = 0; q < kStage; q++) {
      const int e = (step - g * nch) * span + (int)threadIdx.x + q * blockDim.x, col = e / oo;
      if (e < o3) r[q] = Wg[e - col * oo + Mg * col];
    }
  };
  load(0, x);
  for (int step = 0; step < 3 * nch; step++) {
    if (step + 1 < 3 * nch) load(step + 1, y);
    // (u, s, t) = (i, j, k), (j, i, k), (k, i, j): strides in Ws
    const int g = step / nch, su = g == 0 ? 1 : (g == 1 ? p1 : p2), ss = g == 0 ? p1 : 1, st = g == 2 ? p1 : p2;
#pragma unroll
    for (int q = 0; q < kStage; q++) {
      const int e = (step - g * nch) * span + (int)threadIdx.x + q * blockDim.x, col = e / oo, t = col / oo;
      if (e < o3) {
        double *p = Ws + (e - col * oo) * su + (col - t * oo) * ss + t * st;
        *p = g == 0 ? x[q] : *p + x[q];
      }
      x[q] = y[q];
    }
    if (step + 1 == (g + 1) * nch) __syncthreads();
  }
  const double evirt = eps[o + a] + eps[o + b] + eps[o + c];
  double acc = 0.0;
  for (int q = threadIdx.x; q < norbits; q += blockDim.x) {
    const uint32_t code = __ldg(orbits + q);
    const int i = code & 255, j = (code >> 8) & 255, k = (code >> 16) & 255, m = code >> 24;
    const double ai = ta[i], aj = ta[j], ak = ta[k], bi = tb[i], bj = tb[j], bk = tb[k], ci = tc[i], cj = tc[j],
                 ck = tc[k];
    const int pi = p1 * i, pj = p1 * j, pk = p1 * k, qi = p2 * i, qj = p2 * j, qk = p2 * k;
    // V_xyz = t1_xa (yb|zc) + t1_yb (xa|zc) + t1_zc (xa|yb)                       :70-75
    const double we0 = Ws[i + pj + qk], we1 = Ws[j + pk + qi], we2 = Ws[k + pi + qj];
    const double wo0 = Ws[i + pk + qj], wo1 = Ws[k + pj + qi], wo2 = Ws[j + pi + qk];
    const double ye0 = fma(ai, Sbc[j + pk], fma(bj, Sac[i + pk], fma(ck, Sab[i + pj], we0)));
    const double ye1 = fma(aj, Sbc[k + pi], fma(bk, Sac[j + pi], fma(ci, Sab[j + pk], we1)));
    const double ye2 = fma(ak, Sbc[i + pj], fma(bi, Sac[k + pj], fma(cj, Sab[k + pi], we2)));
    const double yo0 = fma(ai, Sbc[k + pj], fma(bk, Sac[i + pj], fma(cj, Sab[i + pk], wo0)));
    const double yo1 = fma(ak, Sbc[j + pi], fma(bj, Sac[k + pi], fma(ci, Sab[k + pj], wo1)));
    const double yo2 = fma(aj, Sbc[i + pk], fma(bi, Sac[j + pk], fma(ck, Sab[j + pi], wo2)));
    const double Se = (ye0 + ye1) + ye2, So = (yo0 + yo1) + yo2;
    const double ce = fma(-2.0, So, Se), co = fma(-2.0, Se, So);                   // :152-154
    double num = we0 * fma(3.0, ye0, ce);
    num = fma(we1, fma(3.0, ye1, ce), num);
    num = fma(we2, fma(3.0, ye2, ce), num);
    num = fma(wo0, fma(3.0, yo0, co), num);
    num = fma(wo1, fma(3.0, yo1, co), num);
    num = fma(wo2, fma(3.0, yo2, co), num);
    const double d = ((eo[i] + eo[j]) + eo[k]) - evirt;                             // :155
    // an orbit with two (three) equal indices visits its elements twice (six times)
    acc += num * (m == 0 ? 1.0 : (m == 1 ? 0.5 : 1.0 / 6.0)) / d;                   // :156
  }
  // the CTA's sum in one warp: eight warps' shuffles cost more FP64 issue than this
  __syncthreads();  // (W is read)
  Ws[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double sum = 0.0;
    for (int q = threadIdx.x; q < (int)blockDim.x; q += 32) sum += Ws[q];
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
    if (threadIdx.x == 0) {
      // degeneracy of the virtual indices                                            :135-139
      if (a == c) sum /= 6.0;
      else if (a == b || b == c) sum *= 0.5;
      energies[triple_id(a, b, c)] = sum;
    }
  }
}

__global__ void sum_energies_kernel(int64_t n, const double *__restrict__ e, double *out) {
  __shared__ double red[32];
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += e[i];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) t += red[q];
    out[0] = 2.0 * t;                                                              // :167
  }
}

// Offset table over a list of (extent, stride) dims, first fastest:
// entry e = sum_d i_d stride_d for e = i_0 + ext_0 (i_1 + ext_1 (...)).  Kept
// as a spec and filled on the device (DevTables::build).
struct TableSpec {
  int nd = 0;
  int64_t ext[6] = {1, 1, 1, 1, 1, 1}, str[6] = {0, 0, 0, 0, 0, 0};
  // first dimension: entries from `valid` on are padding, and read the last valid index
  // or (skip) get kNoOffset
  int64_t valid = INT64_MAX;
  bool skip = false;
  int64_t size() const {
    int64_t n = 1;
    for (int d = 0; d < nd; d++) n *= ext[d];
    return n;
  }
};

TableSpec table(std::initializer_list<std::pair<int64_t, int64_t>> dims) {
  TableSpec t;
  if (dims.size() > 6) throw Error(SCESS_ERR_INVALID, "offset table: too many dims");
  for (auto &d : dims) {
    t.ext[t.nd] = d.first;
    t.str[t.nd] = d.second;
    t.nd++;
  }
  return t;
}

TableSpec padded(TableSpec t, int64_t valid, bool skip) {
  t.valid = valid;
  t.skip = skip;
  return t;
}
constexpr int64_t kNoOffset = -(int64_t(1) << 60);  // negative with every base added

constexpr int kMaxTables = 24;
struct TableBatch {
  int nt = 0;
  int64_t start[kMaxTables + 1] = {};
  TableSpec spec[kMaxTables];
  int64_t *out = nullptr;
};

__global__ void fill_tables_kernel(const __grid_constant__ TableBatch b) {
  const int64_t total = b.start[b.nt];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int t = 0;
    while (e >= b.start[t + 1]) t++;
    const TableSpec &sp = b.spec[t];
    int64_t r = e - b.start[t], off = 0;
    bool none = false;
    for (int d = 0; d < sp.nd; d++) {
      const int64_t q = r / sp.ext[d];
      int64_t i = r - q * sp.ext[d];
      if (d == 0 && i >= sp.valid) {
        none = sp.skip;
        i = sp.valid - 1;
      }
      off += i * sp.str[d];
      r = q;
    }
    b.out[e] = none ? kNoOffset : off;
  }
}

struct DevTables {
  DevMem mem;
  std::vector<const int64_t *> ptr;
  // One allocation, filled by one kernel per kMaxTables tables on ctx's stream.
  void build(Ctx &ctx, const std::vector<TableSpec> &ts) {
    size_t tot = 0;
    for (auto &t : ts) tot += (size_t)t.size();
    mem.alloc(std::max<size_t>(tot, 1) * sizeof(int64_t));
    ptr.clear();
    size_t off = 0;
    for (size_t i0 = 0; i0 < ts.size(); i0 += kMaxTables) {
      TableBatch b;
      b.out = mem.as<int64_t>() + off;
      b.nt = (int)std::min<size_t>(kMaxTables, ts.size() - i0);
      int64_t n = 0;
      for (int t = 0; t < b.nt; t++) {
        b.spec[t] = ts[i0 + t];
        b.start[t] = n;
        ptr.push_back(mem.as<int64_t>() + off + n);
        n += ts[i0 + t].size();
      }
      b.start[b.nt] = n;
      if (n > 0) {
        fill_tables_kernel<<<(unsigned)std::min<int64_t>(ceil_div(n, 256), 8 * kNumSMs), 256, 0,
                             ctx.stream>>>(b);
        SCESS_CHECK_LAUNCH();
      }
      off += (size_t)n;
    }
  }
};

// The six simultaneous permutations of Symmetrise, as position maps: the raw
// term w^{u[p0] u[p1] u[p2]}_{w[p0] w[p1] w[p2]} feeds W^{abc}_{ijk}.
const int kPerm[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};

int choose_nb(int64_t o, int64_t v, size_t welem_bytes, size_t budget) {
  const int64_t forced = tune_value("t_nb", 0);  // block size override (tests, tuning)
  if (forced >= 1) return (int)std::min<int64_t>(forced, v);
  const double o3 = (double)o * o * o;
  int nb = (int)std::floor(std::cbrt((double)budget / (welem_bytes * o3)));
  nb = std::max(1, std::min<int>(nb, (int)v));
  // balance the blocks over v
  const int64_t nblk = ceil_div(v, nb);
  nb = (int)ceil_div(v, nblk);
  return nb;
}

// W tables: W's unit-stride index i is kept first on the lane side (GEMM rows)
// or on the per-thread side (GEMM columns) of every epilogue: when i is the k'
// of a permutation the Q operand is taken in (k', j', z) column order, when it
// is the j' of an R product the R operand is taken in (j', i', x) row order.
bool q_swapped(const int *pi) { return pi[2] == 0; }
bool r_swapped(const int *pi) { return pi[1] == 0; }

// FP64 repacks of RCCSD_T.cpp:30-56 (virtuals padded to vp) and the offset
// tables of the block-triple GEMMs: per permutation p the W rows / columns of
// its P.Q and R.t2 products (dt.ptr[4p .. 4p+3]), then the operand tables
// (dt.ptr[kOperand + 0 .. 9]).
struct TriplesSetup {
  int64_t o = 0, v = 0, N = 0, nb = 0, NB = 0, vp = 0;
  DTensor P, Qt, Rt, T2p;
  DTensor S;  // S(i,j,a,b) = (ia|jb), o x o x v x v
  DevTables dt;
  size_t kOperand = 0;
  // integrals from the eri (views) or, when d_B is given, from the DF factors
  // B (naux x N x N): P, R, S are single B.B contractions (be: FP64 or tensor
  // cores), so the N^4 eri is never formed
  void build(Ctx &ctx, const double *d_eri, const double *d_t2, const double *d_B = nullptr,
             int64_t naux = 0, Backend be = Backend::FP64);
  int64_t Mpq() const { return o * nb * nb; }
  int64_t Npq() const { return o * o * nb; }
  int64_t Mr() const { return o * o * nb; }
  int64_t Nr() const { return o * nb * nb; }
};

void TriplesSetup::build(Ctx &ctx, const double *d_eri, const double *d_t2, const double *d_B,
                         int64_t naux, Backend be) {
  cudaStream_t s = ctx.stream;
  const int64_t o2 = o * o, o3 = o2 * o, N2 = N * N, N3 = N2 * N;
  S = DTensor({o, o, v, v});
  // Zero-padded FP64 repacks (RCCSD_T.cpp:30-56), virtual indices padded to vp.
  P = DTensor({o, v, vp, vp});   // P(i,f,a,b) = (ia|bf) = eri(i, o+b, o+a, o+f)
  Qt = DTensor({v, o, o, vp});   // Q(f,j,k,c) = t2(k,j,c,f)
  Rt = DTensor({o, o, o, vp});   // R(i,j,m,a) = (ia|mj) = eri(i, m, o+a, j)
  T2p = DTensor({o, o, vp, vp}); // t2(m,k,b,c)
  SCESS_CUDA(cudaMemsetAsync(P.p(), 0, P.size() * sizeof(double), s));
  SCESS_CUDA(cudaMemsetAsync(Qt.p(), 0, Qt.size() * sizeof(double), s));
  SCESS_CUDA(cudaMemsetAsync(Rt.p(), 0, Rt.size() * sizeof(double), s));
  SCESS_CUDA(cudaMemsetAsync(T2p.p(), 0, T2p.size() * sizeof(double), s));
  {
    TV Pv = P.v;
    Pv.ext[2] = v;
    Pv.ext[3] = v;
    TV Rv = Rt.v;
    Rv.ext[3] = v;
    if (d_B) {
      // (pq|rs) = sum_Q B(Q,p,q) B(Q,r,s): P(i,f,a,b) = (ia|bf), R(i,j,m,a) = (ia|mj),
      // S(i,j,a,b) = (ia|jb)
      auto bview = [&](int64_t p0, int64_t q0, int64_t np, int64_t nq) {
        TV b;
        b.p = const_cast<double *>(d_B) + naux * p0 + naux * N * q0;
        b.nd = 3;
        const int64_t be3[3] = {naux, np, nq}, bs3[3] = {1, naux, naux * N};
        std::memcpy(b.ext, be3, sizeof(be3));
        std::memcpy(b.str, bs3, sizeof(bs3));
        return b;
      };
      const TV Bov = bview(0, o, o, v), Bvv = bview(o, o, v, v), Boo = bview(0, 0, o, o);
      einsum(ctx, "Qia,Qbf->ifab", 1.0, Bov, Bvv, 0.0, Pv, be);
      einsum(ctx, "Qia,Qmj->ijma", 1.0, Bov, Boo, 0.0, Rv, be);
      einsum(ctx, "Qia,Qjb->ijab", 1.0, Bov, Bov, 0.0, S.v, be);
    } else {
      TV e;  // (i, b, a, f) -> eri(i, o+b, o+a, o+f)
      e.p = const_cast<double *>(d_eri) + o * N + o * N2 + o * N3;
      e.nd = 4;
      int64_t ee[4] = {o, v, v, v}, es[4] = {1, N, N2, N3};
      std::memcpy(e.ext, ee, sizeof(ee));
      std::memcpy(e.str, es, sizeof(es));
      permute(ctx, "ibaf->ifab", 1.0, e, 0.0, Pv);
      TV r;  // (i, m, a, j) -> eri(i, m, o+a, j)
      r.p = const_cast<double *>(d_eri) + o * N2;
      r.nd = 4;
      int64_t re[4] = {o, o, v, o}, rs[4] = {1, N, N2, N3};
      std::memcpy(r.ext, re, sizeof(re));
      std::memcpy(r.str, rs, sizeof(rs));
      permute(ctx, "imaj->ijma", 1.0, r, 0.0, Rv);
      TV sv = r;  // (i, j, a, b) -> eri(i, j, o+a, o+b)
      sv.p = const_cast<double *>(d_eri) + o * N2 + o * N3;
      sv.ext[2] = v;
      sv.ext[3] = v;
      permute(ctx, "ijab->ijab", 1.0, sv, 0.0, S.v);
    }
    const TV t2 = cm(const_cast<double *>(d_t2), {o, o, v, v});
    TV Qv = Qt.v;
    Qv.ext[3] = v;
    permute(ctx, "kjcf->fjkc", 1.0, t2, 0.0, Qv);
    TV Tv = T2p.v;
    Tv.ext[2] = v;
    Tv.ext[3] = v;
    permute(ctx, "mkbc->mkbc", 1.0, t2, 0.0, Tv);
  }

  // Output positions in W[(a_l,b_l,c_l)][i,j,k]: strides of (a_l,b_l,c_l) and (i,j,k).
  const int64_t su[3] = {o3 * nb * nb, o3 * nb, o3};
  const int64_t sw[3] = {1, o, o2};
  // Tables per permutation: PQ rows/cols and R rows/cols in W.  W's unit-stride
  // index i is kept first on the lane side (GEMM rows) or on the per-thread side
  // (GEMM columns) of every epilogue: when i is the k' of a permutation the Q
  // operand is taken in (k', j', z) column order, when it is the j' of an R
  // product the R operand is taken in (j', i', x) row order.
  std::vector<TableSpec> ts;
  for (int p = 0; p < 6; p++) {
    const int *pi = kPerm[p];
    ts.push_back(table({{o, sw[pi[0]]}, {nb, su[pi[0]]}, {nb, su[pi[1]]}}));      // PQ rows (i',x,y)
    if (q_swapped(pi))
      ts.push_back(table({{o, sw[pi[2]]}, {o, sw[pi[1]]}, {nb, su[pi[2]]}}));     // PQ cols (k',j',z)
    else
      ts.push_back(table({{o, sw[pi[1]]}, {o, sw[pi[2]]}, {nb, su[pi[2]]}}));     // PQ cols (j',k',z)
    if (r_swapped(pi))
      ts.push_back(table({{o, sw[pi[1]]}, {o, sw[pi[0]]}, {nb, su[pi[0]]}}));     // R rows (j',i',x)
    else
      ts.push_back(table({{o, sw[pi[0]]}, {o, sw[pi[1]]}, {nb, su[pi[0]]}}));     // R rows (i',j',x)
    ts.push_back(table({{o, sw[pi[2]]}, {nb, su[pi[1]]}, {nb, su[pi[2]]}}));      // R cols (k',y,z)
  }
  kOperand = ts.size();
  // operand tables (FP64 path): P rows (i',x,y), f; Q cols (j',k',z), f; R rows, m; t2 cols, m
  ts.push_back(table({{o, 1}, {nb, o * v}, {nb, o * v * vp}}));                  // +0: P rows
  ts.push_back(table({{v, o}}));                                                 // +1: P k (f)
  ts.push_back(table({{o, v}, {o, v * o}, {nb, v * o2}}));                       // +2: Q cols (j,k,z)
  ts.push_back(table({{v, 1}}));                                                 // +3: Q k (f)
  ts.push_back(table({{o, 1}, {o, o}, {nb, o3}}));                               // +4: R rows (i,j,x)
  ts.push_back(table({{o, o2}}));                                                // +5: R k (m)
  ts.push_back(table({{o, o}, {nb, o2}, {nb, o2 * vp}}));                        // +6: t2 cols
  ts.push_back(table({{o, 1}}));                                                 // +7: t2 k (m)
  ts.push_back(table({{o, v * o}, {o, v}, {nb, v * o2}}));                       // +8: Q cols (k,j,z)
  ts.push_back(table({{o, o}, {o, 1}, {nb, o3}}));                               // +9: R rows (j,i,x)
  dt.build(ctx, ts);
}

// The 12 FP64 GEMMs of block triple U = (A, B, C): W[(a_l,b_l,c_l)][i,j,k] =
// sum over the six permutations of the raw P.Q - R.t2 product (GetW,
// RCCSD_T.cpp:62-68), each added at its permuted position (Symmetrise :78-106).
// tc: the same GEMMs on the tensor cores (TcEngine::table_gemm).
void w_block_fp64(Ctx &ctx, const TriplesSetup &T, const int64_t U[3], double *W,
                  bool tc = false) {
  const int64_t o = T.o, v = T.v, nb = T.nb, vp = T.vp, o2 = o * o, o3 = o2 * o;
  for (int p = 0; p < 6; p++) {
    const int *pi = kPerm[p];
    const int64_t X = U[pi[0]], Yb = U[pi[1]], Z = U[pi[2]];
    const int64_t *rowPQ = T.dt.ptr[4 * p + 0], *colPQ = T.dt.ptr[4 * p + 1];
    const int64_t *rowR = T.dt.ptr[4 * p + 2], *colR = T.dt.ptr[4 * p + 3];
    TableGemm g;
    g.A = T.P.p();
    g.B = T.Qt.p();
    g.C = W;
    g.rowA = T.dt.ptr[T.kOperand + 0];
    g.kA = T.dt.ptr[T.kOperand + 1];
    g.colB = T.dt.ptr[T.kOperand + (q_swapped(pi) ? 8 : 2)];
    g.kB = T.dt.ptr[T.kOperand + 3];
    g.rowC = rowPQ;
    g.colC = colPQ;
    g.baseA = o * v * (X * nb) + o * v * vp * (Yb * nb);
    g.baseB = v * o2 * (Z * nb);
    g.M = T.Mpq();
    g.N = T.Npq();
    g.K = v;
    g.alpha = 1.0;
    g.beta = p == 0 ? 0.0 : 1.0;
    g.aUnitM = 1;
    g.bUnitN = 0;
    if (tc) ctx.tensor_cores().table_gemm(g, "triples_w");
    else fp64_table_gemm(ctx, g, "slice_gemm[triples_w]");
    TableGemm h;
    h.A = T.Rt.p();
    h.B = T.T2p.p();
    h.C = W;
    h.rowA = T.dt.ptr[T.kOperand + (r_swapped(pi) ? 9 : 4)];
    h.kA = T.dt.ptr[T.kOperand + 5];
    h.colB = T.dt.ptr[T.kOperand + 6];
    h.kB = T.dt.ptr[T.kOperand + 7];
    h.rowC = rowR;
    h.colC = colR;
    h.baseA = o3 * (X * nb);
    h.baseB = o2 * (Yb * nb) + o2 * vp * (Z * nb);
    h.M = T.Mr();
    h.N = T.Nr();
    h.K = o;
    h.alpha = -1.0;
    h.beta = 1.0;
    h.aUnitM = r_swapped(pi) ? 0 : 1;
    h.bUnitN = 0;
    if (tc) ctx.tensor_cores().table_gemm(h, "triples_w");
    else fp64_table_gemm(ctx, h, "slice_gemm[triples_w]");
  }
}

// Gradient of the block triple's energy with respect to its W and V (FP64).
// With L = r3 (a symmetric linear map over the six orderings of (i,j,k): the
// two cyclic shifts are each other's transposes, the three swaps are their own)
// and the triple's term E_abc = (2/deg) sum W L(W + V) / D:
//   dE/dW = (2/deg) [L(Y)/D + L(W/D)],   dE/dV = (2/deg) L(W/D),   Y = W + V.
// G (W's layout) receives gE dE/dW, zero for triples outside a >= b >= c; dE/dV
// flows into t1 and the (ia|jb) slices S (o x o x v x v) through
// V_ijk = t1_ia S(j,k,b,c) + t1_jb S(i,k,a,c) + t1_kc S(i,j,a,b) (:70-75, :132)
// with global FP64 atomics.  Also writes the triple's energy like the energy
// kernel.  One CTA per (a_l, b_l, c_l); threads own (i, j) pairs and walk k.
__global__ void __launch_bounds__(256) triples_grad_kernel(
    const double *__restrict__ W, double *__restrict__ G, int64_t o, int64_t v, int64_t nb,
    int64_t A, int64_t Bk, int64_t C, const double *__restrict__ eps,
    const double *__restrict__ t1, const double *__restrict__ Sg, double gE,
    double *__restrict__ energies, double *__restrict__ g_t1, double *__restrict__ g_S) {
  const int64_t al = blockIdx.x / (nb * nb), bl = (blockIdx.x / nb) % nb, cl = blockIdx.x % nb;
  const int64_t a = A * nb + al, b = Bk * nb + bl, c = C * nb + cl;
  const int oo = (int)o, o2 = oo * oo, o3 = o2 * oo;
  const double *Wt = W + ((al * nb + bl) * nb + cl) * (int64_t)o3;
  double *Gt = G + ((al * nb + bl) * nb + cl) * (int64_t)o3;
  if (a >= v || b >= v || c >= v || b > a || c > b) {
    for (int e = threadIdx.x; e < o3; e += blockDim.x) Gt[e] = 0.0;
    return;
  }
  extern __shared__ __align__(16) unsigned char sm_raw[];
  __shared__ double red[32];
  const int p1 = oo | 1, p2 = (p1 * oo) | 1;
  double *Y = reinterpret_cast<double *>(sm_raw);
  double *Sbc = Y + p2 * oo, *Sac = Sbc + o2, *Sab = Sac + o2;
  double *gSbc = Sab + o2, *gSac = gSbc + o2;
  double *ta = gSac + o2, *tb = ta + oo, *tc = tb + oo, *eo = tc + oo;
  double *gta = eo + oo, *gtb = gta + oo, *gtc = gtb + oo;
  for (int e = threadIdx.x; e < o2; e += blockDim.x) {
    Sbc[e] = Sg[e + o2 * (b + v * c)];
    Sac[e] = Sg[e + o2 * (a + v * c)];
    Sab[e] = Sg[e + o2 * (a + v * b)];
    gSbc[e] = 0.0;
    gSac[e] = 0.0;
  }
  for (int i = threadIdx.x; i < oo; i += blockDim.x) {
    ta[i] = t1[i + o * a];
    tb[i] = t1[i + o * b];
    tc[i] = t1[i + o * c];
    eo[i] = eps[i];
    gta[i] = gtb[i] = gtc[i] = 0.0;
  }
  __syncthreads();
  const double evirt = eps[o + a] + eps[o + b] + eps[o + c];
  double deg = 1.0;                                                                 // :135-139
  if (a == c) deg = 6.0;
  else if (a == b || b == c) deg = 2.0;
  const double fac = gE * 2.0 / deg;
  auto L = [&](int i, int j, int k) {  // r3 at (i,j,k) of the array in Y   :152-154
    return 4.0 * Y[i + p1 * j + p2 * k] + Y[k + p1 * i + p2 * j] + Y[j + p1 * k + p2 * i] -
           2.0 * (Y[k + p1 * j + p2 * i] + Y[i + p1 * k + p2 * j] + Y[j + p1 * i + p2 * k]);
  };
  // Y = W + V
  for (int pr = threadIdx.x; pr < o2; pr += blockDim.x) {
    const int i = pr % oo, j = pr / oo;
    for (int k = 0; k < oo; k++)
      Y[i + p1 * j + p2 * k] = Wt[pr + o2 * k] + ta[i] * Sbc[j + oo * k] + tb[j] * Sac[i + oo * k] +
                               tc[k] * Sab[pr];
  }
  __syncthreads();
  // G = fac L(Y)/D; energy term W L(Y)/D
  double acc = 0.0;
  for (int pr = threadIdx.x; pr < o2; pr += blockDim.x) {
    const int i = pr % oo, j = pr / oo;
    for (int k = 0; k < oo; k++) {
      const double d = ((eo[i] + eo[j]) + eo[k]) - evirt;                           // :155
      const double ly = L(i, j, k) / d;
      Gt[pr + o2 * k] = fac * ly;
      acc += Wt[pr + o2 * k] * ly;                                                  // :156
    }
  }
  __syncthreads();
  // Y = W/D
  for (int pr = threadIdx.x; pr < o2; pr += blockDim.x) {
    const int i = pr % oo, j = pr / oo;
    for (int k = 0; k < oo; k++)
      Y[i + p1 * j + p2 * k] = Wt[pr + o2 * k] / (((eo[i] + eo[j]) + eo[k]) - evirt);
  }
  __syncthreads();
  // G += fac L(W/D); dE/dV = fac L(W/D) into t1 and S
  for (int pr = threadIdx.x; pr < o2; pr += blockDim.x) {
    const int i = pr % oo, j = pr / oo;
    double sa = 0.0, sb = 0.0, sab = 0.0;
    for (int k = 0; k < oo; k++) {
      const double gv = fac * L(i, j, k);
      Gt[pr + o2 * k] += gv;
      sa += gv * Sbc[j + oo * k];      // t1_ia (jb|kc)
      sb += gv * Sac[i + oo * k];      // t1_jb (ia|kc)
      sab += gv * tc[k];               // (ia|jb) t1_kc
      atomicAdd(&gtc[k], gv * Sab[pr]);
      atomicAdd(&gSbc[j + oo * k], gv * ta[i]);
      atomicAdd(&gSac[i + oo * k], gv * tb[j]);
    }
    atomicAdd(&gta[i], sa);
    atomicAdd(&gtb[j], sb);
    atomicAdd(&g_S[pr + o2 * (a + v * b)], sab);  // (i,j) owned by this thread
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  if (lane == 0) red[wi] = acc;
  __syncthreads();
  for (int e = threadIdx.x; e < o2; e += blockDim.x) {
    atomicAdd(&g_S[e + o2 * (b + v * c)], gSbc[e]);
    atomicAdd(&g_S[e + o2 * (a + v * c)], gSac[e]);
  }
  for (int i = threadIdx.x; i < oo; i += blockDim.x) {
    atomicAdd(&g_t1[i + o * a], gta[i]);
    atomicAdd(&g_t1[i + o * b], gtb[i]);
    atomicAdd(&g_t1[i + o * c], gtc[i]);
  }
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) sum += red[q];
    energies[triple_id(a, b, c)] = sum / deg;
  }
}

// Transposed GEMMs of w_block_fp64 for block triple U: with G = dE/dW,
//   gP  += G Q,   gQ  += G^T P,   gR -= G' t2,   gt2 -= G'^T R
// per permutation, G read through that permutation's W tables.
// tc: the same GEMMs on the tensor cores (TcEngine::table_gemm).
void g_block_fp64(Ctx &ctx, const TriplesSetup &T, const int64_t U[3], const double *G, double *gP,
                  double *gQt, double *gRt, double *gT2p, bool integrals,
                  bool tc = false) {
  const int64_t o = T.o, v = T.v, nb = T.nb, vp = T.vp, o2 = o * o, o3 = o2 * o;
  const size_t K0 = T.kOperand;
  auto run = [&](TableGemm &g) {
    if (tc) ctx.tensor_cores().table_gemm(g, "triples_vjp");
    else fp64_table_gemm(ctx, g, "slice_gemm[triples_vjp]");
  };
  for (int p = 0; p < 6; p++) {
    const int *pi = kPerm[p];
    const int64_t X = U[pi[0]], Yb = U[pi[1]], Z = U[pi[2]];
    const int64_t *rowPQ = T.dt.ptr[4 * p + 0], *colPQ = T.dt.ptr[4 * p + 1];
    const int64_t *rowR = T.dt.ptr[4 * p + 2], *colR = T.dt.ptr[4 * p + 3];
    const int64_t *qcols = T.dt.ptr[K0 + (q_swapped(pi) ? 8 : 2)];
    const int64_t *rrows = T.dt.ptr[K0 + (r_swapped(pi) ? 9 : 4)];
    const int64_t baseP = o * v * (X * nb) + o * v * vp * (Yb * nb), baseQ = v * o2 * (Z * nb);
    const int64_t baseR = o3 * (X * nb), baseT = o2 * (Yb * nb) + o2 * vp * (Z * nb);
    if (integrals) {  // gP(m, f) += sum_n G(m, n) Q(n, f)
      TableGemm g;
      g.A = G; g.rowA = rowPQ; g.kA = colPQ;
      g.B = T.Qt.p(); g.colB = T.dt.ptr[K0 + 3]; g.kB = qcols; g.baseB = baseQ;
      g.C = gP; g.rowC = T.dt.ptr[K0 + 0]; g.colC = T.dt.ptr[K0 + 1]; g.baseC = baseP;
      g.M = T.Mpq(); g.N = v; g.K = T.Npq(); g.alpha = 1.0; g.beta = 1.0;
      run(g);
    }
    {  // gQ(n, f) += sum_m G(m, n) P(m, f)
      TableGemm g;
      g.A = G; g.rowA = colPQ; g.kA = rowPQ;
      g.B = T.P.p(); g.colB = T.dt.ptr[K0 + 1]; g.kB = T.dt.ptr[K0 + 0]; g.baseB = baseP;
      g.C = gQt; g.rowC = qcols; g.colC = T.dt.ptr[K0 + 3]; g.baseC = baseQ;
      g.M = T.Npq(); g.N = v; g.K = T.Mpq(); g.alpha = 1.0; g.beta = 1.0;
      run(g);
    }
    if (integrals) {  // gR(r, m) -= sum_n G(r, n) t2(n, m)
      TableGemm g;
      g.A = G; g.rowA = rowR; g.kA = colR;
      g.B = T.T2p.p(); g.colB = T.dt.ptr[K0 + 7]; g.kB = T.dt.ptr[K0 + 6]; g.baseB = baseT;
      g.C = gRt; g.rowC = rrows; g.colC = T.dt.ptr[K0 + 5]; g.baseC = baseR;
      g.M = T.Mr(); g.N = o; g.K = T.Nr(); g.alpha = -1.0; g.beta = 1.0;
      run(g);
    }
    {  // gt2(n, m) -= sum_r G(r, n) R(r, m)
      TableGemm g;
      g.A = G; g.rowA = colR; g.kA = rowR;
      g.B = T.Rt.p(); g.colB = T.dt.ptr[K0 + 5]; g.kB = rrows; g.baseB = baseR;
      g.C = gT2p; g.rowC = T.dt.ptr[K0 + 6]; g.colC = T.dt.ptr[K0 + 7]; g.baseC = baseT;
      g.M = T.Nr(); g.N = o; g.K = T.Mr(); g.alpha = -1.0; g.beta = 1.0;
      run(g);
    }
  }
}

// Block size of the grouped tensor-core form: GEMM rows (u, x_l) = o nb fill
// the units' rows well (256 on cluster pairs, else 128), the padded virtual range
// vp = NB nb stays close to v, and W (nb^3 o^3 floats per buffer) stays within 64 MiB a
// buffer; ties go to the larger block (fewer, larger launches).  With rows counted in
// 128s on pairs, o = 13, v = 117 took nb = 9 (117 of 256 rows, 455 launches, 27.5 ms)
// where nb = 17 (84 launches) takes 16.8 ms.  The tuning key t_nb overrides it.
int choose_nb_grouped(int64_t o, int64_t v) {
  const int64_t forced = tune_value("t_nb", 0);
  if (forced >= 1) return (int)std::min<int64_t>(forced, v);
  int best = 1;
  double best_score = -1.0;
  const double o3 = (double)o * o * pad4(o), bm = TcEngine::pair_available() ? 256.0 : 128.0;
  for (int nb = 1; nb <= std::min<int64_t>(v, 64); nb++) {
    if (nb > 1 && (double)nb * nb * nb * o3 * 4.0 > double(64 << 20)) break;
    const double rows = (double)o * nb;
    const double effM = rows / (bm * std::ceil(rows / bm));
    const double vp = (double)ceil_div(v, nb) * nb;
    const double effV = std::pow((double)v / vp, 3.0);
    const double score = effM * effV;
    if (score >= best_score * (1.0 - 1e-9)) {
      best = nb;
      best_score = std::max(score, best_score);
    }
  }
  return best;
}

// Block size of the sliced FP64 form: rows (u, x_l) in 128-row tiles, padded
// virtuals close to v, the three FP64 W buffers within 96 MiB so that they stay in L2
// between the GEMM and the energy kernel; ties go to the larger block.
int choose_nb_sliced(int64_t o, int64_t v) {
  const int64_t forced = tune_value("t_nb", 0);
  if (forced >= 1) return (int)std::min<int64_t>(forced, v);
  int best = 1;
  double best_score = -1.0;
  const double o3 = (double)o * o * o;
  for (int nb = 1; nb <= std::min<int64_t>(v, 64); nb++) {
    if (nb > 1 && (double)nb * nb * nb * o3 * 24.0 > double(96 << 20)) break;
    const double rows = (double)o * nb;
    const double vp = (double)ceil_div(v, nb) * nb;
    const double score = rows / (128.0 * std::ceil(rows / 128.0)) * std::pow((double)v / vp, 3.0);
    if (score >= best_score * (1.0 - 1e-9)) {
      best = nb;
      best_score = std::max(score, best_score);
    }
  }
  return best;
}

// Exponents of the sliced FP64 form.  All four segments of a group add up in one sum per
// output, so P and t2 rows of a (u, x) share an exponent, and Q (t2 too) and R rows of an (s, t);
// t2 2^s meets R 2^-s there, with one shift s for the call that brings amplitudes and
// integrals to one size on either side (unshifted, amplitudes of 2^-30 had 33 bits of their 53).
// raw: P, t2 ([nA] each), Q, R ([nB] each), 0 for all zeros; out: the exponents to cut P, t2, Q and
// R with, kRowNonFinite kept; mx: the four tensors' largest.
__global__ void __launch_bounds__(1024) triples_exps_kernel(const int *__restrict__ raw, int64_t nA, int64_t nB,
                                                            int *__restrict__ out, int *__restrict__ mx) {
  chain();
  __shared__ int m[4];
  if (threadIdx.x < 4) m[threadIdx.x] = 0;
  __syncthreads();
  const int64_t n[4] = {nA, nA, nB, nB}, at[4] = {0, nA, 2 * nA, 2 * nA + nB};
  for (int q = 0; q < 4; q++) {
    int e = 0;
    for (int64_t i = threadIdx.x; i < n[q]; i += blockDim.x) e = max(e, raw[at[q] + i]);
    atomicMax(&m[q], e);
  }
  __syncthreads();
  if (threadIdx.x < 4) mx[threadIdx.x] = m[threadIdx.x];
  const int s = (m[0] && m[1] && m[2] && m[3]) ? ((m[0] - m[1]) + (m[3] - m[2])) / 2 : 0;
  for (int side = 0; side < 2; side++) {
    const int sh = side ? -s : s;  // of the second tensor of the side
    const int *x = raw + at[2 * side], *y = x + n[2 * side];
    int *ox = out + at[2 * side], *oy = ox + n[2 * side];
    for (int64_t i = threadIdx.x; i < n[2 * side]; i += blockDim.x) {
      const bool bad = x[i] == kRowNonFinite || y[i] == kRowNonFinite;
      const int e = x[i] || y[i] ? max(1, max(x[i] ? x[i] : 1, y[i] ? y[i] + sh : 1)) : 0;
      ox[i] = bad ? kRowNonFinite : e;
      oy[i] = bad ? kRowNonFinite : (e ? e - sh : 0);
    }
  }
}

// Sums of squares of P and Q for every f, t2 and R for every m, relative to the tensor's largest
// exponent: out[column][part], columns P (v), Q (v), t2 (o), R (o).
constexpr int kSquareParts = 8;
struct SquareOps {
  const double *src[4];
  const int64_t *row[4], *k[4];
  int64_t rows[4];
  int v, o;
};
__global__ void __launch_bounds__(256) triples_squares_kernel(SquareOps ops, const int *__restrict__ mx,
                                                              float *__restrict__ out) {
  chain();
  __shared__ float red[8];
  int c = blockIdx.x / kSquareParts;
  const int part = blockIdx.x % kSquareParts;
  const int q = c < ops.v ? 0 : c < 2 * ops.v ? 1 : c < 2 * ops.v + ops.o ? 2 : 3;
  c -= q < 2 ? q * ops.v : 2 * ops.v + (q - 2) * ops.o;
  const int e = mx[q == 0 ? 0 : q == 1 ? 2 : q == 2 ? 1 : 3];  // (mx in the order P, t2, Q, R)
  const double *src = ops.src[q] + ops.k[q][c];
  float s = 0.0f;
  for (int64_t r = part * 256 + threadIdx.x; r < ops.rows[q]; r += 256 * kSquareParts) {
    const float x = __uint_as_float(slice_magnitude(src[ops.row[q][r]], e) << 16);
    s = fmaf(x, x, s);
  }
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) s += red[w];
    out[blockIdx.x] = s;
  }
}

// Whether the sliced form is as accurate as FP64 multiply-adds for the energy, a sum over all W of
// a block: the squared errors of all outputs (see slice_left, gemm_slice.cu) are compared,
//   2^-122 / 3 sum [(column max)^2 a_k^2 + (row max)^2 b_k^2]  <=  0.16 2^-106 sum (a_k b_k)^2
// with a factor of 2 to spare; dense tensors pass by a factor of 50 and more.  False also
// where an exponent leaves the range of FP64's.
// eA: exponents as used, the tensors' largest, the sums of squares.
bool triples_slices_hold(const int *eA, int64_t o, int64_t v, int64_t nA, int64_t nB) {
  const int *eB = eA + 2 * nA, *mx = eB + 2 * nB, *squares = mx + 4;
  for (const int *e = eA; e < mx; e++)
    if (*e >= kRowNonFinite) return false;
  if (mx[1] == 0) return true;  // no t2: every W is exactly zero
  auto col = [&](int64_t c) {
    double s = 0.0;
    for (int p = 0; p < kSquareParts; p++) {
      float x;
      std::memcpy(&x, squares + c * kSquareParts + p, sizeof(x));
      s += x;
    }
    return s;
  };
  int a = 1, b = 1;  // largest exponents of the two sides
  for (int64_t i = 0; i < nA; i++) a = std::max(a, eA[i]);
  for (int64_t i = 0; i < nB; i++) b = std::max(b, eB[i]);
  double ra = 0.0, rb = 0.0;  // sums of (row max)^2, (column max)^2 over (u, x), (s, t)
  for (int64_t i = 0; i < nA; i++)
    if (eA[i]) ra += std::exp2(2.0 * (eA[i] - a));
  for (int64_t i = 0; i < nB; i++)
    if (eB[i]) rb += std::exp2(2.0 * (eB[i] - b));
  // the tensors' largest relative to their side's: t2 and R carry the shift
  int64_t shift = 0;
  for (int64_t i = 0; i < nA; i++)
    if (eA[i]) shift = eA[i] - eA[nA + i];
  const double scale[4] = {2.0 * (mx[0] - a), 2.0 * (mx[2] - b), 2.0 * (mx[1] + shift - a), 2.0 * (mx[3] - shift - b)};
  double norms[2] = {0.0, 0.0}, products = 0.0;
  for (int pair = 0; pair < 2; pair++) {
    const int64_t n = pair ? o : v, c0 = pair ? 2 * v : 0;
    const double fa = std::exp2(scale[2 * pair]), fb = std::exp2(scale[2 * pair + 1]);
    for (int64_t f = 0; f < n; f++) {
      const double x = col(c0 + f) * fa, y = col(c0 + n + f) * fb;
      norms[0] += x;
      norms[1] += y;
      products += x * y;
    }
  }
  return (double)v * (rb * norms[0] + ra * norms[1]) <= 16384.0 * products;
}

// FP64 (T) with the 12 products of a block triple as one grouped launch on the
// tensor cores' exact slices (gemm_slice.h), in the three groups of four K segments
// described in rccsd_triples.  False (nothing computed) when the packs do not fit into device
// memory or the slices do not hold the operands.
bool triples_fp64_sliced(Ctx &ctx, const double *d_eri, int64_t nmo, int64_t o, const double *d_eps,
                         const double *d_t1, const double *d_t2, const Control &ctl, TriplesStats *stats,
                         const double *d_B, int64_t naux, double &e_t) {
  const int64_t v = nmo - o, N = nmo, o2 = o * o, o3 = o2 * o;
  cudaStream_t s = ctx.stream;
  const int nb = choose_nb_sliced(o, v);
  const int64_t NB = ceil_div(v, nb), vp = NB * nb;
  const int64_t Mg = o * nb, Ng = o2, prob = Mg * Ng;
  if (!ctx.slice_engine() || !ctx.slice_engine()->usable(o * vp * vp, o2 * vp, v)) return false;
  const int64_t ntrip = v * (v + 1) * (v + 2) / 6;
  TriplesSetup T;
  T.o = o;
  T.v = v;
  T.N = N;
  T.nb = nb;
  T.NB = NB;
  T.vp = vp;
  SliceEngine &se = *ctx.slice_engine();
  SlicedPack pP, pQ, pQ2, pR, pR2, pTx;
  DevTables pdt, gdt;
  DevMem exps, W, orbits;
  DTensor energies;
  const int64_t nA = o * vp, nexp = 2 * nA + 2 * o2, nsq = (2 * v + 2 * o) * kSquareParts;
  std::vector<uint32_t> ot = orbit_table(o);
  const int norbits = (int)ot.size();
  try {
    {
      TimedScope ts(ctx.timer, "phase:triples_setup", 0.0, 0.0, s);
      T.build(ctx, d_eri, d_t2, d_B, naux, Backend::FP64);
    }
    TimedScope ts(ctx.timer, "phase:triples_pack", 0.0, 0.0, s);
    // rows as in the mixed form: P (i,x | y,Y,X), Q (j,k | z,Z), R (i,j | x,X),
    // t2 (u,x | z,X,Z), Q (k,j | z,Z), R (j,i | x,X); then the exponent index of each:
    // i + o x over all virtuals (P, t2), s + o t (Q, R)
    pdt.build(ctx, {table({{o, 1}, {nb, o * v}, {nb, o * v * vp}, {NB, o * v * vp * nb}, {NB, o * v * nb}}),
                    table({{o, v}, {o, v * o}, {nb, v * o2}, {NB, v * o2 * nb}}),
                    table({{o, 1}, {o, o}, {nb, o3}, {NB, o3 * nb}}),
                    table({{o, o}, {nb, o2 * vp}, {nb, o2}, {NB, o2 * vp * nb}, {NB, o2 * nb}}),
                    table({{o, v * o}, {o, v}, {nb, v * o2}, {NB, v * o2 * nb}}),
                    table({{o, o}, {o, 1}, {nb, o3}, {NB, o3 * nb}}),
                    table({{o, 1}, {nb, o}, {nb, 0}, {NB, 0}, {NB, o * nb}}),
                    table({{o, 1}, {nb, o}, {nb, 0}, {NB, o * nb}, {NB, 0}}),
                    table({{o, 1}, {o, o}, {nb, 0}, {NB, 0}})});
    // P, t2 (o vp each), Q, R (o^2 each): exponents as found, then as used; the largest; the
    // sums of squares
    exps.alloc((size_t)(2 * nexp + 4 + nsq) * sizeof(int));
    int *raw = exps.as<int>(), *use = raw + nexp;
    SCESS_CUDA(cudaMemsetAsync(raw, 0, (size_t)nexp * sizeof(int), s));
    const int64_t *kP = T.dt.ptr[T.kOperand + 1], *kT = T.dt.ptr[T.kOperand + 7], *kQ = T.dt.ptr[T.kOperand + 3],
                  *kR = T.dt.ptr[T.kOperand + 5];
    const int64_t rP = o * vp * vp, rQ = o2 * vp;
    struct Op {
      const DTensor &t;
      int row;
      int64_t rows;
      const int64_t *k;
      int64_t K;
      bool unitK;
      int64_t e;  // of its exponents
      int idx;
      bool neg;
      SlicedPack &out;
    };
    const int64_t oT = nA, oQ = 2 * nA, oR = 2 * nA + o2;
    const Op ops[6] = {{T.P, 0, rP, kP, v, false, 0, 6, false, pP},   {T.T2p, 3, rP, kT, o, true, oT, 7, true, pTx},
                       {T.Qt, 1, rQ, kQ, v, true, oQ, 8, false, pQ},  {T.Qt, 4, rQ, kQ, v, true, oQ, 8, false, pQ2},
                       {T.Rt, 2, rQ, kR, o, false, oR, 8, false, pR}, {T.Rt, 5, rQ, kR, o, false, oR, 8, false, pR2}};
    for (const Op &q : ops)
      se.row_exps(q.t.p(), pdt.ptr[q.row], q.rows, q.k, q.K, q.unitK, raw + q.e, pdt.ptr[q.idx]);
    launch(triples_exps_kernel, 1, 1024, 0, s, (const int *)raw, nA, o2, use, use + nexp);
    SCESS_CHECK_LAUNCH();
    SquareOps sq = {};
    sq.v = (int)v;
    sq.o = (int)o;
    for (int q = 0; q < 4; q++) {
      const Op &x = ops[q == 0 ? 0 : q == 1 ? 2 : q == 2 ? 1 : 4];
      sq.src[q] = x.t.p();
      sq.row[q] = pdt.ptr[x.row];
      sq.k[q] = x.k;
      sq.rows[q] = x.rows;
    }
    launch(triples_squares_kernel, (unsigned)nsq, 256, 0, s, sq, (const int *)(use + nexp),
           reinterpret_cast<float *>(use + nexp + 4));
    SCESS_CHECK_LAUNCH();
    for (const Op &q : ops)
      se.pack_with_exps(q.t.p(), pdt.ptr[q.row], q.rows, q.k, q.K, q.unitK, use + q.e, pdt.ptr[q.idx], q.neg, q.out);
    gdt.build(ctx, {table({{Mg, 1}}), table({{Ng, Mg}})});
    W.alloc((size_t)(3 * nb * nb * prob) * sizeof(double));
    energies = DTensor({std::max<int64_t>(ntrip, 1)});
    orbits.alloc(ot.size() * sizeof(uint32_t));
  } catch (const Error &e) {
    if (e.code != SCESS_ERR_OOM) throw;
    return false;
  }
  SCESS_CUDA(cudaMemsetAsync(energies.p(), 0, energies.size() * sizeof(double), s));
  SCESS_CUDA(cudaMemcpyAsync(orbits.as<void>(), ot.data(), ot.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
  std::vector<int> he(nexp + 4 + nsq);
  const int *use = exps.as<int>() + nexp;
  SCESS_CUDA(cudaMemcpyAsync(he.data(), use, he.size() * sizeof(int), cudaMemcpyDeviceToHost, s));
  ctx.sync();  // (ot and he are host vectors of this scope)
  if (!triples_slices_hold(he.data(), o, v, nA, o2)) return false;
  const int64_t p1 = o | 1, p2 = (p1 * o) | 1;
  const unsigned threads = (unsigned)std::min<int64_t>(256, round_up(norbits, 32));
  const size_t smem = (size_t)std::max<int64_t>(p2 * o + 3 * p1 * o + 4 * o, threads) * 8;
  SCESS_CUDA(cudaFuncSetAttribute(triples_energy_orbit64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  SliceProblemSet ps;
  const SlicedPack *packs[6] = {&pP, &pQ, &pQ2, &pR, &pR2, &pTx};
  const int bn = SliceEngine::tile_n(Ng);
  for (int i = 0; i < 6; i++) ps.maps[i] = SliceEngine::map_of(*packs[i], i == 0 || i == 5 ? 128 : bn);
  ps.nmaps = 6;
  ps.M = Mg;
  ps.N = Ng;
  ps.ny = ps.nz = nb;
  ps.ng = 3;
  ps.nseg = 4;
  const int mA[4] = {0, 0, 5, 5}, mB[4] = {1, 2, 3, 4};
  for (int q = 0; q < 4; q++) {
    ps.seg[q].mapA = mA[q];
    ps.seg[q].mapB = mB[q];
    ps.seg[q].Kpad = q < 2 ? pP.Kpad : pTx.Kpad;
  }
  ps.expA = use;
  ps.expB = use + 2 * nA;
  ps.C = W.d();
  for (int g = 0; g < 3; g++) {
    ps.cy[g] = prob;
    ps.cz[g] = nb * prob;
    ps.cg[g] = g * nb * nb * prob;
    ps.rowC[g] = gdt.ptr[0];
    ps.colC[g] = gdt.ptr[1];
  }
  int64_t blocks_done = 0;
  for (int64_t A = 0; A < NB; A++)
    for (int64_t Bk = 0; Bk <= A; Bk++)
      for (int64_t C = 0; C <= Bk; C++) {
        if ((blocks_done & 15) == 0) ctl.poll();                                     // :123
        const int64_t U[3] = {A, Bk, C};
        const int kRoles[3][3] = {{0, 1, 2}, {1, 0, 2}, {2, 0, 1}};  // (x, y, z) of group g
        const int64_t rp = o * nb * nb, rq = o2 * nb;
        double nprob = 0.0;
        for (int g = 0; g < 3; g++) {
          const int64_t X = U[kRoles[g][0]], Yb = U[kRoles[g][1]], Z = U[kRoles[g][2]];
          SliceSegment &s0 = ps.seg[0], &s1 = ps.seg[1], &s2 = ps.seg[2], &s3 = ps.seg[3];
          s0.rowA0[g] = rp * (Yb + NB * X); s0.rowAy[g] = Mg;   // P(u,f,x,y) Q(f,s,t,z)
          s0.rowB0[g] = rq * Z;             s0.rowBz[g] = o2;
          s1.rowA0[g] = rp * (Z + NB * X);  s1.rowAz[g] = Mg;   // P(u,f,x,z) Q(f,t,s,y)
          s1.rowB0[g] = rq * Yb;            s1.rowBy[g] = o2;
          s2.rowA0[g] = rp * (X + NB * Z);  s2.rowAz[g] = Mg;   // -t2(m,u,z,x) R(s,t,m,y)
          s2.rowB0[g] = rq * Yb;            s2.rowBy[g] = o2;
          s3.rowA0[g] = rp * (X + NB * Yb); s3.rowAy[g] = Mg;   // -t2(m,u,y,x) R(t,s,m,z)
          s3.rowB0[g] = rq * Z;             s3.rowBz[g] = o2;
          ps.expA0[g] = Mg * X;
          ps.tri[g] = Yb == Z;  // problems y < z of a diagonal block feed no unique triple
          nprob += ps.tri[g] ? nb * (nb + 1) / 2.0 : (double)nb * nb;
        }
        se.gemm_grouped(ps, nprob * 2.0 * (double)Mg * Ng * (2.0 * v + 2.0 * o), "slice_gemm[triples]");
        TimedScope ts(ctx.timer, "triples_energy", 0.0, 24.0 * nb * nb * prob, s);
        launch(triples_energy_orbit64_kernel, (unsigned)(nb * nb * nb), threads, smem, s, W.d(), o, v, nb, A, Bk, C,
               d_eps, d_t1, T.S.p(), orbits.as<uint32_t>(), norbits, energies.p());
        SCESS_CHECK_LAUNCH();
        blocks_done++;
      }
  sum_energies_kernel<<<1, 1024, 0, s>>>(ntrip, energies.p(), ctx.dscalars);
  SCESS_CHECK_LAUNCH();
  SCESS_CUDA(cudaMemcpyAsync(ctx.hscalars, ctx.dscalars, sizeof(double), cudaMemcpyDeviceToHost, s));
  ctx.sync();
  if (stats) {
    stats->nb = nb;
    stats->block_triples = blocks_done;
  }
  e_t = ctx.hscalars[0];
  return true;
}

// (T) with blocks of nb virtuals: the mixed form, or FP64 with 12 products a block triple.
double triples_blocked(Ctx &ctx, const double *d_eri, int64_t nmo, int64_t o, const double *d_eps, const double *d_t1,
                       const double *d_t2, bool mixed, const Control &ctl, TriplesStats *stats, const double *d_B,
                       int64_t naux, int nb) {
  const int64_t v = nmo - o, N = nmo;
  cudaStream_t s = ctx.stream;
  const int64_t NB = ceil_div(v, nb), vp = NB * nb;
  const int64_t o2 = o * o, o3 = o2 * o;

  TriplesSetup T;
  T.o = o;
  T.v = v;
  T.N = N;
  T.nb = nb;
  T.NB = NB;
  T.vp = vp;
  {  // (device time of the whole setup; "phase:" timers enclose other timers)
    TimedScope ts(ctx.timer, "phase:triples_setup", 0.0, 0.0, s);
    T.build(ctx, d_eri, d_t2, d_B, naux, mixed ? Backend::TENSOR : Backend::FP64);
  }
  const DTensor &P = T.P, &Qt = T.Qt, &Rt = T.Rt, &T2p = T.T2p;
  const DevTables &dt = T.dt;
  const size_t kOperand = T.kOperand;

  const int64_t ntrip = v * (v + 1) * (v + 2) / 6;
  DTensor energies({std::max<int64_t>(ntrip, 1)});
  SCESS_CUDA(cudaMemsetAsync(energies.p(), 0, energies.size() * sizeof(double), s));
  // FP64: W in FP64.  MIXED: W in FP32 with runs of i padded to op floats (see pad4), either three buffers the groups store into (nw = 3) or
  // one the groups add into with L2 reductions (nw = 1: zeroed here, cleared
  // again by every energy launch after it has read it)
  const int nw = tune_value("t_wbuf", kTriplesWBuffers) == 3 ? 3 : 1;
  const int64_t op = pad4(o), o2p = o * op, o3p = o * o2p;
  const size_t wbytes = (size_t)nb * nb * nb * (mixed ? 4 * nw * o3p : 8 * o3);
  DevMem W(wbytes);
  if (mixed && nw == 1) SCESS_CUDA(cudaMemsetAsync(W.as<void>(), 0, wbytes, s));
  const int64_t p1 = o | 1, p2 = (p1 * o) | 1;
  // the mixed energy kernel keeps (Y, W) in shared memory where two CTAs fit an SM
  const size_t wsmem = (size_t)(16 * o + 12 * o2p + 8 * p2 * o);
  const bool ws = 2 * (wsmem + 1024) <= 228 * 1024;
  const size_t ysmem = mixed ? (ws ? wsmem : (size_t)(16 * o + 12 * p1 * o + 4 * p2 * o + 8))
                             : (size_t)(p2 * o + 3 * o2 + 4 * o) * 8;
  const auto orbit_kernel = nw == 1 ? (ws ? triples_energy_orbit_kernel<1, true> : triples_energy_orbit_kernel<1, false>)
                                    : (ws ? triples_energy_orbit_kernel<3, true> : triples_energy_orbit_kernel<3, false>);
  if (ysmem > 200 * 1024) throw Error(SCESS_ERR_UNSUPPORTED, "(T): o^3 too large for one CTA");
  if (o > 255) throw Error(SCESS_ERR_UNSUPPORTED, "(T): more than 255 occupied orbitals");
  if (mixed && o > kEnergyMaxO)
    throw Error(SCESS_ERR_UNSUPPORTED, "(T), mixed form: more than 32 occupied orbitals");
  DevMem orbits;
  int norbits = 0;
  if (mixed) {
    SCESS_CUDA(cudaFuncSetAttribute(orbit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ysmem));
    const std::vector<uint32_t> ot = orbit_table(o);
    norbits = (int)ot.size();
    orbits.alloc(ot.size() * sizeof(uint32_t));
    SCESS_CUDA(cudaMemcpyAsync(orbits.as<void>(), ot.data(), ot.size() * sizeof(uint32_t),
                               cudaMemcpyHostToDevice, s));
    ctx.sync();  // (ot is a host vector of this scope)
  } else {
    SCESS_CUDA(cudaFuncSetAttribute(triples_energy_kernel<double, double>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ysmem));
  }

  // MIXED: the 12 GEMMs of a block triple regroup into three problem sets.
  // Group g has the roles (x, y, z) = (a, b, c), (b, a, c), (c, a, b) and, for
  // each (y_l, z_l), the GEMM
  //   W_g[(u, x_l), (s, t)] =   sum_f P(u,f,x,y) Q(f,s,t,z) + sum_f P(u,f,x,z) Q(f,t,s,y)
  //                           - sum_m t2(m,u,z,x) R(s,t,m,y) - sum_m t2(m,u,y,x) R(t,s,m,z)
  // where u is x's occupied partner (i, j or k for x = a, b, c) and (s, t) the
  // other two occupied indices in order: the P.Q terms of the permutations
  // that put x's pair on the rows and the R.t2 terms whose t2 carries it (four
  // K segments of one accumulation); W = W_0 + W_1 + W_2, each group adding
  // its product into W at its (a, b, c, i, j, k) positions.  The operands are
  // packed once per call into block-grouped FP16 hi/lo rows; the t2 rows are
  // packed negated, and the A side (P, t2) and the B side (Q, R) each share one
  // scale so that all segments carry the same scale product.
  Packed pP, pQ, pQ2, pR, pR2, pTx;
  const int tbn = 256;
  const int tbk = TcEngine::k_block(tbn);
  // 256 x 256 units on cluster pairs of SMs (each SM stages half of B) where
  // the device runs the pair kernel, else one SM per 128 x 256 unit
  const bool tpair = TcEngine::pair_available();
  const int bbox = tpair ? 128 : tbn;  // B rows staged per CTA
  // K block of the t2.R segments (K = o): 32 in the 64-wide kernel when o <= 32
  // (half-filled stages instead of mostly-padding 64-wide ones)
  const int rbk = (tbk == 64 && o <= 32) ? 32 : tbk;
  CUtensorMap mP{}, mQ{}, mQ2{}, mR{}, mR2{}, mTx{};
  DevTables gdt;  // W_g row / column tables
  DevMem Sf;    // (ia|jb) as FP32 for the energy kernel (padded rows)
  DevMem etab;  // the orbits (uint4), eps as FP32 hi + lo (nmo float2), then t1 in FP32
  uint4 *orb = nullptr;
  float2 *ehl = nullptr;
  float *t1f = nullptr;
  const int64_t Mg = o * nb, Ng = o2p;  // (columns (s, t), s padded to op)
  if (mixed) {
    TimedScope ts(ctx.timer, "phase:triples_pack", 0.0, 0.0, s);
    TcEngine &tc = ctx.tensor_cores();
    std::vector<TableSpec> pt;
    // P rows r = i + o(x + nb(y + nb(Y + NB X))):  P(i, f, X nb + x, Y nb + y)
    pt.push_back(table({{o, 1}, {nb, o * v}, {nb, o * v * vp}, {NB, o * v * vp * nb}, {NB, o * v * nb}}));
    // Q rows r = j + op(k + o(z + nb Z)):  Q(f, j, k, Z nb + z), padding repeated from j = o - 1
    pt.push_back(padded(table({{op, v}, {o, v * o}, {nb, v * o2}, {NB, v * o2 * nb}}), o, false));
    // R rows r = i + op(j + o(x + nb X)):  R(i, j, m, X nb + x)
    pt.push_back(padded(table({{op, 1}, {o, o}, {nb, o3}, {NB, o3 * nb}}), o, false));
    // t2 rows r = u + o(x + nb(z + nb(X + NB Z))):  t2(m, u, Z nb + z, X nb + x)
    pt.push_back(table({{o, o}, {nb, o2 * vp}, {nb, o2}, {NB, o2 * vp * nb}, {NB, o2 * nb}}));
    // Q rows in (k, j) order: r = k + op(j + o(z + nb Z))
    pt.push_back(padded(table({{op, v * o}, {o, v}, {nb, v * o2}, {NB, v * o2 * nb}}), o, false));
    // R rows in (j, i) order: r = j + op(i + o(x + nb X))
    pt.push_back(padded(table({{op, o}, {o, 1}, {nb, o3}, {NB, o3 * nb}}), o, false));
    DevTables pdt;
    pdt.build(ctx, pt);
    DevMem maxw(2 * sizeof(unsigned));
    unsigned *mx = maxw.as<unsigned>();
    SCESS_CUDA(cudaMemsetAsync(mx, 0, 2 * sizeof(unsigned), s));
    tc.maxabs_into(P.p(), pdt.ptr[0], o * vp * vp, dt.ptr[kOperand + 1], v, false, mx);
    tc.maxabs_into(T2p.p(), pdt.ptr[3], o * vp * vp, dt.ptr[kOperand + 7], o, true, mx);
    tc.maxabs_into(Qt.p(), pdt.ptr[1], o2p * vp, dt.ptr[kOperand + 3], v, true, mx + 1);
    tc.maxabs_into(Rt.p(), pdt.ptr[2], o2p * vp, dt.ptr[kOperand + 5], o, false, mx + 1);
    tc.pack_with_max(P.p(), pdt.ptr[0], o * vp * vp, dt.ptr[kOperand + 1], v, false, 128, mx, false, pP);
    tc.pack_with_max(T2p.p(), pdt.ptr[3], o * vp * vp, dt.ptr[kOperand + 7], o, true, 128, mx, true, pTx, rbk);
    tc.pack_with_max(Qt.p(), pdt.ptr[1], o2p * vp, dt.ptr[kOperand + 3], v, true, 128, mx + 1, false, pQ);
    tc.pack_with_max(Qt.p(), pdt.ptr[4], o2p * vp, dt.ptr[kOperand + 3], v, true, 128, mx + 1, false, pQ2);
    tc.pack_with_max(Rt.p(), pdt.ptr[2], o2p * vp, dt.ptr[kOperand + 5], o, false, 128, mx + 1, false, pR, rbk);
    tc.pack_with_max(Rt.p(), pdt.ptr[5], o2p * vp, dt.ptr[kOperand + 5], o, false, 128, mx + 1, false, pR2, rbk);
    ctx.sync();
    // B side (Q, R rows): tiles of tbn columns; 256 halves the A-operand
    // shared-memory traffic per FLOP (SCESS_T_BN=128 selects the narrow tiles).
    // Boxes as wide as the kernel's K block.
    mP = TcEngine::map_of(pP, 128, tbk);
    mQ = TcEngine::map_of(pQ, bbox, tbk);
    mQ2 = TcEngine::map_of(pQ2, bbox, tbk);
    mR = TcEngine::map_of(pR, bbox, rbk);
    mR2 = TcEngine::map_of(pR2, bbox, rbk);
    mTx = TcEngine::map_of(pTx, 128, rbk);
    // Every group writes its (u, s, t) at the triple's (i, j, k), i + op j + o2p k.
    // Rows (u, x_l), columns (s, t): g = 0 (x = a): (u,s,t) = (i,j,k), padding skipped;
    // g = 1 (x = b): (j,i,k); g = 2 (x = c): (k,i,j), both with the padding of i.
    // nw = 3: buffer g holds W_g[(y_l nb + z_l) nb + x_l]; nw = 1:
    // W[(a_l nb + b_l) nb + c_l], the (y_l, z_l) strides being the problem offsets cy, cz.
    const int64_t xa = nw == 3 ? o3p : nb * nb * o3p, xb = nw == 3 ? o3p : nb * o3p;
    gdt.build(ctx, {table({{o, 1}, {nb, xa}}), padded(table({{op, op}, {o, o2p}}), o, true),
                    table({{o, op}, {nb, xb}}), table({{op, 1}, {o, o2p}}),
                    table({{o, o2p}, {nb, o3p}}), table({{op, 1}, {o, op}})});
    Sf.alloc((size_t)o2p * v * v * sizeof(float));
    etab.alloc((size_t)norbits * sizeof(uint4) + (size_t)N * sizeof(float2) + (size_t)o * v * sizeof(float));
    orb = etab.as<uint4>();
    ehl = reinterpret_cast<float2 *>(orb + norbits);
    t1f = reinterpret_cast<float *>(ehl + N);
    energy_tables_kernel<<<(unsigned)std::min<int64_t>(ceil_div(N + o * v + norbits, 256), 4 * kNumSMs), 256, 0, s>>>(
        d_eps, N, d_t1, o * v, orbits.as<uint32_t>(), norbits, ehl, t1f, orb);
    SCESS_CHECK_LAUNCH();
    to_f32_rows_kernel<<<(unsigned)std::min<int64_t>(ceil_div(o2p * v * v, 256), 16 * kNumSMs), 256, 0, s>>>(
        T.S.p(), v * v * o, o, op, Sf.as<float>());
    SCESS_CHECK_LAUNCH();
  }
  // (i, j) pairs spread evenly over at most 256 threads
  const unsigned e3threads =
      (unsigned)round_up(ceil_div(o2, ceil_div(o2, 256)), 32);
  // MIXED: consecutive launches overlap (programmatic dependent launches);
  // SCESS_TUNE t_pdl = 0 serialises them, for comparison
  const bool pdl = tune_value("t_pdl", 1) != 0;
  int64_t blocks_done = 0;
  for (int64_t A = 0; A < NB; A++)
    for (int64_t Bk = 0; Bk <= A; Bk++)
      for (int64_t C = 0; C <= Bk; C++) {
        if ((blocks_done & 15) == 0) ctl.poll();                                   // :123
        const int64_t U[3] = {A, Bk, C};
        if (mixed) {
          TcEngine &tc = ctx.tensor_cores();
          TcProblemSet ps;
          ps.maps[0] = mP;
          ps.maps[1] = mQ;
          ps.maps[2] = mQ2;
          ps.maps[3] = mR;
          ps.maps[4] = mR2;
          ps.maps[5] = mTx;
          ps.nmaps = 6;
          ps.M = Mg;
          ps.N = Ng;
          ps.ny = nb;
          ps.nz = nb;
          ps.ng = 3;
          ps.nseg = 4;
          // TMEM drains per tile.  The FP32 accumulation inside the tensor
          // core truncates, so the error of E_T grows with the products
          // accumulated between drains: measured 1.7e-7 / 4.6e-7 / 1.1e-6
          // relative to FP64 with a drain per 64 / 128 / 256 K.
          ps.kbd = (int)tune_value("t_kbd", kTriplesKbd);
          if (ps.kbd != 1 && ps.kbd != 2 && ps.kbd != 4) ps.kbd = kTriplesKbd;
          ps.bn = tbn;
          ps.bk = tbk;
          ps.pair = tpair;
          // problem offsets of (y_l, z_l): nw = 3, in the group's own buffer;
          // nw = 1, in W with g = 0 (y, z) = (b, c), g = 1 (a, c), g = 2 (a, b)
          for (int g = 0; g < 3; g++) {
            ps.cy[g] = nb * nb * o3p;
            ps.cz[g] = nb * o3p;
          }
          if (nw == 1) {
            ps.cy[0] = nb * o3p;      ps.cz[0] = o3p;
            ps.cy[1] = nb * nb * o3p; ps.cz[1] = o3p;
            ps.cy[2] = nb * nb * o3p; ps.cz[2] = nb * o3p;
          }
          const int kRoles[3][3] = {{0, 1, 2}, {1, 0, 2}, {2, 0, 1}};  // (x, y, z) of group g
          const int64_t rp = o * nb * nb, rq = o2p * nb;                // block strides of the packs
          TcSegment &s0 = ps.seg[0], &s1 = ps.seg[1], &s2 = ps.seg[2], &s3 = ps.seg[3];
          s0.mapA = 0; s0.mapB = 1; s0.Kpad = pP.Kpad;   // P(u,f,x,y) Q(f,s,t,z)
          s1.mapA = 0; s1.mapB = 2; s1.Kpad = pP.Kpad;   // P(u,f,x,z) Q(f,t,s,y)
          s2.mapA = 5; s2.mapB = 3; s2.Kpad = pTx.Kpad;  // -t2(m,u,z,x) R(s,t,m,y)
          s3.mapA = 5; s3.mapB = 4; s3.Kpad = pTx.Kpad;  // -t2(m,u,y,x) R(t,s,m,z)
          s2.bk = s3.bk = rbk;
          for (int g = 0; g < 3; g++) {
            const int64_t X = U[kRoles[g][0]], Yb = U[kRoles[g][1]], Z = U[kRoles[g][2]];
            ps.cg[g] = nw == 3 ? g * nb * nb * nb * o3p : 0;
            s0.rowA0[g] = rp * (Yb + NB * X); s0.rowAy[g] = o * nb;
            s0.rowB0[g] = rq * Z;             s0.rowBz[g] = o2p;
            s1.rowA0[g] = rp * (Z + NB * X);  s1.rowAz[g] = o * nb;
            s1.rowB0[g] = rq * Yb;            s1.rowBy[g] = o2p;
            s2.rowA0[g] = rp * (X + NB * Z);  s2.rowAz[g] = o * nb;
            s2.rowB0[g] = rq * Yb;            s2.rowBy[g] = o2p;
            s3.rowA0[g] = rp * (X + NB * Yb); s3.rowAy[g] = o * nb;
            s3.rowB0[g] = rq * Z;             s3.rowBz[g] = o2p;
          }
          TcOut out;
          out.C = W.as<float>();
          out.fp32 = 1;
          out.rowC = gdt.ptr[0];
          out.colC = gdt.ptr[1];
          for (int g = 0; g < 3; g++) {
            ps.rowC[g] = gdt.ptr[2 * g];
            ps.colC[g] = gdt.ptr[2 * g + 1];
            // i is a column index of groups 1 and 2: quads of it, aligned
            ps.store_quads[g] = g > 0;
          }
          out.alpha = 1.0;
          out.beta = nw == 1 ? 1.0 : 0.0;  // nw = 1: W += each group's product (L2 reductions)
          TcEngine::set_scales(out, pP, pQ);
          // In a diagonal block triple a group's problems with y_l < z_l feed no
          // unique triple a >= b >= c: g0 (y, z) = (b, c) when B = C, g1 (a, c)
          // when A = C, g2 (a, b) when A = B.
          ps.tri[0] = Bk == C;
          ps.tri[1] = A == C;
          ps.tri[2] = A == Bk;
          double nprob = 0.0;
          for (int g = 0; g < 3; g++) nprob += ps.tri[g] ? nb * (nb + 1) / 2.0 : (double)nb * nb;
          const double flops = nprob * 2.0 * (double)Mg * o2 * (2.0 * v + 2.0 * o);
          // behind the previous block triple's energy kernel, the launch starts
          // its MMAs while that kernel finishes (W is stored to only after it)
          ps.pdl = pdl && blocks_done > 0;
          tc.gemm_grouped(ps, out, flops, "tc_gemm[triples]");
        } else {
          w_block_fp64(ctx, T, U, W.d());
        }
        const unsigned nblk = (unsigned)(nb * nb * nb);
        TimedScope ts(ctx.timer, "triples_energy", 0.0,
                      (double)nblk * o3 * (mixed ? (nw == 1 ? 2 : 3) * 4 : 8), s);
        if (mixed) {
          // a programmatic dependent of the grouped GEMM: its CTAs take the SMs
          // that GEMM pairs leave and stage their tables while the last pairs
          // finish; W is read after griddepcontrol.wait
          cudaLaunchConfig_t cfg = {};
          cudaLaunchAttribute at[1];
          at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
          at[0].val.programmaticStreamSerializationAllowed = 1;
          cfg.gridDim = dim3(nblk);
          cfg.blockDim = dim3(e3threads);
          cfg.dynamicSmemBytes = ysmem;
          cfg.stream = s;
          cfg.attrs = at;
          cfg.numAttrs = pdl ? 1 : 0;
          SCESS_CUDA(cudaLaunchKernelEx(&cfg, orbit_kernel, W.as<float>(), (int64_t)o, (int64_t)v, (int64_t)nb,
                                        (int64_t)A, (int64_t)Bk, (int64_t)C, (const float2 *)ehl,
                                        (const float *)t1f, (const float *)Sf.as<float>(), (const uint4 *)orb,
                                        norbits, energies.p()));
        } else
          triples_energy_kernel<double, double><<<nblk, 256, ysmem, s>>>(
              W.d(), o, v, nb, A, Bk, C, d_eps, d_t1, T.S.p(), energies.p());
        SCESS_CHECK_LAUNCH();
        blocks_done++;
      }
  sum_energies_kernel<<<1, 1024, 0, s>>>(ntrip, energies.p(), ctx.dscalars);
  SCESS_CHECK_LAUNCH();
  SCESS_CUDA(cudaMemcpyAsync(ctx.hscalars, ctx.dscalars, sizeof(double), cudaMemcpyDeviceToHost, s));
  ctx.sync();
  if (mixed) ctx.tensor_cores().check_error();
  if (stats) {
    stats->nb = nb;
    stats->block_triples = blocks_done;
  }
  return ctx.hscalars[0];
}

}  // namespace

double rccsd_triples(Ctx &ctx, const double *d_eri, int64_t nmo, int64_t o, const double *d_eps,
                     const double *d_t1, const double *d_t2, bool mixed, const Control &ctl,
                     TriplesStats *stats, const double *d_B, int64_t naux) {
  const int64_t v = nmo - o;
  {
    const int64_t q1 = o | 1, q2 = (q1 * o) | 1;
    if (!mixed && tune_value("f64", 0) != 2 && (q2 * o + 3 * o * o + 4 * o) * 8 <= 200 * 1024 &&
        o <= 255) {  // (else refused below)
      double e_t = 0.0;
      if (triples_fp64_sliced(ctx, d_eri, nmo, o, d_eps, d_t1, d_t2, ctl, stats, d_B, naux, e_t)) return e_t;
    }
  }
  int nb = mixed ? choose_nb_grouped(o, v) : choose_nb(o, v, 8, size_t(128) << 20);
  for (;;) {
    try {
      return triples_blocked(ctx, d_eri, nmo, o, d_eps, d_t1, d_t2, mixed, ctl, stats, d_B, naux, nb);
    } catch (const Error &e) {  // W doesn't fit: smaller blocks (unless a size was asked for)
      if (e.code != SCESS_ERR_OOM || nb == 1 || tune_value("t_nb", 0) >= 1) throw;
      nb = (nb + 1) / 2;
    }
  }
}

double rccsd_triples_vjp(Ctx &ctx, const double *d_eri, int64_t nmo, int64_t o,
                         const double *d_eps, const double *d_t1, const double *d_t2, double gE,
                         const Control &ctl, double *d_gt1, double *d_gt2, double *d_geri,
                         bool mixed) {
  const int64_t v = nmo - o, N = nmo;
  cudaStream_t s = ctx.stream;
  const int nb = choose_nb(o, v, 8, size_t(64) << 20);  // W and G, nb^3 o^3 FP64 each
  const int64_t NB = ceil_div(v, nb), vp = NB * nb;
  const int64_t o2 = o * o, o3 = o2 * o, N2 = N * N, N3 = N2 * N;
  TriplesSetup T;
  T.o = o;
  T.v = v;
  T.N = N;
  T.nb = nb;
  T.NB = NB;
  T.vp = vp;
  T.build(ctx, d_eri, d_t2);
  const bool integrals = d_geri != nullptr;
  DTensor gP, gRt;
  if (integrals) {
    gP = DTensor({o, v, vp, vp});
    gRt = DTensor({o, o, o, vp});
    SCESS_CUDA(cudaMemsetAsync(gP.p(), 0, gP.size() * sizeof(double), s));
    SCESS_CUDA(cudaMemsetAsync(gRt.p(), 0, gRt.size() * sizeof(double), s));
  }
  DTensor gQt({v, o, o, vp}), gT2p({o, o, vp, vp}), gS({o, o, v, v});
  SCESS_CUDA(cudaMemsetAsync(gQt.p(), 0, gQt.size() * sizeof(double), s));
  SCESS_CUDA(cudaMemsetAsync(gT2p.p(), 0, gT2p.size() * sizeof(double), s));
  SCESS_CUDA(cudaMemsetAsync(gS.p(), 0, gS.size() * sizeof(double), s));
  const int64_t ntrip = v * (v + 1) * (v + 2) / 6;
  DTensor energies({std::max<int64_t>(ntrip, 1)});
  SCESS_CUDA(cudaMemsetAsync(energies.p(), 0, energies.size() * sizeof(double), s));
  DevMem W((size_t)o3 * nb * nb * nb * 8), G((size_t)o3 * nb * nb * nb * 8);
  const int64_t p1 = o | 1, p2 = (p1 * o) | 1;
  const size_t gsmem = (size_t)(p2 * o + 5 * o2 + 7 * o) * 8;
  if (gsmem > 200 * 1024) throw Error(SCESS_ERR_UNSUPPORTED, "(T) gradient: o^3 too large for one CTA");
  SCESS_CUDA(cudaFuncSetAttribute(triples_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)gsmem));
  int64_t blocks_done = 0;
  for (int64_t A = 0; A < NB; A++)
    for (int64_t Bk = 0; Bk <= A; Bk++)
      for (int64_t C = 0; C <= Bk; C++) {
        if ((blocks_done & 15) == 0) ctl.poll();
        const int64_t U[3] = {A, Bk, C};
        w_block_fp64(ctx, T, U, W.d(), mixed);
        {
          TimedScope ts(ctx.timer, "triples_grad", 0.0, 0.0, s);
          triples_grad_kernel<<<(unsigned)(nb * nb * nb), 256, gsmem, s>>>(
              W.d(), G.d(), o, v, nb, A, Bk, C, d_eps, d_t1, T.S.p(), gE, energies.p(), d_gt1,
              gS.p());
          SCESS_CHECK_LAUNCH();
        }
        g_block_fp64(ctx, T, U, G.d(), integrals ? gP.p() : nullptr, gQt.p(),
                     integrals ? gRt.p() : nullptr, gT2p.p(), integrals, mixed);
        blocks_done++;
      }
  sum_energies_kernel<<<1, 1024, 0, s>>>(ntrip, energies.p(), ctx.dscalars);
  SCESS_CHECK_LAUNCH();
  SCESS_CUDA(cudaMemcpyAsync(ctx.hscalars, ctx.dscalars, sizeof(double), cudaMemcpyDeviceToHost, s));
  if (mixed) ctx.tensor_cores().check_error();

  // back through the repacks (RCCSD_T.cpp:30-56) into t2 and eri
  const TV g_t2 = cm(d_gt2, {o, o, v, v});
  TV q = gQt.v;  // Q(f,j,k,c) = t2(k,j,c,f)
  q.ext[3] = v;
  permute(ctx, "fjkc->kjcf", 1.0, q, 1.0, g_t2);
  TV t = gT2p.v;
  t.ext[2] = v;
  t.ext[3] = v;
  permute(ctx, "mkbc->mkbc", 1.0, t, 1.0, g_t2);
  if (integrals) {
    auto view = [&](int64_t off, std::initializer_list<int64_t> ext) {
      TV e;
      e.p = d_geri + off;
      e.nd = 4;
      int k = 0;
      for (int64_t x : ext) e.ext[k++] = x;
      const int64_t st[4] = {1, N, N2, N3};
      std::memcpy(e.str, st, sizeof(st));
      return e;
    };
    TV pv = gP.v;  // P(i,f,a,b) = eri(i, o+b, o+a, o+f)
    pv.ext[2] = v;
    pv.ext[3] = v;
    permute(ctx, "ifab->ibaf", 1.0, pv, 1.0, view(o * N + o * N2 + o * N3, {o, v, v, v}));
    TV rv = gRt.v;  // R(i,j,m,a) = eri(i, m, o+a, j)
    rv.ext[3] = v;
    permute(ctx, "ijma->imaj", 1.0, rv, 1.0, view(o * N2, {o, o, v, o}));
    // S(i,j,a,b) = eri(i, j, o+a, o+b)
    permute(ctx, "ijab->ijab", 1.0, gS.v, 1.0, view(o * N2 + o * N3, {o, o, v, v}));
  }
  ctx.sync();
  return ctx.hscalars[0];
}

}  // namespace scess
