// Matvec kernels.  One template per phase, instantiated per precision (T)
// and interpolation order (L).  See kernels.cuh for the memory layout.
#include "kernels.cuh"
#include "device_math.cuh"
#include "green64.cuh"
#include "fmm_kernels.h"
#include "ptx.cuh"

#include <algorithm>
#include <climits>
#include <mutex>
#include <set>
#include <type_traits>
#include <utility>
#include <vector>

namespace dfb {

// --------------------------------------------------------- constant tables --
// Per order L = 2..8: the four L x L interpolation matrices (m2m[0], m2m[1],
// l2l[0], l2l[1]; A(k, p) at k + p L) and the twiddles exp(-2 pi i m / P),
// P = 2L - 1.  Every use sits in a fully unrolled loop, so the operands are
// immediate constant-bank addresses rather than shared-memory loads.
constexpr int kMinOrder = 2, kMaxOrder = 8;
__host__ __device__ constexpr int mat_off(int L) {
  int s = 0;
  for (int l = kMinOrder; l < L; l++) s += 4 * l * l;
  return s;
}
__host__ __device__ constexpr int tw_off(int L) {
  int s = 0;
  for (int l = kMinOrder; l < L; l++) s += 2 * l - 1;
  return s;
}
__constant__ double c_mat64[mat_off(kMaxOrder + 1)];
__constant__ float c_mat32[mat_off(kMaxOrder + 1)];
__constant__ double c_tw64[2 * tw_off(kMaxOrder + 1)];
__constant__ float c_tw32[2 * tw_off(kMaxOrder + 1)];

template <typename T>
__device__ __forceinline__ T cmat(int i);
template <>
__device__ __forceinline__ double cmat<double>(int i) {
  return c_mat64[i];
}
template <>
__device__ __forceinline__ float cmat<float>(int i) {
  return c_mat32[i];
}
// twiddle exp(-2 pi i m / P) of order L, m in [0, P)
template <typename T, int L>
__device__ __forceinline__ typename cpx_t<T>::type ctw(int m) {
  typename cpx_t<T>::type r;
  if constexpr (sizeof(T) == 8) {
    r.x = c_tw64[2 * (tw_off(L) + m)];
    r.y = c_tw64[2 * (tw_off(L) + m) + 1];
  } else {
    r.x = c_tw32[2 * (tw_off(L) + m)];
    r.y = c_tw32[2 * (tw_off(L) + m) + 1];
  }
  return r;
}
// acc += v * conj(w)
template <typename C>
__device__ __forceinline__ void cfmac(C& acc, C v, C w) {
  acc.x = fma(v.x, w.x, acc.x);
  acc.x = fma(v.y, w.y, acc.x);
  acc.y = fma(v.y, w.x, acc.y);
  acc.y = fma(-v.x, w.y, acc.y);
}
// ------------------------------------------------------------- gather/scatter
template <typename T>
__global__ void k_gather(const double2* __restrict__ qin, const int32_t* __restrict__ perm,
                         typename cpx_t<T>::type* __restrict__ q, int64_t n, int64_t nrhs_stride_in,
                         int64_t nrhs_stride_q, int nrhs) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t u = perm[i];
  for (int r = 0; r < nrhs; r++) {
    const double2 v = qin[r * nrhs_stride_in + u];
    typename cpx_t<T>::type w;
    w.x = (T)v.x;
    w.y = (T)v.y;
    q[r * nrhs_stride_q + i] = w;
  }
}

__global__ void k_scatter(const double2* __restrict__ pnear, const double2* __restrict__ pfar,
                          const int32_t* __restrict__ perm, double2* __restrict__ out, int64_t n) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double2 a = pnear[i], b = pfar[i];
  a.x += b.x;
  a.y += b.y;
  out[perm[i]] = a;
}

// -------------------------------------------------------------------- P2M --
// HF leaf (phfP2M, P2M.hpp:114-131), per effective direction d:
//   M_d[l] = conj(sig2_d[l]) * sum_j Z(l, j) exp(-i k d.(y_j - c)) q_j
// LF leaf (plfP2M, P2M.hpp:134-136): M[l] = sum_j Z(l, j) q_j,
// with Z(l, j) = prod_k S_{I_k(l)}(y_jk - c_k) the leaf's interpolation matrix
// (mapOnTrees.hpp:37-83).
//
// Per leaf this is the small GEMM  M[l][s] = sum_j Z[j][l] W[j][s],
// W[j][s] = q_j exp(-i k d_s.(y_j - c)).  One CTA per leaf, in chunks of NPB
// points: Z[j][l] is built once per chunk in shared memory (point-major, l
// padded to LLP = 32 R); each warp takes S of the leaf's slots at a time,
// writes their W column block, and every lane accumulates an R x S register
// tile (expansion entries lane + 32 e, all S slots, so signatures and results
// are read and written at unit stride) over the chunk's points: per point R
// loads of Z and S broadcast loads of W feed 2 R S FMAs.  Latency bounds it
// (the signatures' loads), so an FP64 chunk's Z takes at most 40 KB: with the
// offsets, the basis and W 3 CTAs fit an SM at orders 4 and 5 (57,856 and 57,600
// bytes; 76,288 with several right-hand sides at order 4), 4 at order 6, 5 above.
// Sphere 250k FP64 5.7 -> 4.0 ms against entries R lane .. R lane + R - 1 and
// chunks of 64 points (2 CTAs).  FP32 chunks hold 64 points where they fit: their sums
// are rounded chunk by chunk, and results keep their bits (spheroid 500k mixed
// order 6 9.1 -> 7.0 ms, 5.5 with chunks of 40).
template <typename T, int L>
struct P2MCfg {
  static constexpr int LL = L * L * L;
  static constexpr int R = L >= 5 ? 4 * ((LL + 127) / 128) : (LL + 31) / 32;  // entries per lane
  static constexpr int LLP = 32 * R;
  static constexpr int S0 = (sizeof(T) == 4 ? 32 : 16) / R;
  static constexpr int S = S0 < 1 ? 1 : (S0 > (sizeof(T) == 4 ? 8 : 4) ? (sizeof(T) == 4 ? 8 : 4) : S0);
  static constexpr int NPB0 = (sizeof(T) == 4 ? 65536 : 40960) / (LLP * (int)sizeof(T));
  static constexpr int NPB = NPB0 > 64 ? 64 : NPB0;  // points per chunk
  typedef typename cpx_t<T>::type C;
  // shared memory: Z, point offsets, basis values, W blocks of 4 warps,
  // (with R > 1 right-hand sides) phase blocks of 4 warps, charges (R per point)
  static constexpr size_t smem(int R = 1) {
    return sizeof(T) * (size_t)NPB * LLP + sizeof(double) * NPB * 3 + sizeof(T) * NPB * 3 * L +
           sizeof(C) * 4 * NPB * S * (R > 1 ? 2 : 1) + sizeof(C) * (size_t)NPB * R;
  }
  // W follows Z, the offsets and the basis: an odd chunk could misalign it
  static_assert((sizeof(T) * NPB * LLP + sizeof(double) * NPB * 3 + sizeof(T) * NPB * 3 * L) % sizeof(C) == 0,
                "W blocks are read as complex values");
};

template <typename T, int L, int SS>
__device__ __forceinline__ void p2m_group(const DevPlan& P, int64_t j0, int ns, bool hf, bool first, int np,
                                          const T* __restrict__ Zs, const double* __restrict__ yc,
                                          const typename cpx_t<T>::type* __restrict__ qs,
                                          typename cpx_t<T>::type* __restrict__ Ws,
                                          typename cpx_t<T>::type* __restrict__ Es, const double* dirs,
                                          const typename cpx_t<T>::type* __restrict__ s2,
                                          typename cpx_t<T>::type* __restrict__ M, int R, int lane) {
  typedef typename cpx_t<T>::type C;
  typedef P2MCfg<T, L> G;
  constexpr int RE = G::R, LLP = G::LLP, LL = G::LL;
  __syncwarp();
  // phases exp(-i k d_s.(y_j - c)) of the group's slots, shared by the
  // right-hand sides (with one right-hand side the charge is folded in here)
  for (int idx = lane; idx < np * SS; idx += 32) {
    const int j = idx / SS, s = idx % SS;
    C w;
    if (s >= ns) {
      w = czero<C>();
    } else if (hf) {
      const double* dv = dirs + 3 * P.S_cdir[j0 + s];
      double dp = 0.;
      for (int k = 0; k < 3; k++) dp += dv[k] * yc[3 * j + k];
      w = expi<C>(-P.kappa * dp);
    } else {
      w.x = T(1);
      w.y = T(0);
    }
    if (R == 1)
      Ws[j * SS + s] = cmul(w, qs[j]);
    else
      Es[j * SS + s] = w;
  }
  for (int r = 0; r < R; r++) {
    __syncwarp();
    if (R > 1) {
      for (int idx = lane; idx < np * SS; idx += 32) {
        const int j = idx / SS;
        Ws[idx] = cmul(Es[idx], qs[j * R + r]);
      }
      __syncwarp();
    }
    C acc[RE][SS];
#pragma unroll
    for (int e = 0; e < RE; e++)
#pragma unroll
      for (int s = 0; s < SS; s++) acc[e][s] = czero<C>();
    const T* zl = Zs + lane;
    for (int j = 0; j < np; j++) {
      T z[RE];
      C w[SS];
#pragma unroll
      for (int e = 0; e < RE; e++) z[e] = zl[j * LLP + 32 * e];
#pragma unroll
      for (int s = 0; s < SS; s++) w[s] = Ws[j * SS + s];
#pragma unroll
      for (int e = 0; e < RE; e++)
#pragma unroll
        for (int s = 0; s < SS; s++) rfma(acc[e][s], z[e], w[s]);
    }
#pragma unroll
    for (int s = 0; s < SS; s++) {
      if (s < ns) {
        const int slot = P.S_cslot[j0 + s], d = P.S_cdir[j0 + s];
#pragma unroll
        for (int e = 0; e < RE; e++) {
          const int l = lane + 32 * e;
          if (l < LL) {
            const C a = hf ? cmulc(s2[(int64_t)d * LL + l], acc[e][s]) : acc[e][s];
            C* out = M + ((int64_t)slot * R + r) * LL + l;
            if (first) {
              *out = a;
            } else {
              C o = *out;
              o.x += a.x;
              o.y += a.y;
              *out = o;
            }
          }
        }
      }
    }
  }
}

// M: base of the expansions written here (slot s, right-hand side r at
// M + (s R + r) LL); q: tree-order charges, R per particle (q[j R + r]);
// only the leaf slots with a direction in [d0, d1) are computed.  A leaf's
// slots are shared by `split` CTAs (each builds Z for itself) where there are
// too few leaves to fill the chip.
template <typename T, int L>
__global__ void __launch_bounds__(128) k_p2m(DevPlan P, const int32_t* __restrict__ leaves, int nleaves,
                                             const typename cpx_t<T>::type* __restrict__ q,
                                             const typename cpx_t<T>::type* __restrict__ sig2,
                                             typename cpx_t<T>::type* __restrict__ M, int R, int d0, int d1,
                                             int split) {
  typedef typename cpx_t<T>::type C;
  typedef P2MCfg<T, L> G;
  constexpr int LL = G::LL, LLP = G::LLP, NPB = G::NPB, S = G::S;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Zs = reinterpret_cast<T*>(smem_raw);
  double* yc = reinterpret_cast<double*>(Zs + (size_t)NPB * LLP);
  T* Bs = reinterpret_cast<T*>(yc + NPB * 3);
  C* Wall = reinterpret_cast<C*>(Bs + NPB * 3 * L);
  C* Eall = Wall + 4 * NPB * S;
  C* qs = Eall + (R > 1 ? 4 * NPB * S : 0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  C* Ws = Wall + warp * NPB * S;
  C* Es = Eall + warp * NPB * S;
  for (int64_t w = blockIdx.x; w < (int64_t)nleaves * split; w += gridDim.x) {
    const int c = leaves[w / split], part = (int)(w % split);
    const int n = P.S_nprt[c], f = P.S_first[c];
    const double4 ct = P.S_ctr[c];
    const int lv = P.S_lvl[c];
    const bool hf = P.ishf[lv] != 0;
    const int h = P.hfstage[lv];
    int64_t sb, se;
    dir_range(P.S_cptr, P.S_cdir, c, d0, d1, &sb, &se);
    const int nslots = (int)(se - sb);
    if (nslots <= 4 * S * part) continue;
    const double* dirs = P.dirs + P.dir_off[h] * 3;
    const C* s2 = sig2 + P.sig_off[h];
    for (int p0 = 0; p0 < n; p0 += NPB) {
      const int np = min(NPB, n - p0);
      __syncthreads();  // the previous chunk's Z, W are no longer read
      for (int o = threadIdx.x; o < 3 * np; o += blockDim.x) {
        const int p = o / 3, k = o % 3;
        const double x = P.S_pos[3 * (int64_t)(f + p0 + p) + k] - (&ct.x)[k];
        yc[o] = x;
        T b[L];
        lagrange_all<L, T>((T)x, (T)ct.w, b);
#pragma unroll
        for (int l = 0; l < L; l++) Bs[(p * 3 + k) * L + l] = b[l];
      }
      for (int p = threadIdx.x; p < np * R; p += blockDim.x) qs[p] = q[(int64_t)(f + p0) * R + p];
      __syncthreads();
      for (int o = threadIdx.x; o < np * LLP; o += blockDim.x) {
        const int p = o / LLP, l = o % LLP;
        T z = 0;
        if (l < LL) {
          const int i0 = l / (L * L), i1 = (l / L) % L, i2 = l % L;
          z = Bs[(p * 3 + 0) * L + i0] * Bs[(p * 3 + 1) * L + i1] * Bs[(p * 3 + 2) * L + i2];
        }
        Zs[o] = z;
      }
      __syncthreads();
      for (int g0 = (4 * part + warp) * S; g0 < nslots; g0 += 4 * S * split) {
        const int ns = min(S, nslots - g0);
        if (ns == 1)
          p2m_group<T, L, 1>(P, sb + g0, 1, hf, p0 == 0, np, Zs, yc, qs, Ws, Es, dirs, s2, M, R, lane);
        else
          p2m_group<T, L, S>(P, sb + g0, ns, hf, p0 == 0, np, Zs, yc, qs, Ws, Es, dirs, s2, M, R, lane);
      }
    }
  }
}

// ------------------------------------------------ separable 3-D transfer --
// out[a,b,c] = sum A_s0(a,a') A_s1(b,b') A_s2(c,c') in[a',b',c'] computed in
// three axis passes (axis 2, 1, 0 as interpolation.hpp:311-361); A(k, p) is
// matrix 2*ROLE + s of the order's constant table (ROLE 0: M2M, 1: L2L).
// One warp per transfer; lane ln owns line(s) ln, ln + 32 of each pass:
//   axis 2 on (a, b) lines: input in registers (v), output to buf
//   axis 1 on (a, c) lines: in place in buf (a lane's line is its own)
//   axis 0 on (b, c) lines: from buf to registers (res)
// The branch on each s is warp-uniform and keeps the matrix indices
// compile-time constants.
template <typename T, int L, int ROLE>
struct Sep {
  typedef typename cpx_t<T>::type C;
  static constexpr int NLN = (L * L + 31) / 32;  // lines per lane
  template <int MI>
  __device__ static __forceinline__ void line(const C (&v)[L], C (&o)[L]) {
    constexpr int B = mat_off(L) + MI * L * L;
#pragma unroll
    for (int k = 0; k < L; k++) {
      C acc = czero<C>();
#pragma unroll
      for (int p = 0; p < L; p++) rfma(acc, cmat<T>(B + k + p * L), v[p]);
      o[k] = acc;
    }
  }
  __device__ static __forceinline__ void apply(int s, const C (&v)[L], C (&o)[L]) {
    if (s)
      line<2 * ROLE + 1>(v, o);
    else
      line<2 * ROLE>(v, o);
  }
  // The same transfer with the passes in the order axis 0, 1, 2: the input
  // lines run along axis 0 (v[q][p] = in[p, b, c] for line (b, c) = ln, so a
  // warp reads an expansion with unit stride across lanes), res holds lines
  // (a, b) = ln along axis 2 (res[q][k] = out[a, b, k]).
  __device__ static __forceinline__ void run_a0(int sg0, int sg1, int sg2, const C (&v)[NLN][L], C* buf,
                                                C (&res)[NLN][L], int lane) {
#pragma unroll
    for (int q = 0; q < NLN; q++) {  // axis 0: lines (b, c)
      const int ln = lane + 32 * q;
      if (ln < L * L) {
        C o[L];
        apply(sg0, v[q], o);
#pragma unroll
        for (int k = 0; k < L; k++) buf[k * L * L + ln] = o[k];
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NLN; q++) {  // axis 1: lines (a, c), in place
      const int ln = lane + 32 * q;
      if (ln < L * L) {
        const int a = ln / L, c = ln % L;
        C w[L], o[L];
#pragma unroll
        for (int p = 0; p < L; p++) w[p] = buf[(a * L + p) * L + c];
        apply(sg1, w, o);
#pragma unroll
        for (int k = 0; k < L; k++) buf[(a * L + k) * L + c] = o[k];
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NLN; q++) {  // axis 2: lines (a, b)
      const int ln = lane + 32 * q;
      if (ln < L * L) {
        C w[L];
#pragma unroll
        for (int p = 0; p < L; p++) w[p] = buf[ln * L + p];
        apply(sg2, w, res[q]);
      }
    }
    __syncwarp();
  }
  __device__ static __forceinline__ void run(int sg0, int sg1, int sg2, const C (&v)[NLN][L], C* buf,
                                             C (&res)[NLN][L], int lane) {
#pragma unroll
    for (int q = 0; q < NLN; q++) {  // axis 2: lines (a, b)
      const int ln = lane + 32 * q;
      if (ln < L * L) {
        C o[L];
        apply(sg2, v[q], o);
#pragma unroll
        for (int k = 0; k < L; k++) buf[ln * L + k] = o[k];
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NLN; q++) {  // axis 1: lines (a, c), in place
      const int ln = lane + 32 * q;
      if (ln < L * L) {
        const int a = ln / L, c = ln % L;
        C w[L], o[L];
#pragma unroll
        for (int p = 0; p < L; p++) w[p] = buf[(a * L + p) * L + c];
        apply(sg1, w, o);
#pragma unroll
        for (int k = 0; k < L; k++) buf[(a * L + k) * L + c] = o[k];
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NLN; q++) {  // axis 0: lines (b, c)
      const int ln = lane + 32 * q;
      if (ln < L * L) {
        C w[L];
#pragma unroll
        for (int p = 0; p < L; p++) w[p] = buf[p * L * L + ln];
        apply(sg0, w, res[q]);
      }
    }
    __syncwarp();
  }
};

// -------------------------------------------------------------------- M2M --
// One warp per parent slot with children (upwpass.hpp:49-60):
//   HF parent, direction d (hfM2Mblock M2M.hpp:76-105 / lf2hfM2M :108-124):
//     M_d = conj(sig2_d) o sum_c exp(-i k d.v_c) A_{v_c}(sig_d o M_c)
//   LF parent (lfM2M :35-41): M = sum_c A_{v_c}(M_c);   v_c = ctr_c - ctr_parent
// A lane reads its (b, c) lines (along axis 0) of each child's expansion
// straight into registers, lanes at unit stride (the next child's are
// prefetched during the current transfer); the transfer runs axis 0 first.
// Lane e holds child e's slot, octant and plane-wave phase, computed once
// per parent slot.  With R right-hand sides a warp takes one parent slot and
// runs its transfers for every right-hand side in turn; the parent's
// expansions live at Mp + (slot R + r) LL, the children's at
// Mc0 + (slot R + r) LL (both bases may be the same array).
constexpr int kXferWarps = 4;  // warps (transfers in flight) per CTA

template <typename T, int L>
__global__ void __launch_bounds__(32 * kXferWarps, sizeof(T) == 4 ? (L <= 5 ? 6 : 3) : (L <= 5 ? 3 : 1)) k_m2m(DevPlan P, int64_t s0, int64_t s1,
                                                         const typename cpx_t<T>::type* __restrict__ sig,
                                                         const typename cpx_t<T>::type* __restrict__ sig2,
                                                         typename cpx_t<T>::type* __restrict__ Mp,
                                                         const typename cpx_t<T>::type* __restrict__ Mc0, int R) {
  typedef typename cpx_t<T>::type C;
  typedef Sep<T, L, 0> S;
  constexpr int LL = L * L * L, NW = kXferWarps, NLN = S::NLN;
  __shared__ C sbuf[NW][LL];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t ps = s0 + blockIdx.x * NW + warp; ps < s1; ps += (int64_t)gridDim.x * NW) {
    const int64_t eb = P.m2m_ptr[ps], ee = P.m2m_ptr[ps + 1];
    if (eb == ee) continue;  // leaf slot: written by P2M
    const int pc = P.sS_cell[ps], d = P.sS_dir[ps];
    const int lv = P.S_lvl[pc];
    const bool hf = P.ishf[lv] != 0;
    const int h = P.hfstage[lv];
    const C* sg = sig + P.sig_off[h] + (int64_t)(hf ? d : 0) * LL;
    const C* sg2 = sig2 + P.sig_off[h] + (int64_t)(hf ? d : 0) * LL;
    // child e (<= 8) on lane e: its slot, the octant of its centre (bit k
    // set when v_k >= 0) and its phase exp(-i k d.v)
    const int nch = (int)(ee - eb);
    int my_cs = 0, my_oct = 0;
    C my_ph = czero<C>();
    if (lane < nch) {
      my_cs = P.m2m_child[eb + lane];
      const double4 pct = P.S_ctr[pc], ct = P.S_ctr[P.sS_cell[my_cs]];
      const double v0 = ct.x - pct.x, v1 = ct.y - pct.y, v2 = ct.z - pct.z;
      my_oct = (v0 < 0. ? 0 : 1) | (v1 < 0. ? 0 : 2) | (v2 < 0. ? 0 : 4);
      if (hf) {
        const double* dv = P.dirs + 3 * (P.dir_off[h] + d);
        my_ph = expi<C>(-P.kappa * (dv[0] * v0 + dv[1] * v1 + dv[2] * v2));
      }
    }
    // with one line per lane (L <= 5) the parent's signature line and the
    // next transfer's lines stay in registers; larger orders reload them
    constexpr bool REG = NLN == 1;
    C acc[NLN][L], sgr[REG ? NLN : 1][L];
#pragma unroll
    for (int q = 0; q < NLN; q++) {
      const int ln = lane + 32 * q;
#pragma unroll
      for (int k = 0; k < L; k++) {
        acc[q][k] = czero<C>();
        if (REG) sgr[0][k] = (hf && ln < L * L) ? sg[k * L * L + ln] : czero<C>();
      }
    }
    C nxt[REG ? NLN : 1][L];  // next transfer's (a, b) lines, prefetched
    if (REG) {
      const C* Mc = Mc0 + (int64_t)__shfl_sync(0xffffffffu, my_cs, 0) * R * LL;
#pragma unroll
      for (int k = 0; k < L; k++) nxt[0][k] = lane < L * L ? Mc[k * L * L + lane] : czero<C>();
    }
    // transfers in (right-hand side, child) order
    const int nit = nch * R;
    int e = 0, rr = 0;
    for (int it = 0; it < nit; it++) {
      const int oct = __shfl_sync(0xffffffffu, my_oct, e);
      C in[NLN][L];
      if (REG) {
#pragma unroll
        for (int k = 0; k < L; k++) in[0][k] = hf ? cmul(sgr[0][k], nxt[0][k]) : nxt[0][k];
        const int e1 = e + 1 < nch ? e + 1 : 0, r1 = e + 1 < nch ? rr : rr + 1;
        const int cs1 = __shfl_sync(0xffffffffu, my_cs, e1);
        if (it + 1 < nit) {
          const C* Mc = Mc0 + ((int64_t)cs1 * R + r1) * LL;
#pragma unroll
          for (int k = 0; k < L; k++)
            if (lane < L * L) nxt[0][k] = Mc[k * L * L + lane];
        }
      } else {
        const C* Mc = Mc0 + ((int64_t)__shfl_sync(0xffffffffu, my_cs, e) * R + rr) * LL;
#pragma unroll
        for (int q = 0; q < NLN; q++) {
          const int ln = lane + 32 * q;
#pragma unroll
          for (int k = 0; k < L; k++) {
            const C m = ln < L * L ? Mc[k * L * L + ln] : czero<C>();
            in[q][k] = (hf && ln < L * L) ? cmul(sg[k * L * L + ln], m) : m;
          }
        }
      }
      C res[NLN][L];
      S::run_a0(oct & 1, (oct >> 1) & 1, (oct >> 2) & 1, in, sbuf[warp], res, lane);
      if (hf) {
        C ph;
        ph.x = __shfl_sync(0xffffffffu, my_ph.x, e);
        ph.y = __shfl_sync(0xffffffffu, my_ph.y, e);
#pragma unroll
        for (int q = 0; q < NLN; q++)
#pragma unroll
          for (int k = 0; k < L; k++) cfma(acc[q][k], ph, res[q][k]);
      } else {
#pragma unroll
        for (int q = 0; q < NLN; q++)
#pragma unroll
          for (int k = 0; k < L; k++) {
            acc[q][k].x += res[q][k].x;
            acc[q][k].y += res[q][k].y;
          }
      }
      if (++e == nch) {  // the last child of right-hand side rr
#pragma unroll
        for (int q = 0; q < NLN; q++) {
          const int ln = lane + 32 * q;
#pragma unroll
          for (int k = 0; k < L; k++) {
            if (ln < L * L) {
              const int l = ln * L + k;
              Mp[(ps * R + rr) * LL + l] = hf ? cmulc(sg2[l], acc[q][k]) : acc[q][k];
            }
            acc[q][k] = czero<C>();
          }
        }
        e = 0;
        rr++;
      }
    }
  }
}

// -------------------------------------------------------------------- L2L --
// One warp per child slot with parents (dwnpass.hpp:49-58):
//   HF parent direction d (hfL2Lblock L2L.hpp:78-108 / hf2lfL2L :111-127):
//     L_c += sum_d exp(i k v.d) conj(sig_d) o B_v(sig2_d o L_d)
//   LF parent (lfL2L :35-41): L_c += B_v(L_p);   v = ctr_child - ctr_parent
// Lane e holds parent e's slot, direction and phase, computed once per child
// slot.  With R right-hand sides a warp takes one child slot and runs its
// transfers for every right-hand side in turn; children at
// Lc + (slot R + r) LL, parents at Lp0 + (slot R + r) LL.  Only
// parent slots in [p0, p1) contribute (a pass over part of the directions).
template <typename T, int L>
__global__ void __launch_bounds__(32 * kXferWarps, sizeof(T) == 4 ? (L <= 5 ? 6 : 3) : (L <= 5 ? 4 : 1)) k_l2l(DevPlan P, int64_t s0, int64_t s1,
                                                         const typename cpx_t<T>::type* __restrict__ sig,
                                                         const typename cpx_t<T>::type* __restrict__ sig2,
                                                         typename cpx_t<T>::type* __restrict__ Lc,
                                                         const typename cpx_t<T>::type* __restrict__ Lp0, int R,
                                                         int64_t p0, int64_t p1) {
  typedef typename cpx_t<T>::type C;
  typedef Sep<T, L, 1> S;
  constexpr int LL = L * L * L, NW = kXferWarps, NLN = S::NLN;
  __shared__ C sbuf[NW][LL];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t cs = s0 + blockIdx.x * NW + warp; cs < s1; cs += (int64_t)gridDim.x * NW) {
    const int64_t eb = P.l2l_ptr[cs], ee = P.l2l_ptr[cs + 1];
    if (eb == ee) continue;
    const int cc = P.sT_cell[cs];
    const int pc = P.T_parent[cc];
    const int lv = P.T_lvl[pc];
    const bool hf = P.ishf[lv] != 0;
    const int h = P.hfstage[lv];
    const double4 pct = P.T_ctr[pc], cct = P.T_ctr[cc];
    const double v[3] = {cct.x - pct.x, cct.y - pct.y, cct.z - pct.z};
    const int sg0 = v[0] < 0. ? 0 : 1, sg1 = v[1] < 0. ? 0 : 1, sg2i = v[2] < 0. ? 0 : 1;
    C acc[NLN][L];
#pragma unroll
    for (int q = 0; q < NLN; q++)
#pragma unroll
      for (int k = 0; k < L; k++) acc[q][k] = czero<C>();
    // parents' slots and directions fetched by lane (<= 6 per child slot),
    // only those in [p0, p1), compacted to the first lanes
    const int nall = (int)(ee - eb);
    int all_ps = 0, all_d = 0;
    if (lane < nall) {
      all_ps = P.l2l_parent[eb + lane];
      all_d = P.sT_dir[all_ps];
    }
    int my_ps = 0, my_d = 0, npa = 0;
    for (int e = 0; e < nall; e++) {  // warp-uniform: keep the parents in range, in order
      const int ps_e = __shfl_sync(0xffffffffu, all_ps, e);
      const int d_e = __shfl_sync(0xffffffffu, all_d, e);
      if (ps_e >= p0 && ps_e < p1) {
        if (lane == npa) {
          my_ps = ps_e;
          my_d = d_e;
        }
        npa++;
      }
    }
    if (npa == 0) continue;
    // parent e on lane e: its phase exp(i k v.d_e)
    C my_ph = czero<C>();
    if (hf && lane < npa) {
      const double* dv = P.dirs + 3 * (P.dir_off[h] + my_d);
      my_ph = expi<C>(P.kappa * (v[0] * dv[0] + v[1] * dv[1] + v[2] * dv[2]));
    }
    // with one line per lane (L <= 5) the next transfer's lines are
    // prefetched into registers; larger orders load them when used
    constexpr bool REG = NLN == 1;
    C nxt[REG ? NLN : 1][L];
    if (REG) {
      const C* Lp = Lp0 + (int64_t)__shfl_sync(0xffffffffu, my_ps, 0) * R * LL;
#pragma unroll
      for (int k = 0; k < L; k++) nxt[0][k] = lane < L * L ? Lp[lane * L + k] : czero<C>();
    }
    // transfers in (right-hand side, parent) order
    const int nit = npa * R;
    int e = 0, rr = 0;
    for (int it = 0; it < nit; it++) {
      const int d = __shfl_sync(0xffffffffu, my_d, e);
      const C* sg = sig + P.sig_off[h] + (int64_t)(hf ? d : 0) * LL;
      const C* sgq = sig2 + P.sig_off[h] + (int64_t)(hf ? d : 0) * LL;
      C in[NLN][L];
      if (REG) {
#pragma unroll
        for (int k = 0; k < L; k++) in[0][k] = (hf && lane < L * L) ? cmul(sgq[lane * L + k], nxt[0][k]) : nxt[0][k];
        const int e1 = e + 1 < npa ? e + 1 : 0, r1 = e + 1 < npa ? rr : rr + 1;
        const int ps1 = __shfl_sync(0xffffffffu, my_ps, e1);
        if (it + 1 < nit) {
          const C* Lp = Lp0 + ((int64_t)ps1 * R + r1) * LL;
#pragma unroll
          for (int k = 0; k < L; k++)
            if (lane < L * L) nxt[0][k] = Lp[lane * L + k];
        }
      } else {
        const C* Lp = Lp0 + ((int64_t)__shfl_sync(0xffffffffu, my_ps, e) * R + rr) * LL;
#pragma unroll
        for (int q = 0; q < NLN; q++) {
          const int ln = lane + 32 * q;
#pragma unroll
          for (int k = 0; k < L; k++) {
            const C m = ln < L * L ? Lp[ln * L + k] : czero<C>();
            in[q][k] = (hf && ln < L * L) ? cmul(sgq[ln * L + k], m) : m;
          }
        }
      }
      C res[NLN][L];
      S::run(sg0, sg1, sg2i, in, sbuf[warp], res, lane);
      if (hf) {
        C ph;
        ph.x = __shfl_sync(0xffffffffu, my_ph.x, e);
        ph.y = __shfl_sync(0xffffffffu, my_ph.y, e);
#pragma unroll
        for (int q = 0; q < NLN; q++) {
          const int ln = lane + 32 * q;
          if (ln < L * L)
#pragma unroll
            for (int k = 0; k < L; k++) cfma(acc[q][k], ph, cmulc(sg[k * L * L + ln], res[q][k]));
        }
      } else {
#pragma unroll
        for (int q = 0; q < NLN; q++)
#pragma unroll
          for (int k = 0; k < L; k++) {
            acc[q][k].x += res[q][k].x;
            acc[q][k].y += res[q][k].y;
          }
      }
      if (++e == npa) {  // the last parent of right-hand side rr
#pragma unroll
        for (int q = 0; q < NLN; q++) {
          const int ln = lane + 32 * q;
#pragma unroll
          for (int k = 0; k < L; k++) {
            if (ln < L * L) {
              const int64_t l = (cs * R + rr) * LL + k * L * L + ln;
              C o = Lc[l];
              o.x += acc[q][k].x;
              o.y += acc[q][k].y;
              Lc[l] = o;
            }
            acc[q][k] = czero<C>();
          }
        }
        e = 0;
        rr++;
      }
    }
  }
}

// ---------------------------------------------------------------- M2F/F2L --
// Pruned odd-size 3-D DFT (size P = 2L-1) of the zero-padded expansion
// (circulant.hpp:96-106: M sits at the low corner of the P^3 grid):
//   F[k0,k1,k2] = sum_{a,b,c<L} M[a,b,c] w^(k0 a + k1 b + k2 c),  w = e^{-2 pi i/P}
// One warp per expansion (several per CTA); each axis pass gives one lane one
// line (its L inputs in registers, its P outputs computed from them).
template <typename T, int L>
struct M2FCfg {
  typedef typename cpx_t<T>::type C;
  static constexpr int P = 2 * L - 1, LL = L * L * L;
  static constexpr int PER_WARP = LL + L * L * P + L * P * P;  // complex elements
  // warps per CTA so that a CTA's shared memory stays within ~48 KB
  static constexpr int NW0 = (int)(49152 / (PER_WARP * sizeof(C)));
  static constexpr int NW = NW0 < 1 ? 1 : (NW0 > 8 ? 8 : NW0);
};

// One line of the forward DFT: out(k) = sum_a v[a] w^(k a), k < P = 2 L - 1,
// a < L.  Outputs k and P - k are A - i B and A + i B with A = sum cos v,
// B = sum sin v: 4 (L - 1) FMAs for the two instead of 8 (L - 1) for each.
// Order 7 goes term by term too (the paired sums spill: 6.3 and 5.7 ms).
// FP32 sums go term by term: paired they take 9.3 instead of 11.1 ms (spheroid
// 500k order 6) but round differently, and mixed results keep their bits.
template <typename T, int L, typename C, typename Put>
__device__ __forceinline__ void fdft_line(const C (&v)[L], Put put) {
  constexpr int P = 2 * L - 1;
  if constexpr (sizeof(T) == 4 || L >= 7) {
#pragma unroll
    for (int k = 0; k < P; k++) {
      C o = v[0];
#pragma unroll
      for (int a = 1; a < L; a++) cfma(o, v[a], ctw<T, L>((k * a) % P));
      put(k, o);
    }
  } else {
    C s0 = v[0];
#pragma unroll
    for (int a = 1; a < L; a++) {
      s0.x += v[a].x;
      s0.y += v[a].y;
    }
    put(0, s0);
#pragma unroll
    for (int k = 1; k < L; k++) {
      C A = v[0], B;
#pragma unroll
      for (int a = 1; a < L; a++) {
        const C w = ctw<T, L>((k * a) % P);  // (cos, -sin)
        A.x = fma(w.x, v[a].x, A.x);
        A.y = fma(w.x, v[a].y, A.y);
        B.x = a == 1 ? w.y * v[a].x : fma(w.y, v[a].x, B.x);  // -B
        B.y = a == 1 ? w.y * v[a].y : fma(w.y, v[a].y, B.y);
      }
      C lo, hi;
      lo.x = A.x - B.y;
      lo.y = A.y + B.x;
      hi.x = A.x + B.y;
      hi.y = A.y - B.x;
      put(k, lo);
      put(P - k, hi);
    }
  }
}

template <typename T, int L>
__global__ void __launch_bounds__(256) k_m2f(int64_t nexp, int R, const int32_t* __restrict__ slist,
                                             const typename cpx_t<T>::type* __restrict__ M,
                                             typename cpx_t<T>::type* __restrict__ F) {
  typedef typename cpx_t<T>::type C;
  constexpr int P = 2 * L - 1, LL = L * L * L, PP = P * P * P;
  constexpr int NW = M2FCfg<T, L>::NW, PER = M2FCfg<T, L>::PER_WARP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  C* Mi = reinterpret_cast<C*>(smem_raw) + warp * PER;
  C* A = Mi + LL;
  C* B = A + L * L * P;
  // the next expansion is loaded into registers while the current one is
  // transformed
  constexpr int NV = (LL + 31) / 32;
  // Expansion e is right-hand side r = e mod R of the (i = e / R)-th listed slot.
  // Orders 4 to 6 wait for memory and divide; below and above, i and r go on
  // without a division and the slot's number is read one round ahead of its
  // values (eight right-hand sides, 30,001 points, dividing and not: mixed order
  // 2 0.148 and 0.113 ms, 3 0.231 and 0.210, 7 4.91 and 3.98, 8 8.25 and 7.08,
  // FP64 order 8 15.4 and 14.2; order 5 FP64 2.16 and 2.20).  There counts take
  // 32 bits (the F buffer holds at most 64 GB of spectra), but not in FP32
  // above order 6, where 64-bit ones make the compiler keep more loads in
  // flight (order 7 4.76 and 3.98, order 8 8.02 and 7.08).
  constexpr bool STEP = L < 4 || L > 6;
  typedef typename std::conditional<STEP && (sizeof(T) == 8 || L < 4), int, int64_t>::type E;
  const E n = (E)nexp, e0 = (E)blockIdx.x * NW + warp, de = (E)gridDim.x * NW;
  int i = 0, r = 0, di = 0, dr = 0;
  int32_t slot = 0;
  if constexpr (STEP) {
    i = (int)((unsigned)e0 / (unsigned)R), r = (int)((unsigned)e0 % (unsigned)R);
    di = (int)((unsigned)de / (unsigned)R), dr = (int)((unsigned)de % (unsigned)R);
    if (e0 < n) slot = slist[i];
  }
  // e: e0 first, then each next one
  auto row = [&](E e) {
    if constexpr (STEP) {
      const C* Me = M + ((int64_t)slot * R + r) * LL;
      i += di;
      r += dr;
      if (r >= R) {
        r -= R;
        i++;
      }
      if (e + de < n) slot = slist[i];
      return Me;
    } else {
      return M + ((int64_t)slist[e / R] * R + e % R) * LL;
    }
  };
  C nx[NV];
  if (e0 < n) {
    const C* Me = row(e0);
#pragma unroll
    for (int m = 0; m < NV; m++) {
      const int j = lane + 32 * m;
      nx[m] = j < LL ? Me[j] : czero<C>();
    }
  }
  for (E e = e0; e < n; e += de) {
    __syncwarp();
#pragma unroll
    for (int m = 0; m < NV; m++) {
      const int j = lane + 32 * m;
      if (j < LL) Mi[j] = nx[m];
    }
    __syncwarp();
    if (e + de < n) {
      const C* Me = row(e + de);
#pragma unroll
      for (int m = 0; m < NV; m++) {
        const int j = lane + 32 * m;
        if (j < LL) nx[m] = Me[j];
      }
    }
    for (int ln = lane; ln < L * L; ln += 32) {  // axis 2: (a,b) lines
      C v[L];
#pragma unroll
      for (int c = 0; c < L; c++) v[c] = Mi[ln * L + c];
      fdft_line<T, L>(v, [&](int k2, C o) { A[ln * P + k2] = o; });
    }
    __syncwarp();
    for (int ln = lane; ln < L * P; ln += 32) {  // axis 1: (a,k2) lines
      const int a = ln / P, k2 = ln % P;
      C v[L];
#pragma unroll
      for (int b = 0; b < L; b++) v[b] = A[(a * L + b) * P + k2];
      fdft_line<T, L>(v, [&](int k1, C o) { B[(a * P + k1) * P + k2] = o; });
    }
    __syncwarp();
    for (int ln = lane; ln < P * P; ln += 32) {  // axis 0: (k1,k2) lines
      C v[L];
#pragma unroll
      for (int a = 0; a < L; a++) v[a] = B[a * P * P + ln];
      fdft_line<T, L>(v, [&](int k0, C o) { F[(int64_t)e * PP + k0 * P * P + ln] = o; });
    }
  }
}

// Gather the permuted spectra used by M2L once (permutations.hpp:128-150):
// U_k[i] = tables[key_k >> 6][perm[key_k & 63][i]].
template <typename T>
__global__ void k_permute_tables(int64_t n, int PP, const uint32_t* __restrict__ key, const uint16_t* __restrict__ perm,
                                 const typename cpx_t<T>::type* __restrict__ tables,
                                 typename cpx_t<T>::type* __restrict__ out) {
  for (int64_t k = blockIdx.x; k < n; k += gridDim.x) {
    const uint32_t kk = key[k];
    const typename cpx_t<T>::type* U = tables + (int64_t)(kk >> 6) * PP;
    const uint16_t* pm = perm + (int64_t)(kk & 63) * PP;
    for (int i = threadIdx.x; i < PP; i += blockDim.x) out[k * PP + i] = U[pm[i]];
  }
}

// -------------------------------------------------------------- M2L + F2L --
// One line of the inverse DFT, pruned to its L low outputs:
//   out[a] = sum_k v[k] conj(w)^(k a),  w = exp(-2 pi i / P), P = 2 L - 1.
// The terms k and P - k share their cosine, and their sine up to its sign, so
// they are added and subtracted first: 4 (L - 1) FMAs per output instead of
// 8 (L - 1), none of them multiplications for a = 0.  FP32 sums go term by
// term (fdft_line).
template <typename T, int L, typename C>
__device__ __forceinline__ void idft_line(const C (&v)[2 * L - 1], C (&out)[L]) {
  constexpr int P = 2 * L - 1;
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int a = 0; a < L; a++) {
      C o = v[0];
#pragma unroll
      for (int k = 1; k < P; k++) cfmac(o, v[k], ctw<T, L>((k * a) % P));
      out[a] = o;
    }
  } else {
    C s[L], d[L];
#pragma unroll
    for (int k = 1; k < L; k++) {
      s[k].x = v[k].x + v[P - k].x;
      s[k].y = v[k].y + v[P - k].y;
      d[k].x = v[k].x - v[P - k].x;
      d[k].y = v[k].y - v[P - k].y;
    }
#pragma unroll
    for (int a = 0; a < L; a++) {
      C o = v[0];
#pragma unroll
      for (int k = 1; k < L; k++) {
        if (a == 0) {
          o.x += s[k].x;
          o.y += s[k].y;
        } else {
          const C w = ctw<T, L>((k * a) % P);  // (cos, -sin)
          o.x = fma(w.x, s[k].x, o.x);
          o.y = fma(w.x, s[k].y, o.y);
          o.x = fma(w.y, d[k].y, o.x);
          o.y = fma(-w.y, d[k].x, o.y);
        }
      }
      out[a] = o;
    }
  }
}

// Inverse DFTs of RB spectra of PP entries (acc[k RB + b]: the K values of
// spectrum b, one per thread and k) into their local expansions at dst(b)
// (fourier2geom, circulant.hpp:109-118):
//   L_t[a,b,c] += (1/PP) sum_k J[k] conj(w)^(k0 a + k1 b + k2 c)
// pruned to a,b,c < L, one line per thread per axis pass, in place in Js (RB
// PP entries of shared memory): a line's outputs go to entries that its own
// thread has read.  One buffer instead of one per pass leaves the rest of
// the SM's memory to L1, which serves part of the spectra.  Each axis pass
// runs over the lines of all RB spectra, so the CTA's threads stay busy and
// the transforms take three barriers together.  a() and b() run after the
// first and the second one.  A barrier has to lie between this and the next
// use of Js.
template <typename T, int L, int NT, int RB, typename Dst, typename HookA, typename HookB>
__device__ __forceinline__ void m2l_f2l(const typename cpx_t<T>::type* acc, typename cpx_t<T>::type* Js, Dst dst,
                                        HookA hook_a, HookB hook_b) {
  typedef typename cpx_t<T>::type C;
  constexpr int PD = 2 * L - 1, PP = PD * PD * PD, K = (PP + NT - 1) / NT;
  const T inv = T(1) / T(PP);
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int i = threadIdx.x + k * NT;
    if (i < PP)
#pragma unroll
      for (int b = 0; b < RB; b++) Js[b * PP + i] = acc[k * RB + b];
  }
  __syncthreads();
  hook_a();
  for (int x = threadIdx.x; x < RB * PD * PD; x += NT) {  // axis 0: (k1,k2) lines -> a
    C* q = Js + x / (PD * PD) * PP + x % (PD * PD);
    C v[PD], o[L];
#pragma unroll
    for (int k = 0; k < PD; k++) v[k] = q[k * PD * PD];
    idft_line<T, L>(v, o);
#pragma unroll
    for (int a = 0; a < L; a++) q[a * PD * PD] = o[a];
  }
  __syncthreads();
  hook_b();
  for (int x = threadIdx.x; x < RB * L * PD; x += NT) {  // axis 1: (a,k2) lines -> b
    const int ln = x % (L * PD);
    C* q = Js + x / (L * PD) * PP + ln / PD * (PD * PD) + ln % PD;
    C v[PD], o[L];
#pragma unroll
    for (int k = 0; k < PD; k++) v[k] = q[k * PD];
    idft_line<T, L>(v, o);
#pragma unroll
    for (int b = 0; b < L; b++) q[b * PD] = o[b];
  }
  __syncthreads();
  for (int x = threadIdx.x; x < RB * L * L; x += NT) {  // axis 2: (a,b) lines -> c
    const int r = x / (L * L), ln = x % (L * L);
    const C* q = Js + r * PP + (ln / L * PD + ln % L) * PD;
    C v[PD], s[L];
#pragma unroll
    for (int k = 0; k < PD; k++) v[k] = q[k];
    idft_line<T, L>(v, s);
    C* Lt = dst(r) + ln * L;
#pragma unroll
    for (int c = 0; c < L; c++) {
      C o = Lt[c];
      o.x += s[c].x * inv;
      o.y += s[c].y * inv;
      Lt[c] = o;
    }
  }
}

// Work queue of k_m2l and k_m2l_rhs.  A CTA's first item is its own number, the
// others come from the queue in order, so that the target slots in flight stay
// a window of one cone (F_s and U_k are served from L2); of the CTAs that do
// not fit on the chip at first, the first items run late and outside that
// window.  The next item's index and list are fetched while the current item's
// inverse DFTs run, so that an item starts with its spectra loads instead of a
// chain of three misses (index, pointers, entries): NL lists per item, up to
// kCap entries each, the rest is read directly.  M2L with this and only the
// target slots that have a list: sphere 250k FP64 43.8 -> 38.2 ms, 600k mixed
// 47.1 -> 43.9, eight right-hand sides 160 -> 128.  (Both users have one list.
// Without the list index the compiler orders the spectra loads differently and
// the 250k sphere takes 41.8 ms, the 600k one 46.1.)
template <int NL, int NT>
struct M2LQueue {
  static constexpr int kCap = NT / NL < 64 ? NT / NL : 64;
  struct Shared {
    int64_t item[2], eb[2][NL];
    int len[2][NL];
    int2 e[2][NL][kCap];  // (position in the F batch's list, permuted spectrum)
  };
  Shared& sh;
  const DevPlan& P;
  unsigned long long* queue;
  int64_t nwork;
  int64_t b = 0, fetched = 0;
  int n = 0;
  int2 my;
  __device__ __forceinline__ M2LQueue(Shared& s, const DevPlan& p, unsigned long long* q, int64_t nw)
      : sh(s), P(p), queue(q), nwork(nw) {}
  // every thread: list j's entry i of the next item
  __device__ __forceinline__ int j() const { return threadIdx.x / kCap; }
  __device__ __forceinline__ int i() const { return threadIdx.x % kCap; }
  __device__ __forceinline__ void fetch() {
    if (threadIdx.x == 0) fetched = gridDim.x + (int64_t)atomicAdd(queue, 1ULL);
  }
  // the CTA's first item, without the queue; then a barrier
  __device__ __forceinline__ void first(int64_t u, int64_t u1) {
    fetched = blockIdx.x;
    publish(0);
    pointers(fetched, u, u1);
    entries();
    store(0);
  }
  __device__ __forceinline__ void publish(int ph) {  // before a barrier
    if (threadIdx.x == 0) sh.item[ph] = fetched;
  }
  // after that barrier: pointers of listed target slot u + j (none at or past u1)
  __device__ __forceinline__ void pointers(int64_t item, int64_t u, int64_t u1) {
    n = 0;
    if (j() < NL && item < nwork && u + j() < u1) {
      b = P.m2l_cptr[u + j()];
      n = (int)(P.m2l_cptr[u + j() + 1] - b);
    }
  }
  __device__ __forceinline__ void entries() {
    if (i() < n) my = make_int2(P.m2l_src[b + i()], (int)P.m2l_tab[b + i()]);
  }
  __device__ __forceinline__ void store(int ph) {  // then a barrier
    if (j() >= NL) return;
    if (i() < n) sh.e[ph][j()][i()] = my;
    if (i() == 0) {
      sh.eb[ph][j()] = b;
      sh.len[ph][j()] = n;
    }
  }
  // entry x of list jj of the current item, from memory
  __device__ __forceinline__ int2 direct(int ph, int jj, int x) const {
    const int64_t g = sh.eb[ph][jj] + x;
    return make_int2(P.m2l_src[g], (int)P.m2l_tab[g]);
  }
};

// CTAs per SM of k_m2l (SLOTS = 1) and k_m2l_pair (2): 512 threads in FP64 and
// 1,024 in FP32, but fewer where the accumulators (A registers) would spill and
// more where there is one value per thread and 256 of them (M2L, 30,001-point
// sphere, ms, without and with the exceptions): order 8 FP32 at 128 threads
// (A = 54) 5.99 and 2.86, pairs at 128 threads order 8 FP32 (108) 8.70 and 5.10,
// FP64 (216) 15.7 and 12.6, order 7 FP32 (72) 2.85 and 2.12, FP64 (144) 6.06 and
// 4.03; orders 2 and 3 FP64 at 256 threads 0.71 and 0.54, 1.03 and 0.59.
template <typename T, int L, int NT, int SLOTS>
constexpr int m2l_ctas() {
  constexpr int P = 2 * L - 1, K = (P * P * P + NT - 1) / NT, A = K * SLOTS * 2 * (int)sizeof(T) / 4;
  return (A > 112 ? 256 : sizeof(T) == 8 ? (NT == 256 && K == 1 ? 1536 : 512) : A > 48 ? 512 : 1024) / NT;
}

// One CTA per listed target slot [u0, u1) of a cone batch (M2L.hpp:115-157
// target-stationary, then the inverse DFT above):
//   J[i] = sum_{(s, k) in list(t)} U_k[i] F_s[i]          (registers)
// J never leaves the SM.
template <typename T, int L, int NT>
__global__ void __launch_bounds__(NT, m2l_ctas<T, L, NT, 1>()) k_m2l(DevPlan P, int64_t u0, int64_t u1, int64_t f0, int64_t f1,
                                                       const typename cpx_t<T>::type* __restrict__ F,
                                                       const typename cpx_t<T>::type* __restrict__ ptab,
                                                       typename cpx_t<T>::type* __restrict__ Lx,
                                                       unsigned long long* __restrict__ queue) {
  typedef typename cpx_t<T>::type C;
  typedef M2LQueue<1, NT> Q;
  constexpr int PD = 2 * L - 1, LL = L * L * L, PP = PD * PD * PD, K = (PP + NT - 1) / NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* Js = reinterpret_cast<C*>(smem_raw);
  __shared__ typename Q::Shared qs;
  Q q(qs, P, queue, u1 - u0);
  q.first(u0 + (int64_t)blockIdx.x, u1);
  __syncthreads();
  for (int ph = 0; qs.item[ph] < u1 - u0; ph ^= 1) {
    q.fetch();
    const int64_t t = P.m2l_tlist[u0 + qs.item[ph]];
    const int n = qs.len[ph][0];
    C acc[K];
#pragma unroll
    for (int k = 0; k < K; k++) acc[k] = czero<C>();
    auto add = [&](int2 e) {
      if (e.x < f0 || e.x >= f1) {  // entry outside this cone batch: a plan bug
        if (threadIdx.x == 0) atomicExch(P.err, 1);
        return;
      }
      const C* Fs = F + (e.x - f0) * PP;
      const C* U = ptab + (int64_t)(uint32_t)e.y * PP;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int i = threadIdx.x + k * NT;
        if (i < PP) cfma(acc[k], __ldg(U + i), __ldg(Fs + i));
      }
    };
    const int ns = min(n, Q::kCap);
#pragma unroll 2
    for (int x = 0; x < ns; x++) add(qs.e[ph][0][x]);
    for (int x = ns; x < n; x++) add(q.direct(ph, 0, x));
    q.publish(ph ^ 1);
    m2l_f2l<T, L, NT, 1>(acc, Js, [&](int) { return Lx + t * LL; }, [&] { q.pointers(qs.item[ph ^ 1], u0 + qs.item[ph ^ 1], u1); },
                         [&] { q.entries(); });
    q.store(ph ^ 1);
    __syncthreads();
  }
}

// Two consecutive listed target slots per CTA.  Each slot's list is sorted by
// source slot, so a merge of the two lists finds their common sources
// (about a third of the pairs at order 5), whose spectrum F_s is then read
// once for both.  Every accumulator sees its own list in list order with the
// same operations as k_m2l, so the results are bit-identical to it.  Both lists
// are read from memory as the merge goes on and items all come from the queue:
// M2LQueue for two lists took registers that the second accumulator set needs
// and was the slower one (M2L, ms: sphere 250k FP64 39.7 and 38.5, 600k mixed
// 48.2 and 44.0, 60k mixed order 6 8.6 and 7.0; 30,001 points order 4 FP64 at
// 256 threads 1.74 and 1.19; only order 7 mixed at 256 threads the other way,
// 2.22 and 2.43, where one slot per CTA takes 1.84).
template <typename T, int L, int NT>
__global__ void __launch_bounds__(NT, m2l_ctas<T, L, NT, 2>()) k_m2l_pair(DevPlan P, int64_t u0, int64_t u1, int64_t f0, int64_t f1,
                                                            const typename cpx_t<T>::type* __restrict__ F,
                                                            const typename cpx_t<T>::type* __restrict__ ptab,
                                                            typename cpx_t<T>::type* __restrict__ Lx,
                                                            unsigned long long* __restrict__ queue) {
  typedef typename cpx_t<T>::type C;
  constexpr int PD = 2 * L - 1, LL = L * L * L, PP = PD * PD * PD, K = (PP + NT - 1) / NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* Js = reinterpret_cast<C*>(smem_raw);
  __shared__ int64_t cur;
  for (;;) {
    __syncthreads();  // the previous slots' inverse DFTs are done with Js
    if (threadIdx.x == 0) cur = u0 + 2 * (int64_t)atomicAdd(queue, 1ULL);
    __syncthreads();
    const int64_t u = cur;
    if (u >= u1) break;
    const bool two = u + 1 < u1;
    int64_t a = P.m2l_cptr[u], b = P.m2l_cptr[u + 1];
    const int64_t ae = b, be = two ? P.m2l_cptr[u + 2] : b;
    C acc0[K], acc1[K];
#pragma unroll
    for (int k = 0; k < K; k++) acc0[k] = acc1[k] = czero<C>();
    while (a < ae || b < be) {
      const int sa = a < ae ? P.m2l_src[a] : INT_MAX;
      const int sb = b < be ? P.m2l_src[b] : INT_MAX;
      const int src = sa < sb ? sa : sb;
      if (src < f0 || src >= f1) {  // entry outside this cone batch: a plan bug
        if (threadIdx.x == 0) atomicExch(P.err, 1);
        if (sa == src) a++;
        if (sb == src) b++;
        continue;
      }
      const C* Fs = F + (src - f0) * PP;
      if (sa == sb) {
        const C* U0 = ptab + (int64_t)P.m2l_tab[a] * PP;
        const C* U1 = ptab + (int64_t)P.m2l_tab[b] * PP;
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int i = threadIdx.x + k * NT;
          if (i < PP) {
            const C f = __ldg(Fs + i);
            cfma(acc0[k], __ldg(U0 + i), f);
            cfma(acc1[k], __ldg(U1 + i), f);
          }
        }
        a++;
        b++;
      } else if (sa < sb) {
        const C* U0 = ptab + (int64_t)P.m2l_tab[a] * PP;
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int i = threadIdx.x + k * NT;
          if (i < PP) cfma(acc0[k], __ldg(U0 + i), __ldg(Fs + i));
        }
        a++;
      } else {
        const C* U1 = ptab + (int64_t)P.m2l_tab[b] * PP;
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int i = threadIdx.x + k * NT;
          if (i < PP) cfma(acc1[k], __ldg(U1 + i), __ldg(Fs + i));
        }
        b++;
      }
    }
    m2l_f2l<T, L, NT, 1>(acc0, Js, [&](int) { return Lx + (int64_t)P.m2l_tlist[u] * LL; }, [] {}, [] {});
    if (two) {
      __syncthreads();
      m2l_f2l<T, L, NT, 1>(acc1, Js, [&](int) { return Lx + (int64_t)P.m2l_tlist[u + 1] * LL; }, [] {}, [] {});
    }
  }
}

// Right-hand-side blocks: R charge vectors per pass, F and L holding R
// expansions per slot (F + ((s - f0) R + r) PP, Lx + (t R + r) LL).  A CTA
// takes one (target slot, block of RB right-hand sides) at a time; each
// transfer spectrum entry U_k[i] is loaded once and multiplied into the RB
// spectra of its source slot, so the spectra traffic per right-hand side is
// e P^3 (1 + 1/RB) per far pair instead of 2 e P^3.
// CTAs per SM of k_m2l_rhs, by the registers that its accumulators take
// (A = K RB values of 2 or 4): more CTAs hide more latency until the registers
// left for loads in flight run out.  Of 512, 768 and 1024 threads per SM this
// takes the fastest (M2L, 30,001-point sphere, ms; blocks of 3, 4 or 8
// right-hand sides):
//   128 threads, A <= 22: order 4 FP64 RB = 1 (A = 12) 2.75 / 2.04 / 1.77
//   128 threads, A 24-36: order 5 FP64 RB = 1 (24) 3.64 / 3.37 / 4.77, order 7
//     FP32 RB = 1 (36) 5.79 / 5.42 / 6.31
//   128 threads, A >= 44: order 6 FP64 RB = 1 (44) 6.05 / 7.17 / 8.96, order 6
//     FP32 RB = 2 (44) 7.79 / 8.66 / 13.6, order 8 FP32 RB = 1 (54) 8.51 / 11.8 /
//     16.6; order 7 FP64 RB = 2 (144, more than 128 registers hold) 21.3 / 48 /
//     55 for four right-hand sides, 12.4 at 256
//   256 threads: order 2 FP64 RB = 4 (16, K = 1) 1.63 / 1.12 / 0.85, order 5
//     FP64 RB = 4 (48) 5.22 / 4.42 / 4.78, order 5 FP32 RB = 4 (24) 3.63 / 2.62 /
//     2.12 and RB = 8 (48) 7.31 / 6.92 / 6.26, order 6 FP64 RB = 4 (96) 9.15 /
//     12.3 / 14.5
template <typename T, int L, int NT, int RB>
constexpr int m2l_rhs_ctas() {
  constexpr int P = 2 * L - 1, K = (P * P * P + NT - 1) / NT, A = K * RB * 2 * (int)sizeof(T) / 4;
  constexpr int threads = NT == 128 ? (A <= 22 ? 1024 : A <= 36 ? 768 : A <= 112 ? 512 : 256)
                                    : (A > 48 ? 512 : sizeof(T) == 4 || K == 1 ? 1024 : 768);
  static_assert(A + 16 <= 65536 / threads, "the accumulators alone would spill");
  return threads / NT;
}
// up to 4 right-hand sides per CTA whose spectra take at most 24 KB (FP32 at
// orders <= 5, FP64 <= 4): the inverse DFTs of a target slot's RB spectra run
// together; otherwise one after another
template <typename T, int L, int RB>
__host__ __device__ constexpr bool m2l_rhs_joint() {
  return RB > 1 && RB <= 4 && RB * (2 * L - 1) * (2 * L - 1) * (2 * L - 1) * 2 * sizeof(T) <= 24 * 1024;
}

template <typename T, int L, int NT, int RB>
__global__ void __launch_bounds__(NT, m2l_rhs_ctas<T, L, NT, RB>()) k_m2l_rhs(DevPlan P, int64_t u0, int64_t u1, int64_t f0, int64_t f1, int R,
                                                             const typename cpx_t<T>::type* __restrict__ F,
                                                             const typename cpx_t<T>::type* __restrict__ ptab,
                                                             typename cpx_t<T>::type* __restrict__ Lx,
                                                             unsigned long long* __restrict__ queue) {
  typedef typename cpx_t<T>::type C;
  typedef M2LQueue<1, NT> Q;
  constexpr int PD = 2 * L - 1, LL = L * L * L, PP = PD * PD * PD, K = (PP + NT - 1) / NT;
  constexpr bool JOINT = m2l_rhs_joint<T, L, RB>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* Js = reinterpret_cast<C*>(smem_raw);
  __shared__ typename Q::Shared qs;
  const int nb = R / RB;
  const int64_t nwork = (u1 - u0) * nb;
  Q q(qs, P, queue, nwork);
  q.first(u0 + (int64_t)blockIdx.x / nb, u1);
  __syncthreads();
  for (int ph = 0; qs.item[ph] < nwork; ph ^= 1) {
    q.fetch();
    const int64_t w = qs.item[ph];
    const int64_t t = P.m2l_tlist[u0 + w / nb];
    const int r0 = (int)(w % nb) * RB, n = qs.len[ph][0];
    C acc[K][RB];
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
      for (int b = 0; b < RB; b++) acc[k][b] = czero<C>();
    auto add = [&](int2 e) {
      if (e.x < f0 || e.x >= f1) {  // entry outside this cone batch: a plan bug
        if (threadIdx.x == 0) atomicExch(P.err, 1);
        return;
      }
      const C* Fs = F + ((e.x - f0) * R + r0) * PP;
      const C* U = ptab + (int64_t)(uint32_t)e.y * PP;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int i = threadIdx.x + k * NT;
        if (i < PP) {
          const C u = __ldg(U + i);
#pragma unroll
          for (int b = 0; b < RB; b++) cfma(acc[k][b], u, __ldg(Fs + b * PP + i));
        }
      }
    };
    const int ns = min(n, Q::kCap);
    for (int x = 0; x < ns; x++) add(qs.e[ph][0][x]);
    for (int x = ns; x < n; x++) add(q.direct(ph, 0, x));
    q.publish(ph ^ 1);
    auto hook_a = [&] { q.pointers(qs.item[ph ^ 1], u0 + qs.item[ph ^ 1] / nb, u1); };
    auto hook_b = [&] { q.entries(); };
    if constexpr (JOINT) {
      m2l_f2l<T, L, NT, RB>(&acc[0][0], Js, [&](int r) { return Lx + (t * R + r0 + r) * LL; }, hook_a, hook_b);
    } else {
#pragma unroll
      for (int b = 0; b < RB; b++) {
        C a[K];
#pragma unroll
        for (int k = 0; k < K; k++) a[k] = acc[k][b];
        auto dst = [&](int) { return Lx + (t * R + r0 + b) * LL; };
        if (b == 0) {
          m2l_f2l<T, L, NT, 1>(a, Js, dst, hook_a, hook_b);
        } else {
          __syncthreads();
          m2l_f2l<T, L, NT, 1>(a, Js, dst, [] {}, [] {});
        }
      }
    }
    q.store(ph ^ 1);
    __syncthreads();
  }
}

// Right-hand-side blocks with target groups, fed through shared memory by
// bulk copies (FP32 spectra).  A work item is (G consecutive target slots of
// a cone batch, RB right-hand sides).  Their lists are sorted by source slot;
// merged, every source slot met by any of the G lists is one entry, and its
// RB spectra F_s are loaded once for all the targets that meet it (a group of
// 4 consecutive slots meets 0.45 distinct sources per far pair on a sphere
// at 40 points per wavelength squared, order 5), with the transfer spectrum
// U_k of each such pair.
//
// Warp roles: the last warp produces, the others consume.  The producer
// takes work items from the queue, loads the G lists into shared memory,
// merges them and, per entry, copies the RB spectra of the source and the
// entry's transfer spectra into one of NS stages with 1-D bulk copies
// (cp.async.bulk global -> shared, completing on the stage's "full"
// mbarrier).  Consumer thread c owns spectrum entries c + k NC and keeps the
// G x RB accumulators of its entries in registers; after a stage it arrives
// on the stage's "empty" mbarrier, and after the last entry of an item it
// runs the inverse DFT of every (target, right-hand side) with an entry,
// NSPEC spectra per round, and adds the results into L.  The producer keeps
// filling stages meanwhile.
//
// Every accumulator sees its list in list order with the operations of
// k_m2l_rhs, and the inverse DFT sums in the order of m2l_f2l, so the
// results are bit-identical to k_m2l_rhs (and to the one-right-hand-side
// kernels).  A copy starts at the 16-byte boundary at or below its first
// byte and ends at the one at or above its last (both buffers carry 16 bytes
// of slack at the end); consumers index from the remainder.
//
// Every wait is bounded.  A thread that gives up sets a shared stop flag
// (the other waits then return at once) and the error code 3; the producer
// then waits (bounded) for the copies it issued before it returns.
template <int L>
struct M2LBulk {
  static constexpr int PD = 2 * L - 1, PP = PD * PD * PD, LL = L * L * L;
  static constexpr int G = kM2LGroup;                                   // target slots per work item
  static constexpr int RB = L <= 5 ? 4 : 2;                             // right-hand sides per work item
  static constexpr int K = (PP + 767) / 768;                            // entries per consumer thread
  static constexpr int NC = 32 * ((PP + 32 * K - 1) / (32 * K));        // consumer threads
  static constexpr int NT = NC + 32;                                    // + the producer warp
  static constexpr int NSPEC = L <= 5 ? 4 : 1;                          // spectra per inverse-DFT round
  static constexpr int FB = (RB * PP * 8 + 16 + 15) / 16 * 16;          // stage bytes of the F block
  static constexpr int UB = (PP * 8 + 16 + 15) / 16 * 16;               // stage bytes of one U
  static constexpr int SB = FB + G * UB;
  static constexpr int XB = NSPEC * (PP + L * PD * PD + L * L * PD) * 8;  // inverse-DFT scratch
  static constexpr int LCAP = L <= 4 ? 1024 : 2048;                     // list entries of one work item
  static constexpr int HDR = 1024;                                      // barriers, entry records, twiddles
  static constexpr int NS0 = (232448 - XB - LCAP * 8 - HDR) / SB;
  static constexpr int NS = NS0 > 4 ? 4 : NS0;                          // stages
  static constexpr int CTAS = L <= 3 ? 4 : (L == 4 ? 2 : 1);           // CTAs per SM
  static constexpr size_t smem() { return (size_t)NS * SB + XB + (size_t)LCAP * 8 + HDR; }
};

struct BulkEntry {  // one stage's record, written by the producer
  int64_t tb;       // first target slot of the item
  int mask;         // targets of the item that meet this source
  int flags;        // 1: last entry of the item; 2: no more work
  int nt, r0;       // targets in the item, first right-hand side
  int foff;         // F block: offset (complex entries) from the stage start
  int uoff[kM2LGroup];
};

constexpr uint32_t kBulkWait = 1u << 22;  // polls before a wait counts as failed

template <int L>
__global__ void __launch_bounds__(M2LBulk<L>::NT, M2LBulk<L>::CTAS) k_m2l_bulk(
    DevPlan P, int64_t t0, int64_t t1, int64_t f0, int64_t f1, int R, const float2* __restrict__ F,
    const float2* __restrict__ ptab, float2* __restrict__ Lx, unsigned long long* __restrict__ queue) {
  typedef M2LBulk<L> B;
  constexpr int PD = B::PD, PP = B::PP, LL = B::LL, G = B::G, RB = B::RB, K = B::K, NC = B::NC, NS = B::NS,
                NSPEC = B::NSPEC, FB = B::FB, UB = B::UB, SB = B::SB;
  static_assert(NS >= 2, "at least two stages");
  static_assert((G * RB) % NSPEC == 0, "whole inverse-DFT rounds");
  static_assert(NSPEC * LL <= NC, "one output of the last inverse-DFT pass per thread");
  static_assert(NS * 16 + 8 + NS * sizeof(BulkEntry) + PD * 8 + 8 <= B::HDR, "header");
  extern __shared__ __align__(16) unsigned char smem_raw[];  // stage offsets are multiples of 16 bytes
  unsigned char* stages = smem_raw;
  float2* Js = reinterpret_cast<float2*>(smem_raw + NS * SB);
  float2* Cb = Js + NSPEC * PP;
  float2* D = Cb + NSPEC * L * PD * PD;
  int32_t* ls_src = reinterpret_cast<int32_t*>(D + NSPEC * L * L * PD);
  uint32_t* ls_tab = reinterpret_cast<uint32_t*>(ls_src + B::LCAP);
  uint64_t* full = reinterpret_cast<uint64_t*>(ls_tab + B::LCAP);
  uint64_t* empty = full + NS;
  uint64_t* cbar = empty + NS;
  BulkEntry* rec = reinterpret_cast<BulkEntry*>(cbar + 1);
  float2* tw = reinterpret_cast<float2*>(rec + NS);
  volatile int* stop = reinterpret_cast<volatile int*>(tw + PD);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr unsigned kAll = 0xffffffffu;
  if (tid == 0) {
    for (int i = 0; i < NS; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], NC / 32);
    }
    mbar_init(cbar, NC / 32);
    *stop = 0;
  }
  if (tid < PD) tw[tid] = ctw<float, L>(tid);
  __syncthreads();

  if (warp == NC / 32) {
    // ---------------------------------------------------------- producer
    const int nb = R / RB;
    const int64_t nwork = (t1 - t0 + G - 1) / G * nb;
    uint32_t it = 0;  // stages issued
    bool ok = true;
    for (;;) {
      unsigned long long w = 0;
      if (lane == 0) w = atomicAdd(queue, 1ULL);
      w = __shfl_sync(kAll, w, 0);
      if ((int64_t)w >= nwork) break;
      const int64_t tb = t0 + (int64_t)(w / nb) * G;
      const int r0 = (int)(w % nb) * RB;
      const int nt = (int)(t1 - tb < G ? t1 - tb : G);
      const int64_t eb = P.m2l_ptr[tb], ee = P.m2l_ptr[tb + nt];
      const int64_t n = ee - eb;
      if (n == 0) continue;
      if (n > B::LCAP) {  // the launcher checks the plan's largest group: a plan bug
        if (lane == 0) atomicExch(P.err, 1);
        continue;
      }
      __syncwarp();  // lane 0 is done with the previous item's lists
      for (int64_t i = lane; i < n; i += 32) {
        ls_src[i] = P.m2l_src[eb + i];
        ls_tab[i] = P.m2l_tab[eb + i];
      }
      __syncwarp();
      if (lane == 0) {
        int hd[G], he[G];
#pragma unroll
        for (int j = 0; j < G; j++) {
          hd[j] = j < nt ? (int)(P.m2l_ptr[tb + j] - eb) : 0;
          he[j] = j < nt ? (int)(P.m2l_ptr[tb + j + 1] - eb) : 0;
        }
        // one entry of look-ahead, so the item's last entry is known when issued
        bool have = false;
        int pmask = 0, psrc = 0;
        uint32_t ptabs[G];
        auto issue = [&](bool last) -> bool {
          const int s = (int)(it % NS);
          const uint32_t ph = (it / NS) & 1u;
          if (!mbar_wait_or_stop(&empty[s], ph ^ 1u, kBulkWait, stop)) return false;
          unsigned char* st = stages + (size_t)s * SB;
          BulkEntry& e = rec[s];
          const uintptr_t a = (uintptr_t)(F + ((int64_t)(psrc - f0) * R + r0) * PP);
          const uintptr_t a0 = a & ~(uintptr_t)15, a1 = (a + (uintptr_t)RB * PP * 8 + 15) & ~(uintptr_t)15;
          uint32_t total = (uint32_t)(a1 - a0);
          e.tb = tb;
          e.mask = pmask;
          e.flags = last ? 1 : 0;
          e.nt = nt;
          e.r0 = r0;
          e.foff = (int)((a - a0) >> 3);
          uintptr_t u0[G];
          uint32_t ub[G];
#pragma unroll
          for (int j = 0; j < G; j++) {
            u0[j] = 0;
            ub[j] = 0;
            if ((pmask >> j) & 1) {
              const uintptr_t u = (uintptr_t)(ptab + (int64_t)ptabs[j] * PP);
              u0[j] = u & ~(uintptr_t)15;
              ub[j] = (uint32_t)(((u + (uintptr_t)PP * 8 + 15) & ~(uintptr_t)15) - u0[j]);
              e.uoff[j] = (int)((u - u0[j]) >> 3);
              total += ub[j];
            }
          }
          mbar_arrive_expect_tx(&full[s], total);
          bulk_g2s(st, (const void*)a0, (uint32_t)(a1 - a0), &full[s]);
#pragma unroll
          for (int j = 0; j < G; j++)
            if ((pmask >> j) & 1) bulk_g2s(st + FB + j * UB, (const void*)u0[j], ub[j], &full[s]);
          it++;
          return true;
        };
        for (;;) {
          int src = INT_MAX;
#pragma unroll
          for (int j = 0; j < G; j++)
            if (hd[j] < he[j] && ls_src[hd[j]] < src) src = ls_src[hd[j]];
          if (src == INT_MAX) break;
          int mask = 0;
          uint32_t tabs[G];
#pragma unroll
          for (int j = 0; j < G; j++) {
            tabs[j] = 0;
            if (hd[j] < he[j] && ls_src[hd[j]] == src) {
              mask |= 1 << j;
              tabs[j] = ls_tab[hd[j]];
              hd[j]++;
            }
          }
          if (src < f0 || src >= f1) {  // entry outside this cone batch: a plan bug
            atomicExch(P.err, 1);
            continue;
          }
          if (have && !issue(false)) {
            ok = false;
            break;
          }
          have = true;
          psrc = src;
          pmask = mask;
#pragma unroll
          for (int j = 0; j < G; j++) ptabs[j] = tabs[j];
        }
        if (ok && have && !issue(true)) ok = false;
      }
      ok = __shfl_sync(kAll, ok, 0);
      if (!ok) break;
    }
    if (lane == 0) {
      if (ok) {  // no more work
        const int s = (int)(it % NS);
        if (mbar_wait_or_stop(&empty[s], ((it / NS) & 1u) ^ 1u, kBulkWait, stop)) {
          rec[s].flags = 2;
          mbar_arrive(&full[s]);
        } else {
          ok = false;
        }
      }
      if (!ok) {
        *stop = 1;
        atomicExch(P.err, 3);
        // the copies issued into the last NS stages land before the CTA ends
        for (uint32_t k = it > (uint32_t)NS ? it - NS : 0; k < it; k++) mbar_wait(&full[k % NS], (k / NS) & 1u, kBulkWait);
      }
    }
    return;
  }

  // ------------------------------------------------------------ consumers
  float2 acc[G][RB][K];
#pragma unroll
  for (int j = 0; j < G; j++)
#pragma unroll
    for (int r = 0; r < RB; r++)
#pragma unroll
      for (int k = 0; k < K; k++) acc[j][r][k] = czero<float2>();
  int seen = 0;
  uint32_t cph = 0;
  const float inv = 1.0f / (float)PP;
  // barrier of the consumer warps (bounded; false once any thread gave up)
  auto cbarrier = [&]() -> bool {
    __syncwarp();
    if (lane == 0) mbar_arrive(cbar);
    const bool ok = __all_sync(kAll, mbar_wait_or_stop(cbar, cph, kBulkWait, stop));
    cph ^= 1u;
    if (!ok && lane == 0) {
      *stop = 1;
      atomicExch(P.err, 3);
    }
    return ok;
  };
  for (uint32_t it = 0;; it++) {
    const int s = (int)(it % NS);
    if (!__all_sync(kAll, mbar_wait_or_stop(&full[s], (it / NS) & 1u, kBulkWait, stop))) {
      if (lane == 0) {
        *stop = 1;
        atomicExch(P.err, 3);
      }
      break;
    }
    const BulkEntry e = rec[s];
    if (e.flags & 2) break;
    const float2* st = reinterpret_cast<const float2*>(stages + (size_t)s * SB);
    const float2* Fs = st + e.foff;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int i = tid + k * NC;
      if (i < PP) {
        float2 f[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) f[r] = Fs[r * PP + i];
#pragma unroll
        for (int j = 0; j < G; j++)
          if ((e.mask >> j) & 1) {
            const float2 u = st[(FB + j * UB) / 8 + e.uoff[j] + i];
#pragma unroll
            for (int r = 0; r < RB; r++) cfma(acc[j][r][k], u, f[r]);
          }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    seen |= e.mask;
    if (!(e.flags & 1)) continue;
    // inverse DFT of every (target, right-hand side) with an entry, the
    // passes of m2l_f2l over NSPEC spectra at a time
    bool ok = true;
#pragma unroll
    for (int q0 = 0; q0 < G * RB; q0 += NSPEC) {
      bool live = false;
#pragma unroll
      for (int sp = 0; sp < NSPEC; sp++) {
        const int j = (q0 + sp) / RB;
        live |= j < e.nt && ((seen >> j) & 1);
      }
      if (!live || !ok) continue;
      // this thread's output of the last pass (one per thread): its L entry
      // is loaded now, so the load overlaps the first two passes
      float2* l3 = nullptr;
      float2 lold = czero<float2>();
      if (tid < NSPEC * LL) {
        const int sp = tid / LL, rem = tid - sp * LL;
        const int q = q0 + sp, j = q / RB, r = q - j * RB;
        if (j < e.nt && ((seen >> j) & 1)) {
          l3 = Lx + ((e.tb + j) * R + e.r0 + r) * LL + rem;
          lold = *l3;
        }
      }
#pragma unroll
      for (int sp = 0; sp < NSPEC; sp++)
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int i = tid + k * NC;
          if (i < PP) Js[sp * PP + i] = acc[(q0 + sp) / RB][(q0 + sp) % RB][k];
        }
      if (!(ok = cbarrier())) continue;
      for (int o = tid; o < NSPEC * L * PD * PD; o += NC) {  // axis 0: (k1,k2) lines -> a
        const int sp = o / (L * PD * PD), rem = o - sp * (L * PD * PD);
        const int a = rem / (PD * PD), ln = rem - a * (PD * PD);
        const float2* v = Js + sp * PP + ln;
        float2 sum = v[0];
#pragma unroll
        for (int k0 = 1; k0 < PD; k0++) cfmac(sum, v[k0 * PD * PD], tw[(k0 * a) % PD]);
        Cb[sp * L * PD * PD + a * PD * PD + ln] = sum;
      }
      if (!(ok = cbarrier())) continue;
      for (int o = tid; o < NSPEC * L * L * PD; o += NC) {  // axis 1: (a,k2) lines -> b
        const int sp = o / (L * L * PD), rem = o - sp * (L * L * PD);
        const int a = rem / (L * PD), rem2 = rem - a * (L * PD);
        const int b = rem2 / PD, k2 = rem2 - b * PD;
        const float2* v = Cb + sp * L * PD * PD + a * PD * PD + k2;
        float2 sum = v[0];
#pragma unroll
        for (int k1 = 1; k1 < PD; k1++) cfmac(sum, v[k1 * PD], tw[(k1 * b) % PD]);
        D[sp * L * L * PD + (a * L + b) * PD + k2] = sum;
      }
      if (!(ok = cbarrier())) continue;
      if (l3) {  // axis 2: (a,b) lines -> c, added into L
        const int sp = tid / LL, rem = tid - sp * LL;
        const int ln = rem / L, c = rem - ln * L;
        const float2* v = D + sp * L * L * PD + ln * PD;
        float2 sum = v[0];
#pragma unroll
        for (int k2 = 1; k2 < PD; k2++) cfmac(sum, v[k2], tw[(k2 * c) % PD]);
        lold.x += sum.x * inv;
        lold.y += sum.y * inv;
        *l3 = lold;
      }
    }
    if (!ok) break;
#pragma unroll
    for (int j = 0; j < G; j++)
#pragma unroll
      for (int r = 0; r < RB; r++)
#pragma unroll
        for (int k = 0; k < K; k++) acc[j][r][k] = czero<float2>();
    seen = 0;
  }
}

// -------------------------------------------------------------------- L2P --
// One CTA (4 warps) per target leaf at a precomputed level
// (dwnpass.hpp:39-47): HF (phfL2P, L2P.hpp:122-142)
//   p_j = sum_d exp(i k d.(x_j - c)) sum_l Z(j, l) sig2_d[l] L_d[l]
// LF (plfL2P :165-173): p_j = sum_l Z(j, l) L[l].  Writes p_far.
// Warps take the leaf's slots in turn, lanes its particles; each lane keeps
// its particle's 3 L basis values in registers and accumulates over the
// warp's slots in registers; the 4 warps are summed at the end.
// Lx: base of the local expansions read here (slot s, right-hand side r at
// Lx + (s R + r) LL); only the leaf slots with a direction in [d0, d1)
// contribute; pfar holds R potentials per particle (pfar[j R + r]), written
// (acc = false) or added to (acc = true).  RC right-hand sides per pass over
// the slots (the phase of a slot is computed once per pass).
template <typename T, int L, int RC>
__global__ void __launch_bounds__(128) k_l2p(DevPlan P, const int32_t* __restrict__ leaves, int nleaves,
                                             const typename cpx_t<T>::type* __restrict__ sig2,
                                             const typename cpx_t<T>::type* __restrict__ Lx,
                                             double2* __restrict__ pfar, int R, int d0, int d1, bool accum) {
  typedef typename cpx_t<T>::type C;
  constexpr int LL = L * L * L;
  __shared__ C buf[4][LL];
  __shared__ double2 part[4][RC][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int li = blockIdx.x; li < nleaves; li += gridDim.x) {
    const int c = leaves[li];
    int64_t sb, se;
    dir_range(P.T_cptr, P.T_cdir, c, d0, d1, &sb, &se);
    if (sb == se) continue;
    const int n = P.T_nprt[c], f = P.T_first[c];
    const double4 ct = P.T_ctr[c];
    const int lv = P.T_lvl[c];
    const bool hf = P.ishf[lv] != 0;
    const int h = P.hfstage[lv];
    const double* dirs = P.dirs + P.dir_off[h] * 3;
    const C* s2 = sig2 + P.sig_off[h];
    for (int p0 = 0; p0 < n; p0 += 32) {
      const int np = min(32, n - p0);
      const int pi = f + p0 + min(lane, np - 1);
      double xr[3];
      T B[3][L];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        xr[k] = P.T_pos[3 * (int64_t)pi + k] - (&ct.x)[k];
        lagrange_all<L, T>((T)xr[k], (T)ct.w, B[k]);
      }
      for (int r0 = 0; r0 < R; r0 += RC) {
        const int nr = min(RC, R - r0);
        double2 acc[RC];
#pragma unroll
        for (int u = 0; u < RC; u++) acc[u] = make_double2(0., 0.);
        // units (slot of this warp, right-hand side); the next unit's
        // expansion (and, on a new slot, signature) is loaded into registers
        // while the current one is contracted
        constexpr int NV = (LL + 31) / 32;
        const int64_t nunit = ((se - sb - warp + 3) / 4) * nr;
        C nl[NV], ns[NV];
        int nd = 0;
        auto fetch = [&](int64_t k) {
          const int64_t j = sb + warp + 4 * (k / nr);
          const int u = (int)(k % nr);
          const int slot = P.T_cslot[j];
          const C* Ls = Lx + ((int64_t)slot * R + r0 + u) * LL;
#pragma unroll
          for (int m = 0; m < NV; m++) {
            const int l = lane + 32 * m;
            nl[m] = l < LL ? Ls[l] : czero<C>();
          }
          if (u == 0) {
            nd = P.T_cdir[j];
            const C* Ss = s2 + (int64_t)(hf ? nd : 0) * LL;
#pragma unroll
            for (int m = 0; m < NV; m++) {
              const int l = lane + 32 * m;
              ns[m] = (hf && l < LL) ? Ss[l] : czero<C>();
            }
          }
        };
        if (nunit > 0) fetch(0);
        C ph = czero<C>();
        for (int64_t k = 0; k < nunit; k++) {
          const int u = (int)(k % nr);
          if (u == 0 && hf) {
            const double* dv = dirs + 3 * nd;
            ph = expi<C>(P.kappa * (dv[0] * xr[0] + dv[1] * xr[1] + dv[2] * xr[2]));
          }
          __syncwarp();
#pragma unroll
          for (int m = 0; m < NV; m++) {
            const int l = lane + 32 * m;
            if (l < LL) buf[warp][l] = hf ? cmul(ns[m], nl[m]) : nl[m];
          }
          __syncwarp();
          if (k + 1 < nunit) fetch(k + 1);
          // sum_{a,b,c} B0[a] B1[b] B2[c] X[a,b,c] = sum_a B0[a] (sum_b B1[b] (sum_c B2[c] X[a,b,c]))
          C sum = czero<C>();
#pragma unroll
          for (int a = 0; a < L; a++) {
            C sa = czero<C>();
#pragma unroll
            for (int b = 0; b < L; b++) {
              C sbb = czero<C>();
#pragma unroll
              for (int cc = 0; cc < L; cc++) rfma(sbb, B[2][cc], buf[warp][(a * L + b) * L + cc]);
              rfma(sa, B[1][b], sbb);
            }
            rfma(sum, B[0][a], sa);
          }
          if (hf) sum = cmul(sum, ph);
#pragma unroll
          for (int v = 0; v < RC; v++)
            if (v == u) {
              acc[v].x += (double)sum.x;
              acc[v].y += (double)sum.y;
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < RC; u++) part[warp][u][lane] = acc[u];
        __syncthreads();
        if (threadIdx.x < np) {
#pragma unroll
          for (int u = 0; u < RC; u++) {
            if (r0 + u >= R) break;
            double2 t = part[0][u][threadIdx.x];
            for (int w = 1; w < 4; w++) {
              t.x += part[w][u][threadIdx.x].x;
              t.y += part[w][u][threadIdx.x].y;
            }
            double2* o = pfar + (int64_t)(f + p0 + threadIdx.x) * R + r0 + u;
            if (accum) {
              t.x += o->x;
              t.y += o->y;
            }
            *o = t;
          }
        }
      }
    }
  }
}

// FP64 L2P of high-frequency leaves as a small GEMM per leaf (order 5,
// resident layout),
//   D[j][s] = sum_l Z(j, l) X[l][s],  X[l][s] = sig2_d[l] L_s[l],
//   p_j = sum_s exp(i k d_s.(x_j - c)) D[j][s]:
// one CTA per leaf, Z[l][j] of up to 32 points and X of 16 slots in shared
// memory, a thread on 4 points and a slot.  A warp owns 8 points and all
// slots of a tile, so its points' sums stay in its registers and only warps
// with points issue: 18 points cost 20, where k_l2p's lanes are points, 18 of
// 32.  Per l a thread loads 4 Z (broadcast) and one X for 8 FMAs; a lane of
// k_l2p loads one X for 2.  Half the instructions of k_l2p; the loads of the
// tiles bound it.  k_l2p and this: sphere 250k 5.6 and 5.0 ms.  Elsewhere
// k_l2p is the faster one: order 4 (cube 20k 51 and 66 us), orders from 6 (the
// tiles take twice the memory), blocks of right-hand sides (one staging for
// each), and low-frequency leaves, which have a single slot; FP32 sums (600k
// points 5.4 and 4.2 ms) would round differently, and mixed results keep
// their bits.
template <typename T, int L>
struct L2PHf {
  typedef typename cpx_t<T>::type C;
  static constexpr bool use = L == 5 && sizeof(T) == 8;
  static constexpr int LL = L * L * L;
  static constexpr int NS = 16;       // slots per tile
  static constexpr int NSP = NS + 1;  // row pitch of X
  static constexpr size_t smem() {
    return sizeof(C) * LL * NSP + sizeof(T) * LL * 32 + sizeof(double) * 96 + sizeof(T) * 96 * L;
  }
};

template <typename T, int L>
__global__ void __launch_bounds__(128, 3)
    k_l2p_hf(DevPlan P, const int32_t* __restrict__ leaves, int nleaves, const typename cpx_t<T>::type* __restrict__ sig2,
             const typename cpx_t<T>::type* __restrict__ Lx, double2* __restrict__ pfar) {
  typedef typename cpx_t<T>::type C;
  typedef L2PHf<T, L> G;
  constexpr int LL = G::LL, NS = G::NS, NSP = G::NSP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* X = reinterpret_cast<C*>(smem_raw);
  T* Z = reinterpret_cast<T*>(X + LL * NSP);
  double* xc = reinterpret_cast<double*>(Z + LL * 32);
  T* Bs = reinterpret_cast<T*>(xc + 96);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = 2 * warp + (lane >> 4), si = lane & 15;  // point group, slot of the thread
  for (int li = blockIdx.x; li < nleaves; li += gridDim.x) {
    const int c = leaves[li];
    const int64_t sb = P.T_cptr[c], se = P.T_cptr[c + 1];
    if (sb == se) continue;
    const int n = P.T_nprt[c], f = P.T_first[c], nslots = (int)(se - sb);
    const double4 ct = P.T_ctr[c];
    const int h = P.hfstage[P.T_lvl[c]];
    const double* dirs = P.dirs + P.dir_off[h] * 3;
    const C* s2 = sig2 + P.sig_off[h];
    for (int p0 = 0; p0 < n; p0 += 32) {
      const int np = min(32, n - p0), n4 = (np + 3) & ~3;
      __syncthreads();  // the previous points' Z and offsets are no longer read
      for (int o = threadIdx.x; o < 3 * np; o += 128) {
        const int p = o / 3, k = o % 3;
        const double x = P.T_pos[3 * (int64_t)(f + p0 + p) + k] - (&ct.x)[k];
        xc[o] = x;
        T b[L];
        lagrange_all<L, T>((T)x, (T)ct.w, b);
#pragma unroll
        for (int l = 0; l < L; l++) Bs[o * L + l] = b[l];
      }
      __syncthreads();
      for (int o = threadIdx.x; o < n4 * LL; o += 128) {
        const int l = o / n4, p = o % n4;
        T z = 0;
        if (p < np) {
          const T* b = Bs + p * 3 * L;
          z = b[l / (L * L)] * b[L + l / L % L] * b[2 * L + l % L];
        }
        Z[l * 32 + p] = z;
      }
      const bool act = 4 * g < np;
      double xr[4][3];
#pragma unroll
      for (int v = 0; v < 4; v++)
#pragma unroll
        for (int k = 0; k < 3; k++) xr[v][k] = 4 * g + v < np ? xc[3 * (4 * g + v) + k] : 0.;
      double2 acc[4];
#pragma unroll
      for (int v = 0; v < 4; v++) acc[v] = make_double2(0., 0.);
      for (int s0 = 0; s0 < nslots; s0 += NS) {
        const int nt = min(NS, nslots - s0);
        C ph[4];
        const bool in = act && si < nt;
        const double* dv = dirs + 3 * (in ? P.T_cdir[sb + s0 + si] : 0);
#pragma unroll
        for (int v = 0; v < 4; v++)
          ph[v] = in ? expi<C>(P.kappa * (dv[0] * xr[v][0] + dv[1] * xr[v][1] + dv[2] * xr[v][2])) : czero<C>();
        __syncthreads();  // the previous tile is no longer read (and Z is settled)
#pragma unroll 4
        for (int s = warp; s < NS; s += 4) {
          if (s < nt) {
            const int64_t j = sb + s0 + s;
            const C* Ls = Lx + (int64_t)P.T_cslot[j] * LL;
            const C* Ss = s2 + (int64_t)P.T_cdir[j] * LL;
#pragma unroll
            for (int l = lane; l < LL; l += 32) X[l * NSP + s] = cmul(Ss[l], Ls[l]);
          } else {
            for (int l = lane; l < LL; l += 32) X[l * NSP + s] = czero<C>();
          }
        }
        __syncthreads();
        if (!act) continue;
        C d[4];
#pragma unroll
        for (int v = 0; v < 4; v++) d[v] = czero<C>();
#pragma unroll 5
        for (int l = 0; l < LL; l++) {
          const double2 za = *reinterpret_cast<const double2*>(Z + l * 32 + 4 * g);
          const double2 zb = *reinterpret_cast<const double2*>(Z + l * 32 + 4 * g + 2);
          const C x = X[l * NSP + si];
          rfma(d[0], za.x, x);
          rfma(d[1], za.y, x);
          rfma(d[2], zb.x, x);
          rfma(d[3], zb.y, x);
        }
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const C w = cmul(d[v], ph[v]);
          acc[v].x += w.x;
          acc[v].y += w.y;
        }
      }
#pragma unroll
      for (int v = 0; v < 4; v++) {
        double2 t = acc[v];
#pragma unroll
        for (int o = 8; o; o >>= 1) {
          t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
          t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
        }
        const int p = 4 * g + v;
        if ((lane & 15) == v && p < np) pfar[f + p0 + p] = t;
      }
    }
  }
}

// -------------------------------------------------------------------- P2P --
// Mixed-precision near field.  The phase k r needs ~1e-7 rad absolute
// accuracy at k r up to ~1e2, beyond FP32: the difference vector, r^2, r and
// the reduction of k r to [-pi/2, pi/2] (n = rint(k r / pi)) run in FP64;
// sin/cos of the reduced angle are evaluated in FP32 by their Taylor series
// to degree 13/12, 1/(4 pi r) and the complex products in FP32; every
// product is accumulated in FP64.
// Near field, tiled: one CTA (4 warps) per work item (part of the sources of
// one chunk of <= 32 target particles of one leaf); CTAs take items from a
// global queue in the host's order of decreasing work.  The chunk's source ranges are streamed through shared
// memory in tiles of TS particles loaded with coalesced reads; inside a warp,
// lanes form groups of tp >= nt lanes (one target each) and the 4 warps x
// groups take interleaved sources of the tile, two at a time.  Partial sums
// are reduced in FP64 through shuffles and shared memory; each target is
// written once.
//   MIXED = false: FP64 throughout (P2P.hpp:43-79, green64).
//   MIXED = true : difference vector, r^2, 1/r and the reduction of k r in
//   FP64; sin/cos of the reduced angle, 1/(4 pi r) and the complex products
//   in FP32 with compensated sums (p2p_pair_mixed).
// Source record in shared memory: a = (x, y), b = (z, charge) with the FP32
// charge bits in b.y (mixed) or the FP64 charge in c (FP64 path).

// Compensated (Kahan) FP32 summation: s - c carries the sum.
__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
  const float y = x - c;
  const float t = s + y;
  c = (t - s) - y;
  s = t;
}

// Mixed-precision interaction with FP32 compensated accumulators (the FP64
// path: green64_r).  1/r: approximate FP64 reciprocal square root
// refined once in FP64 (relative error ~1e-14), used for k r, and rounded to
// FP32 for 1/(4 pi r).  k r = n pi + x with n read from the
// low mantissa bits of k r / pi + 1.5 * 2^52 (exact for k r / pi < 2^51) and
// x = k r - n pi in FP64; sin/cos of x by the FP32 Taylor polynomials of
// degree 13 and 12 (truncation below 7e-10 on [-pi/2, pi/2]), (-1)^n applied
// to both.
__device__ __forceinline__ void p2p_pair_mixed(double x0, double x1, double x2, double2 a, double2 b, double kappa,
                                               float& sr, float& cr, float& si, float& ci) {
  const double dx = x0 - a.x, dy = x1 - a.y, dz = x2 - b.x;
  const double R = fma(dx, dx, fma(dy, dy, dz * dz));
  if (R < 1.e-16) return;  // self / duplicate pairs (P2P.hpp:66)
  double yd = rsqrt_approx64(R);
  yd = yd * fma(-0.5 * R * yd, yd, 1.5);
  const float y = (float)yd;
  const double theta = R * yd * kappa;
  const double t = fma(theta, 0.31830988618379067154, 6755399441055744.0);  // + 1.5 * 2^52
  const double n = t - 6755399441055744.0;
  const int odd = __double2loint(t) & 1;
  const float x = (float)fma(-n, 3.14159265358979323846, theta);
  const float xx = x * x;
  float ps = fmaf(xx, 1.6059043836821613e-10f, -2.5052108385441720e-08f);
  ps = fmaf(xx, ps, 2.7557319223985893e-06f);
  ps = fmaf(xx, ps, -1.9841269841269841e-04f);
  ps = fmaf(xx, ps, 8.3333333333333333e-03f);
  ps = fmaf(xx, ps, -1.6666666666666667e-01f);
  ps = fmaf(xx, ps, 1.0f);
  float pc = fmaf(xx, 2.0876756987868099e-09f, -2.7557319223985891e-07f);
  pc = fmaf(xx, pc, 2.4801587301587302e-05f);
  pc = fmaf(xx, pc, -1.3888888888888889e-03f);
  pc = fmaf(xx, pc, 4.1666666666666667e-02f);
  pc = fmaf(xx, pc, -0.5f);
  pc = fmaf(xx, pc, 1.0f);
  const float K = odd ? -0.0795774715459476679f * y : 0.0795774715459476679f * y;  // (-1)^n / (4 pi r)
  const float c = pc * K, s = x * ps * K;
  const float2 q = *reinterpret_cast<const float2*>(&b.y);
  kahan_add(sr, cr, fmaf(c, q.x, -s * q.y));
  kahan_add(si, ci, fmaf(c, q.y, s * q.x));
}

template <bool MIXED>
__global__ void __launch_bounds__(128) k_p2p_tiled(DevPlan P, int64_t nitem, const int32_t* __restrict__ order,
                                                   const int32_t* __restrict__ item_chunk,
                                                   const int32_t* __restrict__ tfirst, const int32_t* __restrict__ tn,
                                                   const int64_t* __restrict__ ptr, const int32_t* __restrict__ sfirst,
                                                   const int32_t* __restrict__ sn, const void* __restrict__ qv,
                                                   double2* __restrict__ pnear, double2* __restrict__ tpart,
                                                   int split, unsigned long long* __restrict__ queue) {
  constexpr int TS = 512;
  typedef typename std::conditional<MIXED, float2, double2>::type Q;
  const Q* q = static_cast<const Q*>(qv);
  __shared__ double2 sa[TS], sb[TS];
  __shared__ double2 sc[MIXED ? 1 : TS];
  __shared__ double2 red[4][32];
  __shared__ int64_t cur;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double kq = P.kappa * 0.63661977236758134308;  // 2 k / pi
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) cur = (int64_t)atomicAdd(queue, 1ULL);
    __syncthreads();
    const int64_t k = cur;
    if (k >= nitem * split) break;
    const int64_t it = order[k / split];
    int tile = split - (int)(k % split);  // tiles until this part's first one, counted from split
    const int64_t ch = item_chunk ? item_chunk[it] : it;
    const int f = tfirst[ch], nt = tn[ch];
    int tp = 1;
    while (tp < nt) tp <<= 1;
    const int groups = 32 / tp, G = 4 * groups;
    const int mt = lane & (tp - 1), gid = warp * groups + lane / tp;
    const int ti = f + min(mt, nt - 1);
    const double x0 = P.T_pos[3 * (int64_t)ti], x1 = P.T_pos[3 * (int64_t)ti + 1], x2 = P.T_pos[3 * (int64_t)ti + 2];
    double pr = 0., pim = 0.;
    float sr = 0.f, cr = 0.f, si = 0.f, ci = 0.f;  // mixed: compensated FP32 sums
    const int64_t rb = ptr[it], re = ptr[it + 1];
    int64_t r = rb;
    int off = 0;  // position inside range r
    while (r < re) {
      // fill one tile from consecutive ranges (uniform control flow)
      int fill = 0;
      const bool mine = tile++ % split == 0;
      if (mine) __syncthreads();
      while (r < re && fill < TS) {
        const int s0 = sfirst[r], ns = sn[r];
        const int take = min(ns - off, TS - fill);
        for (int t = mine ? threadIdx.x : take; t < take; t += blockDim.x) {
          const int64_t sj = (int64_t)s0 + off + t;
          const double* y = P.S_pos + 3 * sj;
          sa[fill + t] = make_double2(y[0], y[1]);
          if (MIXED) {
            const float2 qq = *reinterpret_cast<const float2*>(&q[sj]);
            double qbits;
            *reinterpret_cast<float2*>(&qbits) = qq;
            sb[fill + t] = make_double2(y[2], qbits);
          } else {
            sb[fill + t] = make_double2(y[2], 0.);
            sc[fill + t] = *reinterpret_cast<const double2*>(&q[sj]);
          }
        }
        fill += take;
        off += take;
        if (off == ns) {
          r++;
          off = 0;
        }
      }
      if (!mine) continue;
      __syncthreads();
      int j = gid;
      if constexpr (MIXED) {
        for (; j + G < fill; j += 2 * G) {
          p2p_pair_mixed(x0, x1, x2, sa[j], sb[j], P.kappa, sr, cr, si, ci);
          p2p_pair_mixed(x0, x1, x2, sa[j + G], sb[j + G], P.kappa, sr, cr, si, ci);
        }
        if (j < fill) p2p_pair_mixed(x0, x1, x2, sa[j], sb[j], P.kappa, sr, cr, si, ci);
      } else {
#pragma unroll 4
        for (; j < fill; j += G) {
          const double2 a = sa[j];
          double2 qd = sc[j];
          const double dx = x0 - a.x, dy = x1 - a.y, dz = x2 - sb[j].x;
          const double R = fma(dx, dx, fma(dy, dy, dz * dz));
          const double2 g = green64_r<true>(R, kq);
          // a point's own charge may be infinite or NaN and stays out of its
          // potential: 0 times 0, not 0 times the charge (a select; a branch
          // around the sums took blobs to a sphere, 15,001 points, from 352 to
          // 377 us per matvec)
          if (coincident(R)) qd = make_double2(0., 0.);
          pr = fma(g.x, qd.x, fma(-g.y, qd.y, pr));
          pim = fma(g.x, qd.y, fma(g.y, qd.x, pim));
        }
      }
    }
    if constexpr (MIXED) {
      pr = (double)sr - (double)cr;
      pim = (double)si - (double)ci;
    } else {
      pr *= 1. / (4. * 3.14159265358979323846);
      pim *= 1. / (4. * 3.14159265358979323846);
    }
    for (int o = tp; o < 32; o <<= 1) {
      pr += __shfl_xor_sync(0xffffffffu, pr, o);
      pim += __shfl_xor_sync(0xffffffffu, pim, o);
    }
    if (lane < tp) red[warp][lane] = make_double2(pr, pim);
    __syncthreads();
    if (threadIdx.x < nt) {
      double2 a = red[0][threadIdx.x];
      for (int w = 1; w < 4; w++) {
        a.x += red[w][threadIdx.x].x;
        a.y += red[w][threadIdx.x].y;
      }
      if (tpart)
        tpart[(it * split + k % split) * 32 + threadIdx.x] = a;  // item partial, added per chunk by k_p2p_items
      else
        pnear[f + threadIdx.x] = a;
    }
  }
}

// Item partial sums of the near field into p, per chunk in item order.
__global__ void k_p2p_items(int64_t nchunk, const int32_t* __restrict__ tfirst, const int32_t* __restrict__ tn,
                            const int64_t* __restrict__ chunk_items, const double2* __restrict__ tpart,
                            int split, double2* __restrict__ pnear) {
  const int t = threadIdx.x & 31;
  for (int64_t ch = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); ch < nchunk;
       ch += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    if (t >= tn[ch]) continue;
    double ar = 0., ai = 0.;
    for (int64_t it = chunk_items[ch] * split; it < chunk_items[ch + 1] * split; it++) {
      const double2 v = tpart[it * 32 + t];
      ar += v.x;
      ai += v.y;
    }
    double2 o = pnear[tfirst[ch] + t];
    o.x += ar;
    o.y += ai;
    pnear[tfirst[ch] + t] = o;
  }
}

// ----------------------------------------------------- symmetric near field --
// G(x, y) = exp(i k r) / (4 pi r) of one pair (0 for R < 1e-16, P2P.hpp:66)
// with the arithmetic of p2p_pair_mixed.  Branch-free: a pair with R < 1e-16
// is evaluated at R = 1 and scaled by 0.
__device__ __forceinline__ float2 green32(double dx, double dy, double dz, double kappa) {
  const double R0 = fma(dx, dx, fma(dy, dy, dz * dz));
  const bool skip = R0 < 1.e-16;
  const double R = skip ? 1. : R0;
  double yd = rsqrt_approx64(R);
  yd = yd * fma(-0.5 * R * yd, yd, 1.5);
  const float y = (float)yd;
  const double theta = R * yd * kappa;
  const double t = fma(theta, 0.31830988618379067154, 6755399441055744.0);  // + 1.5 * 2^52
  const double n = t - 6755399441055744.0;
  const int odd = __double2loint(t) & 1;
  const float x = (float)fma(-n, 3.14159265358979323846, theta);
  const float xx = x * x;
  float ps = fmaf(xx, 1.6059043836821613e-10f, -2.5052108385441720e-08f);
  ps = fmaf(xx, ps, 2.7557319223985893e-06f);
  ps = fmaf(xx, ps, -1.9841269841269841e-04f);
  ps = fmaf(xx, ps, 8.3333333333333333e-03f);
  ps = fmaf(xx, ps, -1.6666666666666667e-01f);
  ps = fmaf(xx, ps, 1.0f);
  float pc = fmaf(xx, 2.0876756987868099e-09f, -2.7557319223985891e-07f);
  pc = fmaf(xx, pc, 2.4801587301587302e-05f);
  pc = fmaf(xx, pc, -1.3888888888888889e-03f);
  pc = fmaf(xx, pc, 4.1666666666666667e-02f);
  pc = fmaf(xx, pc, -0.5f);
  pc = fmaf(xx, pc, 1.0f);
  const float K0 = odd ? -0.0795774715459476679f * y : 0.0795774715459476679f * y;
  const float K = skip ? 0.f : K0;
  return make_float2(pc * K, x * ps * K);
}

// Near field for a block of right-hand sides (the target-side form of
// k_p2p_tiled): per work item, the chunk's targets in lanes (groups of
// tp >= nt lanes), sources streamed through shared memory with RB charges
// each; one evaluation of G(x, y) (green64 / green32) is multiplied into the
// RB right-hand sides r0 .. r0 + RB - 1 of the R in q (q[j R + r]).  Mixed:
// FP32 products summed in FP32 over at most 16 sources per lane, those
// partial sums added in FP64.
// Sums go to pnear[(t) R + r] (item_chunk == nullptr: items are chunks) or
// to tpart[(item 32 + t) R + r] for k_p2p_items_rhs.
template <bool MIXED, int RB>
struct P2PRhsCfg {
  static constexpr int TS = 256;  // sources per tile
  typedef typename std::conditional<MIXED, float2, double2>::type Q;
  static constexpr size_t smem() { return sizeof(double2) * 2 * TS + sizeof(Q) * TS * RB + sizeof(double2) * 4 * 32 * RB; }
};

template <bool MIXED, int RB>
__global__ void __launch_bounds__(128) k_p2p_rhs(DevPlan P, int64_t nitem, const int32_t* __restrict__ order,
                                                 const int32_t* __restrict__ item_chunk,
                                                 const int32_t* __restrict__ tfirst, const int32_t* __restrict__ tn,
                                                 const int64_t* __restrict__ ptr, const int32_t* __restrict__ sfirst,
                                                 const int32_t* __restrict__ sn, const void* __restrict__ qv, int R,
                                                 int r0, double2* __restrict__ pnear, double2* __restrict__ tpart,
                                                 int split, unsigned long long* __restrict__ queue) {
  typedef P2PRhsCfg<MIXED, RB> G;
  constexpr int TS = G::TS;
  typedef typename G::Q Q;
  const Q* q = static_cast<const Q*>(qv);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* sa = reinterpret_cast<double2*>(smem_raw);
  double2* sb = sa + TS;
  Q* sq = reinterpret_cast<Q*>(sb + TS);
  double2* red = reinterpret_cast<double2*>(sq + TS * RB);  // [4][32][RB]
  __shared__ int64_t cur;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double kq = P.kappa * 0.63661977236758134308;  // 2 k / pi
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) cur = (int64_t)atomicAdd(queue, 1ULL);
    __syncthreads();
    const int64_t k = cur;
    if (k >= nitem * split) break;
    const int64_t it = order[k / split];
    int tile = split - (int)(k % split);  // as in k_p2p_tiled
    const int64_t ch = item_chunk ? item_chunk[it] : it;
    const int f = tfirst[ch], nt = tn[ch];
    int tp = 1;
    while (tp < nt) tp <<= 1;
    const int groups = 32 / tp, GS = 4 * groups;
    const int mt = lane & (tp - 1), gid = warp * groups + lane / tp;
    const int ti = f + min(mt, nt - 1);
    const double x0 = P.T_pos[3 * (int64_t)ti], x1 = P.T_pos[3 * (int64_t)ti + 1], x2 = P.T_pos[3 * (int64_t)ti + 2];
    double2 acc[RB];
#pragma unroll
    for (int b = 0; b < RB; b++) acc[b] = make_double2(0., 0.);
    const int64_t rb = ptr[it], re = ptr[it + 1];
    int64_t r = rb;
    int off = 0;
    while (r < re) {
      int fill = 0;
      const bool mine = tile++ % split == 0;
      if (mine) __syncthreads();
      while (r < re && fill < TS) {
        const int s0 = sfirst[r], ns = sn[r];
        const int take = min(ns - off, TS - fill);
        for (int t = mine ? threadIdx.x : take; t < take; t += blockDim.x) {
          const int64_t sj = (int64_t)s0 + off + t;
          const double* y = P.S_pos + 3 * sj;
          sa[fill + t] = make_double2(y[0], y[1]);
          sb[fill + t] = make_double2(y[2], 0.);
        }
        for (int t = mine ? threadIdx.x : take * RB; t < take * RB; t += blockDim.x) {
          const int64_t sj = (int64_t)s0 + off + t / RB;
          sq[fill * RB + t] = q[sj * R + r0 + t % RB];
        }
        fill += take;
        off += take;
        if (off == ns) {
          r++;
          off = 0;
        }
      }
      if (!mine) continue;
      __syncthreads();
      if constexpr (MIXED) {
        // FP32 products summed in FP32 over at most kFlush sources of this
        // lane, then added into the FP64 sums
        constexpr int kFlush = 16;
        for (int j0 = gid; j0 < fill; j0 += kFlush * GS) {
          const int j1 = min(fill, j0 + kFlush * GS);
          float2 fs[RB];
#pragma unroll
          for (int b = 0; b < RB; b++) fs[b] = make_float2(0.f, 0.f);
#pragma unroll 8
          for (int j = j0; j < j1; j += GS) {
            const double2 a = sa[j], bz = sb[j];
            const Q* qj = sq + j * RB;
            const float2 g = green32(x0 - a.x, x1 - a.y, x2 - bz.x, P.kappa);
            if constexpr (RB % 2 == 0) {  // two right-hand sides per 16-byte load
              const float4* q4 = reinterpret_cast<const float4*>(qj);
#pragma unroll
              for (int b = 0; b < RB; b += 2) {
                const float4 qq = q4[b / 2];
                fs[b].x = fmaf(g.x, qq.x, fmaf(-g.y, qq.y, fs[b].x));
                fs[b].y = fmaf(g.x, qq.y, fmaf(g.y, qq.x, fs[b].y));
                fs[b + 1].x = fmaf(g.x, qq.z, fmaf(-g.y, qq.w, fs[b + 1].x));
                fs[b + 1].y = fmaf(g.x, qq.w, fmaf(g.y, qq.z, fs[b + 1].y));
              }
            } else {
#pragma unroll
              for (int b = 0; b < RB; b++) {
                const float2 qq = qj[b];
                fs[b].x = fmaf(g.x, qq.x, fmaf(-g.y, qq.y, fs[b].x));
                fs[b].y = fmaf(g.x, qq.y, fmaf(g.y, qq.x, fs[b].y));
              }
            }
          }
#pragma unroll
          for (int b = 0; b < RB; b++) {
            acc[b].x += (double)fs[b].x;
            acc[b].y += (double)fs[b].y;
          }
        }
      } else {
#pragma unroll 4
        for (int j = gid; j < fill; j += GS) {
          const double2 a = sa[j], bz = sb[j];
          const Q* qj = sq + j * RB;
          const double2 g = green64(x0 - a.x, x1 - a.y, x2 - bz.x, kq);
#pragma unroll
          for (int b = 0; b < RB; b++) {
            const double2 qq = qj[b];
            acc[b].x = fma(g.x, qq.x, fma(-g.y, qq.y, acc[b].x));
            acc[b].y = fma(g.x, qq.y, fma(g.y, qq.x, acc[b].y));
          }
        }
      }
    }
#pragma unroll
    for (int b = 0; b < RB; b++) {
      if constexpr (!MIXED) {
        acc[b].x *= 1. / (4. * 3.14159265358979323846);
        acc[b].y *= 1. / (4. * 3.14159265358979323846);
      }
      for (int o = tp; o < 32; o <<= 1) {
        acc[b].x += __shfl_xor_sync(0xffffffffu, acc[b].x, o);
        acc[b].y += __shfl_xor_sync(0xffffffffu, acc[b].y, o);
      }
      if (lane < tp) red[(warp * 32 + lane) * RB + b] = acc[b];
    }
    __syncthreads();
    for (int o = threadIdx.x; o < nt * RB; o += blockDim.x) {
      const int t = o / RB, b = o % RB;
      double2 a = red[t * RB + b];
      for (int w = 1; w < 4; w++) {
        a.x += red[(w * 32 + t) * RB + b].x;
        a.y += red[(w * 32 + t) * RB + b].y;
      }
      if (tpart)
        tpart[((it * split + k % split) * 32 + t) * R + r0 + b] = a;
      else
        pnear[(int64_t)(f + t) * R + r0 + b] = a;
    }
  }
}

// Item partial sums of the near field into p for R right-hand sides, per
// chunk in item order (k_p2p_items with R sums per target).
__global__ void k_p2p_items_rhs(int64_t nchunk, const int32_t* __restrict__ tfirst, const int32_t* __restrict__ tn,
                                const int64_t* __restrict__ chunk_items, const double2* __restrict__ tpart, int split, int R,
                                double2* __restrict__ pnear) {
  const int64_t per = 32 * (int64_t)R;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nchunk * per;
       w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ch = w / per;
    const int t = (int)((w % per) / R), rr = (int)(w % R);
    if (t >= tn[ch]) continue;
    double ar = 0., ai = 0.;
    for (int64_t it = chunk_items[ch] * split; it < chunk_items[ch + 1] * split; it++) {
      const double2 v = tpart[(it * 32 + t) * R + rr];
      ar += v.x;
      ai += v.y;
    }
    double2* o = pnear + (int64_t)(tfirst[ch] + t) * R + rr;
    double2 v = *o;
    v.x += ar;
    v.y += ai;
    *o = v;
  }
}

// Tree-order R-wide charges from R stacked user-order vectors:
// q[i R + r] = qin[r stride + perm[i]].
// Vectors r >= nvec of a partly filled block get zero charges.
template <typename T>
__global__ void k_gather_rhs(const double2* __restrict__ qin, const int32_t* __restrict__ perm,
                             typename cpx_t<T>::type* __restrict__ q, int64_t n, int64_t stride, int R, int nvec) {
  const int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (w >= n * R) return;
  const int64_t i = w / R;
  const int r = (int)(w % R);
  const double2 v = r < nvec ? qin[r * stride + perm[i]] : make_double2(0., 0.);
  typename cpx_t<T>::type o;
  o.x = (T)v.x;
  o.y = (T)v.y;
  q[w] = o;
}

// out[r stride + perm[i]] = pnear[i R + r] + pfar[i R + r].
__global__ void k_scatter_rhs(const double2* __restrict__ pnear, const double2* __restrict__ pfar,
                              const int32_t* __restrict__ perm, double2* __restrict__ out, int64_t n, int64_t stride,
                              int R, int nvec) {
  const int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (w >= n * R) return;
  const int64_t i = w / R;
  const int r = (int)(w % R);
  if (r >= nvec) return;
  double2 a = pnear[w], b = pfar[w];
  a.x += b.x;
  a.y += b.y;
  out[r * stride + perm[i]] = a;
}

// Target charges of the mixed path ride in the second word of (z, w).
__device__ __forceinline__ float2 charge_bits(double w) {
  const long long b = __double_as_longlong(w);
  return make_float2(__int_as_float((int)(b & 0xffffffffLL)), __int_as_float((int)(b >> 32)));
}
__device__ __forceinline__ double charge_word(float2 q) {
  return __longlong_as_double(((long long)(unsigned)__float_as_int(q.y) << 32) | (unsigned)__float_as_int(q.x));
}

// Symmetric blocks of the near field (Plan::sym_*) in FP64: one CTA (4 warps)
// per work item, or part of one (part of the sources of one chunk of <= 32
// targets), taken from a queue in the host's order of decreasing work; of each
// batch of up to 128 ranges, part p of split takes round p of 256 sources and
// every split-th one after it.  (With tiny leaves a batch can have fewer rounds
// than the item has parts; the other parts then only write zeros.  Counting on
// over the batches evens that out but costs more than it gives: 20,000 points
// in leaves of 4, up to 288 ranges per item, 1.94 and 1.95 ms; cube 20k 743 and
// 745 us per matvec.)  A lane owns S sources and meets the chunk's targets in
// blocks of 4, read from shared memory by broadcast.  One evaluation of G feeds
// both
//   the target's partial: 4 sums per block, over the lane's S sources; two
//     exchange steps leave one target per lane (summed over 4 lanes), added
//     to the lane's sum for this block in shared memory, and
//   the source's partial (lane-local over all targets),
// so each mirrored pair of interactions costs one kernel evaluation.  Target
// partials of the item go to tpart (added per chunk by k_p2p_items); source
// partials go to scratch and are added per source leaf by k_p2p_reduce.
//
// The sources of an item (thousands) fill the lanes whatever the number of
// targets, which is only padded to a multiple of 4: 92-95% of the evaluated
// pairs count, where segments of nextpow2(targets) lanes that passed the
// targets' sums around gave 76-86%; and 8 independent evaluations per lane
// keep the FP64 pipe fed (65% of its cycles on a 31k-point sphere).  The near
// field of a 250k-point sphere in FP64 took 20.1 ms with the segments and
// takes 14.1 ms so.
struct P2PSym {
  static constexpr int S = 2;       // sources per lane
  static constexpr int NB = 8;      // blocks of 4 targets in a chunk
};

__global__ void __launch_bounds__(128, 4) k_p2p_sym(DevPlan P, int64_t nwork, const int32_t* __restrict__ order,
                                                 const int32_t* __restrict__ item_chunk,
                                                 const int32_t* __restrict__ tfirst, const int32_t* __restrict__ tn,
                                                 const int64_t* __restrict__ ptr, const int32_t* __restrict__ sfirst,
                                                 const int32_t* __restrict__ sn, const int64_t* __restrict__ soff,
                                                 const double2* __restrict__ q, double2* __restrict__ tpart,
                                                 double2* __restrict__ scr, int split, unsigned long long* __restrict__ queue) {
  typedef double2 Q;
  typedef P2PSym G;
  constexpr int RMAX = 128, S = G::S, NB = G::NB;
  __shared__ double2 trxy[4 * NB], tq[4 * NB];
  __shared__ double trz[4 * NB];
  __shared__ Q tacc[4][NB][32];
  __shared__ int32_t rpre[RMAX + 1], rfst[RMAX];
  __shared__ int64_t roff[RMAX];
  __shared__ double2 red[4][32];
  __shared__ int64_t cur;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double kq = P.kappa * 0.63661977236758134308;  // 2 k / pi
  const double scale = 1. / (4. * 3.14159265358979323846);
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) cur = (int64_t)atomicAdd(queue, 1ULL);
    __syncthreads();
    const int64_t k = cur;
    if (k >= nwork * split) break;
    const int64_t it = order[k / split];
    const int part = (int)(k % split);
    const int64_t ch = item_chunk[it];
    const int f = tfirst[ch], nt = tn[ch];
    const int nb = (nt + 3) >> 2;
    if (threadIdx.x < 4 * NB) {
      const int t = threadIdx.x;
      const double* x = P.T_pos + 3 * (int64_t)(f + (t < nt ? t : 0));
      trxy[t] = make_double2(x[0], x[1]);
      trz[t] = x[2];
      tq[t] = t < nt ? q[f + t] : Q{0, 0};
    }
    for (int b = 0; b < nb; b++) tacc[warp][b][lane] = Q{0, 0};
    const int64_t rb = ptr[it], re = ptr[it + 1];
    for (int64_t r0 = rb; r0 < re; r0 += RMAX) {
      const int nr = (int)min((int64_t)RMAX, re - r0);
      __syncthreads();  // previous batch of ranges (and the target arrays) settled
      for (int m = threadIdx.x; m < nr; m += blockDim.x) {
        rfst[m] = sfirst[r0 + m];
        roff[m] = soff[r0 + m];
        rpre[m + 1] = sn[r0 + m];
      }
      __syncthreads();
      if (warp == 0) {  // inclusive scan of the range lengths
        int carry = 0;
        for (int b0 = 0; b0 < nr; b0 += 32) {
          int v = b0 + lane < nr ? rpre[b0 + lane + 1] : 0;
          for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
          }
          if (b0 + lane < nr) rpre[b0 + lane + 1] = carry + v;
          carry += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) rpre[0] = 0;
      }
      __syncthreads();
      const int ntot = rpre[nr];
      for (int base = (part * 4 + warp) * 32 * S; base < ntot; base += split * 4 * 32 * S) {
        double yx[S], yy[S], yz[S];
        Q qj[S], accT[S];
        int64_t sidx[S];
#pragma unroll
        for (int v = 0; v < S; v++) {
          const int jj = base + 32 * v + lane, jc = min(jj, ntot - 1);
          int lo = 0, hi = nr - 1;  // last range with rpre <= jc
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (rpre[mid] <= jc) lo = mid; else hi = mid - 1;
          }
          const int o = jc - rpre[lo];
          const int64_t sj = (int64_t)rfst[lo] + o;
          const double* y = P.S_pos + 3 * sj;
          yx[v] = y[0];
          yy[v] = y[1];
          yz[v] = y[2];
          qj[v] = jj < ntot ? q[sj] : Q{0, 0};
          accT[v] = Q{0, 0};
          sidx[v] = jj < ntot ? roff[lo] + o : -1;
        }
        // no validity tests: padded targets (copies of the first) and missing
        // sources (copies of the last) carry zero charges, and their sums are
        // never stored
        for (int b = 0; b < nb; b++) {
          // squared distances first: coincident points (R < 1e-16, P2P.hpp:66)
          // are rare, so one test of the block's smallest high word chooses
          // the evaluations without a test of their own
          Q d[4];
          double R[4][S];
          unsigned least = UINT_MAX;
#pragma unroll
          for (int t = 0; t < 4; t++) {
            const double2 a = trxy[4 * b + t];
            const double z = trz[4 * b + t];
            d[t] = Q{0, 0};
#pragma unroll
            for (int v = 0; v < S; v++) {
              const double dx = a.x - yx[v], dy = a.y - yy[v], dz = z - yz[v];
              R[t][v] = fma(dx, dx, fma(dy, dy, dz * dz));
              least = min(least, (unsigned)__double2hiint(R[t][v]));
            }
          }
          auto block = [&](auto guard) {
            constexpr bool GUARD = decltype(guard)::value;
#pragma unroll
            for (int t = 0; t < 4; t++) {
#pragma unroll
              for (int v = 0; v < S; v++) {
                const Q g = green64_r<GUARD>(R[t][v], kq), qi = tq[4 * b + t];
                d[t].x = fma(g.x, qj[v].x, fma(-g.y, qj[v].y, d[t].x));
                d[t].y = fma(g.x, qj[v].y, fma(g.y, qj[v].x, d[t].y));
                accT[v].x = fma(g.x, qi.x, fma(-g.y, qi.y, accT[v].x));
                accT[v].y = fma(g.x, qi.y, fma(g.y, qi.x, accT[v].y));
              }
            }
          };
          if (__any_sync(0xffffffffu, least <= kNearR2Hi))
            block(std::true_type());
          else
            block(std::false_type());
          // lanes with bit 4 keep targets 2, 3, the others 0, 1; then bit 3
          // chooses the odd or the even one
          const bool h1 = lane & 16, h0 = lane & 8;
          Q k0 = h1 ? d[2] : d[0], k1 = h1 ? d[3] : d[1], s0 = h1 ? d[0] : d[2], s1 = h1 ? d[1] : d[3];
          k0.x += __shfl_xor_sync(0xffffffffu, s0.x, 16);
          k0.y += __shfl_xor_sync(0xffffffffu, s0.y, 16);
          k1.x += __shfl_xor_sync(0xffffffffu, s1.x, 16);
          k1.y += __shfl_xor_sync(0xffffffffu, s1.y, 16);
          Q kk = h0 ? k1 : k0;
          s0 = h0 ? k0 : k1;
          kk.x += __shfl_xor_sync(0xffffffffu, s0.x, 8);
          kk.y += __shfl_xor_sync(0xffffffffu, s0.y, 8);
          Q o = tacc[warp][b][lane];
          o.x += kk.x;
          o.y += kk.y;
          tacc[warp][b][lane] = o;
        }
#pragma unroll
        for (int v = 0; v < S; v++)
          if (sidx[v] >= 0) {
            accT[v].x *= scale;
            accT[v].y *= scale;
            scr[sidx[v]] = accT[v];
          }
      }
    }
    for (int b = 0; b < nb; b++) {
      const Q o = tacc[warp][b][lane];
      double pr = o.x * scale, pim = o.y * scale;
#pragma unroll
      for (int w = 4; w; w >>= 1) {
        pr += __shfl_xor_sync(0xffffffffu, pr, w);
        pim += __shfl_xor_sync(0xffffffffu, pim, w);
      }
      if (!(lane & 7)) red[warp][4 * b + (lane >> 3 & 2) + (lane >> 3 & 1)] = make_double2(pr, pim);
    }
    __syncthreads();
    if (threadIdx.x < nt) {
      double2 a = red[0][threadIdx.x];
      for (int w = 1; w < 4; w++) {
        a.x += red[w][threadIdx.x].x;
        a.y += red[w][threadIdx.x].y;
      }
      tpart[(it * split + part) * 32 + threadIdx.x] = a;
    }
  }
}

// The same blocks in mixed precision: their FP32 sums keep one order, pair by
// pair, so they go by segments.  tp steps of a block: lane ls owns one source
// (y, qj) and meets target (ls + step) mod tp; the target's running sum moves
// one lane down per step.  TP = 32 fixes the segment width at compile time.
// Target records in shared memory as two 16-byte arrays, (x, y) and (z, w)
// with w the charge's bits: one conflict-free 16-byte load from each per step.
// Entry j holds target j mod tp (j < 64), so step st of lane ls reads entry
// ls + st without wrapping arithmetic.
template <int TP>
__device__ __forceinline__ void sym_steps(int ls, int tp_rt, double yx, double yy, double yz, float2 qj,
                                          const double2* trxy, const double2* trzw, double kappa, float2& accD,
                                          float2& accT) {
  const int tp = TP ? TP : tp_rt;
  const double2* txy = trxy + ls;
  const double2* tzw = trzw + ls;
#pragma unroll 8
  for (int st = 0; st < tp; st++) {
    const double2 a = txy[st], b = tzw[st];
    const float2 g = green32(a.x - yx, a.y - yy, b.x - yz, kappa);
    const float2 qi = charge_bits(b.y);
    accD.x = fmaf(g.x, qj.x, fmaf(-g.y, qj.y, accD.x));
    accD.y = fmaf(g.x, qj.y, fmaf(g.y, qj.x, accD.y));
    accT.x = fmaf(g.x, qi.x, fmaf(-g.y, qi.y, accT.x));
    accT.y = fmaf(g.x, qi.y, fmaf(g.y, qi.x, accT.y));
    accD.x = __shfl_sync(0xffffffffu, accD.x, ls + 1, tp);
    accD.y = __shfl_sync(0xffffffffu, accD.y, ls + 1, tp);
  }
}

// One CTA (4 warps) per work item; a warp splits into segments of tp =
// nextpow2(nt) lanes; lane l of a segment owns source l of the segment's
// tp-source sub-tile and, over tp steps, meets every target i = (l + step)
// mod tp.  The target's partial is an accumulator that moves one lane down per
// step and ends in lane i (compensated sums over the sub-tiles); the source's
// is lane-local.  Issue bound: 64 instructions per evaluation, 76-86% of the
// evaluated pairs count (600k-point sphere 22.5 ms; sources in lanes as above
// take 19.6 ms, but round the FP32 sums differently by 2e-7).
__global__ void __launch_bounds__(128) k_p2p_sym_mixed(DevPlan P, int64_t nwork, const int32_t* __restrict__ order,
                                                 const int32_t* __restrict__ item_chunk,
                                                 const int32_t* __restrict__ tfirst, const int32_t* __restrict__ tn,
                                                 const int64_t* __restrict__ ptr, const int32_t* __restrict__ sfirst,
                                                 const int32_t* __restrict__ sn, const int64_t* __restrict__ soff,
                                                 const float2* __restrict__ q, double2* __restrict__ tpart,
                                                 float2* __restrict__ scr, unsigned long long* __restrict__ queue) {
  typedef float2 Q;
  constexpr int RMAX = 128;
  __shared__ double2 trxy[64], trzw[64];
  __shared__ int32_t rpre[RMAX + 1], rfst[RMAX];
  __shared__ int64_t roff[RMAX];
  __shared__ double2 red[4][32];
  __shared__ int64_t cur;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) cur = (int64_t)atomicAdd(queue, 1ULL);
    __syncthreads();
    const int64_t k = cur;
    if (k >= nwork) break;
    const int64_t it = order[k];
    const int64_t ch = item_chunk[it];
    const int f = tfirst[ch], nt = tn[ch];
    int tp = 4;
    while (tp < nt) tp <<= 1;
    const int ls = lane & (tp - 1);
    if (threadIdx.x < 64) {
      const int j = threadIdx.x, t = j & (tp - 1);
      if (t < nt) {
        const double* x = P.T_pos + 3 * (int64_t)(f + t);
        const Q qt = q[f + t];
        trxy[j] = make_double2(x[0], x[1]);
        trzw[j] = make_double2(x[2], charge_word(qt));
      } else {
        trxy[j] = make_double2(0., 0.);
        trzw[j] = make_double2(0., 0.);
      }
    }
    float sr = 0.f, cr = 0.f, si = 0.f, ci = 0.f;  // compensated target sums
    const int64_t rb = ptr[it], re = ptr[it + 1];
    for (int64_t r0 = rb; r0 < re; r0 += RMAX) {
      const int nr = (int)min((int64_t)RMAX, re - r0);
      __syncthreads();  // previous batch of ranges (and the target arrays) settled
      for (int m = threadIdx.x; m < nr; m += blockDim.x) {
        rfst[m] = sfirst[r0 + m];
        roff[m] = soff[r0 + m];
        rpre[m + 1] = sn[r0 + m];
      }
      __syncthreads();
      if (warp == 0) {  // inclusive scan of the range lengths
        int carry = 0;
        for (int b0 = 0; b0 < nr; b0 += 32) {
          int v = b0 + lane < nr ? rpre[b0 + lane + 1] : 0;
          for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
          }
          if (b0 + lane < nr) rpre[b0 + lane + 1] = carry + v;
          carry += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) rpre[0] = 0;
      }
      __syncthreads();
      const int ntot = rpre[nr];
      for (int base = warp * 32; base < ntot; base += 4 * 32) {
        const int jj = base + lane;
        const bool vj = jj < ntot;
        double yx = 0., yy = 0., yz = 0.;
        Q qj = Q{0, 0};
        int64_t sidx = 0;
        if (vj) {
          int lo = 0, hi = nr - 1;  // last range with rpre <= jj
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (rpre[mid] <= jj) lo = mid; else hi = mid - 1;
          }
          const int o = jj - rpre[lo];
          const int64_t sj = (int64_t)rfst[lo] + o;
          sidx = roff[lo] + o;
          const double* y = P.S_pos + 3 * sj;
          yx = y[0];
          yy = y[1];
          yz = y[2];
          qj = q[sj];
        }
        Q accD = Q{0, 0}, accT = Q{0, 0};
        // no validity tests: padded targets and missing sources carry zero
        // charges, and their target sums are never stored
        if (tp == 32)
          sym_steps<32>(ls, 32, yx, yy, yz, qj, trxy, trzw, P.kappa, accD, accT);
        else
          sym_steps<0>(ls, tp, yx, yy, yz, qj, trxy, trzw, P.kappa, accD, accT);
        kahan_add(sr, cr, accD.x);
        kahan_add(si, ci, accD.y);
        if (vj) scr[sidx] = accT;
      }
    }
    double pr = (double)sr - (double)cr, pim = (double)si - (double)ci;
    for (int o = tp; o < 32; o <<= 1) {  // segments of the warp hold the same targets
      pr += __shfl_xor_sync(0xffffffffu, pr, o);
      pim += __shfl_xor_sync(0xffffffffu, pim, o);
    }
    if (lane < tp) red[warp][lane] = make_double2(pr, pim);
    __syncthreads();
    if (threadIdx.x < nt) {
      double2 a = red[0][threadIdx.x];
      for (int w = 1; w < 4; w++) {
        a.x += red[w][threadIdx.x].x;
        a.y += red[w][threadIdx.x].y;
      }
      tpart[it * 32 + threadIdx.x] = a;
    }
  }
}

// Source-side partial sums of the symmetric blocks, per source leaf in a
// fixed order (Plan::red_*): p_j += sum_k scratch[off_k + (j - first)].
// One CTA per leaf: 4 groups of 64 threads (one particle each) sum
// contiguous quarters of the leaf's rows, row offsets staged in shared
// memory and four rows in flight per thread; the quarters are added in order.
template <bool MIXED>
__global__ void __launch_bounds__(256) k_p2p_reduce(int64_t nleaf, const int32_t* __restrict__ first,
                                                    const int32_t* __restrict__ n, const int64_t* __restrict__ rptr,
                                                    const int64_t* __restrict__ roff, const void* __restrict__ scratch,
                                                    double2* __restrict__ pnear) {
  typedef typename std::conditional<MIXED, float2, double2>::type Q;
  constexpr int RB = 256;  // row offsets staged per round
  const Q* scr = static_cast<const Q*>(scratch);
  __shared__ int64_t so[RB];
  __shared__ double2 part[4][64];
  const int g = threadIdx.x >> 6, jl = threadIdx.x & 63;
  // (leaf, block of 64 particles): leaves of more than 64 particles take
  // several passes
  for (int64_t l = blockIdx.x; l < nleaf; l += gridDim.x)
  for (int j0 = 0; j0 < n[l]; j0 += 64) {
    const int nl = n[l], j = j0 + jl;
    const int64_t kb = rptr[l], ke = rptr[l + 1];
    double ar = 0., ai = 0.;
    __syncthreads();  // the previous pass is done with part[][]
    for (int64_t k0 = kb; k0 < ke; k0 += RB) {
      const int nr = (int)min((int64_t)RB, ke - k0);
      __syncthreads();
      for (int t = threadIdx.x; t < nr; t += blockDim.x) so[t] = roff[k0 + t];
      __syncthreads();
      // group g takes rows [g*nr/4, (g+1)*nr/4) of this round
      const int r0 = g * nr / 4, r1 = (g + 1) * nr / 4;
      if (j < nl) {
        int r = r0;
        for (; r + 4 <= r1; r += 4) {
          const Q v0 = scr[so[r] + j], v1 = scr[so[r + 1] + j], v2 = scr[so[r + 2] + j], v3 = scr[so[r + 3] + j];
          ar += (double)v0.x;
          ai += (double)v0.y;
          ar += (double)v1.x;
          ai += (double)v1.y;
          ar += (double)v2.x;
          ai += (double)v2.y;
          ar += (double)v3.x;
          ai += (double)v3.y;
        }
        for (; r < r1; r++) {
          const Q v = scr[so[r] + j];
          ar += (double)v.x;
          ai += (double)v.y;
        }
      }
    }
    part[g][jl] = make_double2(ar, ai);
    __syncthreads();
    if (g == 0 && j < nl) {
      double2 o = pnear[first[l] + j];
      for (int q = 0; q < 4; q++) {
        o.x += part[q][jl].x;
        o.y += part[q][jl].y;
      }
      pnear[first[l] + j] = o;
    }
  }
}

// ------------------------------------------------------------ direct sum --
// FP64 direct sum at sampled targets (CheckFULL arithmetic,
// interface.hpp:178-221): one warp per target, lanes over sources.
__global__ void k_direct(int64_t ns, const double* __restrict__ spos, const int32_t* __restrict__ sperm,
                         const double2* __restrict__ qin, int64_t nt, const double* __restrict__ tpos,
                         double kappa, double2* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const double pi4m1 = 1. / (4. * 3.14159265358979323846);
  for (int64_t t = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); t < nt;
       t += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    const double x0 = tpos[3 * t], x1 = tpos[3 * t + 1], x2 = tpos[3 * t + 2];
    double pr = 0., pim = 0.;
    for (int64_t j = lane; j < ns; j += 32) {
      const double dx = x0 - spos[3 * j], dy = x1 - spos[3 * j + 1], dz = x2 - spos[3 * j + 2];
      const double R = dx * dx + dy * dy + dz * dz;
      double K = 1. / sqrt(R);
      if (R < 1.e-16) K = 0.;
      const double rr = K * R * kappa;
      K *= pi4m1;
      double s, c;
      sincos(rr, &s, &c);
      const double2 qq = qin[sperm[j]];
      pr += c * K * qq.x - s * K * qq.y;
      pim += c * K * qq.y + s * K * qq.x;
    }
    for (int off = 16; off; off >>= 1) {
      pr += __shfl_xor_sync(0xffffffffu, pr, off);
      pim += __shfl_xor_sync(0xffffffffu, pim, off);
    }
    if (lane == 0) out[t] = make_double2(pr, pim);
  }
}

// ---------------------------------------------------------------- launch --
namespace {
// twiddles exp(-2 pi i m / P) of every order, computed on the device
__global__ void k_twiddles(double* tw) {
  for (int L = kMinOrder; L <= kMaxOrder; L++) {
    const int P = 2 * L - 1;
    for (int m = threadIdx.x; m < P; m += blockDim.x) {
      double s, c;
      sincospi(-2.0 * m / P, &s, &c);
      tw[2 * (tw_off(L) + m)] = c;
      tw[2 * (tw_off(L) + m) + 1] = s;
    }
  }
}

// Constant tables of the current device: twiddles of every order on first
// use, the interpolation matrices of order L (m2m[0], m2m[1], l2l[0], l2l[1];
// they depend on L only) on first use of L.  Later calls write nothing, so
// kernels of other operators in flight never see a table change.
cudaError_t upload_tables(int L, const double* mats) {
  static std::mutex mu;
  static std::set<std::pair<int, int>> done;  // (device, L); L = 0: twiddles
  std::lock_guard<std::mutex> lock(mu);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!done.count({dev, 0})) {
    constexpr int n = 2 * tw_off(kMaxOrder + 1);
    double* d = nullptr;
    if ((e = cudaMalloc(&d, n * sizeof(double))) != cudaSuccess) return e;
    k_twiddles<<<1, 32>>>(d);
    std::vector<double> h64(n);
    e = cudaMemcpy(h64.data(), d, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return e;
    std::vector<float> h32(h64.begin(), h64.end());
    if ((e = cudaMemcpyToSymbol(c_tw64, h64.data(), n * sizeof(double))) != cudaSuccess ||
        (e = cudaMemcpyToSymbol(c_tw32, h32.data(), n * sizeof(float))) != cudaSuccess)
      return e;
    done.insert({dev, 0});
  }
  if (!done.count({dev, L})) {
    const int n = 4 * L * L;
    std::vector<float> m32(mats, mats + n);
    if ((e = cudaMemcpyToSymbol(c_mat64, mats, n * sizeof(double), mat_off(L) * sizeof(double))) != cudaSuccess ||
        (e = cudaMemcpyToSymbol(c_mat32, m32.data(), n * sizeof(float), mat_off(L) * sizeof(float))) != cudaSuccess)
      return e;
    done.insert({dev, L});
  }
  return cudaSuccess;
}

int grid_for(int64_t n, int per_block, int cap = 148 * 64) {
  int64_t g = (n + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}
}  // namespace

template <typename T, int L>
struct Launch {
  typedef typename cpx_t<T>::type C;
  static constexpr int P = 2 * L - 1, LL = L * L * L, PP = P * P * P;
  static constexpr int NT = PP > 1024 ? 256 : 128;
  static size_t smem_m2f() { return sizeof(C) * M2FCfg<T, L>::PER_WARP * M2FCfg<T, L>::NW; }
  static size_t smem_m2l() { return sizeof(C) * PP; }
  template <int RB>
  static size_t smem_m2l_rhs() { return (m2l_rhs_joint<T, L, RB>() ? RB : 1) * smem_m2l(); }
  static cudaError_t setup(const double* mats) {
    cudaError_t e0 = upload_tables(L, mats);
    if (e0 != cudaSuccess) return e0;
    cudaError_t e = cudaFuncSetAttribute(k_m2f<T, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_m2f());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_m2l<T, L, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_m2l());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_m2l<T, L, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_m2l());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_m2l_pair<T, L, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_m2l());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_m2l_pair<T, L, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_m2l());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_p2m<T, L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)P2MCfg<T, L>::smem(kMaxRhsBlock));
    if (e != cudaSuccess) return e;
    if constexpr (L2PHf<T, L>::use) {
      if ((e = cudaFuncSetAttribute(k_l2p_hf<T, L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)L2PHf<T, L>::smem())) != cudaSuccess)
        return e;
    }
    if ((e = rhs_attr<1, 128>()) != cudaSuccess || (e = rhs_attr<2, 128>()) != cudaSuccess ||
        (e = rhs_attr<4, 256>()) != cudaSuccess || (e = rhs_attr<8, 256>()) != cudaSuccess ||
        (e = bulk_attr()) != cudaSuccess)
      return e;
    return cudaSuccess;
  }
  // largest block of right-hand sides per M2L CTA: K x RB <= 24 complex
  // accumulators per thread at 256 threads
  static constexpr int kMaxRB = (PP + 255) / 256 <= 3 ? 8 : ((PP + 255) / 256 <= 6 ? 4 : ((PP + 255) / 256 <= 12 ? 2 : 1));
  template <int RB, int NT>
  static cudaError_t rhs_attr() {
    if (RB > kMaxRB) return cudaSuccess;
    return cudaFuncSetAttribute(k_m2l_rhs<T, L, NT, (RB <= kMaxRB ? RB : 1)>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_m2l_rhs<(RB <= kMaxRB ? RB : 1)>());
  }
  template <int RB, int NT>
  static void m2l_rhs_go(const DevPlan& dp, int64_t u0, int64_t u1, int64_t f0, int64_t f1, int R, const void* F,
                         const void* ptab, void* Lx, unsigned long long* queue, int nsm, cudaStream_t s) {
    constexpr int RBE = RB <= kMaxRB ? RB : 1;
    const int64_t nwork = (u1 - u0) * (R / RBE);
    const int grid = (int)std::min<int64_t>(nwork, (int64_t)nsm * m2l_rhs_ctas<T, L, NT, RBE>());
    k_m2l_rhs<T, L, NT, RBE><<<grid, NT, smem_m2l_rhs<RBE>(), s>>>(dp, u0, u1, f0, f1, R, (const C*)F, (const C*)ptab,
                                                          (C*)Lx, queue);
  }
  // the shared-memory-staged kernel: FP32, orders 3-6
  static constexpr bool kBulk = std::is_same<T, float>::value && L >= 3 && L <= 6;
  static cudaError_t bulk_attr() {
    if constexpr (kBulk)
      return cudaFuncSetAttribute(k_m2l_bulk<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)M2LBulk<L>::smem());
    return cudaSuccess;
  }
  static bool m2l_bulk(const DevPlan& dp, int64_t t0, int64_t t1, int64_t f0, int64_t f1, int R, const void* F,
                       const void* ptab, void* Lx, unsigned long long* queue, int nsm, int64_t lgroup,
                       cudaStream_t s) {
    if constexpr (kBulk) {
      typedef M2LBulk<L> B;
      if (lgroup <= 0 || lgroup > B::LCAP || R % B::RB) return false;
      const int64_t nwork = (t1 - t0 + B::G - 1) / B::G * (R / B::RB);
      const int grid = (int)std::min<int64_t>(nwork, (int64_t)nsm * B::CTAS);
      k_m2l_bulk<L><<<grid, B::NT, B::smem(), s>>>(dp, t0, t1, f0, f1, R, (const float2*)F, (const float2*)ptab,
                                                   (float2*)Lx, queue);
      return true;
    }
    return false;
  }
  // M2L for R right-hand sides in blocks of rb (1, 2, 4 or 8; a divisor of
  // R, capped by the order's kMaxRB), or staged through shared memory
  static void m2l_rhs(const DevPlan& dp, int64_t u0, int64_t u1, int64_t t0, int64_t t1, int64_t f0, int64_t f1,
                      int R, int rb,
                      const void* F, const void* ptab, void* Lx, unsigned long long* queue, int nsm,
                      int64_t lgroup, cudaStream_t s) {
    if (u1 <= u0) return;
    cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
    if (m2l_bulk(dp, t0, t1, f0, f1, R, F, ptab, Lx, queue, nsm, lgroup, s)) return;
    if (rb > kMaxRB) rb = kMaxRB;
    while (rb > 1 && R % rb) rb >>= 1;
    if (rb >= 8)
      m2l_rhs_go<8, 256>(dp, u0, u1, f0, f1, R, F, ptab, Lx, queue, nsm, s);
    else if (rb >= 4)
      m2l_rhs_go<4, 256>(dp, u0, u1, f0, f1, R, F, ptab, Lx, queue, nsm, s);
    else if (rb >= 2)
      m2l_rhs_go<2, 128>(dp, u0, u1, f0, f1, R, F, ptab, Lx, queue, nsm, s);
    else
      m2l_rhs_go<1, 128>(dp, u0, u1, f0, f1, R, F, ptab, Lx, queue, nsm, s);
  }
  static void p2m(const DevPlan& dp, const int32_t* leaves, int n, const void* q, const void* sig2, void* M, int R,
                  int d0, int d1, cudaStream_t s) {
    if (!n) return;
    // parts until there are 16 CTAs per SM (3 to 6 are resident): the three P2M
    // launches (95, 364 and 938 leaves) of blobs of 15,001 points, order 4,
    // three right-hand sides, FP64 took 134 us whole and take 95 us in parts
    const int split = std::max(1, std::min(4, 148 * 16 / n));
    k_p2m<T, L><<<grid_for((int64_t)n * split, 1), 128, P2MCfg<T, L>::smem(R), s>>>(
        dp, leaves, n, (const C*)q, (const C*)sig2, (C*)M, R, d0, d1, split);
  }
  static void m2m(const DevPlan& dp, int64_t s0, int64_t s1, const void* sig, const void* sig2, void* Mp,
                  const void* Mc, int R, cudaStream_t s) {
    constexpr int NW = kXferWarps;
    if (s1 > s0)
      k_m2m<T, L><<<grid_for(s1 - s0, NW), 32 * NW, 0, s>>>(dp, s0, s1, (const C*)sig, (const C*)sig2, (C*)Mp,
                                                                  (const C*)Mc, R);
  }
  static void l2l(const DevPlan& dp, int64_t s0, int64_t s1, const void* sig, const void* sig2, void* Lc,
                  const void* Lp, int R, int64_t p0, int64_t p1, cudaStream_t s) {
    constexpr int NW = kXferWarps;
    if (s1 > s0)
      k_l2l<T, L><<<grid_for(s1 - s0, NW), 32 * NW, 0, s>>>(dp, s0, s1, (const C*)sig, (const C*)sig2, (C*)Lc,
                                                                  (const C*)Lp, R, p0, p1);
  }
  static void m2f(int64_t n, int R, const int32_t* slist, const void* M, void* F, cudaStream_t s) {
    constexpr int NW = M2FCfg<T, L>::NW;
    if (n)
      k_m2f<T, L><<<grid_for(n * R, NW), 32 * NW, smem_m2f(), s>>>(n * R, R, slist, (const C*)M, (C*)F);
  }
  static void m2l(const DevPlan& dp, int64_t u0, int64_t u1, int64_t f0, int64_t f1, const void* F,
                  const void* ptab, void* Lx, unsigned long long* queue, int nsm, int nt, int pair,
                  cudaStream_t s) {
    if (u1 <= u0) return;
    cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
    if (nt != 128 && nt != 256) nt = NT;
    if (pair) {
      const int grid = (int)std::min<int64_t>((u1 - u0 + 1) / 2, (int64_t)nsm * (2048 / nt));
      if (nt == 256)
        k_m2l_pair<T, L, 256><<<grid, 256, smem_m2l(), s>>>(dp, u0, u1, f0, f1, (const C*)F, (const C*)ptab, (C*)Lx,
                                                            queue);
      else
        k_m2l_pair<T, L, 128><<<grid, 128, smem_m2l(), s>>>(dp, u0, u1, f0, f1, (const C*)F, (const C*)ptab, (C*)Lx,
                                                            queue);
      return;
    }
    const int grid = (int)std::min<int64_t>(u1 - u0, (int64_t)nsm * (2048 / nt));
    if (nt == 256)
      k_m2l<T, L, 256><<<grid, 256, smem_m2l(), s>>>(dp, u0, u1, f0, f1, (const C*)F, (const C*)ptab, (C*)Lx, queue);
    else
      k_m2l<T, L, 128><<<grid, 128, smem_m2l(), s>>>(dp, u0, u1, f0, f1, (const C*)F, (const C*)ptab, (C*)Lx, queue);
  }
  static void permute(int64_t n, const uint32_t* key, const uint16_t* perm, const void* tables, void* out,
                      cudaStream_t s) {
    if (n) k_permute_tables<T><<<grid_for(n, 1), 256, 0, s>>>(n, PP, key, perm, (const C*)tables, (C*)out);
  }
  static void l2p(const DevPlan& dp, const int32_t* leaves, int n, bool hf, const void* sig2, const void* Lx,
                  double2* pfar, int R, int d0, int d1, bool accum, cudaStream_t s) {
    if (!n) return;
    if constexpr (L2PHf<T, L>::use) {
      if (hf) {
        k_l2p_hf<T, L><<<grid_for(n, 1), 128, L2PHf<T, L>::smem(), s>>>(dp, leaves, n, (const C*)sig2, (const C*)Lx,
                                                                        pfar);
        return;
      }
    }
    if (R == 1)
      k_l2p<T, L, 1><<<grid_for(n, 1), 128, 0, s>>>(dp, leaves, n, (const C*)sig2, (const C*)Lx, pfar, R, d0, d1,
                                                    accum);
    else
      k_l2p<T, L, 4><<<grid_for(n, 1), 128, 0, s>>>(dp, leaves, n, (const C*)sig2, (const C*)Lx, pfar, R, d0, d1,
                                                    accum);
  }
};

template <typename T>
const OpTable* op_table_for(int L);

#define DFB_OPS(T, L)                                                                                     \
  {                                                                                                       \
    Launch<T, L>::setup, Launch<T, L>::p2m, Launch<T, L>::m2m, Launch<T, L>::l2l, Launch<T, L>::m2f,       \
        Launch<T, L>::m2l, Launch<T, L>::m2l_rhs, Launch<T, L>::l2p, Launch<T, L>::permute,                 \
        Launch<T, L>::kMaxRB                                                                              \
  }

template <>
const OpTable* op_table_for<double>(int L) {
  static const OpTable t[9] = {{},
                               {},
                               DFB_OPS(double, 2),
                               DFB_OPS(double, 3),
                               DFB_OPS(double, 4),
                               DFB_OPS(double, 5),
                               DFB_OPS(double, 6),
                               DFB_OPS(double, 7),
                               DFB_OPS(double, 8)};
  return (L >= 2 && L <= 8) ? &t[L] : nullptr;
}

template <>
const OpTable* op_table_for<float>(int L) {
  static const OpTable t[9] = {{},
                               {},
                               DFB_OPS(float, 2),
                               DFB_OPS(float, 3),
                               DFB_OPS(float, 4),
                               DFB_OPS(float, 5),
                               DFB_OPS(float, 6),
                               DFB_OPS(float, 7),
                               DFB_OPS(float, 8)};
  return (L >= 2 && L <= 8) ? &t[L] : nullptr;
}

const OpTable* op_table(int L, bool fp64) { return fp64 ? op_table_for<double>(L) : op_table_for<float>(L); }

void launch_gather(bool fp64, const double2* qin, const int32_t* perm, void* q, int64_t n, int64_t sin_, int64_t sq,
                   int nrhs, cudaStream_t s) {
  const int g = (int)((n + 255) / 256);
  if (fp64)
    k_gather<double><<<g, 256, 0, s>>>(qin, perm, (double2*)q, n, sin_, sq, nrhs);
  else
    k_gather<float><<<g, 256, 0, s>>>(qin, perm, (float2*)q, n, sin_, sq, nrhs);
}

void launch_scatter(const double2* pnear, const double2* pfar, const int32_t* perm, double2* out, int64_t n,
                    cudaStream_t s) {
  k_scatter<<<(int)((n + 255) / 256), 256, 0, s>>>(pnear, pfar, perm, out, n);
}

void launch_p2p(bool fp64, const DevPlan& dp, int64_t nitem, const int32_t* order, const int32_t* item_chunk,
                const int32_t* tfirst, const int32_t* tn, const int64_t* ptr, const int32_t* sfirst, const int32_t* sn,
                const void* q, double2* pnear, double2* tpart, int split, unsigned long long* queue, int nsm,
                cudaStream_t s) {
  if (!nitem) return;
  cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
  const int grid = (int)std::min<int64_t>(nitem * split, (int64_t)nsm * 16);
  if (fp64)
    k_p2p_tiled<false><<<grid, 128, 0, s>>>(dp, nitem, order, item_chunk, tfirst, tn, ptr, sfirst, sn, q, pnear,
                                            tpart, split, queue);
  else
    k_p2p_tiled<true><<<grid, 128, 0, s>>>(dp, nitem, order, item_chunk, tfirst, tn, ptr, sfirst, sn, q, pnear,
                                           tpart, split, queue);
}

void launch_p2p_items(int64_t nchunk, const int32_t* tfirst, const int32_t* tn, const int64_t* chunk_items,
                      const double2* tpart, int split, double2* pnear, int nsm, cudaStream_t s) {
  if (nchunk <= 0) return;
  const int grid = (int)std::min<int64_t>((nchunk + 3) / 4, (int64_t)nsm * 16);
  k_p2p_items<<<grid, 128, 0, s>>>(nchunk, tfirst, tn, chunk_items, tpart, split, pnear);
}

void launch_p2p_sym(bool fp64, const DevPlan& dp, int64_t nwork, const int32_t* order, const int32_t* item_chunk,
                    const int32_t* tfirst, const int32_t* tn, const int64_t* ptr, const int32_t* sfirst,
                    const int32_t* sn, const int64_t* soff, const void* q, double2* tpart, void* scratch, int split,
                    unsigned long long* queue, int nsm, int blocks_per_sm, cudaStream_t s) {
  if (nwork <= 0) return;
  cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
  const int grid = (int)std::min<int64_t>(nwork * split, (int64_t)nsm * std::max(1, std::min(blocks_per_sm, 64)));
  if (fp64)
    k_p2p_sym<<<grid, 128, 0, s>>>(dp, nwork, order, item_chunk, tfirst, tn, ptr, sfirst, sn, soff,
                                   (const double2*)q, tpart, (double2*)scratch, split, queue);
  else
    k_p2p_sym_mixed<<<grid, 128, 0, s>>>(dp, nwork, order, item_chunk, tfirst, tn, ptr, sfirst, sn, soff,
                                         (const float2*)q, tpart, (float2*)scratch, queue);
}

void launch_p2p_reduce(bool fp64, int64_t nleaf, const int32_t* first, const int32_t* n, const int64_t* rptr,
                       const int64_t* roff, const void* scratch, double2* pnear, int nsm, cudaStream_t s) {
  if (nleaf <= 0) return;
  const int grid = (int)std::min<int64_t>(nleaf, (int64_t)nsm * 16);
  if (fp64)
    k_p2p_reduce<false><<<grid, 256, 0, s>>>(nleaf, first, n, rptr, roff, scratch, pnear);
  else
    k_p2p_reduce<true><<<grid, 256, 0, s>>>(nleaf, first, n, rptr, roff, scratch, pnear);
}

cudaError_t setup_rhs_kernels() {
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_p2p_rhs<true, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)P2PRhsCfg<true, 8>::smem())) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_p2p_rhs<false, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)P2PRhsCfg<false, 8>::smem())) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_p2p_rhs<true, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)P2PRhsCfg<true, 4>::smem())) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_p2p_rhs<false, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)P2PRhsCfg<false, 4>::smem())) != cudaSuccess)
    return e;
  return cudaSuccess;
}

template <bool MIXED, int RB>
static void p2p_rhs_go(const DevPlan& dp, int64_t nitem, const int32_t* order, const int32_t* item_chunk,
                       const int32_t* tfirst, const int32_t* tn, const int64_t* ptr, const int32_t* sfirst,
                       const int32_t* sn, const void* q, int R, int r0, double2* pnear, double2* tpart,
                       int split, unsigned long long* queue, int grid, cudaStream_t s) {
  k_p2p_rhs<MIXED, RB><<<grid, 128, P2PRhsCfg<MIXED, RB>::smem(), s>>>(dp, nitem, order, item_chunk, tfirst, tn, ptr,
                                                                       sfirst, sn, q, R, r0, pnear, tpart, split,
                                                                       queue);
}

void launch_p2p_rhs(bool fp64, const DevPlan& dp, int64_t nitem, const int32_t* order, const int32_t* item_chunk,
                    const int32_t* tfirst, const int32_t* tn, const int64_t* ptr, const int32_t* sfirst,
                    const int32_t* sn, const void* q, int R, double2* pnear, double2* tpart, int split,
                    unsigned long long* queue, int nsm, int blocks_per_sm, cudaStream_t s) {
  if (!nitem) return;
  const int grid = (int)std::min<int64_t>(nitem * split, (int64_t)nsm * std::max(1, std::min(blocks_per_sm, 64)));
  auto go = [&](auto rb, int r0) {
    constexpr int RB = decltype(rb)::value;
    cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
    if (fp64)
      p2p_rhs_go<false, RB>(dp, nitem, order, item_chunk, tfirst, tn, ptr, sfirst, sn, q, R, r0, pnear, tpart, split,
                            queue, grid, s);
    else
      p2p_rhs_go<true, RB>(dp, nitem, order, item_chunk, tfirst, tn, ptr, sfirst, sn, q, R, r0, pnear, tpart, split,
                           queue, grid, s);
  };
  for (int r0 = 0; r0 < R;) {
    const int left = R - r0;
    const int rb = left >= 8 ? 8 : (left >= 4 ? 4 : left);
    if (rb == 8) go(std::integral_constant<int, 8>(), r0);
    if (rb == 4) go(std::integral_constant<int, 4>(), r0);
    if (rb == 3) go(std::integral_constant<int, 3>(), r0);
    if (rb == 2) go(std::integral_constant<int, 2>(), r0);
    if (rb == 1) go(std::integral_constant<int, 1>(), r0);
    r0 += rb;
  }
}

void launch_p2p_items_rhs(int64_t nchunk, const int32_t* tfirst, const int32_t* tn, const int64_t* chunk_items,
                          const double2* tpart, int split, int R, double2* pnear, int nsm, cudaStream_t s) {
  if (nchunk <= 0) return;
  const int grid = (int)std::min<int64_t>((nchunk * 32 * R + 255) / 256, (int64_t)nsm * 16);
  k_p2p_items_rhs<<<grid, 256, 0, s>>>(nchunk, tfirst, tn, chunk_items, tpart, split, R, pnear);
}

void launch_gather_rhs(bool fp64, const double2* qin, const int32_t* perm, void* q, int64_t n, int64_t stride, int R,
                       int nvec, cudaStream_t s) {
  const int g = (int)((n * R + 255) / 256);
  if (fp64)
    k_gather_rhs<double><<<g, 256, 0, s>>>(qin, perm, (double2*)q, n, stride, R, nvec);
  else
    k_gather_rhs<float><<<g, 256, 0, s>>>(qin, perm, (float2*)q, n, stride, R, nvec);
}

void launch_scatter_rhs(const double2* pnear, const double2* pfar, const int32_t* perm, double2* out, int64_t n,
                        int64_t stride, int R, int nvec, cudaStream_t s) {
  k_scatter_rhs<<<(int)((n * R + 255) / 256), 256, 0, s>>>(pnear, pfar, perm, out, n, stride, R, nvec);
}

void launch_direct(int64_t ns, const double* spos, const int32_t* sperm, const double2* qin, int64_t nt,
                   const double* tpos, double kappa, double2* out, cudaStream_t s) {
  if (nt) k_direct<<<grid_for(nt, 8, 148 * 16), 256, 0, s>>>(ns, spos, sperm, qin, nt, tpos, kappa, out);
}

}  // namespace dfb
