// M2L with the inverse DFT fused, over windows of consecutive target slots.
// Included by fmm_kernels.cu (uses its twiddles).
#pragma once

// ---------------------------------------------------------------- spectra --
// Rows of F and of the permuted transfer spectra hold the PP entries of one
// spectrum padded to whole slabs: a slab is what one warp reads with one
// 16-byte load per lane (512 bytes: 64 FP32 or 32 FP64 complex entries), so
// every load of the M2L is aligned and full.
template <typename T, int L>
struct Spec {
  static constexpr int PD = 2 * L - 1, PP = PD * PD * PD, LL = L * L * L;
  static constexpr int VEC = 16 / (2 * (int)sizeof(T));  // entries per lane
  static constexpr int SLAB = 32 * VEC;
  static constexpr int NS = (PP + SLAB - 1) / SLAB;      // slabs per spectrum
  static constexpr int ROW = NS * SLAB;                  // row stride, entries
};

// One line of the inverse DFT, pruned to its L low outputs:
//   out[a] = sum_k v[k] conj(w)^(k a),  w = exp(-2 pi i / PD).
// The terms k and PD - k share their cosine and their sine up to sign, so
// they are added and subtracted first: 4 (L - 1) FMAs per output, not
// 8 (L - 1).
template <typename T, int L, typename C>
__device__ __forceinline__ void idft_line(const C (&v)[2 * L - 1], C (&out)[L]) {
  constexpr int PD = 2 * L - 1;
  C s[L], d[L];
#pragma unroll
  for (int k = 1; k < L; k++) {
    s[k].x = v[k].x + v[PD - k].x;
    s[k].y = v[k].y + v[PD - k].y;
    d[k].x = v[k].x - v[PD - k].x;
    d[k].y = v[k].y - v[PD - k].y;
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
        const C w = ctw<T, L>((k * a) % PD);  // (cos, -sin)
        o.x = fma(w.x, s[k].x, o.x);
        o.y = fma(w.x, s[k].y, o.y);
        o.x = fma(w.y, d[k].y, o.x);
        o.y = fma(-w.y, d[k].x, o.y);
      }
    }
    out[a] = o;
  }
}

// ------------------------------------------------------------------- M2L --
template <typename T, int L, int RB>
struct M2LWin {
  typedef Spec<T, L> S;
  typedef typename cpx_t<T>::type C;
  static constexpr int JROW = S::PP + (S::VEC - 1);  // PP is odd: 16-byte rows in FP32
  static constexpr int W0 = 98304 / (JROW * RB * (int)sizeof(C));
  static constexpr int W = W0 >= 32 ? 32 : (W0 >= 16 ? 16 : (W0 >= 8 ? 8 : (W0 >= 4 ? 4 : (W0 >= 2 ? 2 : 1))));
  static constexpr int CPT = W >= 16 ? 48 : 96;  // list entries per target and pass (even)
  static constexpr int NT = 512;
  static constexpr size_t smem() { return (size_t)W * RB * JROW * sizeof(C) + (size_t)W * CPT * sizeof(int2); }
};

template <typename T>
__device__ __forceinline__ void ldvec(const char* p, typename cpx_t<T>::type (&v)[16 / (2 * (int)sizeof(T))]) {
  if constexpr (sizeof(T) == 4) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = make_float2(f.x, f.y);
    v[1] = make_float2(f.z, f.w);
  } else {
    v[0] = __ldg(reinterpret_cast<const double2*>(p));
  }
}

template <typename T, int L, int RB>
__global__ void __launch_bounds__(512, 1)
    k_m2l_win(DevPlan P, int64_t t0, int64_t t1, int64_t f0, int64_t f1, int R, int w,
              const typename cpx_t<T>::type* __restrict__ F, const typename cpx_t<T>::type* __restrict__ ptab,
              typename cpx_t<T>::type* __restrict__ Lx, unsigned long long* __restrict__ queue) {
  typedef typename cpx_t<T>::type C;
  typedef M2LWin<T, L, RB> G;
  typedef Spec<T, L> S;
  constexpr int PD = S::PD, PP = S::PP, LL = S::LL, NT = G::NT, VEC = S::VEC, JROW = G::JROW, CPT = G::CPT;
  constexpr int64_t ROWB = (int64_t)S::ROW * sizeof(C);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* J = reinterpret_cast<C*>(smem_raw);
  int2* list = reinterpret_cast<int2*>(J + (size_t)G::W * RB * JROW);
  __shared__ int64_t cur, eb[G::W];
  __shared__ int len[G::W], maxlen, unit;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = R / RB;
  const int64_t nwork = (t1 - t0 + w - 1) / w * nb;
  for (;;) {
    __syncthreads();  // the previous window's transform is done with J
    if (threadIdx.x == 0) cur = (int64_t)atomicAdd(queue, 1ULL);
    __syncthreads();
    if (cur >= nwork) break;
    const int64_t t = t0 + cur / nb * w;
    const int r0 = (int)(cur % nb) * RB;
    const int nt = (int)min((int64_t)w, t1 - t);
    if (warp == 0) {
      int n = 0;
      if (lane < nt) {
        const int64_t b = P.m2l_ptr[t + lane];
        n = (int)(P.m2l_ptr[t + lane + 1] - b);
        eb[lane] = b;
        len[lane] = n;
      }
      n = __reduce_max_sync(0xffffffffu, n);
      if (lane == 0) maxlen = n;
    }
    __syncthreads();
    const int ml = maxlen;
    for (int p0 = 0; p0 < ml; p0 += CPT) {
      if (p0) __syncthreads();
      if (threadIdx.x == 0) unit = 0;
      for (int x = threadIdx.x; x < nt * CPT; x += NT) {
        const int j = x / CPT, e = p0 + x % CPT;
        if (e < len[j]) {
          int64_t s = (int64_t)P.m2l_src[eb[j] + e] - f0;
          if (s < 0 || s >= f1 - f0) {  // entry outside this cone batch: a plan bug
            atomicExch(P.err, 1);
            s = 0;
          }
          list[x] = make_int2((int)s, (int)P.m2l_tab[eb[j] + e]);
        }
      }
      __syncthreads();
      for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(&unit, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= nt * S::NS) break;
        const int sl = u / nt, j = u % nt;
        const int n = min(len[j] - p0, CPT);
        if (n <= 0) continue;
        const char* Fb = reinterpret_cast<const char*>(F) + (int64_t)r0 * ROWB + sl * 512 + lane * 16;
        const char* Ub = reinterpret_cast<const char*>(ptab) + sl * 512 + lane * 16;
        const int4* le = reinterpret_cast<const int4*>(list + j * CPT);
        const int i0 = sl * S::SLAB + lane * VEC;
        C acc[RB][VEC];
#pragma unroll
        for (int b = 0; b < RB; b++)
#pragma unroll
          for (int v = 0; v < VEC; v++) acc[b][v] = czero<C>();
        if (p0) {
          if (i0 < PP)
#pragma unroll
            for (int b = 0; b < RB; b++)
#pragma unroll
              for (int v = 0; v < VEC; v++) acc[b][v] = J[(j * RB + b) * JROW + i0 + v];
        }
        auto one = [&](int s, int k) {
          C uu[VEC], ff[VEC];
          ldvec<T>(Ub + (int64_t)(uint32_t)k * ROWB, uu);
#pragma unroll
          for (int b = 0; b < RB; b++) {
            ldvec<T>(Fb + ((int64_t)s * R + b) * ROWB, ff);
#pragma unroll
            for (int v = 0; v < VEC; v++) cfma(acc[b][v], uu[v], ff[v]);
          }
        };
        int i = 0;
#pragma unroll 2
        for (; i + 1 < n; i += 2) {
          const int4 e = le[i >> 1];
          one(e.x, e.y);
          one(e.z, e.w);
        }
        if (i < n) {
          const int2 e = list[j * CPT + i];
          one(e.x, e.y);
        }
        if (i0 < PP)
#pragma unroll
          for (int b = 0; b < RB; b++) {
            C* o = J + (j * RB + b) * JROW + i0;
            if constexpr (VEC == 2)
              *reinterpret_cast<float4*>(o) = make_float4(acc[b][0].x, acc[b][0].y, acc[b][1].x, acc[b][1].y);
            else
              o[0] = acc[b][0];
          }
      }
    }
    __syncthreads();
    // inverse DFTs of the window's spectra, every axis in place (a line's
    // outputs go to the entries its own thread has read)
    for (int x = threadIdx.x; x < nt * RB * PD * PD; x += NT) {  // axis 0: (k1, k2) lines
      const int r = x / (PD * PD), ln = x % (PD * PD);
      if (!len[r / RB]) continue;
      C* q = J + r * JROW + ln;
      C v[PD], o[L];
#pragma unroll
      for (int k = 0; k < PD; k++) v[k] = q[k * PD * PD];
      idft_line<T, L>(v, o);
#pragma unroll
      for (int a = 0; a < L; a++) q[a * PD * PD] = o[a];
    }
    __syncthreads();
    for (int x = threadIdx.x; x < nt * RB * L * PD; x += NT) {  // axis 1: (a, k2) lines
      const int r = x / (L * PD), ln = x % (L * PD);
      if (!len[r / RB]) continue;
      C* q = J + r * JROW + ln / PD * (PD * PD) + ln % PD;
      C v[PD], o[L];
#pragma unroll
      for (int k = 0; k < PD; k++) v[k] = q[k * PD];
      idft_line<T, L>(v, o);
#pragma unroll
      for (int b = 0; b < L; b++) q[b * PD] = o[b];
    }
    __syncthreads();
    for (int x = threadIdx.x; x < nt * RB * L * L; x += NT) {  // axis 2: (a, b) lines into L
      const int r = x / (L * L), ln = x % (L * L);
      if (!len[r / RB]) continue;
      const C* q = J + r * JROW + (ln / L * PD + ln % L) * PD;
      C v[PD], o[L];
#pragma unroll
      for (int k = 0; k < PD; k++) v[k] = q[k];
      idft_line<T, L>(v, o);
      C* Lt = Lx + ((t + r / RB) * R + r0 + r % RB) * LL + ln * L;
      const T inv = T(1) / T(PP);
#pragma unroll
      for (int c = 0; c < L; c++) {
        C y = Lt[c];
        y.x += o[c].x * inv;
        y.y += o[c].y * inv;
        Lt[c] = y;
      }
    }
  }
}
