// One GMRES cycle as one persistent kernel, for systems whose Arnoldi step is
// bound by latency rather than by bandwidth (see the rule at coop_plan).
//
// A step launched as separate kernels pays a launch, a cold start and a drain
// for each of its six or seven phases, and its orthogonalization kernels
// stream all columns through a handful of blocks when the vectors are short.
// Here every CTA owns a run of consecutive nodes for the whole cycle: its part
// of w stays in shared memory, and so do its rows of the basis and of the
// matrix when they fit; only z (the preconditioned vector that the neighbours
// gather) and the partial sums of the dot products go through L2. The phases
// are separated by a grid barrier. The CTAs are co-resident (cooperative
// launch, one per SM), every wait has a limit, and a CTA whose wait ran out
// sets GState::pad and returns.
//
// The Givens rotations are a serial chain; an extra warp of CTA 0 applies them
// while the other warps go on with the next step, which learns of a finished
// cycle at a barrier it needs anyway.
//
// Included by krylov.cu inside its anonymous namespace.

template <typename T, typename TA, typename TV>
struct CoopArgs {
  int N;                   // nodes
  int chunk;               // nodes of a CTA, a multiple of 8
  int m;                   // most columns
  int two_pass;            // conditional second Gram-Schmidt pass
  double tol_abs;
  const int* brow_ptr;
  const int* bcol;
  const TA* A;
  const T* Dinv;
  const T* Bc;             // blocks of the second sweep, or null
  TV* V;                   // basis columns when shared memory does not hold them
  T *z1, *z2;              // preconditioned vectors, gathered by the neighbours
  T *part1, *part2, *partn;  // partial sums: (m + 1) per CTA, and one per CTA
  T *H, *y;
  unsigned* ctl;           // finished, columns; barrier: arrivals, CTAs that left
  // the cycle starts from src (scaled by sd) and its correction goes to dst:
  // inner solve: src = V_j, dst = Z_j of the outer state; else src = r, dst += correction
  const double* src;
  const double* sd;
  double* dst;
  GState* st;              // outer state (inner solve), or the state of this cycle
  int inner;
  int smem_bytes;
  int limit;               // of a wait
};

__device__ __forceinline__ void coop_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kCoopThreads) : "memory"); }
__device__ __forceinline__ void givens_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kCoopThreads + 32) : "memory");
}
__device__ __forceinline__ void givens_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kCoopThreads + 32) : "memory");
}
constexpr int kBarColumn = 2, kBarRotated = 3;  // a column is ready for the Givens warp; it has been rotated

// The grid barrier (grid_barrier.cuh). Flags that each CTA raises and all poll
// took 5,500 clocks and more against 2,300, and one cluster of 16 CTAs that
// meet at an mbarrier gained nothing (its release waits for the same stores).
struct CoopSync {
  unsigned* count;  // arrivals since the kernel began (cleared by the last CTA to leave)
  unsigned target;
  int* ok;          // shared
  int limit;
};

// Warp 0 of every CTA, after a block barrier.
__device__ __forceinline__ void coop_meet(CoopSync& s) {
  if (threadIdx.x == 0) *s.ok = grid_meet(s.count, s.target, s.limit) ? 1 : 0;
  __syncwarp();
}

// Barrier of all worker threads of all CTAs; false when a wait ran out.
__device__ __forceinline__ bool grid_sync(CoopSync& s) {
  coop_bar();
  s.target += gridDim.x;
  if (threadIdx.x < 32) coop_meet(s);
  coop_bar();
  return *s.ok != 0;
}

// A node's entries of a vector that other CTAs have written in this kernel
// (plain loads: the acquire of the barrier empties L1, which a CTA's
// neighbouring rows then share)
__device__ __forceinline__ void ld_z4(const float* p, float& a, float& b, float& c, float& d) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a = v.x; b = v.y; c = v.z; d = v.w;
}
__device__ __forceinline__ void ld_z4(const double* p, double& a, double& b, double& c, double& d) {
  const double2 u = *reinterpret_cast<const double2*>(p);
  const double2 v = *(reinterpret_cast<const double2*>(p) + 1);
  a = u.x; b = u.y; c = v.x; d = v.y;
}

// Sums of eight values over a warp with 9 additions instead of 40: every
// exchange halves the number of values a lane holds. Returns the sum of value
// coop_col(lane).
template <typename T>
__device__ __forceinline__ T warp_sum8(T (&v)[8], int lane) {
#pragma unroll
  for (int o = 16, h = 4; h >= 1; o >>= 1, h >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const T give = up ? v[i] : v[i + h];
      const T keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  T s = v[0];
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}
__device__ __forceinline__ int coop_col(int lane) {
  return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Rows a lane handles at a time: whole nodes where a basis group is one
// vector load, single rows in FP64 (its pipe is the bound, and short runs of
// rows then leave no lane idle).
template <typename T>
struct CoopRows { static constexpr int R = 4; };
template <>
struct CoopRows<double> { static constexpr int R = 1; };

template <typename T, typename TV>
__device__ __forceinline__ void ld_rows(const TV* p, T (&x)[4]) { load_row<T, TV>(p, x[0], x[1], x[2], x[3]); }
template <typename T, typename TV>
__device__ __forceinline__ void ld_rows(const TV* p, T (&x)[1]) { x[0] = ldv<T, TV>(p); }
template <typename T>
__device__ __forceinline__ void ld_w(const T* p, T (&x)[4]) { Vec4<T>::load(p, x[0], x[1], x[2], x[3]); }
template <typename T>
__device__ __forceinline__ void ld_w(const T* p, T (&x)[1]) { x[0] = *p; }

// This CTA's partial sums of w . V_c for c < ncols, and of w . w as column
// ncols if `self`, to part[CTA][column]. Two mappings:
//  * FP64 with the basis in shared memory: a lane is a column and runs down a
//    share of the rows, so that no addition is spent on a reduction over
//    lanes (one FP64 instruction of a warp takes the SM's pipe 19 clocks);
//  * else eight columns to a warp, lanes across the rows.
// In both, warps left over by the columns share the rows.
template <typename T, typename TV>
__device__ __forceinline__ void coop_dots(const T* w, const TV* V, long long vld, int rows, int ncols, bool self,
                                          bool staged, T* red, T* part, int ldp) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int total = ncols + (self ? 1 : 0);
  int shares;
  if (std::is_same<T, double>::value && staged) {
    const int sets = (total + 31) >> 5;
    shares = max(1, kCoopWarps / 2 / sets);
    const int set = wid % sets, share = wid / sets;
    const int c = 32 * set + lane;
    if (share < shares) {
      T acc = T(0);
      const TV* v = V + (long long)min(c, ncols - 1) * vld;
      if (c == ncols) v = reinterpret_cast<const TV*>(w);
#pragma unroll 4
      for (int r = share; r < rows; r += shares) acc = fma(ldv<T, TV>(v + r), w[r], acc);
      red[share * 32 * sets + c] = acc;
    }
    coop_bar();
    for (int q = threadIdx.x; q < total; q += kCoopThreads) {
      T s = red[q];
      for (int k = 1; k < shares; ++k) s += red[k * 32 * sets + q];
      part[(long long)blockIdx.x * ldp + q] = s;
    }
  } else {
    constexpr int R = CoopRows<T>::R;
    const int sets = (total + 7) >> 3;
    shares = max(1, kCoopWarps / sets);
    for (int s0 = wid; s0 < sets * shares; s0 += kCoopWarps) {
      const int c0 = 8 * (s0 % sets), share = s0 / sets;
      const TV* v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = V + (long long)min(c0 + q, ncols - 1) * vld;
      const int sq = self && c0 <= ncols && ncols < c0 + 8 ? ncols - c0 : -1;
      T acc[8], ww = T(0);
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = T(0);
#pragma unroll 2
      for (int g = (share * 32 + lane) * R; g < rows; g += shares * 32 * R) {
        T x[R], y[8][R];
        ld_w(w + g, x);
#pragma unroll
        for (int q = 0; q < 8; ++q) ld_rows<T, TV>(v[q] + g, y[q]);
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
          for (int e = 0; e < R; ++e) acc[q] = fma(y[q][e], x[e], acc[q]);
        if (sq >= 0) {
#pragma unroll
          for (int e = 0; e < R; ++e) ww = fma(x[e], x[e], ww);
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q == sq) acc[q] = ww;
      const T s = warp_sum8(acc, lane);
      if ((lane & 3) == 0) red[share * 8 * sets + c0 + coop_col(lane)] = s;
    }
    coop_bar();
    for (int q = threadIdx.x; q < total; q += kCoopThreads) {
      T s = red[q];
      for (int k = 1; k < shares; ++k) s += red[k * 8 * sets + q];
      part[(long long)blockIdx.x * ldp + q] = s;
    }
  }
}

// Totals of columns 0..total-1 of part (part[CTA][column]) into out; every CTA
// forms all of them: a lane is a column, the warps share the CTAs' entries.
// Column c < scaled is of a basis vector stored as
// V_c / scale_c: out_c = scale_c x sum, and coef_c = scale_c out_c is its
// coefficient in the update.
template <typename T>
__device__ __forceinline__ void coop_totals(const T* part, int ldp, int total, int scaled, const T* scale, T* red,
                                            T* out, T* coef) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, G = gridDim.x;
  const int sets = (total + 31) >> 5, shares = max(1, kCoopWarps / sets);
  const int set = wid % sets, share = wid / sets, c = 32 * set + lane;
  if (share < shares) {
    T acc = T(0);
    if (c < total) {
      if constexpr (std::is_same<T, double>::value) {
#pragma unroll 8
        for (int k = share; k < G; k += shares) acc += __ldcg(part + (long long)k * ldp + c);
      } else {
        for (int k0 = share; k0 < G; k0 += 10 * shares) {
          T v[10];
#pragma unroll
          for (int u = 0; u < 10; ++u) {
            const int k = k0 + u * shares;
            v[u] = k < G ? __ldcg(part + (long long)k * ldp + c) : T(0);
          }
#pragma unroll
          for (int u = 0; u < 10; ++u)
            if (k0 + u * shares < G) acc += v[u];
        }
      }
    }
    red[share * 32 * sets + c] = acc;
  }
  coop_bar();
  for (int q = threadIdx.x; q < total; q += kCoopThreads) {
    T s = red[q];
    for (int k = 1; k < shares; ++k) s += red[k * 32 * sets + q];
    if (q < scaled) {
      s *= scale[q];
      coef[q] = s * scale[q];
    }
    out[q] = s;
  }
  coop_bar();
}

// The power of two nearest below 1 / sqrt(x), from the exponent bits alone;
// any finite power for x that is no positive number.
__device__ __forceinline__ float pow2_rsqrt(float x) {
  const int e = ((__float_as_int(x) >> 23) & 0xff) - 127;
  return __int_as_float((127 - (e >> 1)) << 23);
}
__device__ __forceinline__ double pow2_rsqrt(double x) {
  const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
  return __hiloint2double((1023 - (e >> 1)) << 20, 0);
}

// w -= V h over this CTA's rows; returns the thread's share of |w|^2. `split`
// lanes share a row group, each with every split-th column.
template <typename T, typename TV>
__device__ __forceinline__ T coop_update(T* w, const TV* V, long long vld, int rows, int ncols, const T* h,
                                         int split, bool staged) {
  constexpr int R = CoopRows<T>::R;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int per = 32 / split, gl = lane & (per - 1), s = lane / per;
  T sq = T(0);
  for (int g0 = wid * per * R; g0 < rows; g0 += kCoopWarps * per * R) {
    const int g = g0 + gl * R;
    const bool live = g < rows;
    T acc[R];
#pragma unroll
    for (int e = 0; e < R; ++e) acc[e] = T(0);
    if (live) {
      if (std::is_same<T, double>::value || staged) {
#pragma unroll 4
        for (int c = s; c < ncols; c += split) {
          const T hc = h[c];
          T v[R];
          ld_rows<T, TV>(V + c * vld + g, v);
#pragma unroll
          for (int e = 0; e < R; ++e) acc[e] = fma(hc, v[e], acc[e]);
        }
      } else {  // from L2 or HBM: whole batches under way (64^3 mesh: 321 -> 301 ms a solve)
        constexpr int B = 8;
        for (int c0 = s; c0 < ncols; c0 += B * split) {
          T v[B][R];
#pragma unroll
          for (int u = 0; u < B; ++u) ld_rows<T, TV>(V + min(c0 + u * split, ncols - 1) * vld + g, v[u]);
#pragma unroll
          for (int u = 0; u < B; ++u)
            if (c0 + u * split < ncols) {
              const T hc = h[c0 + u * split];
#pragma unroll
              for (int e = 0; e < R; ++e) acc[e] = fma(hc, v[u][e], acc[e]);
            }
        }
      }
    }
    for (int o = per; o < 32; o <<= 1)
#pragma unroll
      for (int e = 0; e < R; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    if (live && s == 0) {
#pragma unroll
      for (int e = 0; e < R; ++e) {
        const T v = w[g + e] - acc[e];
        w[g + e] = v;
        sq = fma(v, v, sq);
      }
    }
  }
  return sq;
}

// Norm over all CTAs from the threads' shares of its square, and its
// reciprocal, to all worker threads; a grid barrier as well. Returns false
// when a wait ran out. One warp forms the root and the reciprocal (an FP64
// root by all sixteen takes the pipe 2,300 clocks, by one 600).
template <typename T>
__device__ __forceinline__ bool coop_norm(T v, T* red, T* partn, CoopSync& sync, T& norm, T& inv) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) red[wid] = v;
  coop_bar();
  sync.target += gridDim.x;
  if (wid == 0) {
    T s = warp_sum(lane < kCoopWarps ? red[lane] : T(0));
    if (lane == 0) partn[blockIdx.x] = s;
    __syncwarp();
    coop_meet(sync);
    s = T(0);
    if constexpr (std::is_same<T, double>::value) {
      for (int k = lane; k < (int)gridDim.x; k += 32) s += __ldcg(partn + k);
    } else {
      for (int k0 = lane; k0 < (int)gridDim.x; k0 += 160) {
        T p[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) p[u] = k0 + 32 * u < (int)gridDim.x ? __ldcg(partn + k0 + 32 * u) : T(0);
        s += ((p[0] + p[1]) + (p[2] + p[3])) + p[4];
      }
    }
    s = sqrt(warp_sum(s));
    const T i = T(1) / s;
    if (lane == 0) {
      red[kCoopWarps] = s;
      red[kCoopWarps + 1] = i;
    }
  }
  coop_bar();
  norm = red[kCoopWarps];
  inv = red[kCoopWarps + 1];
  return *sync.ok != 0;
}

// The Givens warp of CTA 0: rotates column after column, publishes whether
// the cycle is finished, and ends with the back substitution.
template <typename T>
struct GivensShared {
  int cols;    // columns so far (set by the workers with the column)
  int last;    // no further column follows
  int quit;    // a wait ran out: leave
  int done;    // set by the Givens warp
  T norm;
  T beta;
};

// y = R^-1 g by one warp, column by column: entry r of g in lane r mod 32, D
// columns of up to 32 Q rows in registers and D more on their way from L2. (One
// column ahead, a step took L2's latency: 50k clocks for 60 columns, 5% of a
// small cycle, while all CTAs wait for y.)
template <typename T, int Q, int D>
__device__ __forceinline__ void back_substitute(int k, const T* g, const T* dinv, const T* H, int ldh, T* y) {
  const int lane = threadIdx.x & 31;
  T gv[Q], dv[Q], c[D][Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int r = lane + 32 * q;
    gv[q] = r < k ? g[r] : T(0);
    dv[q] = r < k ? dinv[r] : T(0);
  }
  auto load = [&](T (&to)[D][Q], int top) {  // the entries above the diagonal of columns top, top - 1, ...
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
      for (int q = 0; q < Q; ++q)
        to[d][q] = lane + 32 * q < top - d ? H[(long long)ldh * (top - d) + lane + 32 * q] : T(0);
  };
  load(c, k - 1);
  for (int top = k - 1; top >= 0; top -= D) {
    T next[D][Q];
    load(next, top - D);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int i = top - d;
      if (i < 0) break;
      T gi = gv[0], di = dv[0];
#pragma unroll
      for (int q = 1; q < Q; ++q)
        if (i >> 5 == q) {
          gi = gv[q];
          di = dv[q];
        }
      const T yi = __shfl_sync(0xffffffffu, gi * di, i & 31);
      if (lane == (i & 31)) y[i] = yi;
#pragma unroll
      for (int q = 0; q < Q; ++q) gv[q] -= c[d][q] * yi;
    }
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
      for (int q = 0; q < Q; ++q) c[d][q] = next[d][q];
  }
}

template <typename T>
__device__ void givens_warp(GivensShared<T>* gs, const T* col, T* rot, T* lows, T* cs, T* sn, T* g, T* dinv, T* H,
                            int ldh, T* y, double tol_abs, GState* st) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    givens_sync(kBarColumn);
    if (gs->quit) return;
    const int j = gs->cols - 1;
    if (j == 0 && lane == 0) g[0] = gs->beta;
    __syncwarp();
    // h_i after the rotations before it, low_i, follows low_{i+1} = c_i h_{i+1} - s_i low_i:
    // one dependent operation a step; the products before and the rotated
    // entries after are formed by all lanes at once
    for (int i = lane; i < j; i += 32) lows[i] = cs[i] * col[i + 1];
    __syncwarp();
    T low = col[0];
    for (int i0 = 0; i0 < j; i0 += 32) {
      T mine = T(0);
      const int e = min(32, j - i0);
#pragma unroll 4
      for (int i = 0; i < e; ++i) {
        if (lane == i) mine = low;
        low = fma(-sn[i0 + i], low, lows[i0 + i]);
      }
      const int i = i0 + lane;
      T r = T(0);
      if (lane < e) r = fma(cs[i], mine, sn[i] * col[i + 1]);
      __syncwarp();
      if (lane < e) rot[i] = r;
    }
    __syncwarp();
    const T a = low, b = gs->norm;
    const T r = c_hypot(a, b);
    const T over = (lane == 0 ? a : lane == 1 ? b : T(1)) / r;  // a / r, b / r, 1 / r
    const T s_r = __shfl_sync(0xffffffffu, over, 1), i_r = __shfl_sync(0xffffffffu, over, 2);
    if (lane == 0) {
      T c = T(1), s = T(0);
      if (r > T(0)) { c = over; s = s_r; }
      cs[j] = c;
      sn[j] = s;
      rot[j] = r;
      dinv[j] = r != T(0) ? i_r : T(0);
      const T gj = g[j];
      g[j + 1] = -s * gj;
      g[j] = c * gj;
      const double res = (double)fabs(g[j + 1]);
      gs->done = (gs->last || res <= tol_abs || b == T(0) || !(res == res)) ? 1 : 0;
      if (st) st->res = res;
    }
    __syncwarp();
    T* h = H + (long long)ldh * j;
    for (int i = lane; i <= j; i += 32) h[i] = rot[i];
    const bool done = gs->done != 0;
    if (done) {
      const int k = j + 1;
      constexpr int D = std::is_same<T, double>::value ? 4 : 8;
      __syncwarp();
      if (k <= 64) back_substitute<T, 2, D>(k, g, dinv, H, ldh, y);
      else if (k <= 128) back_substitute<T, 4, D / 2>(k, g, dinv, H, ldh, y);
      else back_substitute<T, kMaxM / 32, D / 4>(k, g, dinv, H, ldh, y);
    }
    __syncwarp();
    givens_arrive(kBarRotated);
    if (done) return;
  }
}

template <typename T, typename TA, typename TV>
__global__ void __launch_bounds__(kCoopThreads + 32, 1) k_gmres_coop(const CoopArgs<T, TA, TV> a) {
  extern __shared__ __align__(32) unsigned char coop_smem[];
  __shared__ GivensShared<T> gs;
  __shared__ int ok;
  __shared__ T newscale;
  __shared__ int over;
  const int tid = threadIdx.x;
  // The outer cycle is over: every CTA leaves. One thread looks, as a CTA whose
  // wait ran out says so in the same place, and the barriers count all threads.
  if (tid == 0) over = a.inner && *(volatile const int*)&a.st->done;
  __syncthreads();
  if (over) return;
  const int n0 = blockIdx.x * a.chunk, n1 = min(a.N, n0 + a.chunk);
  const int nodes = max(0, n1 - n0), rows = 4 * nodes, cap = 4 * a.chunk;
  const long long n = 4ll * a.N;

  // shared memory: w, h of both passes, the Givens arrays (CTA 0), D^-1, B,
  // then the basis and the matrix rows if they fit
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* p = coop_smem + off;
    off += (bytes + 31) / 32 * 32;
    return p;
  };
  T* w = reinterpret_cast<T*>(take(sizeof(T) * cap));
  T* t = a.Bc ? reinterpret_cast<T*>(take(sizeof(T) * cap)) : nullptr;
  T* h1 = reinterpret_cast<T*>(take(sizeof(T) * (a.m + 2)));
  T* h2 = reinterpret_cast<T*>(take(sizeof(T) * (a.m + 2)));
  T* coef = reinterpret_cast<T*>(take(sizeof(T) * (a.m + 2)));
  T* scale = reinterpret_cast<T*>(take(sizeof(T) * (a.m + 2)));  // V_c = scale_c x the stored column
  T* red = reinterpret_cast<T*>(take(sizeof(T) * kCoopRed));
  T *gcol = nullptr, *grot = nullptr, *glow = nullptr, *gcs = nullptr, *gsn = nullptr, *gg = nullptr, *gdi = nullptr;
  if (blockIdx.x == 0) {
    const size_t bytes = sizeof(T) * (a.m + 2);
    gcol = reinterpret_cast<T*>(take(bytes));
    grot = reinterpret_cast<T*>(take(bytes));
    glow = reinterpret_cast<T*>(take(bytes));
    gcs = reinterpret_cast<T*>(take(bytes));
    gsn = reinterpret_cast<T*>(take(bytes));
    gg = reinterpret_cast<T*>(take(bytes));
    gdi = reinterpret_cast<T*>(take(bytes));
  }
  int* brow = reinterpret_cast<int*>(take(sizeof(int) * (a.chunk + 1)));

  if (tid >= kCoopThreads) {
    if (blockIdx.x == 0)
      givens_warp<T>(&gs, gcol, grot, glow, gcs, gsn, gg, gdi, a.H, a.m + 1, a.y, a.tol_abs, a.inner ? nullptr : a.st);
    return;
  }
  CoopSync sync{a.ctl + 2, 0u, &ok, a.limit};
  const T* Dinv = a.Dinv + 16ll * n0;
  const T* Bc = a.Bc ? a.Bc + 16ll * n0 : nullptr;
  auto stage_blocks = [&](const T* src) -> const T* {
    if (off + sizeof(T) * 4 * cap + 32 > (size_t)a.smem_bytes) return src;
    T* d = reinterpret_cast<T*>(take(sizeof(T) * 4 * cap));
    for (int i = tid; i < 16 * nodes; i += kCoopThreads) d[i] = __ldg(src + i);
    return d;
  };
  Dinv = stage_blocks(Dinv);
  if (Bc) Bc = stage_blocks(Bc);
  TV* V = a.V + 4ll * n0;
  long long vld = n;
  bool staged = false;
  const int vs = cap + (std::is_same<T, double>::value ? 1 : 32);  // FP64: lanes on successive columns, no bank conflicts
  if (off + sizeof(TV) * (size_t)vs * (a.m + 1) + 32 <= (size_t)a.smem_bytes) {
    V = reinterpret_cast<TV*>(take(sizeof(TV) * (size_t)vs * (a.m + 1)));
    vld = vs;
    staged = true;
  }
  const int k0 = nodes ? __ldg(a.brow_ptr + n0) : 0;
  const int nblk = nodes ? __ldg(a.brow_ptr + n1) - k0 : 0;
  for (int i = tid; i <= nodes; i += kCoopThreads) brow[i] = nodes ? __ldg(a.brow_ptr + n0 + i) - k0 : 0;
  const TA* A = a.A + 16ll * k0;
  const int* bcol = a.bcol + k0;
  if (off + (sizeof(TA) * 16 + sizeof(int)) * (size_t)nblk + 64 <= (size_t)a.smem_bytes) {
    TA* As = reinterpret_cast<TA*>(take(sizeof(TA) * 16 * (size_t)nblk));
    int* cs = reinterpret_cast<int*>(take(sizeof(int) * (size_t)nblk));
    constexpr int per = 16 / sizeof(TA);
    for (int i = tid; i < nblk * 16 / per; i += kCoopThreads)
      reinterpret_cast<uint4*>(As)[i] = __ldg(reinterpret_cast<const uint4*>(A) + i);
    for (int i = tid; i < nblk; i += kCoopThreads) cs[i] = __ldg(bcol + i);
    A = As;
    bcol = cs;
  }

  // lanes of a node in the products: 4 rows x P groups of blocks
  int P = 1;
  while (P < 8 && 8 * P * max(nodes, 1) <= kCoopThreads) P *= 2;
  int split = 1;
  {
    const int groups = max(1, rows / CoopRows<T>::R), most = std::is_same<T, double>::value ? 2 : 8;
    while (split < most && 2 * split * groups <= kCoopThreads) split *= 2;
  }
  // out[row] = by (A x)[row] for this CTA's rows. In FP32 whole batches of loads
  // are in flight: the remainder of an unrolled loop waits for L2 block by block
  // (40^3 mesh, ms a solve: unrolled by 4 46.7, batches of 4 41.6, of 5 40.6;
  // 16^3 12.1 -> 9.9). In FP64 the pipe takes a masked block's instructions all
  // the same (4^3 3.25 -> 3.64), so the loop there stays exact.
  constexpr int kBatch = 5;
  auto product = [&](const T* x, T* out, T by) {
    const int r = tid & 3, grp = (tid >> 2) & (P - 1), per = kCoopThreads / (4 * P);
    for (int base = 0; base < nodes; base += per) {
      const int q = base + tid / (4 * P);
      T acc = T(0);
      if (q < nodes) {
        const int b1 = brow[q + 1];
        if constexpr (std::is_same<T, double>::value) {
#pragma unroll 4
          for (int k = brow[q] + grp; k < b1; k += P) {
            T a0, a1, a2, a3, x0, x1, x2, x3;
            load_row<T, TA>(A + 16ll * k + 4 * r, a0, a1, a2, a3);
            ld_z4(x + 4ll * bcol[k], x0, x1, x2, x3);
            acc = fma(a0, x0, acc);
            acc = fma(a1, x1, acc);
            acc = fma(a2, x2, acc);
            acc = fma(a3, x3, acc);
          }
        } else {
          for (int k0 = brow[q] + grp; k0 < b1; k0 += kBatch * P) {
            T m[kBatch][4], z[kBatch][4];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
              const int k = min(k0 + u * P, b1 - 1);  // past the end: the last block again, not added
              load_row<T, TA>(A + 16ll * k + 4 * r, m[u][0], m[u][1], m[u][2], m[u][3]);
              ld_z4(x + 4ll * bcol[k], z[u][0], z[u][1], z[u][2], z[u][3]);
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
              if (k0 + u * P < b1)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc = fma(m[u][e], z[u][e], acc);
          }
        }
      }
      for (int o = 4; o < 4 * P; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (q < nodes && grp == 0) out[4 * q + r] = by * acc;
    }
  };
  // dst[node] = M x[node] (4x4 blocks) for the node of the calling quad's row
  auto block4 = [&](const T* M, int row, T x) {
    const int q0 = (tid & 31) & ~3;
    const T x0 = __shfl_sync(0xffffffffu, x, q0), x1 = __shfl_sync(0xffffffffu, x, q0 + 1);
    const T x2 = __shfl_sync(0xffffffffu, x, q0 + 2), x3 = __shfl_sync(0xffffffffu, x, q0 + 3);
    T d0 = T(0), d1 = T(0), d2 = T(0), d3 = T(0);
    if (row < rows) Vec4<T>::load(M + 4ll * row, d0, d1, d2, d3);
    return fma(d0, x0, fma(d1, x1, fma(d2, x2, d3 * x3)));
  };
  const int rows32 = (rows + 31) & ~31, ldp = a.m + 1;

  // The column that the Givens warp has, if any, has to be back before the next
  // arrival at its barrier, and after its last one it waits no more.
  bool handed = false;
  auto collect = [&]() {
    givens_sync(kBarRotated);
    handed = false;
  };
  auto failed = [&]() {
    if (tid == 0) {
      a.st->pad = 1;
      a.st->done = 1;
    }
    if (blockIdx.x == 0) {
      if (handed) collect();
      if (!gs.done) {
        if (tid == 0) gs.quit = 1;
        coop_bar();
        givens_arrive(kBarColumn);
      }
    }
  };

  // ---- start: r, beta, v_0 and z = D^-1 v_0
  const double* src = a.inner ? a.src + (long long)a.st->j * n : a.src;
  double* dst = a.inner ? a.dst + (long long)a.st->j * n : a.dst;
  if (tid == 0) { gs.cols = 0; gs.last = 0; gs.quit = 0; gs.done = 0; }
  T sq = T(0);
  for (int i = tid; i < rows; i += kCoopThreads) {
    const long long gi = 4ll * n0 + i;
    const T v = a.sd ? (T)(src[gi] * a.sd[gi]) : (T)src[gi];
    w[i] = v;
    sq = fma(v, v, sq);
  }
  T norm = T(0), inv = T(0);
  if (!coop_norm(sq, red, a.partn, sync, norm, inv)) { failed(); return; }
  if (tid == 0) gs.beta = norm;
  int cols = 0;
  bool live = norm > T(0);  // zero or NaN: no step, correction 0
  // The column is stored as w s and z1 = D^-1 (w s) with s a power of two near
  // 1 / |w|, which leaves rounding as it is, and V = scale x stored: so z1 goes
  // out with the partial norms, one barrier for both.
  auto publish = [&](int col, T s) {
    for (int i = tid; i < rows32; i += kCoopThreads) {
      T v = T(0);
      if (i < rows) {
        TV* p = V + (long long)col * vld + i;
        stv<TV, T>(p, w[i] * s);
        v = ldv<T, TV>(p);
      }
      const T z = block4(Dinv, i, v);
      if (i < rows) a.z1[4ll * n0 + i] = z;
    }
  };
  if (live) {
    const T s = pow2_rsqrt(norm * norm);
    publish(0, s);
    if (tid == 0) scale[0] = inv / s;
    if (!grid_sync(sync)) { failed(); return; }
  }

  // z2 = z1 + B (x - A z1), the second sweep on this CTA's rows
  auto second_sweep = [&](auto x_of) {
    product(a.z1, t, T(1));
    coop_bar();
    for (int i = tid; i < rows32; i += kCoopThreads) {
      const T d = i < rows ? x_of(i) - t[i] : T(0);
      const T s = block4(Bc, i, d);
      if (i < rows) a.z2[4ll * n0 + i] = a.z1[4ll * n0 + i] + s;
    }
  };

  while (live) {
    const T* z = a.z1;
    if (Bc) {
      second_sweep([&](int i) { return ldv<T, TV>(V + (long long)cols * vld + i); });
      if (!grid_sync(sync)) { failed(); return; }
      z = a.z2;
    }
    product(z, w, scale[cols]);
    coop_bar();
    const int nc = cols + 1;
    // whether the previous column ended the cycle: asked for before the last
    // barrier of the orthogonalization, where the Givens warp has had the
    // longest time to answer
    auto column_done = [&]() {
      if (blockIdx.x == 0 && cols > 0) {
        collect();
        if (tid == 0) {
          a.ctl[0] = (unsigned)gs.done;
          a.ctl[1] = (unsigned)cols;
        }
      }
    };
    coop_dots<T, TV>(w, V, vld, rows, nc, true, staged, red, a.part1, ldp);
    if (!a.two_pass) column_done();
    if (!grid_sync(sync)) { failed(); return; }
    if (!a.two_pass && cols > 0 && __ldcg(a.ctl)) break;
    coop_totals(a.part1, ldp, nc + 1, nc, scale, red, h1, coef);
    const T before = h1[nc];
    T sq = coop_update<T, TV>(w, V, vld, rows, nc, coef, split, staged);
    const T* hs = h1;  // the projection that the norm estimate takes off
    bool second = false;
    if (a.two_pass) {
      coop_bar();
      coop_dots<T, TV>(w, V, vld, rows, nc, true, staged, red, a.part2, ldp);
      column_done();
      if (!grid_sync(sync)) { failed(); return; }
      if (cols > 0 && __ldcg(a.ctl)) break;
      coop_totals(a.part2, ldp, nc + 1, nc, scale, red, h2, coef);
      second = h2[nc] < T(0.5) * before;
      if (second) sq = coop_update<T, TV>(w, V, vld, rows, nc, coef, split, staged);
      hs = h2;
    }
    if (tid < 32) {  // |w|^2 = |w before|^2 - |h|^2, enough for the storage scale
      T e = T(0);
      if (!a.two_pass || second)
        for (int c = tid; c < nc; c += 32) e = fma(hs[c], hs[c], e);
      e = warp_sum(e);
      if (tid == 0) newscale = pow2_rsqrt(fmax(hs[nc] - e, T(1e-4) * hs[nc]));
    }
    coop_bar();
    T s = newscale;
    if (cols + 1 < a.m) publish(cols + 1, s);
    if (!coop_norm(sq, red, a.partn, sync, norm, inv)) { failed(); return; }
    ++cols;
    live = norm > T(0) && cols < a.m;
    if (blockIdx.x == 0) {
      for (int c = tid; c < nc; c += kCoopThreads) gcol[c] = second ? h1[c] + h2[c] : h1[c];
      if (tid == 0) {
        gs.cols = cols;
        gs.norm = norm;
        gs.last = live ? 0 : 1;
      }
      givens_arrive(kBarColumn);
      handed = true;
    }
    if (!live) {
      if (blockIdx.x == 0) {
        collect();
        if (tid == 0) a.ctl[1] = (unsigned)cols;
      }
      if (!grid_sync(sync)) { failed(); return; }
      break;
    }
    // Where the estimate lost its digits the column is stored again: it is to have
    // unit norm at least, as a normalized one has, or binary16 would hold its small
    // entries to fewer bits.
    if (norm * s > T(8) || norm * s < T(1)) {
      s = pow2_rsqrt(norm * norm);
      publish(cols, s);
      if (!grid_sync(sync)) { failed(); return; }
    }
    if (tid == 0) scale[cols] = inv / s;
    coop_bar();
  }

  // ---- correction: x = V y, u = M^-1 x
  const int k = cols ? (int)__ldcg(a.ctl + 1) : 0;
  for (int c = tid; c < k; c += kCoopThreads) h1[c] = -scale[c] * __ldcg(a.y + c);
  for (int i = tid; i < rows; i += kCoopThreads) w[i] = T(0);
  coop_bar();
  coop_update<T, TV>(w, V, vld, rows, k, h1, split, staged);
  coop_bar();
  for (int i = tid; i < rows32; i += kCoopThreads) {
    const T u = block4(Dinv, i, i < rows ? w[i] : T(0));
    if (i < rows) {
      if (Bc) {
        a.z1[4ll * n0 + i] = u;
      } else {
        const long long gi = 4ll * n0 + i;
        if (a.inner) dst[gi] = (double)u * a.sd[gi];
        else dst[gi] += (double)u;
      }
    }
  }
  if (Bc) {
    if (!grid_sync(sync)) { failed(); return; }
    second_sweep([&](int i) { return w[i]; });
    coop_bar();
    for (int i = tid; i < rows; i += kCoopThreads) {
      const long long gi = 4ll * n0 + i;
      const T u = a.z2[gi];
      if (a.inner) dst[gi] = (double)u * a.sd[gi];
      else dst[gi] += (double)u;
    }
  }
  if (!a.inner && blockIdx.x == 0 && tid == 0) {
    a.st->j = k;
    a.st->done = 1;
  }
  if (blockIdx.x == 0 && cols == 0) {  // no column was handed over: release the Givens warp
    if (tid == 0) gs.quit = 1;
    coop_bar();
    givens_arrive(kBarColumn);
  }
  if (tid == 0) {  // the last CTA to leave clears the count for the next cycle
    __threadfence();
    if (atomicAdd(a.ctl + 3, 1u) == gridDim.x - 1) {
      a.ctl[2] = 0u;
      a.ctl[3] = 0u;
    }
  }
}
