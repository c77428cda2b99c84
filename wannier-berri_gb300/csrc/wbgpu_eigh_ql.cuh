// ---------------------------------------------------------------------------------------
// 2. Implicit QL eigenvalues of the real symmetric tridiagonal (d, e), thread per matrix.
// d and e of thread t live in shared memory at [i * blockDim + t] (conflict-free, no
// local-memory traffic).
// ---------------------------------------------------------------------------------------
// a b, a b + c d and a b - c of the QL rotations.  FP64 names its roundings, so that the two kernels below
// give the same bits whatever the compiler would fuse in each.
template <typename R> WBG_D R ql_mul(R a, R b) { return a * b; }
template <typename R> WBG_D R ql_lin(R a, R b, R c, R d) { return a * b + c * d; }
template <typename R> WBG_D R ql_mulsub(R a, R b, R c) { return a * b - c; }
template <> WBG_D double ql_mul(double a, double b) { return __dmul_rn(a, b); }
template <> WBG_D double ql_lin(double a, double b, double c, double d) { return __fma_rn(a, b, __dmul_rn(c, d)); }
template <> WBG_D double ql_mulsub(double a, double b, double c) { return __fma_rn(a, b, -c); }

// FP64: r = sqrt(q) and 1 / r from one reciprocal square root and a Newton step for r, instead of a square root
// and a division after it on the chain of every rotation: 13 824 matrices of n = 32 2.29 -> 2.09 ms, 512 of n = 8
// 0.139 -> 0.129 ms; errors against 30 digits a tenth smaller.
WBG_D void ql_root(double q, double& r, double& rinv) {
  rinv = rsqrt(q);
  const double t = __dmul_rn(q, rinv);
  r = q == 0.0 ? 0.0 : __fma_rn(__fma_rn(-t, t, q), __dmul_rn(0.5, rinv), t);
}

template <typename R>
__global__ void eigh_ql(const R* __restrict__ dIn, const R* __restrict__ eIn, int n, int nk, double* __restrict__ Eout,
                        int* __restrict__ errflag) {
  typedef Arith<R> A;
  extern __shared__ unsigned char smq[];
  const int B = blockDim.x;
  const long long k = (long long)blockIdx.x * B + threadIdx.x;
  if (k >= nk) return;
  R* ds = reinterpret_cast<R*>(smq) + threadIdx.x;
  R* es = ds + (size_t)n * B;
  auto d = [&](int i) -> R& { return ds[i * B]; };
  auto e = [&](int i) -> R& { return es[i * B]; };
  const R zero = A::from(0.0), one = A::from(1.0), two = A::from(2.0), eps = A::eps();
  for (int i = 0; i < n; ++i) { d(i) = dIn[k * n + i]; e(i) = eIn[k * n + i]; }
  e(n - 1) = zero;
  bool ok = true;
  for (int l = 0; l < n; ++l) {
    int iter = 0, m;
    do {
      for (m = l; m < n - 1; ++m) {
        const R dd = fabs(d(m)) + fabs(d(m + 1));
        if (fabs(e(m)) <= eps * dd) break;
      }
      if (m != l) {
        if (iter++ >= 60) { ok = false; break; }
        R g = (d(l + 1) - d(l)) / (two * e(l));
        R r = sqrt(fma(g, g, one));
        g = d(m) - d(l) + e(l) / (g + copysign(r, g));
        R s = one, c = one, p = zero;
        bool underflow = false;
        for (int i = m - 1; i >= l; --i) {
          const R f = ql_mul(s, e(i));
          const R b = ql_mul(c, e(i));
          // Givens rotation: one sqrt and one reciprocal (f, g are O(|T|): no overflow concern)
          R rinv;
          if constexpr (std::is_same<R, double>::value) ql_root(ql_lin(f, f, g, g), r, rinv);
          else r = sqrt(fma(f, f, ql_mul(g, g)));
          e(i + 1) = r;
          if (r == zero) { d(i + 1) = d(i + 1) - p; e(m) = zero; underflow = true; break; }
          if constexpr (!std::is_same<R, double>::value) rinv = one / r;
          s = ql_mul(f, rinv);
          c = ql_mul(g, rinv);
          g = d(i + 1) - p;
          r = ql_lin(d(i) - g, s, two * c, b);
          p = ql_mul(s, r);
          d(i + 1) = g + p;
          g = ql_mulsub(c, r, b);
        }
        if (underflow) continue;
        d(l) = d(l) - p;
        e(l) = g;
        e(m) = zero;
      }
    } while (m != l);
    if (!ok) break;
  }
  if (!ok) atomicOr(errflag, WBG_FLAG_QL_NOCONV);
  // ascending insertion sort
  for (int i = 1; i < n; ++i) {
    const R x = d(i);
    int j = i - 1;
    while (j >= 0 && d(j) > x) { d(j + 1) = d(j); --j; }
    d(j + 1) = x;
  }
  for (int i = 0; i < n; ++i) Eout[k * n + i] = A::to(d(i));
}

// One implicit QL sweep of the block [l, m] by a single thread: the rotations are a serial chain, and d and e
// are read and written in its program order.
template <typename R>
WBG_D void ql_sweep(R* ds, R* es, int l, int m) {
  typedef Arith<R> A;
  auto d = [&](int i) -> R& { return ds[i]; };
  auto e = [&](int i) -> R& { return es[i]; };
  const R zero = A::from(0.0), one = A::from(1.0), two = A::from(2.0);
  R g = (d(l + 1) - d(l)) / (two * e(l));
  R r = sqrt(fma(g, g, one));
  g = d(m) - d(l) + e(l) / (g + copysign(r, g));
  R s = one, c = one, p = zero;
  // d(i + 1) is the value read as d(i) one step before; the next step's e and d are read ahead of
  // this one's stores, off the chain of dependent operations
  R di1 = d(m), en = e(m - 1), dn = d(m - 1);
  for (int i = m - 1; i >= l; --i) {
    const R ei = en, di = dn;
    if (i > l) {
      en = e(i - 1);
      dn = d(i - 1);
    }
    const R f = ql_mul(s, ei);
    const R b = ql_mul(c, ei);
    // Givens rotation: one sqrt and one reciprocal (f, g are O(|T|): no overflow concern)
    R rinv;
    if constexpr (std::is_same<R, double>::value) ql_root(ql_lin(f, f, g, g), r, rinv);
    else r = sqrt(fma(f, f, ql_mul(g, g)));
    e(i + 1) = r;
    if (r == zero) {  // f^2 + g^2 underflowed: the matrix splits here
      d(i + 1) = di1 - p;
      e(m) = zero;
      return;
    }
    if constexpr (!std::is_same<R, double>::value) rinv = one / r;
    s = ql_mul(f, rinv);
    c = ql_mul(g, rinv);
    g = di1 - p;
    r = ql_lin(di - g, s, two * c, b);
    p = ql_mul(s, r);
    d(i + 1) = g + p;
    g = ql_mulsub(c, r, b);
    di1 = di;
  }
  d(l) = d(l) - p;
  e(l) = g;
  e(m) = zero;
}

// The same sweep with a warp per matrix, for batches too small to fill the SMs otherwise: lane 0 runs the (serial)
// rotations, the search for a negligible off-diagonal element and the final sort, a third of the time in one
// thread, are shared by the lanes.  d and e are written by lane 0 only, between two warp barriers: no lane
// reads them meanwhile.  The same comparisons and rotations as eigh_ql: the same bits.  512 double-float matrices of
// 96 x 96: 4.7 (a thread each) -> 3.7 ms.
constexpr int QW_WARPS = 4;  // matrices per block
template <typename R>
__global__ void __launch_bounds__(32 * QW_WARPS)
    eigh_ql_warp(const R* __restrict__ dIn, const R* __restrict__ eIn, int n, int nk, double* __restrict__ Eout,
                 int* __restrict__ errflag) {
  typedef Arith<R> A;
  extern __shared__ unsigned char smq[];
  const int lane = threadIdx.x & 31;
  const long long k = (long long)blockIdx.x * QW_WARPS + (threadIdx.x >> 5);
  if (k >= nk) return;
  R* ds = reinterpret_cast<R*>(smq) + (size_t)(threadIdx.x >> 5) * 2 * n;
  R* es = ds + n;
  const R zero = A::from(0.0), eps = A::eps();
  for (int i = lane; i < n; i += 32) {
    ds[i] = dIn[k * n + i];
    es[i] = i < n - 1 ? eIn[k * n + i] : zero;
  }
  bool ok = true;
  for (int l = 0; l < n; ++l) {
    int iter = 0, m;
    do {
      __syncwarp();  // the sweep's (at first: the loads') stores are visible
      m = n - 1;
      for (int base = l; base < n - 1; base += 32) {  // the first m >= l with |e(m)| negligible
        const int i = base + lane;
        const bool hit = i < n - 1 && fabs(es[i]) <= eps * (fabs(ds[i]) + fabs(ds[i + 1]));
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (hits) {
          m = base + __ffs(hits) - 1;
          break;
        }
      }
      __syncwarp();  // every lane has read what the sweep is about to change
      if (m != l) {
        if (iter++ >= 60) { ok = false; break; }
        if (lane == 0) ql_sweep<R>(ds, es, l, m);
      }
    } while (m != l);
    if (!ok) break;
  }
  if (!ok && lane == 0) atomicOr(errflag, WBG_FLAG_QL_NOCONV);
  __syncwarp();
  bool nan = false;
  for (int i = lane; i < n; i += 32) nan |= ds[i] != ds[i];
  nan = __any_sync(0xffffffffu, nan);  // not ordered: left as it is
  for (int i = lane; i < n; i += 32) {
    const R x = ds[i];
    int r = 0;
    for (int j = 0; j < n; ++j) r += ds[j] < x || (ds[j] == x && j < i);
    Eout[k * n + (nan ? i : r)] = A::to(x);
  }
}

