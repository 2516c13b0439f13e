// Treecode evaluation on the plan's source tree (the reference's MultipoleSolver::calcA / calcB(current,
// point), FMM/FMMGPU/multipole_solver.cpp:686-700, descending with QuadratureOctreeNode::calcA / calcRot,
// quadrature_octree.cpp:171-258).
//
// For each query point x the source tree is walked from its root: a box whose half-diagonal r and
// distance d from its centre satisfy 4 r^2 < d^2 contributes through its multipole (the reference's
// acceptance test), any other box through its children; a leaf that fails the test is summed directly
// (by default) or contributes nothing (FMM_TREECODE_REFERENCE_NEAR, as the reference, which loses
// 10-19 % near its sources). With box-size scaled multipoles (a box of side h keeps M~_l = M_l / h^l)
// a box's potential at x is (1/h) sum_k M~_k I_k(u), u = (x - c) / h. B = curl A is again a sum of irregular
// harmonics, one degree higher: with T_l^m the complex irregular harmonic of fmm_common.cuh,
//   d/dz T_l^m = -T_{l+1}^m,   (d/dx + i d/dy) T_l^m = -T_{l+1}^{m+1},   (d/dx - i d/dy) T_l^m = T_{l+1}^{m-1} (m >= 1),
// so a box's curl expansion is a fixed combination of at most four multipole coefficients per entry, made
// once per box and group of points, and a point costs one harmonic recurrence. Or B comes by central differences of
// A with step 1e-3 as the reference does (FMM_TREECODE_FD_CURL).
//
// A block takes W query points (1..32, neighbours in Morton order where W > 1) and walks the tree for all of them
// at once: a box on the block's stack carries the mask of the points that reached it. A batch of boxes is tested a
// thread per box; the points a box is far from meet it as one entry of the far list, a leaf's others as
// one of the near list, and the rest go to its children. The far entries are dealt out to the warps (curl
// expansion into shared memory, then a point per lane, 32 / W lanes sharing a point's orders), the near leaves'
// sources are staged in shared memory in FP64 and split over all lanes. The sums meet in a fixed order.
//
// What bounds it: the FP64 near sum (~30 FP64 instructions a pair) and the FP32 far evaluation (~18 instructions a
// harmonic). With a thread per point walking alone, evaluating value and gradient by dual numbers and reading
// its boxes' multipoles itself, the few points near the sources kept their warps for the whole call. Measured, that ->
// this, 262,144 sources, p = 10, FP32: leaves of 1000, 65,536 points 23.4 -> 2.65 ms, 1,000 points 16.6 -> 0.45 ms, one
// point 0.39 -> 0.03 ms; leaves of 100, 65,536 points 11.5 -> 3.9 ms; FP64, leaves of 1000, 65,536 points 40 -> 3.5 ms.
#include <cub/cub.cuh>

#include "fmm_internal.cuh"

namespace fmm {

namespace {

constexpr int TC_NT = 256, TC_WARPS = TC_NT / 32;
// Boxes on a block's stack. A batch pops at most (room left - 200) / 7 boxes, at least one, and pushes at most 8 for
// each; one box at a time adds at most 7 a level (147 in 21 levels) before the stack is shorter again.
constexpr int TC_STACK = 1536;
constexpr int TC_SRC = 256;     // sources staged at a time

// The curl (entries of degree <= p + 1) of the expansion sum_k M_k I_k as terms of the multipole row [3][Lp], with
// the real-basis factors (-1)^l sqrt2 folded in: entry [k'][component], at most four terms.
template <class T>
struct CurlTerm
{
   int idx[4];
   T c[4];
};

template <class T>
std::vector<CurlTerm<T>> curlTerms(int p, int Lp)
{
   const int q = p + 1;
   std::vector<CurlTerm<T>> tab(size_t(nharm(q)) * 4);
   // A = sum a_lm Re T_l^m + b_lm Im T_l^m; a (im = 0) or b (im = 1) of degree l, order m as a multiple of a coefficient
   auto put = [&](CurlTerm<T>& e, int& n, double f, int comp, int l, int m, int im) {
      if(l < 0 || m > l || m < 0 || (im && m == 0)) return;
      e.idx[n] = comp * Lp + hidx(l, im ? -m : m);
      e.c[n] = T(f * ((l & 1) ? -1.0 : 1.0) * (m ? 1.4142135623730950488 : 1.0));
      n++;
   };
   for(int k = 0; k < nharm(q); k++)
   {
      int l = 0;
      while((l + 1) * (l + 1) <= k) l++;
      const int mu = abs(k - l * l - l), im = k - l * l - l < 0;   // entry: Re (im = 0) or Im T_l^mu
      // its coefficient in d/dx_j of component c (times f), from degree l - 1
      auto deriv = [&](CurlTerm<T>& e, int& n, double f, int c, int j) {
         if(j == 2) put(e, n, -f, c, l - 1, mu, im);
         else if(j == 0)
         {
            if(mu >= 1) put(e, n, mu == 1 && !im ? -f : -0.5 * f, c, l - 1, mu - 1, im);
            put(e, n, 0.5 * f, c, l - 1, mu + 1, im);
         }
         else if(im)
         {
            put(e, n, mu == 1 ? -f : -0.5 * f, c, l - 1, mu - 1, 0);
            put(e, n, -0.5 * f, c, l - 1, mu + 1, 0);
         }
         else
         {
            put(e, n, 0.5 * f, c, l - 1, mu - 1, 1);
            put(e, n, 0.5 * f, c, l - 1, mu + 1, 1);
         }
      };
      for(int c = 0; c < 3; c++)
      {
         CurlTerm<T>& e = tab[4 * size_t(k) + c];
         e = CurlTerm<T>{};
         int n = 0;
         deriv(e, n, 1.0, (c + 2) % 3, (c + 1) % 3);
         deriv(e, n, -1.0, (c + 1) % 3, (c + 2) % 3);
      }
      tab[4 * size_t(k) + 3] = CurlTerm<T>{};
   }
   return tab;
}

// Walks T_l^m(ux, uy, uz) for m = g, g + G, .. <= q and l = m..q and calls f(k of (l, m), k of (l, -m), re, im, l). The
// recurrence's integer factors are kept as running sums in T.
template <class T, class F>
__device__ __forceinline__ void visitIrregular(int q, int g, int G, T ux, T uy, T uz, F&& f)
{
   const T r2 = ux * ux + uy * uy + uz * uz;
   const T i2 = T(1) / r2;
   const T zi = uz * i2, xi = ux * i2, yi = uy * i2;
   T dre = sqrt(i2), dim = T(0);   // T_m^m
   int m = 0;
   T odd = T(1);                   // 2 m + 1
   auto diag = [&]() {
      const T nre = odd * (xi * dre - yi * dim), nim = odd * (xi * dim + yi * dre);
      dre = nre; dim = nim;
      odd += T(2);
      m++;
   };
   while(m < g && m < q) diag();
   if(m < g) return;
   while(true)
   {
      T are = dre, aim = dim, bre = T(0), bim = T(0);
      T c1 = odd, c2 = T(0);       // 2 l + 1, l^2 - m^2
      for(int l = m, k0 = m * m + 2 * m, k1 = m * m;; l++)
      {
         f(k0, k1, are, aim, l);
         if(l == q) break;
         const T az = c1 * zi, bz = c2 * i2;
         const T cre = az * are - bz * bre, cim = az * aim - bz * bim;
         bre = are; bim = aim; are = cre; aim = cim;
         c2 += c1;
         c1 += T(2);
         k0 += 2 * l + 2; k1 += 2 * l + 2;
      }
      if(m + G > q) break;
      for(int j = 0; j < G; j++) diag();
   }
}

template <class T>
struct TcSmem
{
   int stackN, stackM, farN, farM, nearN, nearM, pts, src, warp0, perWarp, total;
   __host__ __device__ TcSmem(int p, bool wantA)
   {
      int b = 0;
      auto take = [&](int bytes) { const int at = b; b += (bytes + 15) & ~15; return at; };
      stackN = take(4 * TC_STACK);
      stackM = take(4 * TC_STACK);
      farN = take(4 * TC_NT);
      farM = take(4 * TC_NT);
      nearN = take(4 * TC_NT);
      nearM = take(4 * TC_NT);
      pts = take(8 * (3 * 32 + 2));
      src = take(8 * 8 * TC_SRC);            // also the warps' sums at the end: [TC_WARPS][32][6]
      warp0 = b;
      // per warp: the curl expansion [(p + 2)^2][4] and the potential's [(p + 1)^2][4]
      perWarp = int(sizeof(T)) * (4 * nharm(p + 1) + (wantA ? 4 * nharm(p) : 0));
      perWarp = (perWarp + 31) & ~31;
      b = (b + 31) & ~31;
      warp0 = b;
      total = warp0 + TC_WARPS * perWarp;
   }
};

template <class T>
__global__ void __launch_bounds__(TC_NT) kTreecode(Tree t, const RootBox* __restrict__ rootp, int p, int Lp,
                                                   const T* __restrict__ mult, const CurlTerm<T>* __restrict__ curl,
                                                   const typename Vec4<T>::type* __restrict__ spos,
                                                   const typename Vec4<T>::type* __restrict__ sq, const T* __restrict__ pts,
                                                   const int* __restrict__ order, int64_t m, int W, int flags, T scaleB,
                                                   T scaleA, int want, int bem, T* __restrict__ outB, T* __restrict__ outA)
{
   typedef typename Vec4<T>::type V4;
   typedef cub::BlockScan<int, TC_NT> Scan;
   extern __shared__ __align__(32) unsigned char smraw[];
   __shared__ typename Scan::TempStorage scanTmp;
   const bool refNear = flags & 1, fdCurl = flags & 2;
   const bool wantB = want & 1, wantA = (want & 2) != 0, curlB = wantB && !fdCurl, potA = wantA || fdCurl;
   const TcSmem<T> sm(p, potA);
   int* stackN = reinterpret_cast<int*>(smraw + sm.stackN);
   unsigned* stackM = reinterpret_cast<unsigned*>(smraw + sm.stackM);
   int* farN = reinterpret_cast<int*>(smraw + sm.farN);
   unsigned* farM = reinterpret_cast<unsigned*>(smraw + sm.farM);
   int* nearN = reinterpret_cast<int*>(smraw + sm.nearN);
   unsigned* nearM = reinterpret_cast<unsigned*>(smraw + sm.nearM);
   double* P = reinterpret_cast<double*>(smraw + sm.pts);       // [3][32], then the root's side and its inverse
   double* S = reinterpret_cast<double*>(smraw + sm.src);       // [TC_SRC][8]
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   V4* Cs = reinterpret_cast<V4*>(smraw + sm.warp0 + warp * sm.perWarp);
   V4* As = Cs + nharm(p + 1);
   const int64_t q0 = int64_t(blockIdx.x) * W;
   const int nq = int(min(int64_t(W), m - q0));
   const int G = 32 / W, j = lane % W, g = lane / W;
   if(tid < 32)
   {
      const int64_t i = q0 + min(tid, nq - 1);
      const int64_t src = order ? order[i] : i;
      for(int d = 0; d < 3; d++) P[32 * d + tid] = double(pts[3 * src + d]);
   }
   const RootBox rb = rootp[0];
   if(tid == 0) { P[96] = 2.0 * rb.H; P[97] = 1.0 / (2.0 * rb.H); }
   const unsigned all = nq == 32 ? 0xffffffffu : (1u << nq) - 1u;
   int count = 0;
   for(int r = t.levelStart[0]; r < t.levelStart[1]; r++)
   {
      if(tid == 0) { stackN[count] = r; stackM[count] = all; }
      count++;
   }
   __syncthreads();
   const double x = P[j], y = P[32 + j], z = P[64 + j];
   double A[3] = {0, 0, 0}, B[3] = {0, 0, 0};
   const T eps = T(1e-3);   // the reference's math::eps for the central differences
   // (the side is the root's times a power of two, so neither it nor its inverse takes a division)
   auto power2 = [](int e) { return __longlong_as_double((long long)(1023 + e) << 52); };
   auto centre = [&](int node, double& h, double& cx, double& cy, double& cz) {
      const int level = t.level[node];
      h = P[96] * power2(-level);
      cx = rb.center[0] - rb.H + (double(t.ix[node]) + 0.5) * h;
      cy = rb.center[1] - rb.H + (double(t.iy[node]) + 0.5) * h;
      cz = rb.center[2] - rb.H + (double(t.iz[node]) + 0.5) * h;
      return level;
   };
   while(count > 0)
   {
      // a batch from the top of the stack, a thread per box
      const int batch = min(count, max(1, min(TC_NT, (TC_STACK - 200 - count) / 7)));
      const int base = count - batch;
      int node = -1, c0 = 0, nc = 0;
      unsigned farMask = 0, rest = 0;
      if(tid < batch)
      {
         node = stackN[base + tid];
         const unsigned mask = stackM[base + tid];
         if(t.s1[node] > t.s0[node])
         {
            double h, cx, cy, cz;
            centre(node, h, cx, cy, cz);
            const double r2 = 3.0 * 0.25 * h * h;   // half-diagonal^2: three half-widths h / 2
            for(unsigned left = mask; left; left &= left - 1)
            {
               const int i = __ffs(left) - 1;
               const double dx = P[i] - cx, dy = P[32 + i] - cy, dz = P[64 + i] - cz;
               const double d2 = dx * dx + dy * dy + dz * dz;
               if(4.0 * r2 < d2) farMask |= 1u << i;
            }
            rest = mask & ~farMask;
            if(rest) { nc = t.nchild[node]; c0 = t.child0[node]; }
         }
      }
      const bool near = rest && nc == 0 && !refNear;
      // far entries, near leaves and children in one scan: 9, 9 and 12 bits
      int at, total;
      Scan(scanTmp).ExclusiveSum((farMask ? 1 : 0) | (near ? 1 << 9 : 0) | (rest ? nc << 18 : 0), at, total);
      if(farMask) { farN[at & 511] = node; farM[at & 511] = farMask; }
      if(near) { nearN[at >> 9 & 511] = node; nearM[at >> 9 & 511] = rest; }
      if(rest)
         for(int c = 0; c < nc; c++)
         {
            stackN[base + (at >> 18) + c] = c0 + c;
            stackM[base + (at >> 18) + c] = rest;
         }
      count = base + (total >> 18);
      const int nFar = total & 511, nNear = total >> 9 & 511;
      __syncthreads();
      // far boxes, one a warp at a time
      for(int e = warp; e < nFar; e += TC_WARPS)
      {
         const int box = farN[e];
         const bool on = farM[e] >> j & 1;
         const T* row = mult + int64_t(box) * 3 * Lp;
         __syncwarp();
         if(curlB)
            for(int i = lane; i < 4 * nharm(p + 1); i += 32)
            {
               const CurlTerm<T> ce = curl[i];
               reinterpret_cast<T*>(Cs)[i] =
                  ce.c[0] * row[ce.idx[0]] + ce.c[1] * row[ce.idx[1]] + ce.c[2] * row[ce.idx[2]] + ce.c[3] * row[ce.idx[3]];
            }
         if(potA)
            for(int i = lane; i < 4 * nharm(p); i += 32)
            {
               const int k = i >> 2, c = i & 3;
               int l = int(sqrtf(float(k) + 0.5f));
               const T f = ((l & 1) ? T(-1) : T(1)) * (k != l * l + l ? T(1.4142135623730950488) : T(1));
               reinterpret_cast<T*>(As)[i] = c < 3 ? f * row[c * Lp + k] : T(0);
            }
         __syncwarp();
         double h, cx, cy, cz;
         const double ih = P[97] * power2(centre(box, h, cx, cy, cz));
         const double dx = x - cx, dy = y - cy, dz = z - cz;
         T b[3] = {T(0), T(0), T(0)}, a[3] = {T(0), T(0), T(0)};
         // (for m = 0 the imaginary part is zero, so its k1 = k0 term adds nothing)
         auto addA = [&](int k0, int k1, T re, T im) {
            const V4 u = As[k0], v = As[k1];
            a[0] += u.x * re + v.x * im; a[1] += u.y * re + v.y * im; a[2] += u.z * re + v.z * im;
         };
         const T ux = T(dx * ih), uy = T(dy * ih), uz = T(dz * ih);
         if(curlB)
            visitIrregular<T>(p + 1, g, G, ux, uy, uz, [&](int k0, int k1, T re, T im, int l) {
               const V4 u = Cs[k0], v = Cs[k1];
               b[0] += u.x * re + v.x * im; b[1] += u.y * re + v.y * im; b[2] += u.z * re + v.z * im;
               if(wantA && l <= p) addA(k0, k1, re, im);
            });
         else if(wantA)
            visitIrregular<T>(p, g, G, ux, uy, uz, [&](int k0, int k1, T re, T im, int) { addA(k0, k1, re, im); });
         if(on)
            for(int c = 0; c < 3; c++) { B[c] += double(b[c]) * ih * ih; A[c] += double(a[c]) * ih; }
         if(wantB && fdCurl)
         {
            // central differences of this box's A: dA_c / dx_j
            double D[3][3];
            for(int d = 0; d < 3; d++)
            {
               T s[2][3];
               for(int side = 0; side < 2; side++)
               {
                  const double sh = (side ? -1.0 : 1.0) * (double(eps) * ih);
                  for(int c = 0; c < 3; c++) a[c] = T(0);
                  visitIrregular<T>(p, g, G, T(dx * ih + (d == 0 ? sh : 0.0)), T(dy * ih + (d == 1 ? sh : 0.0)),
                                    T(dz * ih + (d == 2 ? sh : 0.0)), [&](int k0, int k1, T re, T im, int) { addA(k0, k1, re, im); });
                  for(int c = 0; c < 3; c++) s[side][c] = a[c];
               }
               for(int c = 0; c < 3; c++)
               {
                  // the lanes of a point hold different orders: their sums first, then the difference
                  for(int off = W; off < 32; off <<= 1)
                  {
                     s[0][c] += __shfl_xor_sync(0xffffffffu, s[0][c], off);
                     s[1][c] += __shfl_xor_sync(0xffffffffu, s[1][c], off);
                  }
                  D[c][d] = double(s[0][c] - s[1][c]) * ih / (2.0 * double(eps));
               }
            }
            if(on && g == 0)
            {
               B[0] += D[2][1] - D[1][2];
               B[1] += D[0][2] - D[2][0];
               B[2] += D[1][0] - D[0][1];
            }
         }
      }
      // near leaves: their sources staged in FP64, every lane takes every (8 G)-th one
      for(int e = 0; e < nNear; e++)
      {
         const int leaf = nearN[e];
         const bool on = nearM[e] >> j & 1;
         const int s1 = t.s1[leaf];
         for(int sb = t.s0[leaf]; sb < s1; sb += TC_SRC)
         {
            const int n = min(TC_SRC, s1 - sb);
            __syncthreads();
            bool odd = false;
            if(tid < n)
            {
               const V4 a = spos[sb + tid], b = sq[sb + tid];
               double* d = S + 8 * tid;
               d[0] = double(a.x); d[1] = double(a.y); d[2] = double(a.z); d[3] = double(b.w);
               d[4] = double(b.x); d[5] = double(b.y); d[6] = double(b.z);
               odd = !isfinite(b.x + b.y + b.z + b.w);   // (or a sum out of range, which only costs)
            }
            // Coincident points are skipped: by a factor of zero, but in a tile with a strength that is no number the sum
            // goes from one such point to the next.
            const bool skip = __syncthreads_or(odd);
            for(int i = warp * G + g; on && i < n; i += TC_WARPS * G)
            {
               int stop = n;
               if(skip)
                  for(stop = i; stop < n; stop += TC_WARPS * G)
                  {
                     const double ex = x - S[8 * stop], ey = y - S[8 * stop + 1], ez = z - S[8 * stop + 2];
                     if(ex * ex + ey * ey + ez * ez == 0.0) break;
                  }
#pragma unroll 2
               for(; i < stop; i += TC_WARPS * G)
               {
                  const double* d = S + 8 * i;
                  const double2 d0 = *reinterpret_cast<const double2*>(d), d1 = *reinterpret_cast<const double2*>(d + 2);
                  const double2 d2 = *reinterpret_cast<const double2*>(d + 4);
                  const double sx = d2.x, sy = d2.y, sz = d[6];
                  const double ex = x - d0.x, ey = y - d0.y, ez = z - d1.x;
                  const double e2 = ex * ex + ey * ey + ez * ez;
                  const double ri = e2 > 0.0 ? rsqrt(e2) : 0.0, ri3 = ri * ri * ri;   // (coincident points skipped)
                  if(bem)
                  {
                     // the BEM kernel sigma d / |d|^3 + d x s / |d|^3 with d = q - x = -(ex, ey, ez) (fmm_bem.cu)
                     const double sg = d1.y;
                     A[0] -= (sg * ex + (ey * sz - ez * sy)) * ri3;
                     A[1] -= (sg * ey + (ez * sx - ex * sz)) * ri3;
                     A[2] -= (sg * ez + (ex * sy - ey * sx)) * ri3;
                     continue;
                  }
                  if(wantB)
                  {
                     B[0] += (sy * ez - sz * ey) * ri3;
                     B[1] += (sz * ex - sx * ez) * ri3;
                     B[2] += (sx * ey - sy * ex) * ri3;
                  }
                  if(wantA) { A[0] += sx * ri; A[1] += sy * ri; A[2] += sz * ri; }
               }
            }
         }
      }
      __syncthreads();
   }
   // the lanes of a point, then the warps
   double s[6] = {B[0], B[1], B[2], A[0], A[1], A[2]};
   for(int off = W; off < 32; off <<= 1)
      for(int c = 0; c < 6; c++) s[c] += __shfl_xor_sync(0xffffffffu, s[c], off);
   for(int c = 0; c < 6; c++) S[(warp * 6 + c) * 32 + lane] = s[c];
   __syncthreads();
   if(tid < nq)
   {
      for(int w = 1; w < TC_WARPS; w++)
         for(int c = 0; c < 6; c++) s[c] += S[(w * 6 + c) * 32 + tid];
      const int64_t q = order ? order[q0 + tid] : q0 + tid;
      for(int c = 0; c < 3; c++)
      {
         if(wantB) outB[3 * q + c] = T(s[c] * double(scaleB));
         if(wantA) outA[3 * q + c] = T(s[3 + c] * double(scaleA));
      }
   }
}

// Morton keys of the query points, 10 bits an axis over twice the root cube (points outside clamp to its faces).
template <class T>
__global__ void kQueryKeys(const T* __restrict__ pts, int64_t m, const RootBox* __restrict__ rootp, unsigned* keys, int* idx)
{
   const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
   if(i >= m) return;
   const RootBox rb = rootp[0];
   unsigned key = 0;
   for(int d = 0; d < 3; d++)
   {
      const double u = (double(pts[3 * i + d]) - rb.center[d]) / (4.0 * rb.H) + 0.5;
      const unsigned v = unsigned(fmin(1023.0, fmax(0.0, u * 1024.0)));
      for(int b = 0; b < 10; b++) key |= (v >> b & 1u) << (3 * b + d);
   }
   keys[i] = key;
   idx[i] = int(i);
}

}  // namespace

template <class T>
fmm_status treecodeT(Plan& P, double current, int want, const void* pts, int64_t m, void* outB, void* outA, int flags,
                     cudaStream_t st)
{
   typedef typename Vec4<T>::type V4;
   if(m == 0) return FMM_OK;
   // A (and, for BEM sources, the BEM integral) times current / (4 pi), as MultipoleSolver::calcA
   // (multipole_solver.cpp:686-692) scales both
   const T scaleB = T(REF_MU0 / (4 * REF_PI) * current), scaleA = T(1.0 / (4 * REF_PI) * current);
   if(P.tcCurlOrder != P.p)
   {
      const std::vector<CurlTerm<T>> tab = curlTerms<T>(P.p, P.Lp);
      const size_t bytes = tab.size() * sizeof(CurlTerm<T>);
      FMM_TRY(P.tcCurl.reserve(bytes));
      P.tcCurlHost.resize(bytes);
      std::copy_n(reinterpret_cast<const unsigned char*>(tab.data()), bytes, P.tcCurlHost.data());
      FMM_CUDA(cudaMemcpyAsync(P.tcCurl.ptr, P.tcCurlHost.data(), bytes, cudaMemcpyHostToDevice, st));
      P.tcCurlOrder = P.p;
   }
   // Points a block (W): neighbours want mostly the same boxes, and a far box is prepared once for the block's points; few
   // points, or points sparse among the boxes, walk alone (then a point has 256 threads). W grows while the block's
   // points meet up to 32 times as many boxes and 592 blocks (2 points), 296 (4, 8), 1184 (16, 32) remain, or while every box has
   // a point of its own and 296 blocks remain (few large leaves: the near sums fill the lanes). Measured over orders
   // 1-16, leaves of 10-1000, 300-300,000 points, both precisions: on average within 3 % of the best W (the second
   // condition alone 35 %), e.g. 65,536 points, 65,536 sources in leaves of 30, p = 10, FP32: W = 8 4.6 ms, 32 3.1.
   const int64_t nodes = std::max<int64_t>(1, P.tree.nNodes);
   int W = 1;
   auto grow = [&](int w) {
      const int64_t blocks = m / w;
      return (w <= 32 * m / nodes && blocks >= (w == 2 ? 592 : (w <= 8 ? 296 : 1184))) || (w <= m / nodes && blocks >= 296);
   };
   while(W < 32 && grow(2 * W)) W *= 2;
   const int* order = nullptr;
   size_t tmp = 0;
   unsigned* k = nullptr;
   if(W > 1)
   {
      // keys, sorted keys, indexes, sorted indexes, then the sort's scratch; without room for them every point walks alone
      cub::DeviceRadixSort::SortPairs(nullptr, tmp, k, k, (int*)nullptr, (int*)nullptr, int(m), 0, 30, st);
      if(!P.roomFor(P.tcSort, sizeof(unsigned) * 4 * size_t(m)) || !P.roomFor(P.cubTmp, tmp)) W = 1;
   }
   if(W > 1)
   {
      k = (unsigned*)P.tcSort.ptr;
      int* ix = (int*)(k + 2 * m);
      kQueryKeys<T><<<int((m + 255) / 256), 256, 0, st>>>((const T*)pts, m, P.root, k, ix);
      FMM_TRY(launched(P, "kQueryKeys", st));
      tmp = P.cubTmp.bytes;
      FMM_CUDA(cub::DeviceRadixSort::SortPairs(P.cubTmp.ptr, tmp, k, k + m, ix, ix + m, int(m), 0, 30, st));
      order = ix + m;
   }
   const TcSmem<T> sm(P.p, (want & 2) || (flags & 2));
   FMM_CUDA(allowShared(kTreecode<T>));
   kTreecode<T><<<unsigned((m + W - 1) / W), TC_NT, sm.total, st>>>(
      P.tree, P.root, P.p, P.Lp, (const T*)P.mult.ptr, (const CurlTerm<T>*)P.tcCurl.ptr, (const V4*)P.sPos.ptr,
      (const V4*)P.sQ.ptr, (const T*)pts, order, m, W, flags, scaleB, scaleA, want, P.bem ? 1 : 0, (T*)outB, (T*)outA);
   FMM_TRY(launched(P, "kTreecode", st));
   return FMM_OK;
}

template fmm_status treecodeT<float>(Plan&, double, int, const void*, int64_t, void*, void*, int, cudaStream_t);
template fmm_status treecodeT<double>(Plan&, double, int, const void*, int64_t, void*, void*, int, cudaStream_t);

}  // namespace fmm
