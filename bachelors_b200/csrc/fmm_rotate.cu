// Translations through the z axis (M2L, M2M and L2L on the CUDA cores, FP32 and FP64).
//
// A translation by a vector v is a rotation that takes v to the z axis, a translation along z, and the
// rotation back. Rotations keep the degree l and, split into an azimuth turn (2 x 2 blocks on (m, -m)) and
// a turn about y (which keeps the cosine and the sine coefficients apart), cost sum (l+1)^2 + l^2
// multiply-adds; a z translation keeps m and costs as much. One box pair and component takes about 3 x (2/3) p^3
// multiply-adds instead of the (p+1)^4 of the dense operator (p = 12: 4.4k instead of 28.6k, p = 16: 9.8k
// instead of 83.5k), with the same truncation: degrees are kept by the rotations, so m2l_truncate's limit on
// l + lambda keeps the same terms. (The method is White and Head-Gordon's, J. Chem. Phys. 105, 5061, 1996.)
//
// With D the rotation of the solid harmonics, R(rot x) = D R(x), N = diag sqrt((l-m)! (l+m)!) and D^ = N D N^-1,
// which is orthogonal:
//   M2L  L_out = D^T Tz D M                  Tz[l, lambda] = (-1)^(l+m) (l+lambda)! / r^(l+lambda+1)
//   M2M  M_out = N^-1 D^^T N  Tz  D M        Tz[l, lambda] = (-r)^(l-lambda) / (l-lambda)!
//   L2L  L_out = D^T  Tz  N D^ N^-1 L        Tz[l, lambda] = r^(lambda-l) / (lambda-l)!
// with the box-size scaling's powers of two in the last factor. Tz depends on l and lambda only through their
// sum or difference, so an operator is two sets of rotation blocks and a vector of 2p + 1 numbers.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include <cub/cub.cuh>

#include "fmm_internal.cuh"

namespace fmm {

namespace rot {

// ------------------------------------------------------------------------------ operator tables
// Coefficients in two orders. Degree-major: (l, cos m = 0..l) and (l, sin m = 1..l) blocks, each contiguous in
// m. Order-major: (m, cos l = m..p) and (m, sin) blocks, contiguous in l. Blocks of n coefficients are products with
// n x n matrices, taken four outputs at a time: a group's table is [k < n rounded up to even][4], 16-byte loads in
// the kernel (the odd n's last row is zero; it meets the next block's first coefficient).
//
// One operator's table in T: the forward groups, the backward groups (both: for n = 1..p+1 the ceil(n/4) groups of
// the cosine block of degree n - 1, then of the sine block of degree n), H[s][4] for s = 0..2p+1 (four
// neighbouring entries of the z translation's vector: s, s+1, .. for M2L, s, s-1, .. otherwise; no translation has a
// term at the entry an odd block's last row adds, but its coefficient is the next block's, see kRotTranslate) and
// (cos, sin)(m phi).
__host__ __device__ constexpr int grp(int n) { return (n + 3) >> 2; }
__host__ __device__ constexpr int even(int n) { return (n + 1) & ~1; }
__host__ __device__ constexpr int groupBase(int n)   // elements before the groups of blocks of n
{
   int s = 0;
   for(int i = 1; i < n; i++) s += 8 * grp(i) * even(i);
   return s;
}
struct Blob
{
   int half, hOff, zOff, size;
   Blob() = default;
   __host__ __device__ Blob(int p)
   {
      half = groupBase(p + 1) + 4 * grp(p + 1) * even(p + 1);
      hOff = 2 * half;
      zOff = hOff + 4 * (2 * p + 2);
      size = zOff + ((2 * (p + 1) + 3) & ~3);
   }
};
// element offset of group g of the cosine (degree n - 1) or sine (degree n) block
__host__ __device__ inline int groupOff(int n, int sine, int g) { return groupBase(n) + (sine * grp(n) + g) * 4 * even(n); }

// positions in the two orders; order-major blocks are padded to an even number of coefficients
__host__ __device__ inline int degPos(int l, int m) { return l * l + (m >= 0 ? m : l - m); }   // cos 0..l, then sin 1..l
__host__ __device__ inline int ordBase(int p, int m)   // first position of order |m|'s cosine (m < 0: sine) block
{
   const int a = m < 0 ? -m : m;
   int s = 0;
   for(int b = 0; b < a; b++) s += (b ? 2 : 1) * even(p + 1 - b);
   return s + (m < 0 ? even(p + 1 - a) : 0);
}
__host__ __device__ inline int ordPos(int p, int l, int m) { return ordBase(p, m) + l - (m < 0 ? -m : m); }
__host__ __device__ inline int ordSize(int p) { return ordBase(p, p + 1); }

// D^ of the quarter turn about x that takes e_z to e_y, degree blocks [2l+1][2l+1] up to degree p one after the other, by
// integrating products of the orthonormal harmonics over the sphere (Gauss-Legendre x trapezoid, exact for
// these degrees): R_i(Q x) against R_j(x). A product of two harmonics of one degree is even, so the points below the
// equator are left out. Made once for an order (p = 16 1.3 ms, p = 8 0.1).
static int quarterOff(int l) { return l * (4 * l * l - 1) / 3; }   // sum of (2i+1)^2, i < l
static const std::vector<double>& quarterTurn(int p)
{
   static std::vector<double> tabs[MAXORDER + 1];
   static std::once_flag once[MAXORDER + 1];
   std::vector<double>& tab = tabs[p];
   std::call_once(once[p], [&] {
      const int L = nharm(p), nz = p + 1, na = 2 * p + 2;
      // Gauss-Legendre nodes by Newton's method on P_nz
      std::vector<double> zs(nz), ws(nz);
      for(int i = 0; i < nz; i++)
      {
         double x = std::cos(M_PI * (i + 0.75) / (nz + 0.5)), dp = 1;
         for(int it = 0; it < 100; it++)
         {
            double a = 1, b = x;
            for(int n = 2; n <= nz; n++) { const double c = ((2 * n - 1) * x * b - (n - 1) * a) / n; a = b; b = c; }
            dp = nz * (x * b - a) / (x * x - 1);
            const double dx = b / dp;
            x -= dx;
            if(std::fabs(dx) < 1e-16) break;
         }
         zs[i] = x;
         ws[i] = 2 / ((1 - x * x) * dp * dp);
      }
      // orthogonal-basis regular harmonics N R at a unit vector, by the recurrence of visitRegular
      std::vector<double> norm(L);
      for(int l = 0; l <= p; l++)
         for(int m = -l; m <= l; m++)
         {
            double f = 1;
            for(int k = 2; k <= l - std::abs(m); k++) f *= k;
            double g = 1;
            for(int k = 2; k <= l + std::abs(m); k++) g *= k;
            norm[hidx(l, m)] = std::sqrt(f) * std::sqrt(g);
         }
      auto harm = [&](double x, double y, double z, double* out) {
         double dre = 1, dim = 0;
         for(int m = 0; m <= p; m++)
         {
            if(m > 0)
            {
               const double s = 1.0 / (2 * m), nre = (dre * x - dim * y) * s, nim = (dre * y + dim * x) * s;
               dre = nre; dim = nim;
            }
            double are = dre, aim = dim, bre = 0, bim = 0;
            for(int l = m; l <= p; l++)
            {
               const double s = (l & 1) ? -1 : 1, q = std::sqrt(2.0);
               if(m == 0) out[hidx(l, 0)] = s * are * norm[hidx(l, 0)];
               else
               {
                  out[hidx(l, m)] = s * q * are * norm[hidx(l, m)];
                  out[hidx(l, -m)] = s * q * aim * norm[hidx(l, m)];
               }
               const double inv = 1.0 / ((l - m + 1.0) * (l + m + 1.0));
               const double cre = ((2 * l + 1) * z * are - bre) * inv, cim = ((2 * l + 1) * z * aim - bim) * inv;
               bre = are; bim = aim; are = cre; aim = cim;
            }
         }
      };
      tab.assign(quarterOff(p + 1), 0.0);
      std::vector<double> a(L), b(L);
      for(int i = 0; i < (nz + 1) / 2; i++)   // (the nodes come in decreasing order; an odd number's middle one is the equator)
         for(int j = 0; j < na; j++)
         {
            const double s = std::sqrt(1 - zs[i] * zs[i]), f = 2 * M_PI * j / na;
            const double x = s * std::cos(f), y = s * std::sin(f), z = zs[i];
            harm(x, y, z, b.data());
            harm(x, z, -y, a.data());   // Q x: e_z -> e_y, e_y -> -e_z
            const double w = ws[i] / (2 * i + 1 == nz ? 2 : 1) / na;
            for(int l = 0; l <= p; l++)
               for(int u = 0; u <= 2 * l; u++)
                  for(int v = 0; v <= 2 * l; v++)
                     tab[quarterOff(l) + u * (2 * l + 1) + v] += w * (2 * l + 1) * a[l * l + u] * b[l * l + v];
         }
   });
   return tab;
}

// One block per operator: 0..7 M2M octants, 8..15 L2L octants, 16.. the M2L offset slots.
// The turn about y by -theta is Q Z(-theta) Q^T with Q the quarter turn and Z the azimuth turn.
template <class T>
__global__ void kBuildRotations(int p, int cut, const double* __restrict__ quarter, T* __restrict__ out)
{
   constexpr int M1 = MAXORDER + 1;
   const Blob B(p);
   const int op = blockIdx.x;
   const int kind = op < 8 ? 0 : (op < 16 ? 1 : 2);
   double v[3];
   if(kind == 2)
   {
      const int o = d_m2lOffset[op - 16];
      v[0] = o % 7 - 3; v[1] = (o / 7) % 7 - 3; v[2] = o / 49 - 3;
   }
   else
      for(int d = 0; d < 3; d++) v[d] = (((op >> d) & 1) - 0.5) * (kind == 0 ? 0.5 : -0.5);
   const double r = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
   const double theta = acos(fmin(1.0, fmax(-1.0, v[2] / r)));
   const double phi = v[0] == 0 && v[1] == 0 ? 0.0 : atan2(v[1], v[0]);
   __shared__ double norm[M1 * M1];   // N of (l, m), m >= 0, at l M1 + m
   __shared__ double ct[M1], sn[M1];
   for(int e = threadIdx.x; e < M1 * M1; e += blockDim.x)
   {
      const int l = e / M1, m = e % M1;
      double f = 1, g = 1;
      for(int k = 2; k <= l - m; k++) f *= k;
      for(int k = 2; k <= l + m; k++) g *= k;
      norm[e] = sqrt(f) * sqrt(g);
   }
   if(threadIdx.x <= p) { ct[threadIdx.x] = cos(threadIdx.x * theta); sn[threadIdx.x] = sin(threadIdx.x * theta); }
   T* o = out + int64_t(op) * B.size;
   for(int e = threadIdx.x; e < B.size; e += blockDim.x) o[e] = T(0);
   __syncthreads();
   for(int l = 0; l <= p; l++)
   {
      const int w = 2 * l + 1;
      int q0 = 0;
      for(int i = 0; i < l; i++) q0 += (2 * i + 1) * (2 * i + 1);
      const double* Q = quarter + q0;
      // entries (a, b) of D^'s cosine (a, b = 0..l) and sine (a, b = 1..l) blocks
      for(int e = threadIdx.x; e < (l + 1) * (l + 1) + l * l; e += blockDim.x)
      {
         const int sine = e < (l + 1) * (l + 1) ? 0 : 1;
         const int f = sine ? e - (l + 1) * (l + 1) : e, n = sine ? l : l + 1;
         const int i = f / n, j = f % n;
         const int ma = i + sine, mb = j + sine;
         const int a = sine ? -ma : ma, b = sine ? -mb : mb;
         // sum over c of Q[a, c] (Z(-theta) Q^T)[c, b], Z on (m, -m): x_m' = cos x_m + sin x_-m, x_-m' = cos x_-m - sin x_m
         double s = Q[(l + a) * w + l] * Q[(l + b) * w + l];
         for(int m = 1; m <= l; m++)
         {
            const double ap = Q[(l + a) * w + l + m], an = Q[(l + a) * w + l - m];
            const double bp = Q[(l + b) * w + l + m], bn = Q[(l + b) * w + l - m];
            s += ap * (ct[m] * bp + sn[m] * bn) + an * (ct[m] * bn - sn[m] * bp);
         }
         const double nab = norm[l * M1 + mb] / norm[l * M1 + ma];   // N_b / N_a
         // forward, output a from input b: D = N^-1 D^ N for multipoles, N D^ N^-1 for locals
         o[groupOff(n, sine, i >> 2) + 4 * j + (i & 3)] = T(kind == 1 ? s / nab : s * nab);
         // backward, output b from input a: D^T with M2L's sign, N^-1 D^^T N (M2M), N D^^T N^-1 = D^T (L2L)
         double t = kind == 0 ? s / nab : s * nab;
         if(kind == 2) { if((l + ma) & 1) t = -t; }
         else t = ldexp(t, kind == 0 ? -l : -(l + 1));
         o[B.half + groupOff(n, sine, j >> 2) + 4 * i + (j & 3)] = T(t);
      }
   }
   // the z translation's vector: entry l + lambda (M2L), lambda - l + p (M2M, L2L)
   for(int e = threadIdx.x; e < 4 * (2 * p + 2); e += blockDim.x)
   {
      const int i = kind == 2 ? (e >> 2) + (e & 3) : (e >> 2) - (e & 3);
      double s = 0;
      if(kind == 2)
      {
         if(i <= cut)
         {
            s = 1 / r;
            for(int k = 1; k <= i; k++) s *= k / r;
         }
      }
      else
      {
         const int d = kind == 0 ? p - i : i - p;
         if(i >= 0 && d > 0)   // (d = 0, the coefficient itself, is added exactly: see kRotTranslate)
         {
            s = 1;
            for(int k = 1; k <= d; k++) s *= (kind == 0 ? -2 * r : r) / k;   // M2M: 2^-lambda = 2^-l 2^(l - lambda)
         }
      }
      o[B.hOff + e] = T(s);
   }
   for(int m = threadIdx.x; m <= p; m += blockDim.x)
   {
      o[B.zOff + 2 * m] = T(cos(m * phi));
      o[B.zOff + 2 * m + 1] = T(sin(m * phi));
   }
}

// ------------------------------------------------------------------------------ kernel
// A task of one quarter-warp: four outputs of a block of K coefficients.
struct __align__(16) Task
{
   unsigned short in, K, op, pad;   // first input position, inputs (even), operator offset / 4
   unsigned short out[4];           // output positions (0xFFFF: none)
};
constexpr int MAXTASK = 88;         // quarter-warp tasks of one step (p = 16)
constexpr int MAXTILE = 100;        // target boxes of an M2L or M2M tile at most
struct TaskTable
{
   int n[3];                        // warp tasks (four tasks of equal K) of each step
   Task t[3][MAXTASK];
};

// The tasks of the three steps, longest first.
static void makeTasks(int p, int mode, TaskTable& tab)
{
   const Blob B(p);
   for(int step = 0; step < 3; step++)
   {
      std::vector<Task> v;
      for(int K = even(p + 1); K >= 2; K -= 2)
      {
         for(int n = K; n >= K - 1; n--)
         {
            if(n > p + 1) continue;
            for(int g = 0; g < grp(n); g++)
               for(int sine = 0; sine < 2; sine++)
               {
                  // the two blocks of n coefficients: cosine of degree n - 1 and sine of degree n (rotations),
                  // cosine and sine of order p + 1 - n (z translation)
                  if(sine && n == p + 1) continue;
                  Task t{};
                  t.K = (unsigned short)K;
                  const int l = n - 1 + sine, m = p + 1 - n;
                  if(step == 1)
                  {
                     t.in = (unsigned short)ordBase(p, sine ? -m : m);
                     t.op = (unsigned short)((B.hOff + 4 * (mode == 0 ? 2 * m + 4 * g : p - 4 * g)) / 4);
                  }
                  else
                  {
                     t.in = (unsigned short)degPos(l, sine ? -1 : 0);
                     t.op = (unsigned short)(((step == 2 ? B.half : 0) + groupOff(n, sine, g)) / 4);
                  }
                  for(int q = 0; q < 4; q++)
                  {
                     const int i = 4 * g + q;
                     int pos = 0xFFFF;
                     if(i < n)
                     {
                        const int mm = sine ? -(i + 1) : i;
                        pos = step == 1 ? degPos(m + i, sine ? -m : m) : step == 0 ? ordPos(p, l, mm) : degPos(l, mm);
                     }
                     t.out[q] = (unsigned short)pos;
                  }
                  v.push_back(t);
               }
         }
         while(v.size() & 3)
         {
            Task t = v.back();
            for(int q = 0; q < 4; q++) t.out[q] = 0xFFFF;
            v.push_back(t);
         }
      }
      tab.n[step] = int(v.size() / 4);
      std::copy(v.begin(), v.end(), tab.t[step]);
   }
}

// A lane's rows of one coefficient: R groups of V (FP32: 4, as two packed pairs; FP64: 2) consecutive rows, 8 V
// rows apart.
template <class T> constexpr int laneRows() { return 16 / int(sizeof(T)); }
template <class T> constexpr int chunkPairs() { return sizeof(T) == 4 ? 20 : 10; }
template <class T> constexpr int rowStride() { return 3 * chunkPairs<T>(); }   // 60 (FP64: 30): a multiple of V, 2-way conflicts transposed

template <class T, int R> struct Rows;
template <int R> struct Rows<float, R>
{
   f2p v[2 * R];
   __device__ __forceinline__ void zero()
   {
#pragma unroll
      for(int i = 0; i < 2 * R; i++) v[i] = 0;
   }
   __device__ __forceinline__ void load(const float* p)
   {
#pragma unroll
      for(int g = 0; g < R; g++)
      {
         const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(p + 32 * g);
         v[2 * g] = x.x; v[2 * g + 1] = x.y;
      }
   }
   // (the last group's last lane has no rows)
   __device__ __forceinline__ void store(float* p, bool all) const
   {
#pragma unroll
      for(int g = 0; g < R; g++)
         if(g == 0 || all) *reinterpret_cast<ulonglong2*>(p + 32 * g) = make_ulonglong2(v[2 * g], v[2 * g + 1]);
   }
   __device__ __forceinline__ void mac(float a, const Rows& x)
   {
      const f2p aa = pk2(a, a);
#pragma unroll
      for(int i = 0; i < 2 * R; i++) v[i] = fma2(aa, x.v[i], v[i]);
   }
   // a x + b y
   __device__ __forceinline__ void comb(float a, const Rows& x, float b, const Rows& y)
   {
      const f2p aa = pk2(a, a), bb = pk2(b, b);
#pragma unroll
      for(int i = 0; i < 2 * R; i++) v[i] = fma2(bb, y.v[i], mul2(aa, x.v[i]));
   }
};
template <int R> struct Rows<double, R>
{
   double v[2 * R];
   __device__ __forceinline__ void zero()
   {
#pragma unroll
      for(int i = 0; i < 2 * R; i++) v[i] = 0;
   }
   __device__ __forceinline__ void load(const double* p)
   {
#pragma unroll
      for(int g = 0; g < R; g++)
      {
         const double2 x = *reinterpret_cast<const double2*>(p + 16 * g);
         v[2 * g] = x.x; v[2 * g + 1] = x.y;
      }
   }
   __device__ __forceinline__ void store(double* p, bool all) const
   {
#pragma unroll
      for(int g = 0; g < R; g++)
         if(g == 0 || all) *reinterpret_cast<double2*>(p + 16 * g) = make_double2(v[2 * g], v[2 * g + 1]);
   }
   __device__ __forceinline__ void mac(double a, const Rows& x)
   {
#pragma unroll
      for(int i = 0; i < 2 * R; i++) v[i] = fma(a, x.v[i], v[i]);
   }
   __device__ __forceinline__ void comb(double a, const Rows& x, double b, const Rows& y)
   {
#pragma unroll
      for(int i = 0; i < 2 * R; i++) v[i] = fma(b, y.v[i], a * x.v[i]);
   }
};
__device__ __forceinline__ void loadOps(const float* p, float (&e)[4])
{
   const float4 x = *reinterpret_cast<const float4*>(p);
   e[0] = x.x; e[1] = x.y; e[2] = x.z; e[3] = x.w;
}
__device__ __forceinline__ void loadOps(const double* p, double (&e)[4])
{
   const double2 x = reinterpret_cast<const double2*>(p)[0], y = reinterpret_cast<const double2*>(p)[1];
   e[0] = x.x; e[1] = x.y; e[2] = y.x; e[3] = y.y;
}

// One step: the quarter-warps of every warp task compute four outputs of a block for their 8 lanes' rows.
template <class T, int R>
__device__ __forceinline__ void runStep(const Task* tasks, int nTasks, int warp, int NW, int lane, const T* ops, const T* Win, T* Wout)
{
   constexpr int RS = rowStride<T>();
   const int hl = lane & 7, quarter = lane >> 3;
   const bool all = hl < 7;
   Win += laneRows<T>() * hl;
   Wout += laneRows<T>() * hl;
   // dealt out back and forth: the tasks come longest first
   for(int t0 = 0, t = warp; t0 < nTasks; t0 += NW, t = t0 + ((t0 / NW) & 1 ? NW - 1 - warp : warp))
   {
      if(t >= nTasks) continue;
      const uint4 d = *reinterpret_cast<const uint4*>(tasks + 4 * t + quarter);
      const T* x = Win + int(d.x & 0xFFFF) * RS;
      const T* o = ops + 4 * int(d.y & 0xFFFF);
      const int K = int(d.x >> 16);
      Rows<T, R> acc[4];
#pragma unroll
      for(int q = 0; q < 4; q++) acc[q].zero();
#pragma unroll 2
      for(int k = 0; k < K; k += 2)
      {
#pragma unroll
         for(int h = 0; h < 2; h++)
         {
            Rows<T, R> xv;
            xv.load(x + (k + h) * RS);
            T e[4];
            loadOps(o + 4 * (k + h), e);
#pragma unroll
            for(int q = 0; q < 4; q++) acc[q].mac(e[q], xv);
         }
      }
      const int out[4] = {int(d.z & 0xFFFF), int(d.z >> 16), int(d.w & 0xFFFF), int(d.w >> 16)};
#pragma unroll
      for(int q = 0; q < 4; q++)
         if(out[q] != 0xFFFF) acc[q].store(Wout + out[q] * RS, all);
   }
}

// Azimuth turn of the pairs (l, m), (l, -m) in degree-major order, in place: into the z frame (back = false) or out of it.
template <class T, int R>
__device__ __forceinline__ void turn(const unsigned* pairs, int nPairs, int warp, int NW, int lane, const T* Z, T* W, bool back)
{
   constexpr int RS = rowStride<T>();
   const int hl = lane & 7, quarter = lane >> 3;
   W += laneRows<T>() * hl;
   for(int i = 4 * warp + quarter; i < nPairs; i += 4 * NW)
   {
      const unsigned d = pairs[i];
      T* wc = W + int(d & 0x3FF) * RS;
      T* ws = W + int(d >> 10 & 0x3FF) * RS;
      const T c = Z[2 * (d >> 20)], s0 = Z[2 * (d >> 20) + 1], s = back ? -s0 : s0;
      Rows<T, R> x, y, u, v;
      x.load(wc);
      y.load(ws);
      u.comb(c, x, s, y);
      v.comb(c, y, -s, x);
      u.store(wc, hl < 7);
      v.store(ws, hl < 7);
   }
}

constexpr int MAXT = MAXTILE;
constexpr int MAXTL = 160;    // of an L2L tile
template <class T>
struct Smem   // byte offsets in the block's dynamic shared memory
{
   int w0, w1, tasks, pairs, pos, pads, total;
   __host__ __device__ explicit Smem(int p)
   {
      constexpr int RS = rowStride<T>();
      const int L = nharm(p);
      int b = int(sizeof(T)) * Blob(p).size;
      // one more position after the last block, and the last lane's reads past the last row
      w0 = b; b += int(sizeof(T)) * (L + 2) * RS;
      w1 = b; b += int(sizeof(T)) * (ordSize(p) + 1) * RS;
      b = (b + 15) & ~15;
      tasks = b; b += 3 * MAXTASK * int(sizeof(Task));
      pairs = b; b += 4 * (p * (p + 1) / 2);
      pads = b; b += 4 * (MAXORDER + 2);
      pos = b; b += 2 * (padded(L));
      total = (b + 15) & ~15;
   }
};

__device__ __forceinline__ void cpAsync16(void* dst, const void* src)
{
   const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
   asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// one element, asynchronously
__device__ __forceinline__ void cpAsyncElem(float* dst, const float* src)
{
   const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
   asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncElem(double* dst, const double* src)
{
   const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
   asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

// 2^-l of coefficient k's degree l (half that with `less`): a coefficient's own term in the M2M (L2L)
template <class T>
__device__ __forceinline__ T boxScale(int k, bool less)
{
   const int e = int(sqrtf(float(k) + 0.5f)) + (less ? 1 : 0);
   if constexpr(sizeof(T) == 4) return __int_as_float((127 - e) << 23);
   else return __longlong_as_double((1023ll - e) << 52);
}

struct L2LSegR { int start[9]; };

// The M2L operators of every tile, in order: their number, the operators and the work of those before each; over the tiles
// the work before each tile (start[tiles]: all); and how the tiles are dealt out to the blocks: the first `whole` in turn,
// then of the rest block b takes the work from share[b] to share[b + 1].
struct TileOps
{
   int tiles, whole, blocks;
   int* n;
   int* before;          // [tile][316]
   unsigned short* op;   // [tile][316]
   int64_t* start;       // [tiles + 1]
   int64_t* share;       // [blocks + 1]
};

// The work of an operator with n pairs in the tile, in twentieths of a full chunk: its chunks, a half chunk being one with a
// single group of rows, and its table. (The weights that served best of those around a fit to the blocks' times; they
// move the M2L by a few per cent.)
template <class T>
__device__ __forceinline__ int opWork(int n, int p)
{
   constexpr int CH = chunkPairs<T>();
   const int rest = n % CH, half = sizeof(T) == 8 ? 13 : (p <= 6 ? 12 : 9);
   return n == 0 ? 0 : 1 + 20 * (n / CH) + (3 * rest > 8 * laneRows<T>() ? 20 : (rest ? half : 0));
}

// start[] from the tiles' work at start[tile + 1], then the shares, by one block: every block's whole tiles and share together
// are to make the same work (a block whose whole tiles alone are more than that gets an empty share).
constexpr int TILEOPS_NT = 320;
__device__ void tileStarts(const TileOps ops)
{
   typedef cub::BlockScan<int64_t, TILEOPS_NT> Scan;
   __shared__ typename Scan::TempStorage tmp;
   const int tid = threadIdx.x;
   int64_t base = 0;
   if(tid == 0) ops.start[0] = 0;
   for(int t0 = 0; t0 < ops.tiles; t0 += TILEOPS_NT)
   {
      const int t = t0 + tid;
      int64_t v = t < ops.tiles ? __ldcg(ops.start + t + 1) : 0, sum;
      Scan(tmp).InclusiveSum(v, v, sum);
      if(t < ops.tiles) ops.start[t + 1] = base + v;
      base += sum;
      __syncthreads();
   }
   if(ops.whole == 0)
   {
      for(int b = tid; b <= ops.blocks; b += TILEOPS_NT) ops.share[b] = base / ops.blocks * b + base % ops.blocks * b / ops.blocks;
      return;
   }
   // what each block still needs, summed up to each block's end; then scaled to the work that is left
   const int64_t first = ops.start[ops.whole];
   int64_t needed = 0;
   for(int b0 = 0; b0 < ops.blocks; b0 += TILEOPS_NT)
   {
      const int b = b0 + tid;
      int64_t need = 0, sum;
      if(b < ops.blocks)
      {
         need = base / ops.blocks + 1;
         for(int t = b; t < ops.whole; t += ops.blocks) need -= ops.start[t + 1] - ops.start[t];
         if(need < 0) need = 0;
      }
      Scan(tmp).InclusiveSum(need, need, sum);
      if(b < ops.blocks) ops.share[b + 1] = needed + need;
      needed += sum;
      __syncthreads();
   }
   for(int b = tid; b < ops.blocks; b += TILEOPS_NT)
      ops.share[b + 1] = b + 1 == ops.blocks ? base : first + int64_t(double(base - first) * double(ops.share[b + 1]) / double(max(needed, int64_t(1))));
   if(tid == 0) ops.share[0] = first;
}

// TileOps of one tile a block, a thread per operator; the last block to end (done counts them, from 0 back to 0) makes the starts.
template <class T>
__global__ void __launch_bounds__(TILEOPS_NT) kTileOps(const int* __restrict__ targets, int nTargets, const int* __restrict__ vtab,
                                                       int TT, int p, const TileOps ops, unsigned* done)
{
   __shared__ int node[MAXTILE];
   __shared__ int warpSum[TILEOPS_NT / 32][2];
   const int tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   const int nTile = min(TT, nTargets - tile * TT);
   for(int t = tid; t < nTile; t += TILEOPS_NT) node[t] = targets[tile * TT + t];
   __syncthreads();
   int n = 0;
   if(tid < 316)
      for(int t0 = 0; t0 < nTile; t0 += 50)
      {
         int v[50];   // loads that are all in flight: a small tree waits for this one block
#pragma unroll
         for(int u = 0; u < 50; u++) v[u] = t0 + u < nTile ? vtab[int64_t(node[t0 + u]) * 316 + tid] : -1;
#pragma unroll
         for(int u = 0; u < 50; u++) n += v[u] >= 0;
      }
   // positions in the list and the work before, over the block
   const int mine = opWork<T>(n, p);
   const unsigned bits = __ballot_sync(0xffffffffu, n > 0);
   int incl = mine;
   for(int d = 1; d < 32; d <<= 1)
   {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if(lane >= d) incl += v;
   }
   if(lane == 31) { warpSum[warp][0] = __popc(bits); warpSum[warp][1] = incl; }
   __syncthreads();
   int at = __popc(bits & ((1u << lane) - 1)), work = incl - mine, count = 0, all = 0;
   for(int w = 0; w < TILEOPS_NT / 32; w++)
   {
      if(w < warp) { at += warpSum[w][0]; work += warpSum[w][1]; }
      count += warpSum[w][0];
      all += warpSum[w][1];
   }
   if(n > 0)
   {
      ops.op[int64_t(tile) * 316 + at] = (unsigned short)tid;
      ops.before[int64_t(tile) * 316 + at] = work;
   }
   __shared__ bool last;
   if(tid == 0)
   {
      ops.n[tile] = count;
      ops.start[tile + 1] = all;
      __threadfence();
      last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;
      __threadfence();
   }
   __syncthreads();
   if(last) tileStarts(ops);
}

// the tile that holds unit w of the work (w < start[tiles])
__device__ __forceinline__ int tileOf(const int64_t* __restrict__ start, int tiles, int64_t w)
{
   int a = 0, b = tiles;   // start[a] <= w < start[b]
   while(b - a > 1)
   {
      const int m = (a + b) >> 1;
      if(start[m] <= w) a = m;
      else b = m;
   }
   return a;
}

// Y of the tiles that several blocks share: the slots' sums added in block order. blockIdx.x: the tile, of those behind the
// whole ones; blockIdx.y of gridDim.y: boxes of it. Bound by latency where tiles are few (16 slots' loads in flight).
template <class T>
__global__ void __launch_bounds__(512) kAddParts(const int* __restrict__ targets, int nTargets, int TT, const TileOps ops, int Lp,
                                                 const T* __restrict__ ws, T* __restrict__ Y)
{
   const int tile = ops.whole + blockIdx.x;
   const int64_t a = ops.start[tile], e = ops.start[tile + 1];
   int b0 = 0, b1 = 0;   // the blocks that begin inside the tile
   for(int c = 0; c < ops.blocks; c += blockDim.x)
   {
      const int64_t at = c + int(threadIdx.x) < ops.blocks ? ops.share[c + threadIdx.x] : INT64_MAX;
      b0 += __syncthreads_count(at <= a);
      b1 += __syncthreads_count(at < e);
   }
   if(b0 >= b1) return;
   const int nTile = min(TT, nTargets - tile * TT), n = 3 * Lp;
   for(int t = blockIdx.y; t < nTile; t += gridDim.y)
   {
      T* y = Y + int64_t(targets[tile * TT + t]) * n;
      for(int k = threadIdx.x; k < n; k += blockDim.x)
      {
         T s = y[k];
         for(int b = b0; b < b1; b += 16)
         {
            T v[16];
#pragma unroll
            for(int u = 0; u < 16; u++) v[u] = b + u < b1 ? ws[(int64_t(b + u) * TT + t) * n + k] : T(0);
#pragma unroll
            for(int u = 0; u < 16; u++) s += v[u];
         }
         y[k] = s;
      }
   }
}

// A tile of TT target boxes and its operators, or some of them. For every
// operator with a source for some box of the tile the pairs are taken a chunk at a time, 20 (FP64: 10) pairs of 3
// vectors, none of them empty: their source rows are gathered into shared memory [coefficient][vector],
// turned about z in place, then the three steps (rotation, z translation, rotation back) alternate between two
// such buffers, and the result is turned back and added to the targets' rows in global memory (one block owns
// them; they stay in L2). A lane holds 8 (FP64: 4) vectors, a quarter-warp four outputs: per input
// coefficient and lane three (FP64: four) 16-byte shared loads for 32 (16) multiply-adds, FP32 ones in
// packed pairs. 16 warps an SM, in one to four blocks.
// What bounds it (p = 12): ~17,000 warp instructions and ~3,500 shared-memory wavefronts a full chunk, half of the issue
// slots used, the rest fixed latencies and barriers; fewer warps were slower (8 an SM: 23.0 ms a solve of 2^20 points and targets,
// 12: 20.3, 16: 19.1), as was a lane per vector with the inputs in registers and every block size unrolled (31.4 ms,
// instruction fetch).
// Measured, dense operators on the CUDA cores -> this: M2L of 2^20 torus points, p = 12, FP32 55.4 -> 15.1 ms; 2^19
// points, p = 16, 61.5 -> 20.1 ms; 65,536 points, p = 12, FP64 24.1 -> 2.3 ms; 2,000 points, p = 10, 3.4 -> 0.05 ms; L2L
// of 2^24 points, p = 16, 13.4 -> 9.3 ms.
//   MODE 0: M2L, X = multipoles, Y = locals (zero before); vtab[box][316], the tile's boxes are targets[..]
//   MODE 1: M2M, X = Y = multipoles, the boxes are parents (zero before), vtab[parent][8] their children with sources
//   MODE 2: L2L, X = Y = locals, one octant's operator (blockIdx.z); the boxes are its children, the source their parent
// In the M2M and L2L a coefficient's own term (lambda = l) is the coefficient times a power of two: it is added as
// it is, and only the other, smaller terms go through the rotations and their rounding (with it among them the
// 2^24-point solve at p = 16 was 8.5e-7 off, without 7.7e-7 as with the dense operators).
// M2L: a block takes every gridDim.x-th of the first tiles, so that those in flight are neighbours and share their sources
// in L2, and of the rest a share of operators that evens out the blocks' work (TileOps). The block with a tile's first
// operator adds to the rows of Y, one that begins inside a tile keeps its sums there in its slot of ws ([3 TT][Lp])
// for kAddParts: a slot a block, whatever the tree. Without SHARED the grid is a block per tile.
// (Before, every tile was split into as many equal parts as made eight rounds of blocks, up to 64 copies of the locals:
// 0.43 to 0.57 GB, now 75 MB at most. M2L of 65,536 points and targets, FP32 p = 12 1.24 -> 1.02 ms, FP64 p = 9 1.49 -> 1.23;
// 131,072, FP32 p = 16 5.37 -> 4.95; 2^20, p = 4 4.6 both, p = 8 11.7 -> 12.0, p = 12 24.8 both, p = 16 51.0 -> 46.1.)
// M2M: blockIdx.y of gridDim.y parts of a tile's operators, their sums go to ws[part][3 nTargets][Lp] (zero before) for kSumParts.
template <class T, int MODE, bool SHARED = false>
__global__ void __launch_bounds__(512) kRotTranslate(const int* __restrict__ targets, int nTargets,
                                                    const int* __restrict__ vtab, const int* __restrict__ parent,
                                                    const L2LSegR seg, const TileOps tileOps, int TT, int p, int Lp,
                                                    const TaskTable* __restrict__ tasks, const T* __restrict__ ops, const T* X,
                                                    T* Y, T* ws)
{
   constexpr int NOP = MODE == 0 ? 316 : 8;
   constexpr int RS = rowStride<T>(), CH = chunkPairs<T>(), V = laneRows<T>();
   extern __shared__ __align__(16) unsigned char smraw[];
   constexpr int MT = MODE == 2 ? MAXTL : MAXT;
   __shared__ int tileNode[MT];
   __shared__ uint32_t present[10];
   __shared__ int offs[NOP];
   __shared__ int nOffS;
   __shared__ int slotT[2][MAXT], slotS[2][MT], nSlot[2];
   __shared__ int srcRow[2][RS], dstRow[2][RS];
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   const int NT = blockDim.x, NW = NT >> 5;
   const int L = nharm(p);
   const Blob B(p);
   int first = blockIdx.x * TT, end = nTargets;
   if(MODE == 2)
   {
      first = seg.start[blockIdx.z] + blockIdx.x * TT;
      end = seg.start[blockIdx.z + 1];
      if(first >= end) return;
   }
   // M2L: the tile in which this block's share begins (tiles: its share is empty)
   auto shareTile = [&]() {
      const int64_t w = tileOps.share[blockIdx.x];
      return w < tileOps.share[blockIdx.x + 1] || w > tileOps.start[tileOf(tileOps.start, tileOps.tiles, w)] ? tileOf(tileOps.start, tileOps.tiles, w)
                                                                                                          : tileOps.tiles;
   };
   if(SHARED && blockIdx.x >= tileOps.whole)
   {
      first = shareTile() * TT;
      if(first >= end) return;
   }
   int nTile = min(TT, end - first);
   const Smem<T> sm(p);
   T* D = reinterpret_cast<T*>(smraw);
   T* W0 = reinterpret_cast<T*>(smraw + sm.w0);
   T* W1 = reinterpret_cast<T*>(smraw + sm.w1);
   Task* task = reinterpret_cast<Task*>(smraw + sm.tasks);
   unsigned* pairs = reinterpret_cast<unsigned*>(smraw + sm.pairs);       // positions of (l, m), (l, -m), and m
   int* pads = reinterpret_cast<int*>(smraw + sm.pads);                   // order-major pad positions, their number at [MAXORDER + 1]
   unsigned short* pos = reinterpret_cast<unsigned short*>(smraw + sm.pos);   // degree-major position of k (L: none)
   const int nTask[3] = {tasks->n[0], tasks->n[1], tasks->n[2]};
   for(int e = tid; e < 3 * MAXTASK; e += NT)
      reinterpret_cast<uint4*>(task)[e] = reinterpret_cast<const uint4*>(&tasks->t[0][0])[e];
   for(int k = tid; k < Lp; k += NT)
   {
      int l = int(sqrtf(float(k)));
      while(l * l > k) l--;
      while((l + 1) * (l + 1) <= k) l++;
      const int m = k - l * l - l;
      pos[k] = (unsigned short)(k < L ? degPos(l, m) : 0xFFFF);
      if(k < L && m > 0) pairs[l * (l - 1) / 2 + m - 1] = unsigned(degPos(l, m)) | unsigned(degPos(l, -m)) << 10 | unsigned(m) << 20;
   }
   if(tid == 0)
   {
      int n = 0;
      for(int a = 0; a <= p; a++)
         if((p + 1 - a) & 1)
         {
            pads[n++] = ordBase(p, a) + p + 1 - a;
            if(a) pads[n++] = ordBase(p, -a) + p + 1 - a;
         }
      pads[MAXORDER + 1] = n;
   }
   // (a zero operator row meets these: they must be numbers)
   for(int e = tid; e < 2 * RS; e += NT) W0[L * RS + e] = T(0);
   for(int e = tid; e < RS; e += NT) W1[ordSize(p) * RS + e] = T(0);
   // the tiles of the block's share (M2M, L2L: its one tile)
   for(;;)
   {
      for(int t = tid; t < nTile; t += NT) tileNode[t] = targets[first + t];
      if(MODE == 1 && tid < 10) present[tid] = 0;
      __syncthreads();
      int o0 = 0, o1 = 1;
      bool toParts = false;   // the sums of this tile go to ws
      if(MODE == 2)
      {
         // every box has its pair: its parent
         if(tid == 0) { offs[0] = blockIdx.z; nSlot[0] = nTile; }
         for(int t = tid; t < nTile; t += NT) slotS[0][t] = parent[tileNode[t]];
         __syncthreads();
      }
      else if(MODE == 0)
      {
         // the tile's operators, those whose work begins in the share
         const int tile = first / TT, n = tileOps.n[tile];
         const bool all = !SHARED || tile < tileOps.whole;
         const int64_t lo = all ? 0 : tileOps.share[blockIdx.x] - tileOps.start[tile];
         const int64_t hi = all ? INT64_MAX : tileOps.share[blockIdx.x + 1] - tileOps.start[tile];
         o1 = 0;
         for(int e0 = 0; e0 < n; e0 += NT)
         {
            const int e = e0 + tid;
            const int64_t at = e < n ? tileOps.before[int64_t(tile) * NOP + e] : INT64_MAX;
            if(e < n) offs[e] = tileOps.op[int64_t(tile) * NOP + e];
            o0 += __syncthreads_count(at < lo);
            o1 += __syncthreads_count(at < hi);
         }
         toParts = SHARED && o0 > 0;
      }
      else
      {
         // a warp per box, its table row in loads that are all in flight
         constexpr int NWORD = (NOP + 31) / 32;
         uint32_t have[NWORD] = {};
         for(int t = warp; t < nTile; t += NW)
         {
            const int* row = vtab + int64_t(tileNode[t]) * NOP;
            int v[NWORD];
#pragma unroll
            for(int w = 0; w < NWORD; w++) v[w] = lane + 32 * w < NOP ? row[lane + 32 * w] : -1;
#pragma unroll
            for(int w = 0; w < NWORD; w++) have[w] |= __ballot_sync(0xffffffffu, v[w] >= 0);
         }
         if(lane == 0)
#pragma unroll
            for(int w = 0; w < NWORD; w++)
               if(have[w]) atomicOr(&present[w], have[w]);
         __syncthreads();
         if(warp == 0)
         {
            // the operators present, in order
            int base = 0;
            for(int w = 0; w * 32 < NOP; w++)
            {
               const uint32_t bits = present[w];
               if(bits >> lane & 1) offs[base + __popc(bits & ((1u << lane) - 1))] = 32 * w + lane;
               base += __popc(bits);
            }
            if(lane == 0) nOffS = base;
         }
         __syncthreads();
         const int nOff = nOffS, parts = gridDim.y, part = blockIdx.y;
         o0 = int(int64_t(nOff) * part / parts);
         o1 = int(int64_t(nOff) * (part + 1) / parts);
         toParts = parts > 1;
      }
      // source of the tile's box t for operator o
      auto sourceOf = [&](int t, int o) {
         if(t >= nTile) return -1;
         return vtab[int64_t(tileNode[t]) * NOP + o];
      };
      // warp 0: the pairs of operator oi, compacted; the sources were loaded one operator earlier
      constexpr int AH = (MAXT + 31) / 32;
      int ahead[AH];
      auto loadAhead = [&](int oi) {
#pragma unroll
         for(int h = 0; h < AH; h++) ahead[h] = sourceOf(lane + 32 * h, offs[oi]);
      };
      auto compact = [&](int b) {
         int n = 0;
#pragma unroll
         for(int h = 0; h < AH; h++)
         {
            const uint32_t bits = __ballot_sync(0xffffffffu, ahead[h] >= 0);
            if(ahead[h] >= 0)
            {
               const int k = n + __popc(bits & ((1u << lane) - 1));
               slotT[b][k] = lane + 32 * h;
               slotS[b][k] = ahead[h];
            }
            n += __popc(bits);
         }
         if(lane == 0) nSlot[b] = n;
      };
      T* out = !toParts ? Y : ws + (MODE == 0 ? int64_t(blockIdx.x) * TT : int64_t(blockIdx.y) * nTargets + first) * 3 * Lp;
      if(SHARED && toParts)
      {
         for(int e = tid; e < 3 * nTile * Lp; e += NT) out[e] = T(0);
         __syncthreads();
      }
      if(o0 < o1)
      {
         // the rows of X a chunk's vectors come from and the rows of Y (or of this part's sums) they are added to
         auto setRows = [&](int b, int c0, int nr, int db) {
            if(tid < nr)
            {
               const int t = c0 + tid / 3, cmp = tid % 3;
               srcRow[db][tid] = 3 * slotS[b][t] + cmp;
               dstRow[db][tid] = 3 * (MODE == 2 ? tileNode[t] : toParts ? slotT[b][t] : tileNode[slotT[b][t]]) + cmp;
            }
         };
         // Gather: element copies that all stay in flight while the previous chunk's sums are added, 8 consecutive
         // coefficients (a 32-byte sector in FP32) of 4 rows a warp.
         const int nk8 = (L + 7) >> 3, k8 = lane & 7, r4 = lane >> 3;
         auto gather = [&](const int* rows, int nr) {
            const int nq = (nr + 3) >> 2;
            for(int j = warp; j < nk8; j += NW)
            {
               const int k = 8 * j + k8;
               if(k >= L) continue;
               T* w = W0 + int(pos[k]) * RS + r4;
               const T* src = X + k;
#pragma unroll 4
               for(int q = 0; q < nq; q++)
                  if(4 * q + r4 < nr) cpAsyncElem(w + 4 * q, src + int64_t(rows[4 * q + r4]) * Lp);
            }
         };
         // Sums: 4 lanes of V consecutive coefficients by 8 rows a warp and item, BT items' loads in flight together.
         const int kl = V * (lane & 3), rl = lane >> 2, nkb = (Lp + 4 * V - 1) / (4 * V);
         typedef typename std::conditional<sizeof(T) == 4, float4, double2>::type VT;
         constexpr int BT = MODE != 0 ? 4 : (SHARED ? 5 : 6);   // (6 would spill beside the loop over tiles)
         auto addOut = [&](int db, int nr) {
            const int* rows = dstRow[db];
            const int nItems = nkb * ((nr + 7) >> 3);
            for(int i0 = warp; i0 < nItems; i0 += BT * NW)
            {
               VT y[BT], id[BT];
               T* q[BT];
#pragma unroll
               for(int h = 0; h < BT; h++)
               {
                  const int it = i0 + h * NW, r = 8 * (it / nkb) + rl, k = 4 * V * (it % nkb) + kl;
                  q[h] = nullptr;
                  if(it < nItems && r < nr)
                  {
                     q[h] = out + int64_t(rows[r]) * Lp + k;
                     y[h] = *reinterpret_cast<const VT*>(q[h]);
                     if(MODE != 0) id[h] = *reinterpret_cast<const VT*>(X + int64_t(srcRow[db][r]) * Lp + k);
                  }
               }
#pragma unroll
               for(int h = 0; h < BT; h++)
               {
                  if(!q[h]) continue;
                  const int it = i0 + h * NW, r = 8 * (it / nkb) + rl, k = 4 * V * (it % nkb) + kl;
                  T* ys = reinterpret_cast<T*>(&y[h]);
#pragma unroll
                  for(int i = 0; i < V; i++)
                  {
                     const int w = pos[k + i];
                     if(w == 0xFFFF) continue;
                     T v = W1[w * RS + r];
                     if(MODE != 0) v = fma(reinterpret_cast<const T*>(&id[h])[i], boxScale<T>(k + i, MODE == 2), v);
                     ys[i] += v;
                  }
                  *reinterpret_cast<VT*>(q[h]) = y[h];
               }
            }
         };
         if(MODE != 2 && warp == 0)
         {
            loadAhead(o0);
            compact(0);
            if(o0 + 1 < o1) loadAhead(o0 + 1);
         }
         __syncthreads();
         int oi = o0, b = 0, c0 = 0, nPairs = nSlot[0], nr = 3 * min(CH, nPairs), prevRows = 0, chunk = 0;
         setRows(0, 0, nr, 0);
         __syncthreads();
         const T* Z = D + B.zOff;
         const int nTurn = p * (p + 1) / 2;
         while(true)
         {
            if(c0 == 0)
            {
               const T* src = ops + int64_t(offs[oi]) * B.size;
               for(int e = tid * V; e < B.size; e += NT * V) cpAsync16(D + e, src + e);
               asm volatile("cp.async.commit_group;" ::: "memory");
            }
            gather(srcRow[chunk & 1], nr);
            asm volatile("cp.async.commit_group;" ::: "memory");
            if(chunk) addOut((chunk - 1) & 1, prevRows);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if(MODE != 2 && c0 == 0 && warp == 0 && oi + 1 < o1)
            {
               compact(b ^ 1);
               if(oi + 2 < o1) loadAhead(oi + 2);
            }
            for(int e = tid; e < pads[MAXORDER + 1] * RS; e += NT) W1[pads[e / RS] * RS + e % RS] = T(0);
            if(nr > 8 * V)
            {
               turn<T, 2>(pairs, nTurn, warp, NW, lane, Z, W0, false);
               __syncthreads();
               runStep<T, 2>(task, nTask[0], warp, NW, lane, D, W0, W1);
               __syncthreads();
               runStep<T, 2>(task + MAXTASK, nTask[1], warp, NW, lane, D, W1, W0);
               __syncthreads();
               runStep<T, 2>(task + 2 * MAXTASK, nTask[2], warp, NW, lane, D, W0, W1);
               __syncthreads();
               turn<T, 2>(pairs, nTurn, warp, NW, lane, Z, W1, true);
            }
            else
            {
               // at most one group of rows
               turn<T, 1>(pairs, nTurn, warp, NW, lane, Z, W0, false);
               __syncthreads();
               runStep<T, 1>(task, nTask[0], warp, NW, lane, D, W0, W1);
               __syncthreads();
               runStep<T, 1>(task + MAXTASK, nTask[1], warp, NW, lane, D, W1, W0);
               __syncthreads();
               runStep<T, 1>(task + 2 * MAXTASK, nTask[2], warp, NW, lane, D, W0, W1);
               __syncthreads();
               turn<T, 1>(pairs, nTurn, warp, NW, lane, Z, W1, true);
            }
            // the next chunk
            prevRows = nr;
            chunk++;
            c0 += CH;
            if(c0 >= nPairs)
            {
               c0 = 0;
               b ^= 1;
               if(++oi < o1) nPairs = nSlot[b];
            }
            if(oi < o1)
            {
               nr = 3 * min(CH, nPairs - c0);
               setRows(b, c0, nr, chunk & 1);
            }
            __syncthreads();
            if(oi >= o1) break;
         }
         addOut((chunk - 1) & 1, prevRows);
      }
      // the block's next tile
      if(!SHARED) break;
      int next = first / TT;
      if(next < tileOps.whole)
      {
         next += gridDim.x;
         if(next >= tileOps.whole) next = tileOps.whole < tileOps.tiles ? shareTile() : tileOps.tiles;
      }
      else if(++next < tileOps.tiles && tileOps.start[next] >= tileOps.share[blockIdx.x + 1]) next = tileOps.tiles;
      if(next >= tileOps.tiles) break;
      first = next * TT;
      nTile = min(TT, end - first);
      __syncthreads();
   }
}

// Y of every target row = the parts' sums in order.
template <class T>
__global__ void kSumParts(const int* __restrict__ targets, int nTargets, int parts, int Lp, const T* __restrict__ ws,
                          T* __restrict__ Y)
{
   const int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
   const int64_t rowElems = 3 * int64_t(nTargets) * Lp;
   if(e >= rowElems) return;
   const int64_t row = e / Lp;
   T s = T(0);
   for(int q = 0; q < parts; q++) s += ws[q * rowElems + e];
   Y[(int64_t(targets[row / 3]) * 3 + row % 3) * Lp + int(e % Lp)] = s;
}

}  // namespace rot

// The rotation tables of the plan's order: the full M2L operator, or with m2l_truncate the terms up to l + lambda = p.
// (fmm_config.m2l_tc_degree_cutoff is the tensor-core M2L's: here a cutoff would save nothing.) Tensor-core M2L plans take
// the M2M's and L2L's operators alone.
template <class T>
fmm_status ensureRotations(Plan& P, cudaStream_t st)
{
   const int cut = P.cfg.m2l_truncate ? P.p : 2 * P.p;
   if(P.rotCut == cut) return FMM_OK;
   const int count = !P.fp64 && P.cfg.m2l_mode != FMM_M2L_SIMT ? 16 : 16 + 316;
   const rot::Blob B(P.p);
   const std::vector<double>& q = rot::quarterTurn(P.p);
   FMM_TRY(P.rotQuarter.reserve(sizeof(double) * q.size()));
   FMM_TRY(P.rotOps.reserve(sizeof(T) * size_t(B.size) * count));
   // the step tasks of the M2L and of the M2M / L2L
   P.rotTaskHost.resize(2 * sizeof(rot::TaskTable));
   for(int mode = 0; mode < 2; mode++)
      rot::makeTasks(P.p, mode, reinterpret_cast<rot::TaskTable*>(P.rotTaskHost.data())[mode]);
   FMM_TRY(P.rotTasks.reserve(P.rotTaskHost.size()));
   FMM_CUDA(cudaMemcpyAsync(P.rotTasks.ptr, P.rotTaskHost.data(), P.rotTaskHost.size(), cudaMemcpyHostToDevice, st));
   FMM_CUDA(cudaMemcpyAsync(P.rotQuarter.ptr, q.data(), sizeof(double) * q.size(), cudaMemcpyHostToDevice, st));
   rot::kBuildRotations<T><<<count, 256, 0, st>>>(P.p, cut, (const double*)P.rotQuarter.ptr, (T*)P.rotOps.ptr);
   FMM_TRY(launched(P, "kBuildRotations", st));
   P.rotCut = cut;
   return FMM_OK;
}

// Boxes of a tile, the blocks of a launch and their threads. An M2L tile has five chunks' boxes (FP64: six): an operator
// has partners for about half of them, so its chunks are mostly full (tiles of one chunk: M2L of 2^19 points and
// targets, p = 12, 9.3 ms, of five 7.5; FP64, 131,072, p = 12, 4.3 and 3.6). Threads: 16 warps an SM (the registers' limit)
// as two blocks, from p = 13 on as one; for the M2L blocks of 4 warps where three or four fit, p <= 9 in FP32 (8 warps a block at
// p = 4: 2.4 ms, 4 warps 1.7; at p = 8 4.3 and 3.9; at p = 10, where two fit, 6.0 and 7.4).
template <class T> static int rotTile(int mode) { return rot::chunkPairs<T>() * (mode == 0 ? (sizeof(T) == 8 ? 6 : 5) : 1); }
template <class T>
static int rotPerSM(const Plan& P, int mode)
{
   const int fit = (227 * 1024) / (rot::Smem<T>(P.p).total + 6 * 1024);
   return fit >= 3 && mode == 0 ? std::min(fit, 4) : (fit >= 2 ? 2 : 1);
}
template <class T> static int rotTiles(int mode, int count) { return (count + rotTile<T>(mode) - 1) / rotTile<T>(mode); }
template <class T> static int rotThreads(const Plan& P, int mode)
{
   const int perSM = rotPerSM<T>(P, mode);
   return perSM >= 3 ? 128 : 512 / perSM;
}
// M2L: the blocks of a launch, all resident at once (fewer in trees of a few tiles: 64 a tile)
template <class T> static int rotBlocks(Plan& P, int tiles)
{
   if(P.rotResident == 0)
   {
      auto kern = rot::kRotTranslate<T, 0, true>;
      const int smem = rot::Smem<T>(P.p).total;
      int n = 0;
      if(allowShared(kern) != cudaSuccess ||
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, rotThreads<T>(P, 0), smem) != cudaSuccess)
         cudaGetLastError();
      P.rotResident = std::max(1, n);
   }
   return std::min(148 * P.rotResident, 64 * tiles);
}
// M2M: parts of a tile's operators, four rounds of blocks
template <class T>
static int rotParts(const Plan& P, int count)
{
   const int tiles = rotTiles<T>(1, count);
   return tiles ? std::max(1, std::min(8, 4 * 148 * rotPerSM<T>(P, 1) / tiles)) : 1;
}
template <class T> static size_t rotRowBytes(const Plan& P) { return sizeof(T) * 3 * size_t(P.Lp); }

// The M2L's tile lists in rotTiles. The last one to two rounds of tiles are shared, those before them whole (half a round to one
// and a half: 2^19 points, p = 16, 15.3 ms against 13.8, as blocks whose whole tiles exceed the mean get no share).
template <class T> static rot::TileOps rotTileOps(Plan& P)
{
   rot::TileOps o;
   o.tiles = rotTiles<T>(0, P.nM2LTargets);
   o.blocks = rotBlocks<T>(P, o.tiles);
   o.whole = std::max(0, o.tiles / o.blocks - 1) * o.blocks;
   o.start = (int64_t*)P.rotTiles.ptr;
   o.share = o.start + o.tiles + 1;
   o.before = (int*)(o.share + o.blocks + 1);
   o.n = o.before + size_t(o.tiles) * 316;
   o.op = (unsigned short*)(o.n + o.tiles);
   return o;
}

// What the launches on the current tree need, so that none of them allocates: the M2L's tile lists and room for the blocks' and
// parts' sums, at most 75 MB whatever the tree and order. Without that room the M2L takes a block per tile and the M2M does not
// split, which is slower but needs none.
template <class T>
fmm_status reserveRotations(Plan& P, cudaStream_t st)
{
   const bool tc = !P.fp64 && P.cfg.m2l_mode != FMM_M2L_SIMT;   // M2L (and M2M) on the tensor cores
   if(tc && P.tcTranslations(1)) return FMM_OK;
   size_t bytes = 0;
   if(!tc && P.nM2LTargets > 0)
   {
      const int tiles = rotTiles<T>(0, P.nM2LTargets), blocks = rotBlocks<T>(P, tiles);
      FMM_TRY(P.rotTiles.reserve(size_t(tiles) * (8 + 4 + 316 * 6) + 8 * size_t(blocks + 2)));
      const rot::TileOps ops = rotTileOps<T>(P);
      rot::kTileOps<T><<<tiles, rot::TILEOPS_NT, 0, st>>>((const int*)P.m2lTargets.ptr, P.nM2LTargets, P.lists.vtab, rotTile<T>(0),
                                                              P.p, ops, (unsigned*)P.err + 2);
      FMM_TRY(launched(P, "kTileOps", st));
      bytes = rotRowBytes<T>(P) * rotTile<T>(0) * blocks;
   }
   for(int level = 0; level + 1 < P.tree.nLevels; level++)
   {
      const int count = P.parStart[level + 1] - P.parStart[level], parts = rotParts<T>(P, count);
      if(parts > 1) bytes = std::max(bytes, rotRowBytes<T>(P) * parts * size_t(count));
   }
   if(bytes) P.roomFor(P.rotWs, bytes);
   return FMM_OK;
}

template <class T, int MODE>
static fmm_status launchRot(Plan& P, cudaStream_t st, const int* targets, int count, const int* vtab, const rot::L2LSegR& seg,
                            int most, const T* X, T* Y)
{
   const rot::Blob B(P.p);
   const size_t smem = rot::Smem<T>(P.p).total;
   const int THREADS = rotThreads<T>(P, MODE);
   auto kern = rot::kRotTranslate<T, MODE>;
   if(MODE != 0) FMM_CUDA(allowShared(kern));
   const T* ops = (const T*)P.rotOps.ptr + size_t(B.size) * (MODE == 0 ? 16 : MODE == 1 ? 0 : 8);
   const rot::TaskTable* tasks = (const rot::TaskTable*)P.rotTasks.ptr + (MODE == 0 ? 0 : 1);
   const int tile = rotTile<T>(MODE);
   if(MODE == 2)
   {
      // up to eight chunks a block, which loads the octant's tables once, while that leaves four rounds of blocks
      const int chunk = rot::chunkPairs<T>(), all = seg.start[8] - seg.start[0];
      const int tl = chunk * std::max(1, std::min(rot::MAXTL / chunk, all / (chunk * 4 * 148 * rotPerSM<T>(P, MODE))));
      kern<<<dim3((most + tl - 1) / tl, 1, 8), THREADS, smem, st>>>(targets, 0, nullptr, P.tree.parent, seg, rot::TileOps{}, tl, P.p,
                                                                   P.Lp, tasks, ops, X, Y, nullptr);
      return launched(P, "kRotTranslate<L2L>", st);
   }
   const int tiles = rotTiles<T>(MODE, count);
   T* ws = (T*)P.rotWs.ptr;
   if(MODE == 0)
   {
      const rot::TileOps tileOps = rotTileOps<T>(P);
      auto run = [&](auto kernel, int grid) -> fmm_status {
         FMM_CUDA(allowShared(kernel));
         kernel<<<grid, THREADS, smem, st>>>(targets, count, vtab, P.tree.parent, seg, tileOps, tile, P.p, P.Lp, tasks, ops, X, Y, ws);
         return launched(P, "kRotTranslate<M2L>", st);
      };
      // A block per tile where the last round of blocks counts for little against the registers that the loop over tiles
      // costs, or without room for the slots. In shares / a block per tile, ms: one block an SM (p = 16) 2^21 points, 8 rounds,
      // 74 / 78, 2^22, 17 rounds, 213 / 206, 2^24 669 / 621; two (p = 12) 2^20, 2 rounds, 25 / 29, 2^21, 4 rounds, 43.4 / 42.4,
      // 2^22 117 / 111; four (p = 8) 2^21, 2 rounds, 19 / 22, 2^22, 4 rounds, 54.9 / 54.6, 2^23 75 / 71.
      const int shared = tiles - tileOps.whole, perTile = P.rotResident == 1 ? 12 : 4;
      if(tiles >= perTile * tileOps.blocks || P.rotWs.bytes < rotRowBytes<T>(P) * tile * tileOps.blocks) return run(rot::kRotTranslate<T, 0>, tiles);
      FMM_TRY(run(rot::kRotTranslate<T, 0, true>, tileOps.blocks));
      const int n = 3 * P.Lp, rounds = (n + 511) / 512, threads = ((n + rounds - 1) / rounds + 31) / 32 * 32;
      rot::kAddParts<T><<<dim3(shared, std::max(8, std::min(tile, 4736 / shared))), threads, 0, st>>>(targets, count, tile, tileOps,
                                                                                                    P.Lp, ws, Y);
      return launched(P, "kAddParts", st);
   }
   const int64_t n = 3 * int64_t(count) * P.Lp;
   int parts = rotParts<T>(P, count);
   if(P.rotWs.bytes < sizeof(T) * size_t(parts) * n) parts = 1;
   if(parts > 1) FMM_CUDA(cudaMemsetAsync(ws, 0, sizeof(T) * size_t(parts) * n, st));
   kern<<<dim3(tiles, parts), THREADS, smem, st>>>(targets, count, vtab, P.tree.parent, seg, rot::TileOps{}, tile, P.p, P.Lp, tasks,
                                                   ops, X, Y, ws);
   FMM_TRY(launched(P, "kRotTranslate<M2M>", st));
   if(parts > 1)
   {
      rot::kSumParts<T><<<int((n + 255) / 256), 256, 0, st>>>(targets, count, parts, P.Lp, ws, Y);
      FMM_TRY(launched(P, "kSumParts", st));
   }
   return FMM_OK;
}

template <class T>
fmm_status rotM2L(Plan& P, cudaStream_t st)
{
   if(P.nM2LTargets <= 0) return FMM_OK;
   return launchRot<T, 0>(P, st, (const int*)P.m2lTargets.ptr, P.nM2LTargets, P.lists.vtab, rot::L2LSegR{}, 0,
                          (const T*)P.mult.ptr, (T*)P.local.ptr);
}

template <class T>
fmm_status rotM2M(Plan& P, cudaStream_t st)
{
   for(int level = P.tree.nLevels - 2; level >= 0; level--)
   {
      const int a = P.parStart[level], b = P.parStart[level + 1];
      if(b <= a) continue;
      FMM_TRY((launchRot<T, 1>(P, st, (const int*)P.parList.ptr + a, b - a, (const int*)P.vtabUp.ptr, rot::L2LSegR{}, 0,
                               (const T*)P.mult.ptr, (T*)P.mult.ptr)));
   }
   FMM_CHECK_LAUNCH();
   return FMM_OK;
}

template <class T>
fmm_status rotL2L(Plan& P, cudaStream_t st)
{
   for(int level = 0; level + 1 < P.tree.nLevels; level++)
   {
      rot::L2LSegR seg;
      int most = 0;
      for(int o = 0; o <= 8; o++) seg.start[o] = P.l2lStart[8 * (level + 1) + o];
      for(int o = 0; o < 8; o++) most = std::max(most, seg.start[o + 1] - seg.start[o]);
      if(most == 0) continue;
      FMM_TRY((launchRot<T, 2>(P, st, (const int*)P.l2lTargets.ptr, 0, nullptr, seg, most, (const T*)P.local.ptr, (T*)P.local.ptr)));
   }
   FMM_CHECK_LAUNCH();
   return FMM_OK;
}

template fmm_status ensureRotations<float>(Plan&, cudaStream_t);
template fmm_status ensureRotations<double>(Plan&, cudaStream_t);
template fmm_status reserveRotations<float>(Plan&, cudaStream_t);
template fmm_status reserveRotations<double>(Plan&, cudaStream_t);
template fmm_status rotM2L<float>(Plan&, cudaStream_t);
template fmm_status rotM2L<double>(Plan&, cudaStream_t);
template fmm_status rotM2M<float>(Plan&, cudaStream_t);
template fmm_status rotM2M<double>(Plan&, cudaStream_t);
template fmm_status rotL2L<float>(Plan&, cudaStream_t);
template fmm_status rotL2L<double>(Plan&, cudaStream_t);

}  // namespace fmm
