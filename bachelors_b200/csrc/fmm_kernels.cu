// FMM kernels for sm_100a: dense translation-operator tables (FP64), P2M, and the L2P and direct near field.
// (The translations are in fmm_rotate.cu and fmm_m2l_tc.cu.)
//
// Every expansion is stored box-size scaled: a node of side h keeps M~_l = M_l / h^l and
// L~_l = L_l h^(l+1). With that scaling the M2M, L2L and M2L operators do not depend on the
// level: 8 M2M and 8 L2L operators (one per child octant) and 316 M2L operators (one per
// offset o in [-3,3]^3 outside [-1,1]^3), all built once per order in FP64.
//
// Reference counterparts (FMM/FMMGPU/):
//   P2M   math::calcIntegralContribution                     integration.cpp:137-161
//   M2M   MultipoleTranslator::translateMultipoleWithComplex  multipole_translator.cpp:3-32,111-125,143-146
//   M2L   multipoleToLocalWithComplex (l + lambda <= p)       multipole_translator.cpp:148-199
//   L2L   translateLocalWithComplex                          multipole_translator.cpp:201-255
//   L2P   CalculationPointOctreeNode::calcA / calcRot        calculation_point_octree.cpp:192-275
//         (B from analytic gradients here, finite differences there)
//   near  bioSavartLaplaceFunction                           integration.cpp:113-120
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include <cuda_bf16.h>

#include <cub/cub.cuh>

#include "fmm_internal.cuh"

namespace fmm {

__constant__ int d_m2lIndex[NOFF];
__constant__ int d_m2lOffset[316];
__constant__ int d_m2lFarFirst[316];

// Constant memory is per device context: fill it once on every device that uses the library.
fmm_status initOffsetTables()
{
   static bool done[64] = {false};
   int dev = 0;
   FMM_CUDA(cudaGetDevice(&dev));
   if(dev < 64 && done[dev]) return FMM_OK;
   int idx[NOFF], off[316];
   int k = 0;
   for(int oz = -3; oz <= 3; oz++)
      for(int oy = -3; oy <= 3; oy++)
         for(int ox = -3; ox <= 3; ox++)
         {
            int o = offsetIndex(ox, oy, oz);
            if(abs(ox) <= 1 && abs(oy) <= 1 && abs(oz) <= 1) idx[o] = -1;
            else { idx[o] = k; off[k] = o; k++; }
         }
   int far[316];
   for(int i = 0; i < 316; i++) far[i] = i;
   auto len2 = [&](int slot) {
      int o = off[slot];
      int ox = o % 7 - 3, oy = (o / 7) % 7 - 3, oz = o / 49 - 3;
      return ox * ox + oy * oy + oz * oz;
   };
   std::stable_sort(far, far + 316, [&](int a, int b) { return len2(a) > len2(b); });
   FMM_CUDA(cudaMemcpyToSymbol(d_m2lFarFirst, far, sizeof(far)));
   FMM_CUDA(cudaMemcpyToSymbol(d_m2lIndex, idx, sizeof(idx)));
   FMM_CUDA(cudaMemcpyToSymbol(d_m2lOffset, off, sizeof(off)));
   if(dev < 64) done[dev] = true;
   return FMM_OK;
}

// ====================================================================================
// Operator tables. Entry (i, j) of a translation in the real basis, derived from the
// reference's complex form res(l,m) = sum a(lambda,mu) G(l,m,lambda,mu) between the
// realToComplex / complexToReal conversions (harmonics.cpp:340-379), with exact 1/sqrt2.
// ====================================================================================
struct C2 { double re, im; };

__device__ inline C2 cplxOf(const double* H, int n, int k)
{
   const double s = 0.70710678118654752440;
   if(k == 0) return {H[hidx(n, 0)], 0.0};
   int a = abs(k);
   return {s * H[hidx(n, a)], (k > 0 ? s : -s) * H[hidx(n, -a)]};
}

__device__ inline double signPow(int t) { int e = (-t) / 2; return (e & 1) ? -1.0 : 1.0; }

// kind 0 = M2M, 1 = L2L, 2 = M2L. H = real harmonics of the translation (regular for
// M2M / L2L, irregular to order `lim` for M2L).
__device__ C2 translationG(int kind, int l, int m, int lam, int mu, const double* H, int lim)
{
   if(kind == 0)
   {
      int dl = l - lam, dm = m - mu;
      if(dl < 0 || abs(dm) > dl) return {0, 0};
      C2 b = cplxOf(H, dl, dm);
      double f = signPow(abs(m) - abs(m - mu) - abs(mu));
      return {b.re * f, b.im * f};
   }
   if(kind == 1)
   {
      int dl = lam - l, dm = m - mu;
      if(dl < 0 || abs(dm) > dl) return {0, 0};
      C2 b = cplxOf(H, dl, dm);
      double f = signPow(abs(mu) - abs(m - mu) - abs(m)) * (((lam + l) & 1) ? -1.0 : 1.0);
      return {b.re * f, b.im * f};
   }
   int dl = l + lam, dm = m - mu;
   if(dl > lim) return {0, 0};
   C2 b = cplxOf(H, dl, dm);
   double f = signPow(abs(m - mu) - abs(m) - abs(mu)) * ((lam & 1) ? -1.0 : 1.0);
   return {b.re * f, b.im * f};
}

__device__ double operatorEntry(int kind, int i, int j, const double* H, int lim)
{
   const double s = 0.70710678118654752440;
   int l = int(sqrt(double(i))); while(l * l > i) l--; while((l + 1) * (l + 1) <= i) l++;
   int mi = i - l * l - l;
   int lam = int(sqrt(double(j))); while(lam * lam > j) lam--; while((lam + 1) * (lam + 1) <= j) lam++;
   int mj = j - lam * lam - lam;
   // complex input of the unit real vector e_j
   int mus[2]; C2 as[2]; int nin;
   if(mj == 0) { mus[0] = 0; as[0] = {1, 0}; nin = 1; }
   else if(mj > 0) { mus[0] = mj; as[0] = {s, 0}; mus[1] = -mj; as[1] = {s, 0}; nin = 2; }
   else { mus[0] = -mj; as[0] = {0, s}; mus[1] = mj; as[1] = {0, -s}; nin = 2; }
   auto res = [&](int m) {
      C2 r = {0, 0};
      for(int e = 0; e < nin; e++)
      {
         C2 g = translationG(kind, l, m, lam, mus[e], H, lim);
         r.re += as[e].re * g.re - as[e].im * g.im;
         r.im += as[e].re * g.im + as[e].im * g.re;
      }
      return r;
   };
   if(mi == 0) return res(0).re;
   if(mi > 0) return s * (res(mi).re + res(-mi).re);
   return s * (res(-mi).im - res(mi).im);
}

// One block per operator. op < 8: M2M octant, op < 16: L2L octant, else M2L slot.
__global__ void kBuildOperators(int p, int lim, int first, int count, double* m2m, double* l2l, double* m2l)
{
   extern __shared__ double Hs[];
   int op = first + blockIdx.x;
   if(blockIdx.x >= count) return;
   int L = nharm(p);
   int kind = op < 8 ? 0 : (op < 16 ? 1 : 2);
   if(threadIdx.x == 0)
   {
      if(kind < 2)
      {
         int oct = op & 7;
         double t[3] = {((oct & 1) - 0.5) * 0.5, (((oct >> 1) & 1) - 0.5) * 0.5, (((oct >> 2) & 1) - 0.5) * 0.5};
         if(kind == 1) { t[0] = -t[0]; t[1] = -t[1]; t[2] = -t[2]; }
         realRegular<double>(p, t[0], t[1], t[2], Hs);
      }
      else
      {
         int o = d_m2lOffset[op - 16];
         int ox = o % 7 - 3, oy = (o / 7) % 7 - 3, oz = o / 49 - 3;
         realIrregular<double>(lim, double(ox), double(oy), double(oz), Hs);
      }
   }
   __syncthreads();
   double* out = kind == 0 ? m2m + int64_t(op) * L * L : kind == 1 ? l2l + int64_t(op - 8) * L * L
                                                                   : m2l + int64_t(op - 16) * L * L;
   for(int e = threadIdx.x; e < L * L; e += blockDim.x)
   {
      int i = e / L, j = e % L;
      double v = operatorEntry(kind, i, j, Hs, lim);
      int li = int(sqrt(double(i))); while(li * li > i) li--; while((li + 1) * (li + 1) <= i) li++;
      int lj = int(sqrt(double(j))); while(lj * lj > j) lj--; while((lj + 1) * (lj + 1) <= j) lj++;
      if(kind == 0) v = ldexp(v, -lj);        // scaled M2M: columns times 2^-lambda
      else if(kind == 1) v = ldexp(v, -(li + 1));  // scaled L2L: rows times 2^-(l+1)
      out[e] = v;
   }
}

// The gradient coefficients of kL2PNear's gradCoeff as terms: its value is sum_i c[i] Lv[idx[i]]
// (the same case analysis, for tables).
struct GradTerms
{
   int n;
   int idx[2];
   double c[2];
};
inline GradTerms gradTerms(int j, int lp, int mu)
{
   const int l = lp + 1;
   const double h = 0.5, r2 = 0.70710678118654752440;
   GradTerms g{0, {0, 0}, {0.0, 0.0}};
   auto add = [&](double c, int m) {
      if(std::abs(m) <= l) { g.idx[g.n] = hidx(l, m); g.c[g.n] = c; g.n++; }
   };
   if(j == 2) add(-1.0, mu);
   else if(j == 0)
   {
      if(mu == 0) add(-r2, 1);
      else if(mu == 1) { add(-h, 2); add(r2, 0); }
      else if(mu >= 2) { add(-h, mu + 1); add(h, mu - 1); }
      else if(mu == -1) add(-h, -2);
      else { add(-h, mu - 1); add(h, mu + 1); }
   }
   else
   {
      if(mu == 0) add(-r2, -1);
      else if(mu == 1) add(-h, -2);
      else if(mu >= 2) { add(-h, -(mu + 1)); add(-h, -(mu - 1)); }
      else if(mu == -1) { add(h, 2); add(r2, 0); }
      else { add(h, 1 - mu); add(h, -mu - 1); }
   }
   return g;
}
// One entry of the L2P curl table: curl-expansion coefficient k' (degree <= p - 1), component c,
// with the real-basis factor (-1)^l' (sqrt2 for m != 0) folded in, as <= 4 terms of the local
// expansion row [3][Lp] of a box. Entries are [k'][4]; the fourth of each k' is empty.
template <class T>
struct CurlEntry
{
   int idx[4];
   T c[4];
};

// The dense FP64 operator tables: the tensor-core operator images are made from them, and fmm_get_operator
// returns them. The CUDA-core translations (fmm_rotate.cu) have tables of their own.
fmm_status buildDenseOperators(Plan& P, cudaStream_t st)
{
   if(P.denseOrder == P.p) return FMM_OK;
   FMM_TRY(initOffsetTables());
   const int p = P.p, L = P.L;
   const int lim = P.cfg.m2l_truncate ? p : 2 * p;
   FMM_TRY(P.opM2M64.reserve(sizeof(double) * 8 * L * L));
   FMM_TRY(P.opL2L64.reserve(sizeof(double) * 8 * L * L));
   FMM_TRY(P.opM2L64.reserve(sizeof(double) * 316 * L * L));
   size_t shm = sizeof(double) * nharm(std::max(lim, p));
   kBuildOperators<<<16 + 316, 256, shm, st>>>(p, lim, 0, 16 + 316, (double*)P.opM2M64.ptr, (double*)P.opL2L64.ptr,
                                               (double*)P.opM2L64.ptr);
   FMM_TRY(launched(P, "kBuildOperators", st));
   FMM_CHECK_LAUNCH();
   P.denseOrder = p;
   P.opImgOrder = -1;
   return FMM_OK;
}

// What every solve of the plan's order needs, built once: the rotation tables, the L2P's curl table and, in
// tensor-core plans, the dense operators.
fmm_status buildOperators(Plan& P, cudaStream_t st)
{
   if(P.opOrder == P.p) return FMM_OK;
   FMM_TRY(initOffsetTables());
   const int p = P.p, Lp = P.Lp;
   if(!P.fp64 && P.cfg.m2l_mode != FMM_M2L_SIMT) FMM_TRY(buildDenseOperators(P, st));
   FMM_TRY(P.fp64 ? ensureRotations<double>(P, st) : ensureRotations<float>(P, st));
   // the L2P curl table in the plan's precision
   {
      const int Lb = nharm(p - 1);
      const size_t esz = P.fp64 ? sizeof(CurlEntry<double>) : sizeof(CurlEntry<float>);
      P.curlHost.assign(esz * 4 * Lb, 0);
      for(int k = 0; k < Lb; k++)
      {
         int lp = 0;
         while((lp + 1) * (lp + 1) <= k) lp++;
         const int mu = k - lp * lp - lp;
         const double f = ((lp & 1) ? -1.0 : 1.0) * (mu != 0 ? 1.4142135623730950488 : 1.0);
         for(int c = 0; c < 3; c++)
         {
            // B_x = dAz/dy - dAy/dz, B_y = dAx/dz - dAz/dx, B_z = dAy/dx - dAx/dy
            const int cp = (c + 2) % 3, cm = (c + 1) % 3, jp = (c + 1) % 3, jm = (c + 2) % 3;
            const GradTerms gp = gradTerms(jp, lp, mu), gm = gradTerms(jm, lp, mu);
            int idx[4] = {0, 0, 0, 0};
            double cf[4] = {0, 0, 0, 0};
            int n = 0;
            for(int i = 0; i < gp.n; i++) { idx[n] = cp * Lp + gp.idx[i]; cf[n] = f * gp.c[i]; n++; }
            for(int i = 0; i < gm.n; i++) { idx[n] = cm * Lp + gm.idx[i]; cf[n] = -f * gm.c[i]; n++; }
            unsigned char* dst = P.curlHost.data() + esz * (4 * k + c);
            if(P.fp64)
            {
               CurlEntry<double> e;
               for(int i = 0; i < 4; i++) { e.idx[i] = idx[i]; e.c[i] = cf[i]; }
               memcpy(dst, &e, sizeof(e));
            }
            else
            {
               CurlEntry<float> e;
               for(int i = 0; i < 4; i++) { e.idx[i] = idx[i]; e.c[i] = float(cf[i]); }
               memcpy(dst, &e, sizeof(e));
            }
         }
      }
      FMM_TRY(P.curlTab.reserve(P.curlHost.size()));
      FMM_CUDA(cudaMemcpyAsync(P.curlTab.ptr, P.curlHost.data(), P.curlHost.size(), cudaMemcpyHostToDevice, st));
   }
   P.opOrder = p;
   return FMM_OK;
}

// ====================================================================================
// Geometry helpers
// ====================================================================================
__device__ __forceinline__ void nodeCenter(const RootBox& rb, int level, int ix, int iy, int iz, double c[3], double& h)
{
   h = 2.0 * rb.H / double(int64_t(1) << level);
   c[0] = rb.center[0] - rb.H + (double(ix) + 0.5) * h;
   c[1] = rb.center[1] - rb.H + (double(iy) + 0.5) * h;
   c[2] = rb.center[2] - rb.H + (double(iz) + 0.5) * h;
}

// ====================================================================================
// P2M: one block of NT threads per leaf holding sources, one source point per thread. Each
// thread runs the harmonic recurrence of its point as explicit state in registers (RegularIter,
// the visit order of visitRegular). Every CV visits the block reduces the values of those
// visits over its points through a small shared tile (the values of a visit are the same
// coefficient for every thread, so the tile's columns are coefficients) and adds them to the
// leaf's multipole, kept in shared memory until the end. Leaves with more than NT points take
// their points NT at a time.
// ====================================================================================
template <class T>
struct RegularIter
{
   T x, y, z, r2;
   T dre, dim;       // S_m^m
   T are, aim;       // S_l^m (the current visit)
   T bre, bim;       // S_{l-1}^m
   int l, m, p;
   __device__ __forceinline__ void start(int p_, T x_, T y_, T z_)
   {
      p = p_; x = x_; y = y_; z = z_; r2 = x * x + y * y + z * z;
      dre = T(1); dim = T(0); are = T(1); aim = T(0); bre = T(0); bim = T(0); l = 0; m = 0;
   }
   // moves to the next (l, m) of the visit order: l = m..p for m = 0..p
   __device__ __forceinline__ void next()
   {
      if(l < p)
      {
         T cre, cim;
         if(l == m) { cre = z * are; cim = z * aim; }
         else
         {
            const T inv = T(1) / T((l - m + 1) * (l + m + 1));
            const T a = T(2 * l + 1) * inv;
            cre = a * z * are - inv * r2 * bre;
            cim = a * z * aim - inv * r2 * bim;
         }
         bre = are; bim = aim; are = cre; aim = cim;
         l++;
      }
      else
      {
         m++;
         const T s = T(1) / T(2 * m);
         const T nre = (dre * x - dim * y) * s;
         const T nim = (dre * y + dim * x) * s;
         dre = nre; dim = nim;
         are = dre; aim = dim; bre = T(0); bim = T(0);
         l = m;
      }
   }
};

template <class T, int NT, int CV>
__global__ void __launch_bounds__(NT) kP2M(Tree t, const RootBox* __restrict__ rootp,
                                           const typename Vec4<T>::type* __restrict__ pos,
                                           const typename Vec4<T>::type* __restrict__ q, int p, int Lp, T* __restrict__ M)
{
   __shared__ T R[NT][2 * CV + 1];   // the chunk's real-basis values per point (odd stride)
   __shared__ T Q[NT][3];            // w J per point
   __shared__ int kOf[2 * CV];       // coefficient index of each column of R (-1: none)
   extern __shared__ unsigned char smraw[];
   T* Macc = (T*)smraw;              // [3][Lp] the leaf's multipole
   const int node = blockIdx.x;
   if(t.nchild[node] != 0) return;
   const int s0 = t.s0[node], s1 = t.s1[node];
   if(s1 == s0) return;
   const int tid = threadIdx.x;
   const int L = nharm(p);
   const int nVisits = (p + 1) * (p + 2) / 2;
   for(int e = tid; e < 3 * Lp; e += NT) Macc[e] = T(0);
   const RootBox rb = rootp[rootOf(t, node)];
   double c[3], h;
   nodeCenter(rb, t.level[node], t.ix[node], t.iy[node], t.iz[node], c, h);
   const double ih = 1.0 / h;
   const T sq2 = T(1.4142135623730950488);
   for(int base = s0; base < s1; base += NT)
   {
      const int cnt = min(NT, s1 - base);
      RegularIter<T> it;
      T qx = T(0), qy = T(0), qz = T(0);
      if(tid < cnt)
      {
         const auto xp = pos[base + tid];
         const auto w = q[base + tid];
         it.start(p, T((double(xp.x) - c[0]) * ih), T((double(xp.y) - c[1]) * ih), T((double(xp.z) - c[2]) * ih));
         qx = w.x; qy = w.y; qz = w.z;
      }
      else
         it.start(p, T(0), T(0), T(0));
      Q[tid][0] = qx; Q[tid][1] = qy; Q[tid][2] = qz;
      int vl = 0, vm = 0;   // (l, m) of the chunk's first visit, tracked uniformly by every thread
      for(int v0 = 0; v0 < nVisits; v0 += CV)
      {
         const int nv = min(CV, nVisits - v0);
         // this thread's values for visits v0 .. v0 + nv - 1, and the columns' coefficients
         int cl = vl, cm = vm;
         for(int j = 0; j < nv; j++)
         {
            const T sgn = (it.l & 1) ? T(-1) : T(1);
            if(it.m == 0) { R[tid][2 * j] = sgn * it.are; R[tid][2 * j + 1] = T(0); }
            else { R[tid][2 * j] = sgn * sq2 * it.are; R[tid][2 * j + 1] = sgn * sq2 * it.aim; }
            if(tid == 0)
            {
               kOf[2 * j] = hidx(cl, cm);
               kOf[2 * j + 1] = cm > 0 ? hidx(cl, -cm) : -1;
            }
            if(v0 + j + 1 < nVisits) it.next();
            if(cl < p) cl++;
            else { cm++; cl = cm; }
         }
         vl = cl; vm = cm;
         __syncthreads();
         // reduce over the points: output (column, component) pairs split over the threads
         for(int o = tid; o < 2 * nv * 3; o += NT)
         {
            const int col = o / 3, comp = o - 3 * col;
            const int k = kOf[col];
            if(k < 0) continue;
            T acc = T(0);
            for(int i = 0; i < cnt; i++) acc += Q[i][comp] * R[i][col];
            Macc[comp * Lp + k] += acc;
         }
         __syncthreads();
      }
   }
   T* out = M + int64_t(node) * 3 * Lp;
   for(int e = tid; e < 3 * Lp; e += NT) out[e] = (e % Lp) < L ? Macc[e] : T(0);
}

// ====================================================================================
// P2M, one warp per leaf. Lane (u, c), u < U = p / 2 + 1, c < 3, owns component c of the
// complex coefficients S_l^m of the two orders m_a = u and m_b = p - u (p + 2 values; p / 2 + 1
// when m_a = m_b), so the U units cover every order once and the 3 U <= 27 lanes have equal
// work. The leaf's points go 32 at a time: lane j scales point j to the box and writes its
// diagonal values S_m^m (m = 0..p, the recurrence's first step) to shared memory; then every lane
// walks the points in order, running the l-recurrence of m_a and then of m_b and adding
// q_c S_l^m into registers. Step j of a lane uses the coefficients (a, b, e) of its table row:
//   S_j = a z S_{j-1} - b r^2 S_{j-2} + e S_{m_b}^{m_b}
// with e = 1, a = b = 0 at the step that starts the m_b chain and b = 0 at the first step of
// each chain, so no lane branches. At the end the real coefficients (-1)^l sqrt2 (Re, Im) S_l^m
// (m > 0) and (-1)^l S_l^0 go through shared memory to one coalesced store of the leaf's
// multipole.
// Bound by the issue of the recurrence (a step depends on the last one, 16 warps a SM). Points go two at a time,
// interleaved in shared memory; in FP32 a pair is one packed f32x2 operand of every step (12 instructions a step
// against 21 for two scalar chains), the chain is one FMA deep, the table is kept by u and not by lane, and a
// block serves many leaves per table. 2^24 points in leaves of 18, p = 16: 10.1 -> 8.0 ms; 2^23
// points of 256 coils: 8.1 -> 5.1 ms (128 registers; a chain of scalar operands or the table kept in registers spills).
// ====================================================================================
// A warp's walk over the leaves that hold points: its nodes are first, first + stride, ...; 32 of them are looked at
// together, a lane each, so a leaf's range is in a register when its turn comes and the other nodes cost nothing.
struct LeafWalk
{
   int base, stride;
   unsigned todo = 0;
   int a = 0, b = 0;   // the lane's node
   struct Leaf
   {
      int node, a, b;
   };
   __device__ LeafWalk(int first, int stride_) : base(first - 32 * stride_), stride(stride_) {}
   // The next leaf with [p0, p1) not empty (node < 0: none); all lanes of the warp together.
   __device__ __forceinline__ Leaf next(const Tree& t, const int* __restrict__ p0, const int* __restrict__ p1)
   {
      while(!todo)
      {
         base += 32 * stride;
         if(base >= t.nNodes) return Leaf{-1, 0, 0};
         const int64_t mine = base + int64_t(threadIdx.x & 31) * stride;
         bool in = mine < t.nNodes && t.nchild[mine] == 0;
         if(in)
         {
            a = p0[mine]; b = p1[mine];
            in = b > a;
         }
         todo = __ballot_sync(0xffffffffu, in);
      }
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      return Leaf{base + l * stride, __shfl_sync(0xffffffffu, a, l), __shfl_sync(0xffffffffu, b, l)};
   }
};

// Blocks of a kernel whose warps walk the leaves: every SM filled four times over, so that blocks that meet small
// leaves are replaced, and a block still sets up its tables once for many leaves.
template <class K>
int walkBlocks(K kernel, int threads, size_t shm, int64_t n)
{
   int perSM = 1;
   if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kernel, threads, shm) != cudaSuccess || perSM < 1)
   {
      cudaGetLastError();
      perSM = 1;
   }
   return int(std::max<int64_t>(1, std::min<int64_t>((n + threads / 32 - 1) / (threads / 32), 4 * 148 * int64_t(perSM))));
}

constexpr int P2MW_WARPS = 4;               // a leaf each
constexpr int P2MW_SPLIT_WARPS = 8;         // of one leaf
constexpr int P2MW_STEPS = MAXORDER + 2;
constexpr int P2MW_U = MAXORDER / 2 + 1;   // the step table's row

template <class T>
constexpr size_t p2mTableBytes = (sizeof(T) * P2MW_STEPS * P2MW_U * (sizeof(T) == 4 ? 6 : 3) + 15) / 16 * 16;

// Shared-memory loads that stay where they are written: the step table does not change from pair to pair, and the
// compiler would otherwise keep as many of its rows in registers as fit, and spill.
__device__ __forceinline__ ulonglong2 ldsPair(const void* p)
{
   ulonglong2 v;
   asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(uint32_t(__cvta_generic_to_shared(p))) : "memory");
   return v;
}
__device__ __forceinline__ f2p ldsOne(const void* p)
{
   f2p v;
   asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(uint32_t(__cvta_generic_to_shared(p))) : "memory");
   return v;
}

template <class T>
inline size_t p2mWarpSmem(int p, int Lp, int warps)
{
   const size_t perWarp = 32 * 8 + std::max<size_t>(size_t(32) * 2 * (p + 1), size_t(3) * Lp);
   return p2mTableBytes<T> + sizeof(T) * (warps * perWarp);
}

// SPLIT: the block's warps share one leaf, warp w taking every eighth group of 32 points, and their sums meet in shared
// memory in warp order (few large leaves: 38,400 points in leaves of up to 1000, p = 10, 270 -> 54 us).
template <class T, bool SPLIT>
__global__ void __launch_bounds__(32 * (SPLIT ? P2MW_SPLIT_WARPS : P2MW_WARPS), (sizeof(T) == 4 ? 4 : 3) / (SPLIT ? 2 : 1))
   kP2MWarp(Tree t, const RootBox* __restrict__ rootp, const typename Vec4<T>::type* __restrict__ pos,
            const typename Vec4<T>::type* __restrict__ q, int p, int Lp, T* __restrict__ M,
            uint8_t* __restrict__ Mpieces, int np)
{
   typedef typename Vec4<T>::type V4;
   constexpr bool PK = sizeof(T) == 4;
   constexpr int WARPS = SPLIT ? P2MW_SPLIT_WARPS : P2MW_WARPS;
   extern __shared__ __align__(16) unsigned char smraw[];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int U = p / 2 + 1;
   // the step table, [step][u]: (a, -b), then e; FP32: each value twice, as the packed operands
   T* AB = (T*)smraw;
   T* EE = AB + P2MW_STEPS * P2MW_U * (PK ? 4 : 2);
   const size_t perWarp = 32 * 8 + max(32 * 2 * (p + 1), 3 * Lp);
   T* Pt0 = (T*)(smraw + p2mTableBytes<T>);
   T* Pt = Pt0 + warp * perWarp;                         // [16 pairs][8][2] points: u, r^2, q
   T* Ds = Pt + 32 * 8;                                  // [16][p + 1][re, im][2] S_m^m; later [3][Lp]
   const int u = lane % U, c = min(lane / U, 2);
   const int ma = u, mb = p - u;
   const int jb = p + 2 - U;                             // no lane's m_b chain starts before this step
   for(int e = threadIdx.x; e < P2MW_STEPS * P2MW_U; e += 32 * WARPS)
   {
      const int j = e / P2MW_U, uu = min(e % P2MW_U, U - 1);
      const int a0 = uu, b0 = p - uu, n0 = p + 1 - a0;
      const int n = n0 + (b0 != a0 ? p + 1 - b0 : 0);
      T a = T(0), b = T(0), ee = T(0);
      if(j == n0 && j < n) ee = T(1);
      else if(j > 0 && j < n)
      {
         const int m = j < n0 ? a0 : b0;
         const int l = j < n0 ? a0 + j - 1 : b0 + (j - n0) - 1;
         const T inv = T(1) / T((l - m + 1) * (l + m + 1));
         a = T(2 * l + 1) * inv;
         b = l == m ? T(0) : -inv;
      }
      if constexpr(PK)
      {
         AB[4 * e] = AB[4 * e + 1] = a;
         AB[4 * e + 2] = AB[4 * e + 3] = b;
         EE[2 * e] = EE[2 * e + 1] = ee;
      }
      else
      {
         AB[2 * e] = a;
         AB[2 * e + 1] = b;
         EE[e] = ee;
      }
   }
   __syncthreads();
   // SPLIT: the block's node; else the warp's nodes, dealt out over the grid
   LeafWalk walk(SPLIT ? int(blockIdx.x) : int(blockIdx.x) * WARPS + warp, int(gridDim.x) * (SPLIT ? 1 : WARPS));
   for(;;)
   {
      const LeafWalk::Leaf leaf = walk.next(t, t.s0, t.s1);
      if(leaf.node < 0) break;
      const int node = leaf.node, s0 = leaf.a, s1 = leaf.b;
      double cen[3], h;
      nodeCenter(rootp[rootOf(t, node)], t.level[node], t.ix[node], t.iy[node], t.iz[node], cen, h);
      const double ih = 1.0 / h;
      typedef typename std::conditional<PK, f2p, T>::type Acc;   // FP32: the two points of a pair summed apart
      Acc accR[P2MW_STEPS], accI[P2MW_STEPS];
#pragma unroll
      for(int j = 0; j < P2MW_STEPS; j++) { accR[j] = Acc(0); accI[j] = Acc(0); }
      for(int base = s0 + (SPLIT ? 32 * warp : 0); base < s1; base += SPLIT ? 32 * WARPS : 32)
      {
         const int cnt = min(32, s1 - base);
         if(lane < ((cnt + 1) & ~1))
         {
            // (an odd count's last partner: a zero-strength point at the box centre)
            T x = T(0), y = T(0), z = T(0);
            V4 w{T(0), T(0), T(0), T(0)};
            if(lane < cnt)
            {
               const V4 xp = pos[base + lane];
               w = q[base + lane];
               x = T((double(xp.x) - cen[0]) * ih);
               y = T((double(xp.y) - cen[1]) * ih);
               z = T((double(xp.z) - cen[2]) * ih);
            }
            T* pt = Pt + (lane >> 1) * 16 + (lane & 1);
            pt[0] = x; pt[2] = y; pt[4] = z; pt[6] = x * x + y * y + z * z;
            pt[8] = w.x; pt[10] = w.y; pt[12] = w.z;
            T dre = T(1), dim = T(0);
            T* d = Ds + (lane >> 1) * 4 * (p + 1) + (lane & 1);
            d[0] = dre; d[2] = dim;
#pragma unroll
            for(int m = 1; m <= MAXORDER; m++)
            {
               if(m > p) break;
               const T sc = T(1) / T(2 * m);
               const T nre = (dre * x - dim * y) * sc;
               const T nim = (dre * y + dim * x) * sc;
               dre = nre; dim = nim;
               d[4 * m] = dre; d[4 * m + 2] = dim;
            }
         }
         __syncwarp();
         for(int i = 0; 2 * i < cnt; i++)
         {
            const T* pt = Pt + i * 16;
            const T* d = Ds + i * 4 * (p + 1);
            if constexpr(PK)
            {
               const ulonglong2 da = *(const ulonglong2*)(d + 4 * ma), db = *(const ulonglong2*)(d + 4 * mb);
               const f2p Z = *(const f2p*)(pt + 4), R2 = *(const f2p*)(pt + 6), Q = *(const f2p*)(pt + 8 + 2 * c);
               f2p are = da.x, aim = da.y, bre = 0, bim = 0;
               accR[0] = fma2(Q, are, accR[0]);
               accI[0] = fma2(Q, aim, accI[0]);
#pragma unroll
               for(int j = 1; j < P2MW_STEPS; j++)
               {
                  if(j > p + 1) break;
                  const ulonglong2 k = ldsPair(AB + 4 * (j * P2MW_U + u));
                  const f2p az = mul2(k.x, Z), br = mul2(k.y, R2);
                  f2p tre = mul2(br, bre), tim = mul2(br, bim);
                  if(j >= jb)
                  {
                     const f2p e = ldsOne(EE + 2 * (j * P2MW_U + u));
                     tre = fma2(e, db.x, tre);
                     tim = fma2(e, db.y, tim);
                  }
                  bre = are; bim = aim;
                  are = fma2(az, are, tre);
                  aim = fma2(az, aim, tim);
                  accR[j] = fma2(Q, are, accR[j]);
                  accI[j] = fma2(Q, aim, accI[j]);
               }
            }
            else
            {
               const T z = pt[4], r2 = pt[6], qc = pt[8 + 2 * c], z2 = pt[5], r22 = pt[7], qc2 = pt[9 + 2 * c];
               T are = d[4 * ma], aim = d[4 * ma + 2], are2 = d[4 * ma + 1], aim2 = d[4 * ma + 3];
               const T bdr = d[4 * mb], bdi = d[4 * mb + 2], bdr2 = d[4 * mb + 1], bdi2 = d[4 * mb + 3];
               T bre = T(0), bim = T(0), bre2 = T(0), bim2 = T(0);
               accR[0] += qc * are + qc2 * are2;
               accI[0] += qc * aim + qc2 * aim2;
#pragma unroll
               for(int j = 1; j < P2MW_STEPS; j++)
               {
                  if(j > p + 1) break;
                  const ulonglong2 kk = ldsPair(AB + 2 * (j * P2MW_U + u));
                  const T ka = __longlong_as_double(kk.x), kb = __longlong_as_double(kk.y);
                  const T ke = __longlong_as_double(ldsOne(EE + j * P2MW_U + u));
                  const T az = ka * z, br = kb * r2;
                  const T az2 = ka * z2, br2 = kb * r22;
                  const T cre = ke * bdr + br * bre + az * are;
                  const T cim = ke * bdi + br * bim + az * aim;
                  const T cre2 = ke * bdr2 + br2 * bre2 + az2 * are2;
                  const T cim2 = ke * bdi2 + br2 * bim2 + az2 * aim2;
                  bre = are; bim = aim; are = cre; aim = cim;
                  bre2 = are2; bim2 = aim2; are2 = cre2; aim2 = cim2;
                  accR[j] += qc * are + qc2 * are2;
                  accI[j] += qc * aim + qc2 * aim2;
               }
            }
         }
         __syncwarp();
      }
      auto sum = [](Acc v) -> T {
         if constexpr(PK)
         {
            T a, b;
            upk2(v, a, b);
            return a + b;
         }
         else return v;
      };
      // real coefficients through shared memory, then one coalesced store
      T* Mst = Ds;
      for(int e = (p + 1) * (p + 1) + lane; e < Lp; e += 32) Mst[e] = Mst[Lp + e] = Mst[2 * Lp + e] = T(0);
      if(lane < 3 * U)
      {
         int ma1 = ma;
         asm volatile("" : "+r"(ma1));   // (else every coefficient's address is kept across the leaves)
         const int mb1 = p - ma1, na1 = p + 1 - ma1;
         const int nb = mb1 != ma1 ? p + 1 - mb1 : 0;
         const T sq2 = T(1.4142135623730950488);
#pragma unroll
         for(int j = 0; j < P2MW_STEPS; j++)
         {
            if(j >= na1 + nb) break;
            const int m = j < na1 ? ma1 : mb1;
            const int l = j < na1 ? ma1 + j : mb1 + (j - na1);
            const T sg = (l & 1) ? T(-1) : T(1);
            T* mc = Mst + c * Lp;
            if(m == 0) mc[hidx(l, 0)] = sg * sum(accR[j]);
            else
            {
               mc[hidx(l, m)] = sg * sq2 * sum(accR[j]);
               mc[hidx(l, -m)] = sg * sq2 * sum(accI[j]);
            }
         }
      }
      __syncwarp();
      T* out = M + int64_t(node) * 3 * Lp;
      if(SPLIT)
      {
         // the warps' sums into the first warp's
         __syncthreads();
         T* first = Pt0 + 32 * 8;
         for(int e = threadIdx.x; e < 3 * Lp; e += 32 * WARPS)
         {
            T v = first[e];
            for(int w = 1; w < WARPS; w++) v += first[w * perWarp + e];
            first[e] = v;
         }
         __syncthreads();
         if(warp) continue;   // (no further leaf)
      }
      for(int e = lane; e < 3 * Lp; e += 32) out[e] = Mst[e];
      // the same coefficients as tensor-core operand pieces (the M2M's and M2L's input format), so the
      // upward pass needs no separate split of the leaves
      if constexpr(sizeof(T) == 4)
         if(Mpieces)
            for(int d = 0; d < 3; d++)
               for(int e = 4 * lane; e < Lp; e += 128)
                  storePieces4(Mpieces, int64_t(node) * 3 + d, e, Lp, np, *(const float4*)(Mst + d * Lp + e));
      __syncwarp();
   }
}

__device__ __forceinline__ void cpAsync16Simt(void* dst, const void* src, uint32_t srcBytes)
{
   const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
   asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(srcBytes) : "memory");
}

// ====================================================================================
// L2P + near field: one block per target leaf. The local expansion is turned into the
// expansion of B = curl A (order p - 1) in shared memory, evaluated per target by the
// harmonic recurrence, then the direct sum over the leaf's source list is added.
//
// Real-basis derivatives used for the curl (R = regular harmonics, standard convention):
//   d/dz R_l^{+-m} = -R_{l-1}^{+-m}
//   d/dx, d/dy move m by one; see gradCoeff below.
// ====================================================================================
template <class T>
__device__ inline T coefAt(const T* Lv, int l, int m)
{
   return (abs(m) <= l) ? Lv[hidx(l, m)] : T(0);
}

// Coefficient of R_{l'}^{mu} in d/dx_j (sum_k L_k R_k), j = 0 (x), 1 (y), 2 (z); l = l' + 1.
template <class T>
__device__ inline T gradCoeff(const T* Lv, int j, int lp, int mu)
{
   const int l = lp + 1;
   const T h = T(0.5), r2 = T(0.70710678118654752440);
   if(j == 2) return -coefAt(Lv, l, mu);
   if(j == 0)
   {
      if(mu == 0) return -r2 * coefAt(Lv, l, 1);
      if(mu == 1) return -h * coefAt(Lv, l, 2) + r2 * coefAt(Lv, l, 0);
      if(mu >= 2) return -h * coefAt(Lv, l, mu + 1) + h * coefAt(Lv, l, mu - 1);
      if(mu == -1) return -h * coefAt(Lv, l, -2);
      return -h * coefAt(Lv, l, mu - 1) + h * coefAt(Lv, l, mu + 1);
   }
   if(mu == 0) return -r2 * coefAt(Lv, l, -1);
   if(mu == 1) return -h * coefAt(Lv, l, -2);
   if(mu >= 2) return -h * coefAt(Lv, l, -(mu + 1)) - h * coefAt(Lv, l, -(mu - 1));
   if(mu == -1) return h * coefAt(Lv, l, 2) + r2 * coefAt(Lv, l, 0);
   return h * coefAt(Lv, l, 1 - mu) + h * coefAt(Lv, l, -mu - 1);
}

// 1/sqrt(x) by the PTX approximate reciprocal square root (flushes subnormal inputs to zero).
__device__ __forceinline__ float rsqrtApprox(float x)
{
   float y;
   asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
   return y;
}
__device__ __forceinline__ void cpAsync4(void* dst, const void* src, uint32_t srcBytes)
{
   const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
   asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(srcBytes) : "memory");
}
// Bytes of one near-field source tile of TS points: FP32 tiles hold source pairs
// [x0 x1 y0 y1 z0 z1 wx0 wx1 wy0 wy1 wz0 wz1] (24 bytes a point), FP64 tiles two [TS] arrays of
// (x, y, z, -) and (wx, wy, wz, -).
template <class T>
__host__ __device__ constexpr int nearTileBytes(int TS)
{
   return sizeof(T) == 4 ? 24 * TS : 2 * 4 * int(sizeof(T)) * TS;
}

// Largest 1/r whose cube is finite in T, for the coincident-pair cap of the near field.
template <class T> __device__ __forceinline__ T riCap();
template <> __device__ __forceinline__ float riCap<float>() { return 6.0e12f; }
template <> __device__ __forceinline__ double riCap<double>() { return 1.0e100; }

// L2P alone, one warp per target leaf, one target per lane (32 at a time). The leaf's curl
// expansion (and, for A, its local expansion) is stored as [k] (x, y, z, 0) with the real-basis
// factors (-1)^l sqrt2 folded in, so each visited harmonic costs one broadcast 16-byte shared
// load and three FMAs per coefficient. The recurrence's coefficients come from a table shared by
// the block (visit order: m outer, l inner): 1/(2m) at l = m, else the (a, b) of
// S_l^m = a z S_{l-1}^m - b r^2 S_{l-2}^m, so no lane divides. The far field is written to the
// outputs unscaled; kL2PNear<..., FAR = false> adds the near field and applies the scale.
// Bound by latency (a leaf's setup, then a recurrence with shared-memory loads in its chain): a warp walks many leaves,
// so the table is built once, and the next leaf's local row is on its way while this one is evaluated. 2^24 targets,
// p = 16: 12.5 -> 11.3 ms; 2^23 targets of 256 coils: 3.6 -> 2.1 ms (against four leaves a block, loaded in turn).
constexpr int L2PW_WARPS = 4;

template <class T, bool WANTA>
inline size_t l2pWarpSmem(int p)
{
   const int L = nharm(p), Lb = nharm(p - 1), nV = (p + 1) * (p + 2) / 2;
   const size_t perWarp = size_t(4) * Lb + (WANTA ? size_t(4) * L : 0) + size_t(3) * padded(L);
   return sizeof(T) * (size_t(4) * nV + L2PW_WARPS * perWarp);
}

template <class T, bool WANTA>
__global__ void __launch_bounds__(32 * L2PW_WARPS, sizeof(T) == 4 ? (WANTA ? 5 : 6) : 3) kL2PWarp(Tree t, const RootBox* __restrict__ rootp, int p,
                                                          int Lp, const T* __restrict__ Lc,
                                                          const typename Vec4<T>::type* __restrict__ tpos,
                                                          const int* __restrict__ tOrder,
                                                          const CurlEntry<T>* __restrict__ curl, int want,
                                                          T* __restrict__ outB, T* __restrict__ outA)
{
   typedef typename Vec4<T>::type V4;
   extern __shared__ __align__(16) unsigned char smraw[];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int L = nharm(p), Lb = nharm(p - 1);
   const int q = WANTA ? p : p - 1;                     // highest degree visited
   const int nV = (p + 1) * (p + 2) / 2;                // table: degrees 0..p
   V4* tab = (V4*)smraw;
   const int perWarp = 4 * Lb + (WANTA ? 4 * L : 0) + 3 * Lp;
   T* wbase = (T*)(tab + nV) + warp * perWarp;
   V4* Cs = (V4*)wbase;                                 // [Lb] curl expansion
   V4* As = Cs + Lb;                                    // [L] local expansion (WANTA)
   T* Ls = wbase + 4 * Lb + (WANTA ? 4 * L : 0);        // [3][Lp] the box's local row
   for(int v = threadIdx.x; v < nV; v += 32 * L2PW_WARPS)
   {
      int m = 0, r = v;
      while(r >= p + 1 - m) { r -= p + 1 - m; m++; }
      const int l = m + r;
      T a = T(0), b = T(0);
      if(l == m) a = m > 0 ? T(1) / T(2 * m) : T(1);
      else
      {
         const int lp = l - 1;
         const T inv = T(1) / T((lp - m + 1) * (lp + m + 1));
         a = T(2 * lp + 1) * inv;
         b = lp == m ? T(0) : inv;
      }
      tab[v] = V4{a, b, T(0), T(0)};
   }
   __syncthreads();
   // a box's local row copied asynchronously (Lp is a multiple of 16): the next leaf's while this one is evaluated
   auto fetch = [&](int node) {
      if(node >= 0)
      {
         const char* src = (const char*)(Lc + int64_t(node) * 3 * Lp);
         for(int e = 16 * lane; e < 3 * Lp * int(sizeof(T)); e += 512) cpAsync16Simt((char*)Ls + e, src + e, 16u);
      }
   };
   LeafWalk walk(int(blockIdx.x) * L2PW_WARPS + warp, int(gridDim.x) * L2PW_WARPS);
   LeafWalk::Leaf leaf = walk.next(t, t.t0, t.t1);
   fetch(leaf.node);
   while(leaf.node >= 0)
   {
      const int node = leaf.node, t0 = leaf.a, t1 = leaf.b;
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      const T* lc = Ls;
      // the curl expansion from the table: each entry <= 4 terms of the box's local row
#pragma unroll 4
      for(int e = lane; e < 4 * Lb; e += 32)
      {
         const CurlEntry<T> ce = curl[e];
         ((T*)Cs)[e] = ce.c[0] * lc[ce.idx[0]] + ce.c[1] * lc[ce.idx[1]] + ce.c[2] * lc[ce.idx[2]] +
                       ce.c[3] * lc[ce.idx[3]];
      }
      if(WANTA)
      {
         const T sq2 = T(1.4142135623730950488);
         for(int e = lane; e < 4 * L; e += 32)
         {
            const int k = e >> 2, c = e & 3;
            int l = int(sqrtf(float(k)));
            while(l * l > k) l--;
            while((l + 1) * (l + 1) <= k) l++;
            const int mu = k - l * l - l;
            const T f = ((l & 1) ? T(-1) : T(1)) * (mu != 0 ? sq2 : T(1));
            ((T*)As)[e] = c < 3 ? f * lc[c * Lp + k] : T(0);
         }
      }
      __syncwarp();
      double cen[3], h;
      nodeCenter(rootp[rootOf(t, node)], t.level[node], t.ix[node], t.iy[node], t.iz[node], cen, h);
      leaf = walk.next(t, t.t0, t.t1);
      fetch(leaf.node);
      const T ih = T(1.0 / h), ih2 = T(1.0 / (h * h));
      // G lanes per target when the leaf is small (G = 4 up to 8 targets, 2 up to 16): group g of the
      // W = 32 / G lanes visits the orders m = g, g + G, ..., and the groups' sums meet by shuffles
      const int nt = t1 - t0;
      const int G = nt <= 8 ? 4 : (nt <= 16 ? 2 : 1), W = 32 / G;
      const int g = lane / W, jl = lane % W;
      auto vStart = [&](int m) { return m * (p + 1) - m * (m - 1) / 2; };   // first visit of order m
      for(int base = t0; base < t1; base += W)
      {
         const int ti = base + jl;
         const bool act = ti < t1;
         const V4 x = act ? tpos[ti] : V4{T(0), T(0), T(0), T(0)};
         const T ux = T((double(x.x) - cen[0]) / h), uy = T((double(x.y) - cen[1]) / h),
                 uz = T((double(x.z) - cen[2]) / h);
         const T r2 = ux * ux + uy * uy + uz * uz;
         T B0 = T(0), B1 = T(0), B2 = T(0), A0 = T(0), A1 = T(0), A2 = T(0);
         T dre = T(1), dim = T(0);   // S_m^m, advanced to this group's first order
         for(int j = 1; j <= g; j++)
         {
            const T sc = tab[vStart(j)].x;
            const T nre = (dre * ux - dim * uy) * sc;
            const T nim = (dre * uy + dim * ux) * sc;
            dre = nre; dim = nim;
         }
         // S_l^0 stays real (the imaginary parts are zero), so order 0 needs no case of its own: its
         // k1 = k0 term adds zero
         // the contribution of one visited harmonic (l, m): coefficients k0 = hidx(l, m), k1 = hidx(l, -m)
         auto visit = [&](int l, int k0, int k1, T are, T aim) {
            if(!WANTA || l < p)
            {
               const V4 c0 = Cs[k0], c1 = Cs[k1];
               B0 += c0.x * are + c1.x * aim; B1 += c0.y * are + c1.y * aim; B2 += c0.z * are + c1.z * aim;
            }
            if(WANTA)
            {
               const V4 a0 = As[k0], a1 = As[k1];
               A0 += a0.x * are + a1.x * aim; A1 += a0.y * are + a1.y * aim; A2 += a0.z * are + a1.z * aim;
            }
         };
         // S_{j-1}^{j-1} -> S_j^j
         auto diag = [&](T& re, T& im, int j) {
            const T sc = tab[vStart(j)].x;
            const T nre = (re * ux - im * uy) * sc;
            const T nim = (re * uy + im * ux) * sc;
            re = nre; im = nim;
         };
         // orders m and m2 = m + G walked together: two independent recurrences in flight per lane
         for(int m = g; m <= q; m += 2 * G)
         {
            const int m2 = m + G;
            const bool two = m2 <= q;
            T e2re = dre, e2im = dim;   // S_{m2}^{m2}
            for(int j = m + 1; j <= m2 && j <= q; j++) diag(e2re, e2im, j);
            int v = vStart(m), v2 = two ? vStart(m2) : 0;
            T are = dre, aim = dim, bre = T(0), bim = T(0);
            T are2 = e2re, aim2 = e2im, bre2 = T(0), bim2 = T(0);
            int k0 = m * m + 2 * m, k1 = m * m, k02 = m2 * m2 + 2 * m2, k12 = m2 * m2;
            visit(m, k0, k1, are, aim);
            v++;
            if(two)
            {
               visit(m2, k02, k12, are2, aim2);
               v2++;
            }
            const int n2 = two ? q - m2 : 0;   // steps both orders take
#pragma unroll 2
            for(int st = 1; st <= n2; st++, v++, v2++)
            {
               const int l = m + st, l2 = m2 + st;
               const V4 ab = tab[v], ab2 = tab[v2];
               k0 += 2 * l; k1 += 2 * l; k02 += 2 * l2; k12 += 2 * l2;
               const T az = ab.x * uz, br = ab.y * r2, az2 = ab2.x * uz, br2 = ab2.y * r2;
               const T cre = az * are - br * bre, cim = az * aim - br * bim;
               const T cre2 = az2 * are2 - br2 * bre2, cim2 = az2 * aim2 - br2 * bim2;
               bre = are; bim = aim; are = cre; aim = cim;
               bre2 = are2; bim2 = aim2; are2 = cre2; aim2 = cim2;
               visit(l, k0, k1, are, aim);
               visit(l2, k02, k12, are2, aim2);
            }
            // the rest of order m (all of it when m2 > q)
#pragma unroll 4
            for(int l = m + n2 + 1; l <= q; l++, v++)
            {
               const V4 ab = tab[v];
               k0 += 2 * l; k1 += 2 * l;
               const T az = ab.x * uz, br = ab.y * r2;
               const T cre = az * are - br * bre, cim = az * aim - br * bim;
               bre = are; bim = aim; are = cre; aim = cim;
               visit(l, k0, k1, are, aim);
            }
            // S_m^m -> S_{m+2G}^{m+2G}
            dre = e2re; dim = e2im;
            for(int j = m2 + 1; j <= m2 + G && j <= q; j++) diag(dre, dim, j);
         }
         for(int off = 16; off >= W; off >>= 1)
         {
            B0 += __shfl_down_sync(0xffffffffu, B0, off);
            B1 += __shfl_down_sync(0xffffffffu, B1, off);
            B2 += __shfl_down_sync(0xffffffffu, B2, off);
            if(WANTA)
            {
               A0 += __shfl_down_sync(0xffffffffu, A0, off);
               A1 += __shfl_down_sync(0xffffffffu, A1, off);
               A2 += __shfl_down_sync(0xffffffffu, A2, off);
            }
         }
         if(act && g == 0)
         {
            const int o = tOrder[ti];
            if(want & 1)
            {
               outB[3 * int64_t(o)] = B0 * ih2; outB[3 * int64_t(o) + 1] = B1 * ih2; outB[3 * int64_t(o) + 2] = B2 * ih2;
            }
            if(WANTA)
            {
               outA[3 * int64_t(o)] = A0 * ih; outA[3 * int64_t(o) + 1] = A1 * ih; outA[3 * int64_t(o) + 2] = A2 * ih;
            }
         }
      }
   }
}

// L2P and the direct near field: one block of NT threads per target leaf. The far field comes from
// the leaf's local expansion (analytic curl, one target per thread). The near field packs the
// points of the leaf's direct-interaction source nodes into shared tiles of TS points; when the
// leaf has fewer targets than threads, the G = NT / targets thread groups each take every G-th
// source of a tile and their partial sums are added in a fixed order at the end. Each thread
// sums one tile in T and the tile sums in FP64, so no single-precision chain is longer than a tile.
template <class T, int NT, int TS, int NE, bool WANTA, bool FAR>
__global__ void __launch_bounds__(NT, FAR ? 1 : (sizeof(T) == 4 ? (WANTA ? 12 : 16) : 8) * 64 / NT) kL2PNear(Tree t, const RootBox* __restrict__ rootp, int p, int Lp,
                                               const T* __restrict__ Lc,
                                               const typename Vec4<T>::type* __restrict__ tpos,
                                               const typename Vec4<T>::type* __restrict__ spos,
                                               const typename Vec4<T>::type* __restrict__ sq,
                                               const int* __restrict__ p2pOff, const int* __restrict__ p2pList,
                                               const int* __restrict__ tOrder, T scaleB, T scaleA, int want,
                                               T* __restrict__ outB, T* __restrict__ outA, double* __restrict__ part,
                                               int mTargets)
{
   typedef typename Vec4<T>::type V4;
   extern __shared__ __align__(32) unsigned char smraw[];
   const int node = blockIdx.x;
   // the tiles of a leaf's list dealt out to gridDim.y blocks (!FAR); their sums then go to part
   const int nParts = FAR ? 1 : int(gridDim.y), myPart = FAR ? 0 : int(blockIdx.y);
   if(t.nchild[node] != 0 || t.t1[node] == t.t0[node]) return;
   const int tid = threadIdx.x;
   const int L = nharm(p);
   const int Lb = nharm(p - 1);
   T* Ls = (T*)smraw;          // [3][L] local
   T* Cs = Ls + 3 * L;         // [3][Lb] curl expansion
   // source tiles start on a 32-byte boundary after the two coefficient arrays (none without FAR)
   const size_t coefBytes = FAR ? (sizeof(T) * (3 * L + 3 * Lb) + 31) & ~size_t(31) : 0;
   unsigned char* tiles = smraw + coefBytes;                          // two source tiles
   double* red = (double*)(tiles + 2 * nearTileBytes<T>(TS));        // [6][NT] group partial sums
   typedef cub::BlockScan<int, NT> ScanT;
   __shared__ typename ScanT::TempStorage scanTmp;
   __shared__ int ePre[NE + 1];        // prefix sums of the batch's source counts
   __shared__ int eSrc[NE];            // first sorted source of each batch entry
   if(FAR)
   {
   for(int e = tid; e < 3 * L; e += NT) Ls[e] = Lc[int64_t(node) * 3 * Lp + (e / L) * Lp + e % L];
   __syncthreads();
   for(int e = tid; e < 3 * Lb; e += NT)
   {
      const int c = e / Lb, k = e % Lb;
      int lp = int(sqrtf(float(k)));
      while(lp * lp > k) lp--;
      while((lp + 1) * (lp + 1) <= k) lp++;
      const int mu = k - lp * lp - lp;
      // B_x = dAz/dy - dAy/dz, B_y = dAx/dz - dAz/dx, B_z = dAy/dx - dAx/dy
      const int cp = (c + 2) % 3, cm = (c + 1) % 3;   // (z,y) for x; (x,z) for y; (y,x) for z
      const int jp = (c + 1) % 3, jm = (c + 2) % 3;
      Cs[e] = gradCoeff(Ls + cp * L, jp, lp, mu) - gradCoeff(Ls + cm * L, jm, lp, mu);
   }
   __syncthreads();
   }
   const RootBox rb = rootp[rootOf(t, node)];
   double c[3], h;
   nodeCenter(rb, t.level[node], t.ix[node], t.iy[node], t.iz[node], c, h);
   const T ih = T(1.0 / h), ih2 = T(1.0 / (h * h));
   const int t0 = t.t0[node], t1 = t.t1[node];
   const int e0 = p2pOff[node], e1 = p2pOff[node + 1];
   constexpr bool wantA = WANTA;
   for(int base = t0; base < t1; base += NT)
   {
      const int nt = min(NT, t1 - base);     // targets in this pass
      const int G = NT / nt;                 // thread groups sharing a tile's sources
      const int tt = tid % nt, g = tid / nt;
      const bool inGroup = g < G;
      const int ti = base + tt;
      V4 x = inGroup ? tpos[ti] : V4{T(0), T(0), T(0), T(0)};
      double Bd[3] = {0, 0, 0}, Ad[3] = {0, 0, 0};
      if(!FAR && inGroup && g == 0 && nParts == 1)
      {
         // the far field, already evaluated by kL2PWarp into the outputs (unscaled)
         const int o = tOrder[ti];
         if(want & 1) for(int d = 0; d < 3; d++) Bd[d] = double(outB[3 * int64_t(o) + d]);
         if(WANTA) for(int d = 0; d < 3; d++) Ad[d] = double(outA[3 * int64_t(o) + d]);
      }
      if(FAR && inGroup && g == 0)
      {
         T B[3] = {T(0), T(0), T(0)}, A[3] = {T(0), T(0), T(0)};
         const T ux = T((double(x.x) - c[0]) / h), uy = T((double(x.y) - c[1]) / h), uz = T((double(x.z) - c[2]) / h);
         const T sq2 = T(1.4142135623730950488);
         visitRegular<T>(p, ux, uy, uz, [&](int l, int m, T re, T im) {
            const T s = (l & 1) ? T(-1) : T(1);
            T r0, r1;
            if(m == 0) { r0 = s * re; r1 = T(0); }
            else { r0 = s * sq2 * re; r1 = s * sq2 * im; }
            if(l < p)
            {
               const int k0 = hidx(l, m), k1 = hidx(l, -m);
               for(int d = 0; d < 3; d++)
               {
                  B[d] += Cs[d * Lb + k0] * r0;
                  if(m) B[d] += Cs[d * Lb + k1] * r1;
               }
            }
            if(wantA)
            {
               const int k0 = hidx(l, m), k1 = hidx(l, -m);
               for(int d = 0; d < 3; d++)
               {
                  A[d] += Ls[d * L + k0] * r0;
                  if(m) A[d] += Ls[d * L + k1] * r1;
               }
            }
         });
         for(int d = 0; d < 3; d++) { Bd[d] = double(B[d] * ih2); Ad[d] = double(A[d] * ih); }
      }
      // near field over packed tiles of the direct-list source nodes
      auto tileSum = [&](int n, int b) {
         if(!inGroup) return;
         T pb[3] = {T(0), T(0), T(0)}, pa[3] = {T(0), T(0), T(0)};
         if constexpr(sizeof(T) == 4)
         {
            // two sources per step in packed f32x2 arithmetic; the cross product's two products are
            // accumulated in separate sums (no negation in the packed FMA)
            const ulonglong2* tq = (const ulonglong2*)(tiles + b * nearTileBytes<T>(TS));
            const int nPairs = (n + 1) >> 1;
            const f2p X = pk2(x.x, x.x), Y = pk2(x.y, x.y), Z = pk2(x.z, x.z);
            f2p sxp = 0, sxn = 0, syp = 0, syn = 0, szp = 0, szn = 0, ax = 0, ay = 0, az = 0;
#pragma unroll 2
            for(int P = g; P < nPairs; P += G)
            {
               const ulonglong2 q0 = tq[3 * P], q1 = tq[3 * P + 1], q2 = tq[3 * P + 2];
               const f2p DX = sub2(X, q0.x), DY = sub2(Y, q0.y), DZ = sub2(Z, q1.x);
               f2p R2 = mul2(DX, DX);
               R2 = fma2(DY, DY, R2);
               R2 = fma2(DZ, DZ, R2);
               float r2a, r2b;
               upk2(R2, r2a, r2b);
               float ria = rsqrtApprox(r2a), rib = rsqrtApprox(r2b);
               // coincident pair (the target itself) and the empty slot of an odd tile: no
               // contribution. For B the capped 1/r (whose cube still fits a float) meets a zero
               // difference vector or a zero weight; A needs the explicit test.
               if constexpr(WANTA)
               {
                  ria = r2a > 0.f ? ria : 0.f;
                  rib = r2b > 0.f ? rib : 0.f;
               }
               else
               {
                  ria = fminf(ria, riCap<float>());
                  rib = fminf(rib, riCap<float>());
               }
               const f2p RI = pk2(ria, rib);
               const f2p RI3 = mul2(mul2(RI, RI), RI);
               const f2p UX = mul2(q1.y, RI3), UY = mul2(q2.x, RI3), UZ = mul2(q2.y, RI3);
               sxp = fma2(UY, DZ, sxp); sxn = fma2(UZ, DY, sxn);
               syp = fma2(UZ, DX, syp); syn = fma2(UX, DZ, syn);
               szp = fma2(UX, DY, szp); szn = fma2(UY, DX, szn);
               if constexpr(WANTA)
               {
                  ax = fma2(q1.y, RI, ax); ay = fma2(q2.x, RI, ay); az = fma2(q2.y, RI, az);
               }
            }
            float u0, u1, v0, v1;
            upk2(sxp, u0, u1); upk2(sxn, v0, v1); pb[0] = (u0 + u1) - (v0 + v1);
            upk2(syp, u0, u1); upk2(syn, v0, v1); pb[1] = (u0 + u1) - (v0 + v1);
            upk2(szp, u0, u1); upk2(szn, v0, v1); pb[2] = (u0 + u1) - (v0 + v1);
            if constexpr(WANTA)
            {
               upk2(ax, u0, u1); pa[0] = u0 + u1;
               upk2(ay, u0, u1); pa[1] = u0 + u1;
               upk2(az, u0, u1); pa[2] = u0 + u1;
            }
         }
         else
         {
            const V4* tp = (const V4*)(tiles + b * nearTileBytes<T>(TS));
            const V4* tq = tp + TS;
#pragma unroll 4
            for(int i = g; i < n; i += G)
            {
               const V4 y = tp[i], w = tq[i];
               const T dx = x.x - y.x, dy = x.y - y.y, dz = x.z - y.z;
               const T r2 = dx * dx + dy * dy + dz * dz;
               T ri = rsqrt(r2);
               if constexpr(WANTA) ri = r2 > T(0) ? ri : T(0);
               else ri = min(ri, riCap<T>());
               const T ri3 = ri * ri * ri;
               pb[0] += (w.y * dz - w.z * dy) * ri3;
               pb[1] += (w.z * dx - w.x * dz) * ri3;
               pb[2] += (w.x * dy - w.y * dx) * ri3;
               if(wantA) { pa[0] += w.x * ri; pa[1] += w.y * ri; pa[2] += w.z * ri; }
            }
         }
         for(int d = 0; d < 3; d++) { Bd[d] += double(pb[d]); Ad[d] += double(pa[d]); }
      };
      // the list in batches of NE entries: their point ranges are read together into shared memory
      // and prefix-summed, so every tile position finds its source by a shared-memory search and
      // all of a tile's loads are independent
      int firstTile = myPart;   // this block's first tile of the batch
      for(int eb = e0; eb < e1; eb += NE)
      {
         const int ne = min(NE, e1 - eb);
         int sz[NE / NT];
#pragma unroll
         for(int r = 0; r < NE / NT; r++)
         {
            const int k = tid * (NE / NT) + r;
            int a = 0, n = 0;
            if(k < ne)
            {
               const int S = p2pList[eb + k];
               a = t.s0[S];
               n = t.s1[S] - a;
            }
            if(k < NE) eSrc[k] = a;
            sz[r] = n;
         }
         int total;
         ScanT(scanTmp).ExclusiveSum(sz, sz, total);
#pragma unroll
         for(int r = 0; r < NE / NT; r++) ePre[tid * (NE / NT) + r] = sz[r];
         if(tid == 0) ePre[NE] = total;
         __syncthreads();
         // tiles double-buffered: tile k + 1's copies (cp.async) are in flight while tile k is summed
         auto issueTile = [&](int pos, int b) {
            const int n = min(TS, total - pos);
            const int nf = sizeof(T) == 4 ? (n + 1) & ~1 : n;   // FP32: the odd tile's last pair slot zero-filled
            unsigned char* tb = tiles + b * nearTileBytes<T>(TS);
            for(int j = tid; j < nf; j += NT)
            {
               const bool in = j < n;
               int src = 0;
               if(in)
               {
                  const int qpos = pos + j;
                  int lo = 0, hi = ne;  // last entry with ePre <= qpos
                  while(hi - lo > 1)
                  {
                     const int mid = (lo + hi) >> 1;
                     if(ePre[mid] <= qpos) lo = mid;
                     else hi = mid;
                  }
                  src = eSrc[lo] + (qpos - ePre[lo]);
               }
               if constexpr(sizeof(T) == 4)
               {
                  float* d = (float*)tb + 12 * (j >> 1) + (j & 1);
                  const float* ps = (const float*)(spos + src);
                  const float* qs = (const float*)(sq + src);
                  const uint32_t by = in ? 4u : 0u;
                  cpAsync4(d, ps, by); cpAsync4(d + 2, ps + 1, by); cpAsync4(d + 4, ps + 2, by);
                  cpAsync4(d + 6, qs, by); cpAsync4(d + 8, qs + 1, by); cpAsync4(d + 10, qs + 2, by);
               }
               else
               {
                  V4* tp = (V4*)tb;
#pragma unroll
                  for(int h = 0; h < int(sizeof(V4)) / 16; h++)
                  {
                     cpAsync16Simt((char*)(tp + j) + 16 * h, (const char*)(spos + src) + 16 * h, 16u);
                     cpAsync16Simt((char*)(tp + TS + j) + 16 * h, (const char*)(sq + src) + 16 * h, 16u);
                  }
               }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
         };
         const int nTiles = (total + TS - 1) / TS;
         if(firstTile < nTiles) issueTile(firstTile * TS, 0);
         int k = firstTile;
         for(int b = 0; k < nTiles; k += nParts, b ^= 1)
         {
            if(k + nParts < nTiles)
            {
               issueTile((k + nParts) * TS, b ^ 1);
               asm volatile("cp.async.wait_group 1;" ::: "memory");
            }
            else
               asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            tileSum(min(TS, total - k * TS), b);
            __syncthreads();
         }
         firstTile = k - nTiles;
         // (a block without a tile in this batch must not overwrite its prefix sums while others read them)
         if(nParts > 1) __syncthreads();
      }
      // add the groups' partial sums in group order
      if(G > 1)
      {
         for(int d = 0; d < 3; d++)
         {
            red[d * NT + tid] = Bd[d];
            if(WANTA) red[(3 + d) * NT + tid] = Ad[d];
         }
         __syncthreads();
         if(g == 0)
            for(int gg = 1; gg < G; gg++)
               for(int d = 0; d < 3; d++)
               {
                  Bd[d] += red[d * NT + gg * nt + tt];
                  if(WANTA) Ad[d] += red[(3 + d) * NT + gg * nt + tt];
               }
         __syncthreads();
      }
      if(g == 0 && nParts > 1)
      {
         double* o = part + int64_t(myPart) * 6 * mTargets + ti;
         for(int d = 0; d < 3; d++)
         {
            o[int64_t(d) * mTargets] = Bd[d];
            if(WANTA) o[int64_t(3 + d) * mTargets] = Ad[d];
         }
      }
      else if(g == 0)
      {
         const int o = tOrder[ti];
         if(want & 1) for(int d = 0; d < 3; d++) outB[3 * int64_t(o) + d] = T(Bd[d] * double(scaleB));
         if(want & 2) for(int d = 0; d < 3; d++) outA[3 * int64_t(o) + d] = T(Ad[d] * double(scaleA));
      }
   }
}

// The outputs' far field plus the near field's parts in order, scaled (kL2PNear with gridDim.y > 1).
template <class T>
__global__ void kNearParts(const double* __restrict__ part, int parts, int m, const int* __restrict__ tOrder, T scaleB, T scaleA,
                           int want, T* __restrict__ outB, T* __restrict__ outA)
{
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if(i >= m) return;
   const int64_t o = 3 * int64_t(tOrder[i]);
   for(int c = 0; c < 6; c++)
   {
      if(!(want & (c < 3 ? 1 : 2))) continue;
      T* out = c < 3 ? outB + o + c : outA + o + c - 3;
      double v = double(*out);
      for(int q = 0; q < parts; q++) v += part[(int64_t(q) * 6 + c) * m + i];
      *out = T(v * double(c < 3 ? scaleB : scaleA));
   }
}

// ====================================================================================
// Direct sums over all sources (fmm_direct): one thread per target, sources staged through shared memory in the
// arithmetic's type. The sources of a coil are split over blockIdx.z where the targets alone leave the chip
// idle; a part's sums then go to part[z][6][targets] and kDirectSum adds the parts in order.
// Bound: the FP64 (FP32) pipe, about 30 FP64 instructions a pair with the library's rsqrt. With 1 / sqrt, the
// potential summed whether wanted or not and no split, 38,400 sources x 10,000 targets in FP64 took 6.5 ms.
// ====================================================================================
template <class U> __device__ __forceinline__ U rsqrtOf(U x);
template <> __device__ __forceinline__ float rsqrtOf<float>(float x) { return rsqrtf(x); }
template <> __device__ __forceinline__ double rsqrtOf<double>(double x) { return rsqrt(x); }

template <class T, class U, int NT, bool WANTB, bool WANTA>
__global__ void __launch_bounds__(NT) kDirect(const typename Vec4<T>::type* __restrict__ spos,
                                              const typename Vec4<T>::type* __restrict__ sq, int n,
                                              const U* __restrict__ tgt, int m, const int* __restrict__ sseg,
                                              const int* __restrict__ tseg, U scaleB, U scaleA, U* __restrict__ outB,
                                              U* __restrict__ outA, U* __restrict__ part)
{
   typedef typename Vec4<U>::type U4;
   __shared__ U4 Sp[NT];          // x, y, z, s_x
   __shared__ U Sy[NT][2];        // s_y, s_z
   // blockIdx.y selects a coil: its targets [tseg[c], tseg[c+1]) see only its sources
   // [sseg[c], sseg[c+1]); without segments every target sees every source
   const int c = blockIdx.y;
   const int tBeg = tseg ? tseg[c] : 0, tEnd = tseg ? tseg[c + 1] : m;
   const int s0 = sseg ? sseg[c] : 0, s1 = sseg ? sseg[c + 1] : n;
   const int ti = tBeg + blockIdx.x * NT + threadIdx.x;
   if(tBeg + int(blockIdx.x) * NT >= tEnd) return;
   const int sBeg = s0 + int(int64_t(s1 - s0) * blockIdx.z / gridDim.z);
   const int sEnd = s0 + int(int64_t(s1 - s0) * (blockIdx.z + 1) / gridDim.z);
   const bool active = ti < tEnd;
   U x = 0, y = 0, z = 0;
   if(active) { x = tgt[3 * int64_t(ti)]; y = tgt[3 * int64_t(ti) + 1]; z = tgt[3 * int64_t(ti) + 2]; }
   U B[3] = {0, 0, 0}, A[3] = {0, 0, 0};
   auto add = [&](U sx, U sy, U sz, U dx, U dy, U dz, U ri) {
      if constexpr(WANTB)
      {
         const U ri3 = ri * ri * ri;
         B[0] += (sy * dz - sz * dy) * ri3;
         B[1] += (sz * dx - sx * dz) * ri3;
         B[2] += (sx * dy - sy * dx) * ri3;
      }
      if constexpr(WANTA) { A[0] += sx * ri; A[1] += sy * ri; A[2] += sz * ri; }
   };
   for(int sb = sBeg; sb < sEnd; sb += NT)
   {
      const int cnt = min(NT, sEnd - sb);
      __syncthreads();
      if(threadIdx.x < cnt)
      {
         const auto a = spos[sb + threadIdx.x];
         const auto b = sq[sb + threadIdx.x];
         Sp[threadIdx.x] = U4{U(a.x), U(a.y), U(a.z), U(b.x)};
         Sy[threadIdx.x][0] = U(b.y);
         Sy[threadIdx.x][1] = U(b.z);
      }
      __syncthreads();
      if(active)
#pragma unroll 4
         for(int i = 0; i < cnt; i++)
         {
            const U4 p = Sp[i];
            const U dx = x - p.x, dy = y - p.y, dz = z - p.z;
            const U r2 = dx * dx + dy * dy + dz * dz;
            add(p.w, Sy[i][0], Sy[i][1], dx, dy, dz, r2 == U(0) ? U(0) : rsqrtOf<U>(r2));
         }
   }
   // Coincident pairs are skipped: by a factor of zero, or, if that left a sum that is no number (a coincident source's strength
   // may be none), by a branch in a second run (in every pair the branch took 7 % more, zeroed strengths 4 %). The second run
   // is rare and reads the sources from memory: staged like the first one, from one loop body with it, it cost the first run 2 %
   // (38,400 sources x 10,000 targets, B in FP64, 852 against 834 us; FP32, 432 against 417, both fields 470 against 494).
   if(active && !isfinite(B[0] + B[1] + B[2] + A[0] + A[1] + A[2]))
   {
      for(int d = 0; d < 3; d++) B[d] = A[d] = U(0);
#pragma unroll 1
      for(int i = sBeg; i < sEnd; i++)
      {
         const U dx = x - U(spos[i].x), dy = y - U(spos[i].y), dz = z - U(spos[i].z);
         const U r2 = dx * dx + dy * dy + dz * dz;
         if(r2 != U(0)) add(U(sq[i].x), U(sq[i].y), U(sq[i].z), dx, dy, dz, rsqrtOf<U>(r2));
      }
   }
   if(!active) return;
   if(gridDim.z > 1)
   {
      U* o = part + int64_t(blockIdx.z) * 6 * m + ti;
      for(int d = 0; d < 3; d++)
      {
         if constexpr(WANTB) o[int64_t(d) * m] = B[d];
         if constexpr(WANTA) o[int64_t(3 + d) * m] = A[d];
      }
      return;
   }
   if constexpr(WANTB) for(int d = 0; d < 3; d++) outB[3 * int64_t(ti) + d] = B[d] * scaleB;
   if constexpr(WANTA) for(int d = 0; d < 3; d++) outA[3 * int64_t(ti) + d] = A[d] * scaleA;
}

// out[3 i + d] = scale * the parts' sums of quantity d (0..2) of target i, first = 0 (B) or 3 (A)
template <class U>
__global__ void kDirectSum(const U* __restrict__ part, int parts, int m, int first, U scale, U* __restrict__ out)
{
   const int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
   if(e >= 3 * int64_t(m)) return;
   const int d = int(e / m), i = int(e % m);
   U s = U(0);
   for(int q = 0; q < parts; q++) s += part[(int64_t(q) * 6 + first + d) * m + i];
   out[3 * int64_t(i) + d] = s * scale;
}

// ====================================================================================
// Host drivers
// ====================================================================================
template <class T>
fmm_status upwardT(Plan& P, cudaStream_t st)
{
   FMM_TRY(buildOperators(P, st));
   const int64_t N = P.tree.nNodes;
   const int Lp = P.Lp;
   FMM_TRY(P.mult.reserve(sizeof(T) * N * 3 * Lp));
   FMM_CUDA(cudaMemsetAsync(P.mult.ptr, 0, sizeof(T) * N * 3 * Lp, st));
   typedef typename Vec4<T>::type V4;
   constexpr int NT = 64;
   const size_t shm = sizeof(T) * 3 * Lp;
   if(P.bem)
   {
      // dipole multipoles of the BEM sources (fmm_bem.cu); the translations below are the same
      P.p2mPiecesTag = -1;
      FMM_TRY(bemP2MT<T>(P, st));
   }
   else if(P.p2mChunk == 0)
   {
      // a warp per leaf, or a block where leaves are large and too few to fill the chip with warps
      const bool split = N <= 16 * 148 && P.n / std::max<int64_t>(1, N) >= 64;
      auto kern = split ? kP2MWarp<T, true> : kP2MWarp<T, false>;
      const int warps = split ? P2MW_SPLIT_WARPS : P2MW_WARPS;
      const size_t shw = p2mWarpSmem<T>(P.p, Lp, warps);
      if(shw > 48 * 1024) FMM_CUDA(allowShared(kern));
      // tensor-core M2M plans: the leaves' multipoles also leave as the M2M's operand pieces
      int np = 0;
      if(sizeof(T) == 4 && P.tcTranslations(1) && P.tcDrainMode != 0) np = m2mPieces(P);
      if(np)
         FMM_TRY(P.multBf.reserve(size_t(np == 1 ? 4 : 2 * np) * size_t(N) * 3 * Lp));
      kern<<<split ? int(N) : walkBlocks(kern, 32 * warps, shw, N), 32 * warps, shw, st>>>(
         P.tree, P.root, (const V4*)P.sPos.ptr, (const V4*)P.sQ.ptr, P.p, Lp, (T*)P.mult.ptr,
         np ? (uint8_t*)P.multBf.ptr : nullptr, np);
      P.p2mPiecesTag = np ? (np == 1 ? 3 : 2 * np) : -1;
   }
   else
   {
      P.p2mPiecesTag = -1;
      if(P.p2mChunk == 32)
         kP2M<T, NT, 32><<<int(N), NT, shm, st>>>(P.tree, P.root, (const V4*)P.sPos.ptr, (const V4*)P.sQ.ptr, P.p,
                                                 Lp, (T*)P.mult.ptr);
      else
         kP2M<T, NT, 16><<<int(N), NT, shm, st>>>(P.tree, P.root, (const V4*)P.sPos.ptr, (const V4*)P.sQ.ptr, P.p,
                                                 Lp, (T*)P.mult.ptr);
   }
   FMM_TRY(launched(P, "kP2M", st));
   FMM_CHECK_LAUNCH();
   if(P.tcTranslations(1)) return m2mTensorCore(P, st);
   return rotM2M<T>(P, st);
}

template <class T>
fmm_status downwardT(Plan& P, cudaStream_t st)
{
   const int64_t N = P.tree.nNodes;
   const int Lp = P.Lp;
   FMM_TRY(P.local.reserve(sizeof(T) * N * 3 * Lp));
   FMM_CUDA(cudaMemsetAsync(P.local.ptr, 0, sizeof(T) * N * 3 * Lp, st));
   if(sizeof(T) == 4 && P.cfg.m2l_mode != FMM_M2L_SIMT) FMM_TRY(m2lTensorCore(P, st));
   else FMM_TRY(rotM2L<T>(P, st));
   if(P.eventsMade && !P.capturing) cudaEventRecord(P.ev[3], st);
   if(P.tcTranslations(2)) return l2lTensorCore(P, st);
   return rotL2L<T>(P, st);
}

// Into how many blocks a leaf's direct list is split: with few leaves of many sources a block per leaf leaves the chip idle
// while the longest list is summed (38,400 points in leaves of up to 1000 and 4,001 targets: near field 0.86 ms with
// one block a leaf, 0.12 split). Two rounds of 16 blocks a SM, only where lists average two tiles, and at most 50 MB of
// partial sums (more than 2^20 targets in so few leaves keep a block busy by themselves).
int nearParts(const Plan& P)
{
   const int64_t N = std::max<int64_t>(1, P.tree.nNodes);
   if(double(P.nP2P) / double(N) * (double(P.n) / double(N)) < 512 || P.m == 0) return 1;
   return int(std::max<int64_t>(1, std::min({int64_t(16), int64_t(2 * 16 * 148) / N, (int64_t(1) << 20) / P.m})));
}

// Threads of a near-field block. 128 where lists are long (a leaf's targets fill 128 threads better than 64, and a
// tile's fill is shared by more: 2^18 points, 478 sources a list, 0.43 -> 0.365 ms; in FP64 1.28 -> 1.02 ms with the
// L2P; 2^24 points, 465, the same within the clock's drift) and where all blocks run at once, so that the longest one
// counts (2,048 points 25 -> 14 us; 239 large leaves 99 -> 90 us); 64 where a block mostly pays for its set-up (256
// coils, 31 sources a list: 6.5 ms against 7.6 with 128; 2^20 points and targets, 112: 0.48 against 0.54 ms).
int nearThreads(const Plan& P)
{
   const int64_t N = std::max<int64_t>(1, P.tree.nNodes);
   return N <= 16 * 148 || double(P.nP2P) / double(N) * (double(P.n) / double(N)) >= 256 ? 128 : 64;
}

template <class T>
fmm_status evaluateT(Plan& P, double current, int want, cudaStream_t st)
{
   typedef typename Vec4<T>::type V4;
   const int64_t N = P.tree.nNodes;
   const int L = P.L, Lb = nharm(P.p - 1);
   constexpr int NE = 128;
   const int TS = P.nearTile == 128 ? 128 : 256;
   const bool split = P.l2pSplit != 0;
   const int NT = split ? nearThreads(P) : 64;
   const size_t coef = split ? 0 : (sizeof(T) * (3 * L + 3 * Lb) + 31) & ~size_t(31);
   size_t shm = coef + 2 * size_t(nearTileBytes<T>(TS)) + sizeof(double) * (want & 2 || !split ? 6 : 3) * NT;
   T scaleB = T(REF_MU0 / (4 * REF_PI) * current), scaleA = T(1.0 / (4 * REF_PI) * current);
   if(P.bem)
   {
      // BEM: the far field sum_k L_k R_k (the A form of the L2P), then the BEM kernel's near field and
      // the 1 / (4 pi) of calcBEM (fast_multipole_solver.cpp:233-250; no current factor there)
      const size_t sh = l2pWarpSmem<T, true>(P.p);
      if(sh > 48 * 1024) FMM_CUDA(allowShared(kL2PWarp<T, true>));
      kL2PWarp<T, true><<<walkBlocks(kL2PWarp<T, true>, 32 * L2PW_WARPS, sh, N), 32 * L2PW_WARPS, sh, st>>>(
         P.tree, P.root, P.p, P.Lp, (const T*)P.local.ptr, (const V4*)P.tPos.ptr, (const int*)P.tIdx.ptr,
         (const CurlEntry<T>*)P.curlTab.ptr, 2, (T*)P.outB.ptr, (T*)P.outA.ptr);
      FMM_TRY(launched(P, "kL2PWarp", st));
      return bemNearT<T>(P, st);
   }
   if(split)
   {
      auto runL2P = [&](auto kernel, size_t sh) -> fmm_status {
         if(sh > 48 * 1024) FMM_CUDA(allowShared(kernel));
         kernel<<<walkBlocks(kernel, 32 * L2PW_WARPS, sh, N), 32 * L2PW_WARPS, sh, st>>>(
            P.tree, P.root, P.p, P.Lp, (const T*)P.local.ptr, (const V4*)P.tPos.ptr, (const int*)P.tIdx.ptr,
            (const CurlEntry<T>*)P.curlTab.ptr, want, (T*)P.outB.ptr, (T*)P.outA.ptr);
         return FMM_OK;
      };
      if(want & 2) FMM_TRY(runL2P(kL2PWarp<T, true>, l2pWarpSmem<T, true>(P.p)));
      else FMM_TRY(runL2P(kL2PWarp<T, false>, l2pWarpSmem<T, false>(P.p)));
      FMM_TRY(launched(P, "kL2PWarp", st));
   }
   int parts = split ? nearParts(P) : 1;
   if(P.nearPart.bytes < nearPartBytes(P, parts)) parts = 1;   // (reserved at tree build)
   auto run = [&](auto kernel) -> fmm_status {
      if(shm > 48 * 1024) FMM_CUDA(allowShared(kernel));
      kernel<<<dim3(int(N), parts), NT, shm, st>>>(P.tree, P.root, P.p, P.Lp, (const T*)P.local.ptr, (const V4*)P.tPos.ptr,
                                      (const V4*)P.sPos.ptr, (const V4*)P.sQ.ptr, (const int*)P.p2pOff.ptr,
                                      (const int*)P.p2pList.ptr, (const int*)P.tIdx.ptr, scaleB, scaleA, want,
                                      (T*)P.outB.ptr, (T*)P.outA.ptr, (double*)P.nearPart.ptr, int(P.m));
      return FMM_OK;
   };
   auto pick = [&](auto nt, auto ts, auto far) -> fmm_status {
      if(want & 2) return run(kL2PNear<T, decltype(nt)::value, decltype(ts)::value, NE, true, decltype(far)::value>);
      return run(kL2PNear<T, decltype(nt)::value, decltype(ts)::value, NE, false, decltype(far)::value>);
   };
   constexpr std::integral_constant<int, 64> n64;
   constexpr std::integral_constant<int, 128> n128, t128;
   constexpr std::integral_constant<int, 256> t256;
   if(!split) FMM_TRY(TS == 128 ? pick(n64, t128, std::true_type()) : pick(n64, t256, std::true_type()));
   else if(NT == 64) FMM_TRY(TS == 128 ? pick(n64, t128, std::false_type()) : pick(n64, t256, std::false_type()));
   else FMM_TRY(TS == 128 ? pick(n128, t128, std::false_type()) : pick(n128, t256, std::false_type()));
   FMM_TRY(launched(P, "kL2PNear", st));
   if(parts > 1)
   {
      kNearParts<T><<<int((P.m + 255) / 256), 256, 0, st>>>((const double*)P.nearPart.ptr, parts, int(P.m), (const int*)P.tIdx.ptr,
                                                            scaleB, scaleA, want, (T*)P.outB.ptr, (T*)P.outA.ptr);
      FMM_TRY(launched(P, "kNearParts", st));
   }
   FMM_CHECK_LAUNCH();
   return FMM_OK;
}

// kDirect over coils of at most maxT targets and maxS sources (m targets in all), the sources split so that the
// launch has about eight blocks a SM and a part keeps at least 512 sources.
template <class T, class U>
static fmm_status launchDirect(Plan& P, DevBuf& partBuf, int coils, int maxT, int maxS, const U* tgt, int m, const int* sseg,
                               const int* tseg, U scaleB, U scaleA, int want, U* outB, U* outA, cudaStream_t st)
{
   typedef typename Vec4<T>::type V4;
   constexpr int NT = 128;
   const int blocks = (maxT + NT - 1) / NT;
   if(blocks == 0) return FMM_OK;
   const int64_t wantParts = (8 * 148 + int64_t(blocks) * coils - 1) / (int64_t(blocks) * coils);
   int parts = int(std::max<int64_t>(1, std::min<int64_t>(wantParts, maxS / 512)));
   if(parts > 1 && !P.roomFor(partBuf, sizeof(U) * 6 * size_t(parts) * size_t(m))) parts = 1;
   U* part = (U*)partBuf.ptr;
   auto run = [&](auto kern) {
      kern<<<dim3(blocks, coils, parts), NT, 0, st>>>((const V4*)P.sPos.ptr, (const V4*)P.sQ.ptr, int(P.n), tgt, m, sseg, tseg,
                                                      scaleB, scaleA, outB, outA, part);
   };
   if(want == 1) run(kDirect<T, U, NT, true, false>);
   else if(want == 2) run(kDirect<T, U, NT, false, true>);
   else run(kDirect<T, U, NT, true, true>);
   FMM_TRY(launched(P, "kDirect", st));
   if(parts > 1)
   {
      const int sumBlocks = int((3 * int64_t(m) + 255) / 256);
      if(want & 1) kDirectSum<U><<<sumBlocks, 256, 0, st>>>(part, parts, m, 0, scaleB, outB);
      if(want & 2) kDirectSum<U><<<sumBlocks, 256, 0, st>>>(part, parts, m, 3, scaleA, outA);
      FMM_TRY(launched(P, "kDirectSum", st));
   }
   FMM_CHECK_LAUNCH();
   return FMM_OK;
}

template <class T>
fmm_status directT(Plan& P, double current, int want, cudaStream_t st)
{
   T scaleB = T(REF_MU0 / (4 * REF_PI) * current), scaleA = T(1.0 / (4 * REF_PI) * current);
   if(P.bem) return bemDirectT<T>(P, st);
   int maxT = 0, maxS = 0;
   for(int c = 0; c < P.nCoils; c++)
   {
      maxT = std::max(maxT, P.tgtOff[c + 1] - P.tgtOff[c]);
      maxS = std::max(maxS, P.srcOff[c + 1] - P.srcOff[c]);
   }
   const int* seg = (const int*)P.segb.ptr;   // srcOff then tgtOff, uploaded by the tree build or with the packed sources
   return launchDirect<T, T>(P, P.directPart, P.nCoils, maxT, maxS, (const T*)P.tgtXYZ, int(P.m), seg, seg + P.nCoils + 1, scaleB, scaleA,
                             want, (T*)P.outB.ptr, (T*)P.outA.ptr, st);
}

fmm_status directFp64Subset(Plan& P, double current, const double* tgtDev, int k, double* outDev, cudaStream_t st)
{
   const double scaleB = REF_MU0 / (4 * REF_PI) * current;
   if(P.fp64)
      return launchDirect<double, double>(P, P.subsetPart, 1, k, int(P.n), tgtDev, k, nullptr, nullptr, scaleB, 0.0, 1, outDev, nullptr, st);
   return launchDirect<float, double>(P, P.subsetPart, 1, k, int(P.n), tgtDev, k, nullptr, nullptr, scaleB, 0.0, 1, outDev, nullptr, st);
}

// New strengths w J for the same source positions, in the tree's sorted order.
template <class T>
__global__ void kRegatherStrengths(const T* __restrict__ xyz, const T* __restrict__ w, const T* __restrict__ J,
                                   const T* __restrict__ sigma, const int* __restrict__ order, int64_t n,
                                   typename Vec4<T>::type* q)
{
   int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
   if(i >= n) return;
   int64_t s = order[i];
   T jx, jy, jz;
   if(J) { jx = J[3 * s]; jy = J[3 * s + 1]; jz = J[3 * s + 2]; }
   else
   {
      const T x = xyz[3 * s], y = xyz[3 * s + 1];
      const T l = sqrt(x * x + y * y);
      jx = l != T(0) ? -y / l : T(0);
      jy = l != T(0) ? x / l : T(0);
      jz = T(0);
   }
   const T ww = w[s];
   q[i] = {ww * jx, ww * jy, ww * jz, sigma ? ww * sigma[s] : T(0)};
}

template <class T>
__global__ void kScaleCopy(const T* __restrict__ src, T* __restrict__ dst, int64_t count, T scale)
{
   int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
   if(i < count) dst[i] = src[i] * scale;
}

template <class T>
fmm_status regatherStrengthsT(Plan& P, cudaStream_t st)
{
   typedef typename Vec4<T>::type V4;
   if(P.n == 0) return FMM_OK;
   kRegatherStrengths<T><<<int((P.n + 255) / 256), 256, 0, st>>>((const T*)P.srcXYZ, (const T*)P.srcW,
                                                                 (const T*)(P.hasJ ? P.srcJ : nullptr),
                                                                 (const T*)(P.bem ? P.srcSigma : nullptr),
                                                                 (const int*)P.sIdx.ptr, P.n, (V4*)P.sQ.ptr);
   FMM_TRY(launched(P, "kRegatherStrengths", st));
   return FMM_OK;
}

template <class T>
fmm_status scaleCopyT(Plan& P, const void* src, void* dst, int64_t count, double scale, cudaStream_t st)
{
   if(count == 0) return FMM_OK;
   kScaleCopy<T><<<int((count + 255) / 256), 256, 0, st>>>((const T*)src, (T*)dst, count, T(scale));
   FMM_TRY(launched(P, "kScaleCopy", st));
   return FMM_OK;
}

template fmm_status regatherStrengthsT<float>(Plan&, cudaStream_t);
template fmm_status regatherStrengthsT<double>(Plan&, cudaStream_t);
template fmm_status scaleCopyT<float>(Plan&, const void*, void*, int64_t, double, cudaStream_t);
template fmm_status scaleCopyT<double>(Plan&, const void*, void*, int64_t, double, cudaStream_t);

template fmm_status upwardT<float>(Plan&, cudaStream_t);
template fmm_status upwardT<double>(Plan&, cudaStream_t);
template fmm_status downwardT<float>(Plan&, cudaStream_t);
template fmm_status downwardT<double>(Plan&, cudaStream_t);
template fmm_status evaluateT<float>(Plan&, double, int, cudaStream_t);
template fmm_status evaluateT<double>(Plan&, double, int, cudaStream_t);
template fmm_status directT<float>(Plan&, double, int, cudaStream_t);
template fmm_status directT<double>(Plan&, double, int, cudaStream_t);

}  // namespace fmm
