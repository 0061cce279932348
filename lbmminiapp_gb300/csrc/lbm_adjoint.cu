// Discrete adjoint of the collide-stream step (no reference counterpart).
//
// Forward model, one step from the pre-collision state f^t (AB push storage,
// slot s = direction s):
//   rho = sum f, j = sum c f + F/2, u = j / rho           (F = F_uniform + F_field(x))
//   C_s = (1 - omega) f_s + omega eq_s(rho, j) + (1 - omega/2) fd_s(rho, j, F)
//   post_s = (1 - sig) C_s + sig f_opp(s)                  (partial bounce-back, sig(x))
//   f^{t+1}_s(x + c_s) = post_s(x), or f^{t+1}_opp(s)(x) = post_s(x) when x + c_s
//   is blocked (half-way bounce-back)
// with eq_s = w_s (rho + 3 c.j + 9/2 (c.j)^2/rho - 3/2 |j|^2/rho) and
// fd_s = w_s (3 c.F - 3 F.u + 9 (c.u)(c.F)).
//
// Adjoint, lam^t = dL/df^t, from lam^{t+1}:
//   mu_s(x)  = lam^{t+1}_s(x + c_s), or lam^{t+1}_opp(s)(x) when blocked   (streaming transposed)
//   nu_s     = (1 - sig) mu_s
//   A_rho    = sum_s nu_s (omega deq_s/drho + (1 - omega/2) dfd_s/drho)
//   A_j      = sum_s nu_s (omega deq_s/dj   + (1 - omega/2) dfd_s/dj)
//   lam^t_k  = (1 - omega) nu_k + sig mu_opp(k) + A_rho + A_j . c_k + dL_t/df_k
//   dL/dF   += (1 - omega/2) sum_s nu_s dfd_s/dF|_j + A_j / 2 + dL_t/dF
//   dL/dsig += sum_s mu_s (f_opp(s) - C_s)
// where deq_s/drho = w_s (1 - 9/2 (c.u)^2 + 3/2 |u|^2),
//       deq_s/dj   = w_s (3 c + 9 (c.u) c - 3 u),
//       dfd_s/dj   = w_s (9 (c.F) c - 3 F) / rho,
//       dfd_s/drho = w_s (3 F.u - 9 (c.u)(c.F)) / rho,
//       dfd_s/dF   = w_s (3 c - 3 u + 9 (c.u) c).
// Loss terms at step t (weight tw, spatial weights W):
//   velocity:  L_t = tw sum_x W(x) . u(x)        dL/df_k = tw W.(c_k - u)/rho, dL/dF = tw W/(2 rho)
//   energy:    L_t = tw sum_x W_0(x) rho|u|^2/2   dL/df_k = tw W_0 (u.c_k - |u|^2/2), dL/dF = tw W_0 u/2
// The sums over s need mu only through the weighted moments
//   m0 = sum w mu, m1 = sum w mu c, m2 = sum w mu c c^T
// (with nu = (1 - sig) mu a common factor):
//   T     = 3 m1 + 9 m2 u - 3 m0 u
//   A_rho = (1 - sig) [omega ((1 + 3/2 uu) m0 - 9/2 u.m2.u) + (1 - omega/2)/rho (3 F.u m0 - 9 F.m2.u)]
//   A_j   = (1 - sig) [omega T + (1 - omega/2)/rho (9 m2 F - 3 m0 F)]
//   sum_s nu_s (1 - omega/2) dfd_s/dF = (1 - sig) (1 - omega/2) T
//   sum_s mu_s C_s from m0, m1, m2 and sum mu_s f_s
// and opposite directions enter them by their sum and difference.  That is about
// 265 operations per D3Q19 cell; direction by direction it was 1180, and the
// FP64 form is bound by the FP64 pipe (76 cycles per instruction, warp and
// sub-partition).  The sums over f run on deviations g_s = f_s - w_s r,
//   sum_s mu_s (f_s - eq_s) = sum_s mu_s g_s - sum_s mu_s (eq_s - w_s r),
// so that f_opp(s) - C_s has no cancellation against w r: r = 1 for the shifted
// storage formats, which hold exactly these, and in FP32; in FP64 on FP64 storage
// r is the density that the rest population stands for, so that a cell of small
// density loses no bits against 1.
//
// One kernel for both adjoints: R = double, and R = float with lam and the
// arithmetic in FP32.  The gradients are accumulated in FP64 either way; f^t may
// be stored in any storage format.
#include <cuda_runtime.h>

#include "../../include/lbm_gb300.h"
#include "lbm_adjoint.cuh"
#include "lbm_aux.cuh"
#include "lbm_moments.cuh"
#include "lbm_step.cuh"

namespace lbm {

// Whether r is the cell's own, not 1.
template <int ST, typename R>
constexpr bool adj_scaled() { return ST == ST_F64 && sizeof(R) == 8; }

// A stored population (adj_scaled), or its deviation f - w.
template <int ST, typename R>
__device__ __forceinline__ R load_adj(const void* buf, int64_t idx, double w)
{
   if constexpr (adj_scaled<ST, R>()) {
      return static_cast<const double*>(buf)[idx];
   } else if constexpr (ST == ST_F64) {
      return (R)(static_cast<const double*>(buf)[idx] - w);
   } else {
      return (R)load_shifted(static_cast<const typename Store<ST>::T*>(buf) + idx);
   }
}

// The adjoint buffers and the launch constants in the kernel's arithmetic.
template <typename R> struct AdjBuffers;
template <> struct AdjBuffers<double> {
   __device__ static const double* next(const AdjParams& a) { return a.lam_next; }
   __device__ static double* out(const AdjParams& a) { return a.lam; }
   __device__ static const AdjConsts<double>& k(const AdjParams& a) { return a.k; }
};
template <> struct AdjBuffers<float> {
   __device__ static const float* next(const AdjParams& a) { return a.lam_next_f; }
   __device__ static float* out(const AdjParams& a) { return a.lam_f; }
   __device__ static const AdjConsts<float>& k(const AdjParams& a) { return a.kf; }
};

// This thread's cell: its position and neighbour offsets (32-bit: fewer than 2^31
// cells).  Threads take consecutive cells across row ends, so that no lane idles
// whatever nx is; with a row per block an nx of 129 left half of them idle and an nx
// of 1 all but one (D3Q19 FP32, 65,536 cells: 92 us, 8.4 us this way).
__device__ __forceinline__ bool adj_cell(const AdjParams& a, CellIndex& ci)
{
   const GridDims& g = a.g;
   const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
   if (c >= a.ag.ncell) return false;
   const uint32_t row = div_magic(c, (uint32_t)g.nx, a.ag.m_nx), z = div_magic(row, (uint32_t)g.ny, a.ag.m_ny);
   const int x = (int)(c - row * (uint32_t)g.nx), y = (int)(row - z * (uint32_t)g.ny);
   ci.c = (int64_t)c;
   ci.dxm = (x == 0) ? g.nx - 1 : -1;
   ci.dxp = (x == g.nx - 1) ? -(g.nx - 1) : 1;
   ci.dym = (y == 0) ? (g.ny - 1) * g.nx : -g.nx;
   ci.dyp = (y == g.ny - 1) ? -(g.ny - 1) * g.nx : g.nx;
   const int nxy = g.nx * g.ny;
   ci.dzm = (z == 0) ? (g.nz - 1) * nxy : -nxy;
   ci.dzp = ((int)z == g.nz - 1) ? -(g.nz - 1) * nxy : nxy;
   return true;
}

// Small blocks, for the last wave (D3Q19, 64x40x40, FP64 67.9 -> 66.5 us, FP32 with the
// velocity loss 10.3 -> 9.0 us from 128; equal on larger grids).
constexpr int kAdjThreads = 64;

template <int Q, int ST, typename R>
__global__ void __launch_bounds__(kAdjThreads) adjoint_step_kernel(const AdjParams a)
{
   CellIndex ci;
   if (!adj_cell(a, ci)) return;
   const int64_t c = ci.c, plane = a.g.plane;
   const uint32_t lk = a.links ? a.links[c] : 0u;
   R* lam = AdjBuffers<R>::out(a);
   const AdjConsts<R>& K = AdjBuffers<R>::k(a);
   if (lk & kSolidBit) {
#pragma unroll
      for (int s = 0; s < Q; s++) lam[(int64_t)s * plane + c] = R(0);
      return;
   }
   constexpr int NP = (Q - 1) / 2, RD = lat_rest(Q);
   const R* next = AdjBuffers<R>::next(a);
   // mu (streaming transposed): per pair its sum and difference
   R p[NP], d[NP], mur = R(0);
#pragma unroll
   for (int q = 0; q < NP; q++) {
      p[q] = d[q] = R(0);
      if (a.collide) {
         const int s = pair_dir(Q, q), o = lat_opp(Q, s);
         const bool bs = (lk >> s) & 1u, bo = (lk >> o) & 1u;
         const int off = nbr_off(ci, lat_c(Q, s, 0), lat_c(Q, s, 1), lat_c(Q, s, 2));
         const int ofo = nbr_off(ci, lat_c(Q, o, 0), lat_c(Q, o, 1), lat_c(Q, o, 2));
         const R ms = next[(int64_t)(bs ? o : s) * plane + (c + (bs ? 0 : off))];
         const R mo = next[(int64_t)(bo ? s : o) * plane + (c + (bo ? 0 : ofo))];
         p[q] = ms + mo;
         d[q] = ms - mo;
      }
   }
   if (a.collide) mur = next[(int64_t)RD * plane + c];

   // sum g, j and the products with mu of the porosity gradient, in one pass: dot1 =
   // sum over pairs (f_s - f_o)(mu_s - mu_o), dot0 = sum of (g_s + g_o)(mu_s + mu_o)
   constexpr bool kScaled = adj_scaled<ST, R>();
   R gr = load_adj<ST, R>(a.state, (int64_t)RD * plane + c, lat_w(Q, RD)), r = R(1);
   if constexpr (kScaled) {
      r = gr * (1.0 / lat_w(Q, RD));
      gr -= lat_w(Q, RD) * r;
   }
   // g_s + g_o from the loaded pair
   const auto pair_sum = [&](R vs, R vo, double w) { return kScaled ? (vs + vo) - R(2.0 * w) * r : vs + vo; };
   R total = gr, j[3] = {R(0), R(0), R(0)}, dot1 = R(0), dot0 = R(0);
   R m0 = (R)lat_w(Q, RD) * mur, m1[3] = {R(0), R(0), R(0)}, md[3] = {R(0), R(0), R(0)}, mo_[3] = {R(0), R(0), R(0)};
   // axes
   {
      R ps = R(0);
#pragma unroll
      for (int k = 0; k < 3; k++) {
         const int s = 2 * k, o = 2 * k + 1;
         const double w = lat_w(Q, s);
         const R gs = load_adj<ST, R>(a.state, (int64_t)s * plane + c, w);
         const R go = load_adj<ST, R>(a.state, (int64_t)o * plane + c, w);
         const R S = pair_sum(gs, go, w), D = gs - go;
         total += S;
         j[k] = D;
         dot1 += D * d[k];
         dot0 += S * p[k];
         ps += p[k];
         m1[k] = (R)w * d[k];
         md[k] = (R)w * p[k];
      }
      m0 += (R)lat_w(Q, 0) * ps;
   }
   // planes: pairs c = e_a + e_b (q1) and e_a - e_b (q2)
   {
      constexpr double w = lat_w(Q, 6);
      R ps = R(0);
#pragma unroll
      for (int k = 0; k < 3; k++) {
         const int A = k < 2 ? 0 : 1, B = k == 0 ? 1 : 2;
         const int q1 = 3 + 2 * k, q2 = q1 + 1;
         R S[2], D[2];
#pragma unroll
         for (int h = 0; h < 2; h++) {
            const int s = pair_dir(Q, q1 + h), o = lat_opp(Q, s);
            const R gs = load_adj<ST, R>(a.state, (int64_t)s * plane + c, w);
            const R go = load_adj<ST, R>(a.state, (int64_t)o * plane + c, w);
            S[h] = pair_sum(gs, go, w);
            D[h] = gs - go;
            total += S[h];
            dot1 += D[h] * d[q1 + h];
            dot0 += S[h] * p[q1 + h];
         }
         j[A] += D[0] + D[1];
         j[B] += D[0] - D[1];
         const R pp = p[q1] + p[q2];
         ps += pp;
         m1[A] += (R)w * (d[q1] + d[q2]);
         m1[B] += (R)w * (d[q1] - d[q2]);
         md[A] += (R)w * pp;
         md[B] += (R)w * pp;
         mo_[k] = (R)w * (p[q1] - p[q2]);
      }
      m0 += (R)w * ps;
   }
   // bodies: c = (1, +-1, +-1)
   if constexpr (Q == 27) {
      constexpr double w = lat_w(Q, 18);
#pragma unroll
      for (int h = 0; h < 4; h++) {
         const int q = 9 + h, s = pair_dir(Q, q), o = lat_opp(Q, s);
         const R gs = load_adj<ST, R>(a.state, (int64_t)s * plane + c, w);
         const R go = load_adj<ST, R>(a.state, (int64_t)o * plane + c, w);
         const R S = pair_sum(gs, go, w), D = gs - go;
         const R cy = (R)lat_c(Q, s, 1), cz = (R)lat_c(Q, s, 2);   // +-1
         total += S;
         j[0] += D;
         j[1] += cy * D;
         j[2] += cz * D;
         dot1 += D * d[q];
         dot0 += S * p[q];
         const R wd = (R)w * d[q], wp = (R)w * p[q];
         m0 += wp;
         m1[0] += wd;
         m1[1] += cy * wd;
         m1[2] += cz * wd;
         md[0] += wp;
         md[1] += wp;
         md[2] += wp;
         mo_[0] += cy * wp;
         mo_[1] += cz * wp;
         mo_[2] += (cy * cz) * wp;
      }
   }

   // force: (R)(F + field), the fields' FP32 copies where they hold that value
   R F[3];
#pragma unroll
   for (int k = 0; k < 3; k++) {
      if (sizeof(R) == 4 && a.force_field_f) F[k] = a.force_field_f[k * plane + c];
      else F[k] = a.force_field ? (R)(a.F[k] + a.force_field[k * plane + c]) : K.F[k];
   }
   R sig = R(0);
   if (sizeof(R) == 4 && a.porosity_f) sig = a.porosity_f[c];
   else if (a.porosity) sig = (R)a.porosity[c];
   const R rho = r + total;
   const R ir = R(1) / rho;
   R u[3];
#pragma unroll
   for (int k = 0; k < 3; k++) {
      j[k] += R(0.5) * F[k];
      u[k] = j[k] * ir;
   }
   const R uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
   const R Fu = F[0] * u[0] + F[1] * u[1] + F[2] * u[2];
   const R om = K.om, om1 = K.om1, om2 = K.om2;

   R even = R(0), odd[3] = {R(0), R(0), R(0)};   // lam_k = (1-omega) nu_k + sig mu_opp + even + odd . c_k
   R gF[3] = {R(0), R(0), R(0)}, gsig = R(0);
   const R keep = R(1) - sig;
   if (a.collide) {
      const R mu_u[3] = {md[0] * u[0] + mo_[0] * u[1] + mo_[1] * u[2], mo_[0] * u[0] + md[1] * u[1] + mo_[2] * u[2],
                         mo_[1] * u[0] + mo_[2] * u[1] + md[2] * u[2]};
      const R mu_F[3] = {md[0] * F[0] + mo_[0] * F[1] + mo_[1] * F[2], mo_[0] * F[0] + md[1] * F[1] + mo_[2] * F[2],
                         mo_[1] * F[0] + mo_[2] * F[1] + md[2] * F[2]};
      const R uMu = u[0] * mu_u[0] + u[1] * mu_u[1] + u[2] * mu_u[2];
      const R FMu = F[0] * mu_u[0] + F[1] * mu_u[1] + F[2] * mu_u[2];
      const R o2r = om2 * ir;
      const R ffe = R(3) * Fu * m0 - R(9) * FMu;
      even = keep * (om * ((R(1) + R(1.5) * uu) * m0 - R(4.5) * uMu) + o2r * ffe);
      R jm = R(0), Fm = R(0);
#pragma unroll
      for (int k = 0; k < 3; k++) {
         const R T = R(3) * (m1[k] + R(3) * mu_u[k] - m0 * u[k]);
         odd[k] = keep * (om * T + o2r * (R(9) * mu_F[k] - R(3) * m0 * F[k]));
         gF[k] = keep * (om2 * T) + R(0.5) * odd[k];
         jm += m1[k] * j[k];
         Fm += m1[k] * F[k];
      }
      // sum_s mu_s (f_opp(s) - C_s) = -dot1 + omega (sum mu g - sum mu (eq - w r)) - om2 sum mu fd
      const R mug = R(0.5) * (dot0 + dot1) + mur * gr;
      const R mueq = (total - R(1.5) * uu * rho) * m0 + R(3) * jm + R(4.5) * rho * uMu;
      const R mufd = R(3) * Fm - ffe;
      gsig = om * (mug - mueq) - dot1 - om2 * mufd;
   }
   // loss at this step
   if (a.loss_kind == LBM_LOSS_VELOCITY && a.loss_weight) {
      const R W[3] = {(R)a.loss_weight[c], (R)a.loss_weight[plane + c], (R)a.loss_weight[2 * plane + c]};
      const R tw = K.tw * ir;
      even -= tw * (W[0] * u[0] + W[1] * u[1] + W[2] * u[2]);
#pragma unroll
      for (int k = 0; k < 3; k++) {
         odd[k] += tw * W[k];
         gF[k] += R(0.5) * tw * W[k];
      }
   } else if (a.loss_kind == LBM_LOSS_ENERGY && a.loss_weight) {
      const R tw = (R)(a.time_weight * a.loss_weight[c]);
      even -= R(0.5) * tw * uu;
#pragma unroll
      for (int k = 0; k < 3; k++) {
         odd[k] += tw * u[k];
         gF[k] += R(0.5) * tw * u[k];
      }
   }

   const R k1 = om1 * keep;
   const R al = R(0.5) * (k1 + sig), be = R(0.5) * (k1 - sig);
   lam[(int64_t)RD * plane + c] = (k1 + sig) * mur + even;
   R op[3] = {odd[0] + odd[1], odd[0] + odd[2], odd[1] + odd[2]};
   R om_[3] = {odd[0] - odd[1], odd[0] - odd[2], odd[1] - odd[2]};
#pragma unroll
   for (int q = 0; q < NP; q++) {
      const int s = pair_dir(Q, q), o = lat_opp(Q, s);
      R O;
      if (q < 3) O = odd[q];
      else if (q < 9) O = (q - 3) % 2 == 0 ? op[(q - 3) / 2] : om_[(q - 3) / 2];
      else O = (lat_c(Q, s, 1) > 0 ? op[0] : om_[0]) + (lat_c(Q, s, 2) > 0 ? odd[2] : -odd[2]);
      const R X = al * p[q] + even, Y = be * d[q] + O;
      lam[(int64_t)s * plane + c] = X + Y;
      lam[(int64_t)o * plane + c] = X - Y;
   }
   if (a.grad_force) {
#pragma unroll
      for (int k = 0; k < 3; k++) a.grad_force[(int64_t)k * plane + c] += widen(gF[k]);
   }
   if (a.grad_porosity) a.grad_porosity[c] += widen(gsig);
}

// Loss value of the current state (FP64 partial sums per block).
template <int Q, int ST>
__global__ void __launch_bounds__(kReduceThreads) loss_partial_kernel(AdjParams a, double* partials)
{
   double acc = 0.0;
   for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < a.g.ncell;
        c += (int64_t)gridDim.x * blockDim.x) {
      const uint32_t lk = a.links ? a.links[c] : 0u;
      if (lk & kSolidBit) continue;
      double W[3] = {a.loss_weight[c], 0.0, 0.0};
      if (a.loss_kind == LBM_LOSS_VELOCITY) {
         W[1] = a.loss_weight[a.g.plane + c];
         W[2] = a.loss_weight[2 * a.g.plane + c];
      }
      const auto load = [&](int s) { return moment_value<ST>(a.state, (int64_t)s * a.g.plane + c); };
      const CellMoments<Q, ST, decltype(load)> mom(load);
      double ff[3] = {0.0, 0.0, 0.0};
      if (a.force_field) {
#pragma unroll
         for (int d = 0; d < 3; d++) ff[d] = a.force_field[d * a.g.plane + c];
      }
      // a cell of zero weight adds +-0 as long as its u is finite: a warp of them
      // (a loss on one plane) leaves out its FP64 operations
      const bool regular = mom.regular() && finite_bits(ff[0]) && finite_bits(ff[1]) && finite_bits(ff[2]);
      if (!__any_sync(__activemask(), !regular || W[0] != 0.0 || W[1] != 0.0 || W[2] != 0.0)) continue;
      double rho, j[3], F[3] = {a.F[0], a.F[1], a.F[2]};
      mom.get(rho, j);
      if (a.force_field) {
#pragma unroll
         for (int d = 0; d < 3; d++) F[d] += ff[d];
      }
#pragma unroll
      for (int d = 0; d < 3; d++) j[d] += 0.5 * F[d];
      if (a.loss_kind == LBM_LOSS_VELOCITY) acc += (W[0] * j[0] + W[1] * j[1] + W[2] * j[2]) / rho;
      else acc += W[0] * 0.5 * (j[0] * j[0] + j[1] * j[1] + j[2] * j[2]) / rho;
   }
   __shared__ double sh[kReduceThreads / 32];
   for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xFFFFFFFFu, acc, off);
   if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
   __syncthreads();
   if (threadIdx.x == 0) {
      double v = 0.0;
      for (int w = 0; w < kReduceThreads / 32; w++) v += sh[w];
      partials[blockIdx.x] = v * a.time_weight;
   }
}

__global__ void sum_partials_kernel(const double* partials, int n, double* out)
{
   __shared__ double sh[kReduceThreads];
   double v = 0.0;
   for (int i = threadIdx.x; i < n; i += blockDim.x) v += partials[i];
   sh[threadIdx.x] = v;
   __syncthreads();
   for (int stride = blockDim.x / 2; stride > 0; stride >>= 1) {
      if ((int)threadIdx.x < stride) sh[threadIdx.x] += sh[threadIdx.x + stride];
      __syncthreads();
   }
   if (threadIdx.x == 0) out[0] = sh[0];
}

template <int Q, int ST, typename R>
cudaError_t launch_adjoint_r(const AdjParams& a, cudaStream_t st)
{
   AdjParams b = a;
   b.ag = async_geom(a.g.nx, a.g.ny, a.g.nz);
   b.k = {a.omega, 1.0 - a.omega, 1.0 - 0.5 * a.omega, a.time_weight, {a.F[0], a.F[1], a.F[2]}};
   b.kf = {(float)b.k.om, (float)b.k.om1, (float)b.k.om2, (float)b.k.tw, {(float)a.F[0], (float)a.F[1], (float)a.F[2]}};
   adjoint_step_kernel<Q, ST, R><<<(b.ag.ncell + kAdjThreads - 1) / kAdjThreads, kAdjThreads, 0, st>>>(b);
   return cudaGetLastError();
}

template <int Q, int ST>
cudaError_t launch_adjoint_t(const AdjParams& a, cudaStream_t st)
{
   return launch_adjoint_r<Q, ST, double>(a, st);
}

template <int Q, int ST>
cudaError_t launch_adjoint_f32_t(const AdjParams& a, cudaStream_t st)
{
   return launch_adjoint_r<Q, ST, float>(a, st);
}

template <int Q, int ST>
cudaError_t launch_loss_t(const AdjParams& a, double* partials, int nblocks, double* out, cudaStream_t st)
{
   loss_partial_kernel<Q, ST><<<nblocks, kReduceThreads, 0, st>>>(a, partials);
   sum_partials_kernel<<<1, kReduceThreads, 0, st>>>(partials, nblocks, out);
   return cudaGetLastError();
}

#define LBM_ADJ_DISPATCH(FN, ...)                                                        \
   switch (Q * 10 + st) {                                                                \
      case 190: return FN<19, ST_F64>(__VA_ARGS__);                                      \
      case 191: return FN<19, ST_F32>(__VA_ARGS__);                                      \
      case 192: return FN<19, ST_BF16>(__VA_ARGS__);                                     \
      case 193: return FN<19, ST_F16>(__VA_ARGS__);                                      \
      case 270: return FN<27, ST_F64>(__VA_ARGS__);                                      \
      case 271: return FN<27, ST_F32>(__VA_ARGS__);                                      \
      case 272: return FN<27, ST_BF16>(__VA_ARGS__);                                     \
      default: return FN<27, ST_F16>(__VA_ARGS__);                                       \
   }

cudaError_t launch_adjoint(int Q, int st, const AdjParams& a, cudaStream_t stream)
{
   LBM_ADJ_DISPATCH(launch_adjoint_t, a, stream)
}

cudaError_t launch_adjoint_f32(int Q, int st, const AdjParams& a, cudaStream_t stream)
{
   LBM_ADJ_DISPATCH(launch_adjoint_f32_t, a, stream)
}

cudaError_t launch_loss(int Q, int st, const AdjParams& a, double* partials, int nblocks, double* out,
                        cudaStream_t stream)
{
   LBM_ADJ_DISPATCH(launch_loss_t, a, partials, nblocks, out, stream)
}

}  // namespace lbm
