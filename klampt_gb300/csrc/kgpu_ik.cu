// kgpu_ik.cu — batched inverse kinematics, 32 / L problems per warp (L: the
// robot's links rounded up to 8, 16 or 32).
//
// Replaces IKSolver.solve over IKObjective point / transform constraints
// (Python/klampt/src/robotik.cpp:556-689; KrisLibrary RobotIKSolver, absent
// here) for B independent problems in one launch.  The method is this
// project's own (the reference's solver internals are not available):
// Levenberg-Marquardt on the residual
//   e = [p(q) - p*]                                   (position only), or
//   e = [p(q) - p*; 1/2 sum_k R*_k x R_k(q)]           (position + rotation;
//        the second block is sin(theta) u for R = Rot(u, theta) R*),
// with the full Jacobian's rows as derivative (angular rows for the rotation
// block), steps dq = -J^T (J J^T + mu I)^-1 e on the link's ancestor DOFs,
// q clamped to the joint limits after every step, mu / 4 on an accepted step
// (residual norm decreased), mu * 8 on a rejected one.  Converged when
// max |e_i| <= tol.  The FP64 oracle runs the same iteration.
#include <cfloat>

#include "kgpu_device.cuh"

namespace kgpu {

namespace {

struct IkArgs {
  int robot;
  int B;
  float* q;              // [B, L] in: initial guesses, out: results
  const int* links;      // [B] or null (link_all)
  int link_all;
  const float* plocal;   // [B, 3]
  const float* ptarget;  // [B, 3]
  const float* Rtarget;  // [B, 9] row-major or null (position only)
  int max_iters;
  float tol;
  uint8_t* ok;           // [B]
  float* residual;       // [B] max |e_i| at the result
  int* iters;            // [B] iterations used (may be null)
  int per_block;         // problems of a block
};

// sum over a group of L lanes, the first lane's value for all (the lanes'
// orders differ)
template <int L>
__device__ __forceinline__ float group_sum(float v, int gbase)
{
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return __shfl_sync(0xffffffffu, v, gbase);
}

// residual of the link in lane `src` at the FP32 transforms held in lanes
template <int M>
__device__ __forceinline__ void ik_residual(const float* P, int src, float3 pl, const float* pt, const float* Rt,
                                            float* e)
{
  float T[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) T[k] = __shfl_sync(0xffffffffu, P[k], src);
  const float3 p = xform32(T, pl);
  e[0] = p.x - pt[0];
  e[1] = p.y - pt[1];
  e[2] = p.z - pt[2];
  if (M == 6) {
    // 1/2 sum over columns k of R*_k x R_k
    float ex = 0.f, ey = 0.f, ez = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float ax = Rt[k], ay = Rt[3 + k], az = Rt[6 + k];
      const float bx = T[k], by = T[3 + k], bz = T[6 + k];
      ex += ay * bz - az * by;
      ey += az * bx - ax * bz;
      ez += ax * by - ay * bx;
    }
    e[M - 3] = 0.5f * ex;
    e[M - 2] = 0.5f * ey;
    e[M - 1] = 0.5f * ez;
  }
}

// M: residual entries (3 position, 6 position and rotation).  A group of L
// lanes (lane g L + i: link i) iterates on its problem and takes the block's
// next one when it is done, so that the few problems that run to the iteration
// limit do not hold up the others of their warp.  Bound by the dependent
// shuffle, division and square root chains of an iteration (M and L as
// parameters let the 21 group sums overlap).  One warp per problem left 25 of
// 32 lanes idle for a 7-link arm: 65,536 point + rotation problems 1,650 ->
// 532 us for the call, 9,000 552 -> 377 us.
template <int M, int L>
__global__ void __launch_bounds__(256, 2) k_ik(const KWorldDev* __restrict__ W, const IkArgs A)
{
  const int lane = threadIdx.x & 31;
  const KRobotDev& R = W->robots[A.robot];
  const int nl = R.nlinks;
  const int link = lane & (L - 1), gbase = lane & ~(L - 1);
  const bool valid = link < nl;
  const int first = blockIdx.x * A.per_block, count = min(A.per_block, A.B - first);
  __shared__ int taken;
  if (threadIdx.x == 0) taken = 0;
  __syncthreads();
  const float lo = valid ? R.qmin[link] : 0.f, hi = valid ? R.qmax[link] : 0.f;
  const bool weld = !valid || R.jtype[link] == KX_JOINT_WELD;
  const bool revolute = valid && R.jtype[link] == KX_JOINT_REVOLUTE;

  int b = -1, it = 0, li = 0;   // b: problem, -1: none
  bool more = true, start = false, active = false;
  float3 pl = make_float3(0.f, 0.f, 0.f);
  float pt[3] = {0.f, 0.f, 0.f}, Rt[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) Rt[k] = 0.f;
  float q = 0.f, P[12], e[M], E = 0.f, emax = 0.f, mu = 1.f;
#pragma unroll
  for (int k = 0; k < 12; ++k) P[k] = 0.f;
#pragma unroll
  for (int a = 0; a < M; ++a) e[a] = 0.1f;
#pragma unroll 1
  for (;;) {
    // ---- the block's next problem for groups without one
    if (__any_sync(0xffffffffu, b < 0 && more)) {
      int nb = -1;
      if (b < 0 && more && link == 0) nb = atomicAdd(&taken, 1);
      nb = __shfl_sync(0xffffffffu, nb, gbase);
      if (b < 0 && more) {
        if (nb >= count) {
          more = false;
        } else {
          nb += first;
          li = A.links ? __ldg(A.links + nb) : A.link_all;
          if (li < 0 || li >= nl) {
            if (link == 0) set_status(W->status, KGPU_ERR_INVALID);
            li = 0;
          } else {
            b = nb;
            start = true;
            it = 0;
            mu = 1e-4f;
            pl = make_float3(A.plocal[3 * (size_t)b], A.plocal[3 * (size_t)b + 1], A.plocal[3 * (size_t)b + 2]);
#pragma unroll
            for (int k = 0; k < 3; ++k) pt[k] = A.ptarget[3 * (size_t)b + k];
            if (M == 6) {
#pragma unroll
              for (int k = 0; k < 9; ++k) Rt[k] = A.Rtarget[9 * (size_t)b + k];
            }
            // active DOFs: the link and its ancestors (other columns of J are 0)
            active = false;
            if (!weld)
              for (int j = li; j >= 0; j = R.parents[j])
                if (j == link) { active = true; break; }
            q = valid ? A.q[(size_t)b * nl + link] : 0.f;
            q = fminf(fmaxf(q, lo), hi);
          }
        }
      }
    }
    if (!__any_sync(0xffffffffu, b >= 0)) {
      if (!__any_sync(0xffffffffu, more)) break;
      continue;
    }
    // ---- column `link` of J at q (angular rows 0-2, linear rows 3-5 as in
    // k_jacobian); the residual orders position first, so row a of the
    // system is linear row a (a < 3) and angular row a - 3 (a >= 3)
    float c[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    {
      float Ti[12];
#pragma unroll
      for (int k = 0; k < 12; ++k) Ti[k] = __shfl_sync(0xffffffffu, P[k], gbase + li);
      const float3 p = xform32(Ti, pl);
      if (b < 0) {
        // a group without a problem computes along: on harmless values, for
        // zeros, infinities or NaN would take the divisions' slow paths, which
        // the whole warp waits for (2x the time of an iteration)
#pragma unroll
        for (int r = 0; r < 6; ++r) c[r] = 0.1f + 0.02f * (float)((link + 3 * r) & 7);
      } else if (active) {
        const float ax = R.axis[link][0], ay = R.axis[link][1], az = R.axis[link][2];
        const float wx = P[0] * ax + P[1] * ay + P[2] * az;
        const float wy = P[3] * ax + P[4] * ay + P[5] * az;
        const float wz = P[6] * ax + P[7] * ay + P[8] * az;
        if (revolute) {
          const float rx = p.x - P[9], ry = p.y - P[10], rz = p.z - P[11];
          c[0] = wy * rz - wz * ry;
          c[1] = wz * rx - wx * rz;
          c[2] = wx * ry - wy * rx;
          c[3] = wx; c[4] = wy; c[5] = wz;
        } else {
          c[0] = wx; c[1] = wy; c[2] = wz;
        }
      }
    }
    // A = J J^T + mu I (symmetric, lower triangle), y = A^-1 e by Cholesky in
    // place, every lane of the group the same values
    float Lc[M * (M + 1) / 2];
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
      for (int s = 0; s <= r; ++s)
        Lc[r * (r + 1) / 2 + s] = group_sum<L>(c[r] * c[s], gbase) + (r == s ? mu : 0.f);
    float y[M];
    bool spd = true;
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
      for (int s = 0; s <= r; ++s) {
        float v = Lc[r * (r + 1) / 2 + s];
#pragma unroll
        for (int t = 0; t < s; ++t) v -= Lc[r * (r + 1) / 2 + t] * Lc[s * (s + 1) / 2 + t];
        if (s == r) {
          spd = spd && v > 0.f;
          Lc[r * (r + 1) / 2 + s] = sqrtf(fmaxf(v, 1e-30f));
        } else {
          Lc[r * (r + 1) / 2 + s] = v / Lc[s * (s + 1) / 2 + s];
        }
      }
    {
      float z[M];
#pragma unroll
      for (int r = 0; r < M; ++r) {
        float v = e[r];
#pragma unroll
        for (int t = 0; t < r; ++t) v -= Lc[r * (r + 1) / 2 + t] * z[t];
        z[r] = v / Lc[r * (r + 1) / 2 + r];
      }
#pragma unroll
      for (int r = M - 1; r >= 0; --r) {
        float v = z[r];
#pragma unroll
        for (int t = r + 1; t < M; ++t) v -= Lc[t * (t + 1) / 2 + r] * y[t];
        y[r] = v / Lc[r * (r + 1) / 2 + r];
      }
    }
    float dq = 0.f;
#pragma unroll
    for (int r = 0; r < M; ++r) dq -= c[r] * y[r];
    // ---- the trial step (a new problem: its start; not positive definite: none)
    const float qn = !valid ? 0.f : (start || !spd ? q : fminf(fmaxf(q + dq, lo), hi));
    float Pn[12], en[M];
    warp_fk32_group<false>(R, lane, L, valid, qn, 0.f, Pn, nullptr);
    ik_residual<M>(Pn, gbase + li, pl, pt, Rt, en);
    float En = 0.f, enmax = 0.f;
#pragma unroll
    for (int a = 0; a < M; ++a) {
      En += en[a] * en[a];
      enmax = fmaxf(enmax, fabsf(en[a]));
    }
    bool done = false;
    if (b >= 0 && (start || (spd && En < E))) {
      q = qn;
#pragma unroll
      for (int t = 0; t < 12; ++t) P[t] = Pn[t];
#pragma unroll
      for (int a = 0; a < M; ++a) e[a] = en[a];
      E = En;
      emax = enmax;
      if (!start) {
        mu = fmaxf(mu * 0.25f, 1e-10f);
        ++it;
      }
    } else if (b >= 0) {
      mu *= 8.f;
      if (mu > 1e6f) done = true;  // gives up
      else ++it;
    }
    start = false;
    done = done || !(it < A.max_iters && emax > A.tol);
    if (b >= 0 && done) {
      if (valid) A.q[(size_t)b * nl + link] = q;
      if (link == 0) {
        A.ok[b] = emax <= A.tol ? 1 : 0;
        A.residual[b] = emax;
        if (A.iters) A.iters[b] = it;
      }
      b = -1;
      mu = 1.f;
#pragma unroll
      for (int a = 0; a < M; ++a) e[a] = 0.1f;
    }
  }
}

}  // namespace

cudaError_t launch_ik(const KWorldDev* W, int robot, int B, float* q, const int* links, int link_all,
                      const float* plocal, const float* ptarget, const float* Rtarget, int max_iters, float tol,
                      uint8_t* ok, float* residual, int* iters, int nlinks, int num_sms,
                      cudaStream_t s)
{
  if (B <= 0) return cudaSuccess;
  IkArgs A;
  A.robot = robot;
  A.B = B;
  A.q = q;
  A.links = links;
  A.link_all = link_all;
  A.plocal = plocal;
  A.ptarget = ptarget;
  A.Rtarget = Rtarget;
  A.max_iters = max_iters;
  A.tol = tol;
  A.ok = ok;
  A.residual = residual;
  A.iters = iters;
  // one wave of blocks (2 of 8 warps per SM), each with its share of the
  // problems: the queue is the block's own, so calls on several streams do not
  // share anything.  (Fewer problems per warp than fit gain nothing even where
  // warps are left over: 9,000 problems 377 us at 4 per warp, 433 us at 1;
  // 554 problems 250 us either way.)
  const int threads = 256;
  A.per_block = (B + 2 * num_sms - 1) / (2 * num_sms);
  const int blocks = (B + A.per_block - 1) / A.per_block;
  const int width = nlinks <= 8 ? 8 : (nlinks <= 16 ? 16 : 32);
  if (width == 8) {
    if (Rtarget) k_ik<6, 8><<<blocks, threads, 0, s>>>(W, A);
    else k_ik<3, 8><<<blocks, threads, 0, s>>>(W, A);
  } else if (width == 16) {
    if (Rtarget) k_ik<6, 16><<<blocks, threads, 0, s>>>(W, A);
    else k_ik<3, 16><<<blocks, threads, 0, s>>>(W, A);
  } else {
    if (Rtarget) k_ik<6, 32><<<blocks, threads, 0, s>>>(W, A);
    else k_ik<3, 32><<<blocks, threads, 0, s>>>(W, A);
  }
  return cudaGetLastError();
}

}  // namespace kgpu
