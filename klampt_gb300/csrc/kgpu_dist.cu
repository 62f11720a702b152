// kgpu_dist.cu — signed link-obstacle distance, its minimum per configuration,
// the soft-min over a trajectory, and the adjoint (gradient) kernels.
//
// Replaces the per-pair Geometry3D::distance_ext loop
// (Python/klampt/src/robotsim.cpp:1782-1819; DistanceQueryResult conventions
// Python/klampt/src/geometry.h:641-673), WorldPlannerSettings::
// DistanceLowerBound (Cpp/Planning/PlannerSettings.cpp:372-483) and the
// autodiff MinDistance / ADModule path (Python/klampt/math/autodiff/
// geometry_ad.py:613-814, pytorch.py:72-115).
//
// Definition (the FP64 oracle's, bit for bit on the value):
//   d(l, o) = min over triangle pairs of the canonical triangle distance
//             (kx_tri_tri_dist2), ties to the smallest (link triangle, object
//             triangle) index;  if that is 0 (surfaces meet) and o is convex,
//             d = -(largest depth of a link vertex inside o), depth(v) =
//             min over o's faces of (n_f . a_f - n_f . v), 0 if no vertex is
//             strictly inside.
//   min distance  = min over enabled (link, object) pairs, ties to the
//                   smallest (link, object);
//   soft-min      = m - tau log sum exp(-(d - m)/tau) over the trajectory's
//                   pairs with d < m + K tau (K = 30), m the trajectory minimum.
//
// GPU method, one warp per configuration (the soft-min: one warp per pair, see
// below):
//   * FP32 FK with per-link error bounds (warp_fk32);
//   * candidate (link, object) pairs from the object-aware environment tree by
//     box lower bounds, evaluated nearest first; for the minimum, the bound
//     starts at 5 cm and grows x4 until a pair is found below it;
//   * per pair a warp-cooperative BVH-vs-BVH distance traversal in FP32 with
//     conservative pruning; triangle pairs whose FP32 distance lies within the
//     error band of the running minimum become candidates and are finalised
//     in canonical FP64 (one pair per lane, lexicographic warp reduction);
//     a pair certified intersecting in FP32 ends the search (distance 0);
//   * depth: link vertices inside the object's box, FP32 min over faces,
//     FP64 for those within the band of the deepest;
//   * gradient: dd/dq_j = u . (w_j x (p - o_j)) (revolute), u . w_j
//     (prismatic), with u = dd/dp at the link feature point p, accumulated as
//     per-link force/moment sums and pulled back through the chain once per
//     configuration (the adjoint of FK), on FP32 transforms.
#include <algorithm>
#include <cstddef>
#include <cfloat>
#include <climits>

#include "kgpu_device.cuh"
#include "kgpu_pairdist.cuh"

namespace kgpu {

namespace {

constexpr int kDW = 8;         // warps per block
constexpr int kDGStack = 512;  // environment-tree stack for gathering objects
constexpr int kDPairs = 128;   // gathered (link, object) candidates
constexpr double kSoftK = 30.0;  // pairs beyond m + 30 tau weigh < e^-30 of the leading term

struct __align__(16) DistSmem {
  // what a pair's evaluation needs ...
  PairSmem P;
  float T[kMaxLinks][12];
  float delta[kMaxLinks];
  double q64[kMaxLinks];
  const float* item_qa;
  const float* item_qb;
  int item_k, item_n;
  // ... and what gathering the pairs and the gradient need besides: kernels
  // that only evaluate pairs leave it out (kEvalSmem), and the L1 gains it
  // (soft-min over 6,400 waypoints: 3%)
  __align__(16) uint32_t gstack[kDGStack];
  int pobj[kDPairs];
  int plink[kDPairs];
  float plb[kDPairs];
  float F[kMaxLinks][3], M[kMaxLinks][3];
};
constexpr size_t kEvalSmem = offsetof(DistSmem, gstack);

struct DistArgs {
  int robot;
  const float* q;      // [B, L]
  int B;
  double cutoff;
  double* d;           // [B]
  int* pair;           // [B*2]
  double* cp;          // [B*6]
  float* grad;         // [B*L] (mode 0: dd/dq, mode 2: unnormalised soft-min gradient)
  // soft-min (modes 1 and 2): waypoints first .. first + B whose nseg is -1
  // (their pairs did not fit the list), see SoftArgs
  const int* nseg;
  const float *T, *delta;    // FP32 transforms of the chunk
  int first;
  unsigned long long* mkey;  // [T] trajectory minima (double_key)
  double* wsum;        // mode 2: [waypoints] sums
  int W;               // waypoints per trajectory
  double tau;
  unsigned int* head;
  uint2* scratch;
  int scratch_per_warp;
};

// doubles as unsigned integers in the same order, for atomicMin
__device__ __forceinline__ unsigned long long double_key(double d)
{
  const unsigned long long u = (unsigned long long)__double_as_longlong(d);
  return (u >> 63) ? ~u : u | (1ull << 63);
}

constexpr double kSoftCutoff = 1e3;  // pairs farther than this are not looked for

// a trajectory's minimum from its key (all ones: none found yet)
__device__ __forceinline__ double key_min(unsigned long long k)
{
  if (k == ~0ull) return kSoftCutoff;
  return __longlong_as_double((long long)((k >> 63) ? k & ~(1ull << 63) : ~k));
}

struct DCnt {
  unsigned long long pairs = 0;
  PairCnt p;  // per lane
};

// (No distance kernel sets an edge's second end.  Without this branch, the
// soft-min takes 40.4 instead of 39.4 ms over 6,400 waypoints, the same with the
// shared memory's layout kept: its kernels are bound by fetching their code, and
// this moves it.)
__device__ __forceinline__ double item_q64(const DistSmem& S, int lane)
{
  if (S.item_qb == nullptr) return (double)S.item_qa[lane];
  return kx_interp((double)S.item_qa[lane], (double)S.item_qb[lane], S.item_k, S.item_n);
}

__device__ __noinline__ void dist_fk64(DistSmem& S, const KRobotDev& R, double (*T64)[12], int lane, int& fk64)
{
  if (fk64) return;
  if (lane < R.nlinks) S.q64[lane] = item_q64(S, lane);
  __syncwarp();
  warp_fk64(R, S.q64, T64, lane);
  fk64 = 1;
}

// An upper bound on the distance between the surfaces of link l and object
// o: the link vertex nearest the centre of o's box and the vertex of o (the
// first vertex of each of its triangles) nearest that link vertex are both
// surface points; widened by the FP32 placement bounds and rounding.  Seeds
// a pair's running minimum, so that its traversal prunes from the start.
constexpr int kSeedMaxTris = 4096;  // objects up to this size are scanned for a seed

__device__ __noinline__ float pair_seed(DistSmem& S, const KWorldDev* __restrict__ W, const KRobotDev& R, int lane,
                                        int l, int o)
{
  const int ff = W->obj_leaf_first[o], fc = W->obj_leaf_count[o];
  if (fc > kSeedMaxTris) return FLT_MAX;  // large objects (terrains): no seed
  const KNode ob = W->enodes[W->obj_root[o]];
  const float* TA = S.T[l];
  const int vf = R.link_vert_first[l], vc = R.link_vert_count[l];
  float bd = FLT_MAX;
  float3 bv = make_float3(ob.a.x, ob.a.y, ob.a.z);
#pragma unroll 2
  for (int v = lane; v < vc; v += 32) {
    const float4 x = __ldg(W->lvert32 + vf + v);
    const float3 w = xform32(TA, make_float3(x.x, x.y, x.z));
    const float dx = w.x - ob.a.x, dy = w.y - ob.a.y, dz = w.z - ob.a.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    if (d2 < bd) { bd = d2; bv = w; }
  }
  const float m = warp_min(bd);
  if (!(m < FLT_MAX)) return FLT_MAX;  // no vertex: no surface point, no seed
  const unsigned mm = __ballot_sync(0xffffffffu, bd == m);
  const int src = __ffs(mm) - 1;
  bv = make_float3(__shfl_sync(0xffffffffu, bv.x, src), __shfl_sync(0xffffffffu, bv.y, src),
                   __shfl_sync(0xffffffffu, bv.z, src));
  float bo = FLT_MAX;
#pragma unroll 2
  for (int t = lane; t < fc; t += 32) {
    const float4 y = __ldg(W->etri32 + 3 * (size_t)(ff + t));
    const float dx = y.x - bv.x, dy = y.y - bv.y, dz = y.z - bv.z;
    bo = fminf(bo, dx * dx + dy * dy + dz * dz);
  }
  bo = warp_min(bo);
  if (!(bo < FLT_MAX)) return FLT_MAX;
  return sqrtf(bo) * (1.f + 1e-5f) + 2.f * (S.delta[l] + W->eps_env + 2.f * W->eps_extra) + 1e-6f;
}

// FP32 bound of a vertex's depth inside object o against its exact value:
// placement of the vertex, rounding of the planes and of their products
__device__ __forceinline__ float depth_band(const KNode& ob, float dd)
{
  return dd + 32.f * kU * (fabsf(ob.a.x) + fabsf(ob.a.y) + fabsf(ob.a.z) + fabsf(ob.b.x) + fabsf(ob.b.y) +
                           fabsf(ob.b.z) + 1.f);
}

// Whether some vertex of link l may lie at least `need` >= 0 deep inside the
// convex object o; otherwise the pair's signed distance is above -need (or
// not negative, for need = 0).  One pass over the vertices, a few thousand
// cycles; the pair's own evaluation (the search for a certified contact, then
// its deepest vertex in FP64) takes a few hundred thousand.  Among boxes most
// pairs a configuration still has to look at after its first contact are
// shallower contacts: 32,768 terrain clearances 38.9 -> 27.4 ms with this test
// (19-21 by the drawn configurations with the later work on the pair traversal).
__device__ __noinline__ bool may_be_deeper(const DistSmem& S, const KWorldDev* __restrict__ W, const KRobotDev& R,
                                           int lane, int l, int o, float need)
{
  const KNode ob = W->enodes[W->obj_root[o]];
  const float dd = S.delta[l] + W->eps_env + 2.f * W->eps_extra;
  const float tolb = dd + 8.f * kU * (fabsf(ob.a.x) + fabsf(ob.a.y) + fabsf(ob.a.z) + 1.f);
  const float stop = need * (1.f - 1e-6f) - 2.f * depth_band(ob, dd);
  const int ff = W->obj_leaf_first[o], fc = W->obj_leaf_count[o];
  const int vf = R.link_vert_first[l], vc = R.link_vert_count[l];
#pragma unroll 1
  for (int base = 0; base < vc; base += 32) {
    bool deep = false;
    if (base + lane < vc) {
      const float4 x = __ldg(W->lvert32 + vf + base + lane);
      const float3 w = xform32(S.T[l], make_float3(x.x, x.y, x.z));
      deep = fabsf(w.x - ob.a.x) <= ob.b.x + tolb && fabsf(w.y - ob.a.y) <= ob.b.y + tolb &&
             fabsf(w.z - ob.a.z) <= ob.b.z + tolb;
#pragma unroll 1
      for (int f = ff; f < ff + fc && deep; ++f) {
        const float4 pl = __ldg(W->eface32 + f);
        deep = pl.w - (pl.x * w.x + pl.y * w.y + pl.z * w.z) >= stop;
      }
    }
    if (__any_sync(0xffffffffu, deep)) return true;
  }
  return false;
}

struct PairOut {
  int found;
  double d;
  double cp[3], cq[3];
  float dir[3];
};

// The deepest vertex of link l inside the convex object o (canonical FP64
// depth, ties to the smaller vertex) and the face it is nearest to; 0 and no
// vertex when none is strictly inside.  Out of line: contacts are rare in some
// workloads, and its code is larger than the traversal's.
__device__ __noinline__ double link_depth(DistSmem& S, const KWorldDev* __restrict__ W, const KRobotDev& R,
                                          double (*T64)[12], int& fk64, int lane, int l, int o, float dd, int& vbest,
                                          int& fbest)
{
  const float* TA = S.T[l];
  double depth = 0.0;
  // deepest link vertex inside the convex object
  const int vf = R.link_vert_first[l], vc = R.link_vert_count[l];
  const KNode ob = W->enodes[W->obj_root[o]];
  const float tolb = dd + 8.f * kU * (fabsf(ob.a.x) + fabsf(ob.a.y) + fabsf(ob.a.z) + 1.f);
  const int ff = W->obj_leaf_first[o], fc = W->obj_leaf_count[o];
  const float ed = depth_band(ob, dd);
  float lmax = -FLT_MAX;
  // pass 1: FP32 depths, lane-local maximum.  Each lane also keeps the (at
  // most two) vertices whose pass-1 value lies within 2 ed of its running
  // maximum: pass 1's value bounds a vertex's full FP32 minimum from
  // above, and the global maximum is at least the lane's, so every vertex
  // that pass 2 can accept is among them, unless more than two qualified
  // (then the lane rescans all of its vertices)
  int cv0 = 0, cv1 = 0, nc = 0;
  float cd0 = 0.f, cd1 = 0.f;
  bool rescan = false;
#pragma unroll 1
  for (int v = lane; v < vc; v += 32) {
    const float4 x = __ldg(W->lvert32 + vf + v);
    const float3 w = xform32(TA, make_float3(x.x, x.y, x.z));
    if (fabsf(w.x - ob.a.x) > ob.b.x + tolb || fabsf(w.y - ob.a.y) > ob.b.y + tolb ||
        fabsf(w.z - ob.a.z) > ob.b.z + tolb)
      continue;
    // a vertex stops counting once it is no deeper than the deepest so far
    // (or outside the band): its final minimum can only be lower
    const float stop = fmaxf(lmax, -ed);
    float dmin = FLT_MAX;
#pragma unroll 1
    for (int f = ff; f < ff + fc && dmin > stop; ++f) {
      const float4 pl = __ldg(W->eface32 + f);
      dmin = fminf(dmin, pl.w - (pl.x * w.x + pl.y * w.y + pl.z * w.z));
    }
    lmax = fmaxf(lmax, dmin);
    const float thr = lmax - 2.f * ed;
    if (dmin > -ed && dmin >= thr) {
      if (nc == 2 && cd1 < thr) nc = 1;
      if (nc >= 1 && cd0 < thr) {
        if (nc == 2) { cv0 = cv1; cd0 = cd1; }
        --nc;
      }
      if (nc == 0) { cv0 = v; cd0 = dmin; nc = 1; }
      else if (nc == 1) { cv1 = v; cd1 = dmin; nc = 2; }
      else rescan = true;
    }
  }
  const float gmax = -warp_min(-lmax);
  if (gmax > -ed) {
    dist_fk64(S, R, T64, lane, fk64);
    // pass 2: FP64 depth of every vertex within the band of the deepest
    double bd = 0.0;
    int bv = INT_MAX, bf = -1;
    auto depth64 = [&](int v) {
      const float4 x = __ldg(W->lvert32 + vf + v);
      const float3 w = xform32(TA, make_float3(x.x, x.y, x.z));
      if (fabsf(w.x - ob.a.x) > ob.b.x + tolb || fabsf(w.y - ob.a.y) > ob.b.y + tolb ||
          fabsf(w.z - ob.a.z) > ob.b.z + tolb)
        return;
      const float stop = fmaxf(gmax - 2.f * ed, -ed);
      float dmin = FLT_MAX;
#pragma unroll 1
      for (int f = ff; f < ff + fc && dmin >= stop; ++f) {
        const float4 pl = __ldg(W->eface32 + f);
        dmin = fminf(dmin, pl.w - (pl.x * w.x + pl.y * w.y + pl.z * w.z));
      }
      if (dmin < gmax - 2.f * ed || dmin <= -ed) return;
      double w64[3];
      kx_xform_point(T64[l], W->lvert64 + 3 * (size_t)(vf + v), w64);
      double dm = DBL_MAX;
      int fm = -1, fo = INT_MAX;
#pragma unroll 1
      for (int f = ff; f < ff + fc; ++f) {
        // (the nearest face in FP64 lies within the band of the nearest in FP32)
        const float4 pl32 = __ldg(W->eface32 + f);
        if (pl32.w - (pl32.x * w.x + pl32.y * w.y + pl32.z * w.z) > dmin + 2.f * ed) continue;
        const double* pl = W->eface64 + 4 * (size_t)f;
        const double dep = kx_sub(pl[3], kx_dot3(pl, w64));
        const int orig = W->etri_orig[f];
        if (dep < dm || (dep == dm && orig < fo)) { dm = dep; fm = f; fo = orig; }
      }
      if (dm > bd || (dm == bd && dm > 0.0 && v < bv)) { bd = dm; bv = v; bf = fm; }
    };
    if (rescan) {
#pragma unroll 1
      for (int v = lane; v < vc; v += 32) depth64(v);
    } else {
      if (nc >= 1 && cd0 >= gmax - 2.f * ed) depth64(cv0);
      if (nc >= 2 && cd1 >= gmax - 2.f * ed) depth64(cv1);
    }
    // warp maximum of (depth, -vertex)
    double wd = bd;
    int wv = bd > 0.0 ? bv : INT_MAX, wf = bf, src = lane;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double od = __shfl_xor_sync(0xffffffffu, wd, off);
      const int ov = __shfl_xor_sync(0xffffffffu, wv, off);
      const int ofc = __shfl_xor_sync(0xffffffffu, wf, off);
      const int os = __shfl_xor_sync(0xffffffffu, src, off);
      if (od > wd || (od == wd && (ov < wv || (ov == wv && os < src)))) { wd = od; wv = ov; wf = ofc; src = os; }
    }
    if (wd > 0.0) {
      depth = wd;
      vbest = wv;
      fbest = wf;
    }
  }
  return depth;
}

// Signed distance of (link l, object o) below `bound` (found = d < bound).
__device__ __noinline__ void eval_pair(DistSmem& S, const KWorldDev* __restrict__ W, const KRobotDev& R,
                                       double (*T64)[12], int& fk64, int lane, int l, int o, double bound,
                                       PairOut& out, DCnt& cnt, float seed = FLT_MAX)
{
  cnt.pairs++;
  const float dl = S.delta[l] + W->eps_extra;
  const float de = W->eps_env + W->eps_extra;
  // running FP32 upper bound of the minimum: the search bound, or a seed
  float m32 = fminf(seed, bound > 0.0 ? (bound < 1e30 ? (float)bound * 1.000001f + 1e-7f : FLT_MAX) : 0.f);
  int certA = -1;  // link triangle of the certified contact
  __syncwarp();    // (the previous pair's results have been read)
  if (lane == 0) {
    S.P.b2 = DBL_MAX;
    S.P.bA = INT_MAX;
    S.P.bB = INT_MAX;
    S.P.have = 0;
  }
  const float* TA = S.T[l];
  const MeshView A = {W->lnodes, W->lnode_r, W->ltri32, W->ltri64, W->ltri_orig};
  const MeshView B = {W->enodes, nullptr, W->etri32, W->etri64, W->etri_orig};
  const int r = pair_distance<true, true>(S.P, A, B, R.link_root[l], W->obj_root[o], TA, nullptr, T64[l], nullptr,
                                          dl + de, m32, certA, lane, cnt.p,
                                          [&] { dist_fk64(S, R, T64, lane, fk64); });
  if (r == 2) {
    if (lane == 0) set_status(W->status, KGPU_ERR_OVERFLOW);
    out.found = 0;
    return;
  }
  if (r == 0 && !S.P.have) { out.found = 0; return; }
  // unsigned distance: exact zero (certified contact) or the FP64 minimum
  const bool zero = r == 1 || S.P.b2 == 0.0;
  if (!zero) {
    const double d = kx_sqrt(S.P.b2);
    out.found = d < bound;
    out.d = d;
    // (the three divisions on three lanes: one FP64 sequence instead of three)
    const int c = lane < 3 ? lane : 0;
    const float dir = (float)((S.P.bcp[c] - S.P.bcq[c]) / d);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      out.cp[i] = S.P.bcp[i];
      out.cq[i] = S.P.bcq[i];
      out.dir[i] = __shfl_sync(0xffffffffu, dir, i);
    }
    return;
  }
  // ---- surfaces meet
  int vbest = -1, fbest = -1;
  double depth = 0.0;
  if (W->obj_convex[o]) depth = link_depth(S, W, R, T64, fk64, lane, l, o, dl + de, vbest, fbest);
  if (vbest >= 0) {
    double w64[3];
    kx_xform_point(T64[l], W->lvert64 + 3 * (size_t)(R.link_vert_first[l] + vbest), w64);
    const double* pl = W->eface64 + 4 * (size_t)fbest;
    out.d = -depth;
    out.found = -depth < bound;
    for (int i = 0; i < 3; ++i) {
      out.cp[i] = w64[i];
      out.cq[i] = kx_add(w64[i], kx_mul(depth, pl[i]));
      out.dir[i] = (float)pl[i];
    }
    return;
  }
  // contact without a vertex inside (or a non-convex object): d = 0, no direction
  out.d = 0.0;
  out.found = 0.0 < bound;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (certA >= 0) x = __ldg(W->ltri32 + 3 * (size_t)certA);
  const float3 w = xform32(TA, make_float3(x.x, x.y, x.z));
  out.cp[0] = out.cq[0] = w.x;
  out.cp[1] = out.cq[1] = w.y;
  out.cp[2] = out.cq[2] = w.z;
  out.dir[0] = out.dir[1] = out.dir[2] = 0.f;
}

// Gathers objects of group g whose root box is within `bound` of link l's
// world box (lower bound lb in plb) and lb > lower (already handled), into
// S.pobj/plb starting at `count`; stops early when the list is full (the
// caller then evaluates and calls again with `resume` state in the stack).
// Returns the new count; `top` carries the traversal stack between calls.
// ORDERED: the culling sets in which order the pairs are listed, and with it
// the order of a soft-min's FP32 sums, so the soft-min keeps rounded roots (with
// one-instruction ones, 2 of a batch's 44,800 gradient entries moved by 1.4e-9).
// A minimum does not depend on the order: rounded roots there cost 32,768
// clearances 4%.
template <bool ORDERED>
__device__ int gather_objects(DistSmem& S, const KWorldDev* __restrict__ W, const KRobotDev& R, int lane, int l,
                              float bound, float lower, int count, int& top)
{
  const unsigned lt = lanemask_lt();
  const KNode la = W->lnodes[R.link_root[l]];
  const Box32 A = xform_box(S.T[l], la.a, la.b);
  const float slack = (S.delta[l] + W->eps_env + 2.f * W->eps_extra) * 1.7321f +
                      4.f * kU * (fabsf(A.c.x) + fabsf(A.c.y) + fabsf(A.c.z) + 1.f) + 1e-7f;
  const float rad = __ldg(W->lnode_r + R.link_root[l]);
  while (top > 0 && count <= kDPairs - 32) {
    if (top > kDGStack - 64) {
      if (lane == 0) set_status(W->status, KGPU_ERR_OVERFLOW);
      top = 0;
      break;
    }
    const int n = min(top, 32);
    const bool have = lane < n;
    int node = 0;
    if (have) node = (int)S.gstack[top - 1 - lane];
    __syncwarp();
    top -= n;
    int outcome = 0;
    float lbv = 0.f;
    int child = 0;
    if (have) {
      const KNode nb = W->enodes[node];
      const float gx = fmaxf(0.f, fabsf(A.c.x - nb.a.x) - nb.b.x);
      const float gy = fmaxf(0.f, fabsf(A.c.y - nb.a.y) - nb.b.y);
      const float gz = fmaxf(0.f, fabsf(A.c.z - nb.a.z) - nb.b.z);
      const float bx = fmaxf(0.f, fabsf(A.c.x - nb.a.x) - A.h.x - nb.b.x);
      const float by = fmaxf(0.f, fabsf(A.c.y - nb.a.y) - A.h.y - nb.b.y);
      const float bz = fmaxf(0.f, fabsf(A.c.z - nb.a.z) - A.h.z - nb.b.z);
      const float b2 = bx * bx + by * by + bz * bz, g2 = gx * gx + gy * gy + gz * gz;
      lbv = (ORDERED ? fmaxf(sqrtf(b2), sqrtf(g2) * (1.f - 4.f * kU) - rad)
                     : fmaxf(root_below32(b2), root_below32(g2) - rad)) -
            slack;
      if (lbv <= bound) {
        const int o = W->node_obj[node];
        if (o >= 0) {
          outcome = lbv > lower ? 2 : 0;
          child = o;
        } else {
          outcome = 1;
          child = f2i(nb.a.w);
        }
      }
    }
    const unsigned m1 = __ballot_sync(0xffffffffu, outcome == 1);
    const unsigned m2 = __ballot_sync(0xffffffffu, outcome == 2);
    if (outcome == 1) {
      const int r = top + 2 * __popc(m1 & lt);
      S.gstack[r] = (uint32_t)child + 1;
      S.gstack[r + 1] = (uint32_t)child;
    } else if (outcome == 2) {
      const int r = count + __popc(m2 & lt);
      S.pobj[r] = child;
      S.plink[r] = l;
      S.plb[r] = lbv;
    }
    top += 2 * __popc(m1);
    count += __popc(m2);
    __syncwarp();
  }
  return count;
}

// The sums of a gradient, with their roundings spelled out: a soft-min waypoint
// goes through k_soft_reduce or, when its pairs do not fit the list, through
// k_dist<2>; which of the two can depend on the scheduling, and the compiler
// need not fuse the products of two kernels alike.
__device__ __forceinline__ float diff_products(float a, float b, float c, float d)
{
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}
__device__ __forceinline__ float dot_rn(float ax, float ay, float az, float bx, float by, float bz)
{
  return __fmaf_rn(az, bz, __fmaf_rn(ax, bx, __fmul_rn(ay, by)));
}

// Adds the weighted direction u = wgt * d at point p to a link's force and
// moment sums.
__device__ __forceinline__ void wrench_sum(float* F, float* M, float wgt, float dx, float dy, float dz, float px,
                                           float py, float pz)
{
  const float ux = __fmul_rn(wgt, dx), uy = __fmul_rn(wgt, dy), uz = __fmul_rn(wgt, dz);
  F[0] = __fadd_rn(F[0], ux);
  F[1] = __fadd_rn(F[1], uy);
  F[2] = __fadd_rn(F[2], uz);
  M[0] = __fadd_rn(M[0], diff_products(py, uz, pz, uy));
  M[1] = __fadd_rn(M[1], diff_products(pz, ux, px, uz));
  M[2] = __fadd_rn(M[2], diff_products(px, uy, py, ux));
}

// Adds a pair's contribution (weight wgt, feature point p, direction u) to
// the per-link force / moment accumulators.
__device__ __forceinline__ void add_wrench(DistSmem& S, int lane, int l, float wgt, const PairOut& po)
{
  if (lane == 0)
    wrench_sum(S.F[l], S.M[l], wgt, po.dir[0], po.dir[1], po.dir[2], (float)po.cp[0], (float)po.cp[1], (float)po.cp[2]);
  __syncwarp();
}

// Adjoint of FK: gradient g_j = w_j . (M_sub(j) - o_j x F_sub(j)) for a
// revolute joint, w_j . F_sub(j) for a prismatic one, with F_sub/M_sub the
// sums over link j's subtree (children have larger indices than parents).
__device__ void pullback(DistSmem& S, const KRobotDev& R, int lane, float* g_out)
{
  const int nl = R.nlinks;
  if (lane == 0) {
    for (int i = nl - 1; i > 0; --i) {
      const int p = R.parents[i];
      if (p < 0) continue;
      for (int k = 0; k < 3; ++k) {
        S.F[p][k] += S.F[i][k];
        S.M[p][k] += S.M[i][k];
      }
    }
  }
  __syncwarp();
  if (lane < nl && g_out) {
    const float* T = S.T[lane];
    const float* a = R.axis[lane];
    const float wx = dot_rn(T[0], T[1], T[2], a[0], a[1], a[2]);
    const float wy = dot_rn(T[3], T[4], T[5], a[0], a[1], a[2]);
    const float wz = dot_rn(T[6], T[7], T[8], a[0], a[1], a[2]);
    float g = 0.f;
    if (R.jtype[lane] == KX_JOINT_REVOLUTE) {
      const float ox = T[9], oy = T[10], oz = T[11];
      const float* F = S.F[lane];
      const float* M = S.M[lane];
      const float tx = __fsub_rn(M[0], diff_products(oy, F[2], oz, F[1]));
      const float ty = __fsub_rn(M[1], diff_products(oz, F[0], ox, F[2]));
      const float tz = __fsub_rn(M[2], diff_products(ox, F[1], oy, F[0]));
      g = dot_rn(wx, wy, wz, tx, ty, tz);
    } else if (R.jtype[lane] == KX_JOINT_PRISMATIC) {
      g = dot_rn(wx, wy, wz, S.F[lane][0], S.F[lane][1], S.F[lane][2]);
    }
    g_out[lane] = g;
  }
  __syncwarp();
}

// adds a warp's counters to the world's: pairs are counted once per warp
// (lane 0), the rest per lane
__device__ __forceinline__ void count_pairs(const KWorldDev* __restrict__ W, const DCnt& cnt, int lane)
{
  unsigned long long nd = cnt.p.nodes, tp = cnt.p.tri, bd = cnt.p.fp64;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    nd += __shfl_down_sync(0xffffffffu, nd, o);
    tp += __shfl_down_sync(0xffffffffu, tp, o);
    bd += __shfl_down_sync(0xffffffffu, bd, o);
  }
  if (lane == 0 && W->stats) {
    atomicAdd(W->stats + 8, cnt.pairs);
    atomicAdd(W->stats + 9, nd);
    atomicAdd(W->stats + 10, tp);
    atomicAdd(W->stats + 11, bd);
  }
}

// MODE: 0 minimum distance with closest points and gradient; 1 and
// 2 the soft-min's two passes (trajectory minima, every pair below m + K tau)
// for the waypoints whose pairs did not fit the soft-min's list; one
// instantiation each, so that a launch carries only its mode's code
template <int MODE>
__global__ void __launch_bounds__(kDW * 32, 2) k_dist(const KWorldDev* __restrict__ W, const DistArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DistSmem* all = reinterpret_cast<DistSmem*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  DistSmem& S = all[warp];
  const int gwarp = blockIdx.x * kDW + warp;
  double(*T64)[12] = reinterpret_cast<double(*)[12]>(A.scratch + (size_t)gwarp * A.scratch_per_warp);
  const KRobotDev& R = W->robots[A.robot];
  const int nl = R.nlinks;
  DCnt cnt;

  for (;;) {
    unsigned int it = 0;
    if (lane == 0) it = atomicAdd(A.head, 1u);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it >= (unsigned)A.B) break;
    const int b = MODE == 0 ? (int)it : A.first + (int)it;
    if (MODE != 0 && A.nseg[it] >= 0) continue;
    if (lane == 0) {
      S.item_qa = A.q + (size_t)b * nl;
      S.item_qb = nullptr;
      S.item_k = 0;
      S.item_n = 0;
    }
    float q = lane < nl ? __ldg(A.q + (size_t)b * nl + lane) : 0.f;
    __syncwarp();
    if (__any_sync(0xffffffffu, lane < nl && !(fabsf(q) < 1.0e6f))) {
      if (lane == 0) set_status(W->status, KGPU_ERR_NOT_FINITE);
      continue;
    }
    float P[12], delta;
    if (MODE == 0) {
      warp_fk32(R, lane, q, 0.f, P, &delta);
    } else if (lane < nl) {  // the chunk's, so that both ways of a waypoint see the same
      const size_t at = (size_t)it * nl + lane;
      for (int i = 0; i < 12; ++i) P[i] = __ldg(A.T + at * 12 + i);
      delta = __ldg(A.delta + at);
    }
    if (lane < nl) {
      for (int i = 0; i < 12; ++i) S.T[lane][i] = P[i];
      S.delta[lane] = delta;
      S.F[lane][0] = S.F[lane][1] = S.F[lane][2] = 0.f;
      S.M[lane][0] = S.M[lane][1] = S.M[lane][2] = 0.f;
    }
    __syncwarp();
    int fk64 = 0;

    if (MODE == 0 || MODE == 1) {
      // ---- minimum over pairs, iterative deepening of the search bound
      double best = A.cutoff;
      // its FP32 neighbours for the comparisons of the pair loops (an FP64 one
      // costs the SM as much as 40 of FP32): rounded up, the reach of a box
      // bound (boxes bound the unsigned distance: a pair can be negative only
      // when its boxes meet), and whether the rounding was exact
      float best_up, reach;
      bool best_exact;
      auto set_best = [&](double d) {
        best = d;
        best_up = __double2float_ru(d);
        best_exact = (double)best_up == d;
        reach = fmaxf(best_up, 0.f) * 1.00001f + 1e-6f;
      };
      set_best(A.cutoff);
      int bl = -1, bo = -1;
      PairOut bp;
      bp.found = 0;
      // rounds: objects whose box lower bound lies in (lower, bound]; done
      // once the best distance is <= bound (every unvisited object is
      // farther) or the bound reached the cutoff
      float lower = -1.f;
      double round_bound = fmin(A.cutoff, 0.05);
      // evaluates the gathered (link, object) pairs nearest first, over all
      // links at once, so that the closest pair of any link sets the bound
      // that prunes the rest
      auto eval_list = [&](int np) {
        for (int done = 0; done < np; ++done) {
          float v = FLT_MAX;
          int idx = -1;
          for (int k = lane; k < np; k += 32)
            if (S.plb[k] < v) { v = S.plb[k]; idx = k; }
          const float vm = warp_min(v);
          const unsigned mm = __ballot_sync(0xffffffffu, v == vm && idx >= 0);
          if (mm == 0u) break;
          const int owner = __ffs(mm) - 1;
          const int k = __shfl_sync(0xffffffffu, idx, owner);
          if (lane == 0) S.plb[k] = FLT_MAX;
          __syncwarp();
          if (vm > reach) break;
          const int o = S.pobj[k], l = S.plink[k];
          // a pair cannot go below 0 unless its object is convex, and then
          // not below minus the smallest half-extent of the object's box
          // (no point lies deeper inside a convex body that fits in the
          // box): once the best is at or under that, the pair can at most
          // tie, which only a smaller (link, object) would win.  Nor can it
          // go below minus the depth of the link's deepest vertex in it
          if (bl >= 0) {
            const bool convex = W->obj_convex[o] != 0, tie = l < bl || (l == bl && o < bo);
            const float4 oh = W->enodes[W->obj_root[o]].b;
            const float dlow = convex ? -fminf(fminf(oh.x, oh.y), oh.z) : 0.f;
            if (dlow > best_up || (dlow == best_up && !(best_exact && tie))) continue;
            if (convex && best_up <= 0.f && !(best == 0.0 && tie) &&
                !may_be_deeper(S, W, R, lane, l, o, -best_up))
              continue;
          }
          PairOut po;
          // the first pair has no running bound to prune with yet: seed it
          eval_pair(S, W, R, T64, fk64, lane, l, o, nextafter(best, 1e300), po, cnt,
                    bl < 0 ? pair_seed(S, W, R, lane, l, o) : FLT_MAX);
          if (po.found && (po.d < best || (po.d == best && (l < bl || (l == bl && o < bo))))) {
            set_best(po.d);
            bl = l;
            bo = o;
            bp = po;
          }
        }
      };
      for (;;) {
        const float bound = round_bound >= A.cutoff ? FLT_MAX : (float)round_bound * 1.000001f;
        int np = 0;
        for (int l = 0; l < nl; ++l) {
          if (R.link_root[l] < 0) continue;
          for (int g = 0; g < kMaxGroups; ++g) {
            if (!((R.env_mask[l] >> g) & 1u) || W->group_root[g] < 0) continue;
            int top = 1;
            if (lane == 0) S.gstack[0] = (uint32_t)W->group_root[g];
            __syncwarp();
            while (top > 0) {
              np = gather_objects<MODE != 0>(S, W, R, lane, l, fminf(bound, reach), lower, np, top);
              if (top > 0) {
                // list full: evaluate what it holds, then keep gathering
                eval_list(np);
                np = 0;
              }
            }
          }
        }
        eval_list(np);
        if (best <= round_bound || round_bound >= A.cutoff) break;
        lower = bound;
        round_bound = fmin(A.cutoff, round_bound * 4.0);
      }
      if (MODE == 1) {
        if (lane == 0 && bl >= 0) atomicMin(A.mkey + b / A.W, double_key(best));
      } else if (lane == 0) {
        A.d[b] = bl >= 0 ? best : A.cutoff;
        A.pair[2 * (size_t)b] = bl;
        A.pair[2 * (size_t)b + 1] = bo;
        for (int i = 0; i < 3; ++i) {
          A.cp[6 * (size_t)b + i] = bl >= 0 ? bp.cp[i] : 0.0;
          A.cp[6 * (size_t)b + 3 + i] = bl >= 0 ? bp.cq[i] : 0.0;
        }
      }
      if (MODE == 0 && A.grad) {
        if (bl >= 0) add_wrench(S, lane, bl, 1.f, bp);
        pullback(S, R, lane, A.grad + (size_t)b * nl);
      }
    } else {
      // ---- soft-min pass 2: every pair below m + K tau
      const int t = b / A.W;
      const double m = key_min(A.mkey[t]);
      const double bnd = m + kSoftK * A.tau;
      double sum = 0.0;
      const float fbnd = (float)fmax(bnd, 0.0) * 1.000001f + 1e-6f;
      for (int l = 0; l < nl; ++l) {
        if (R.link_root[l] < 0) continue;
        for (int g = 0; g < kMaxGroups; ++g) {
          if (!((R.env_mask[l] >> g) & 1u) || W->group_root[g] < 0) continue;
          int top = 1;
          if (lane == 0) S.gstack[0] = (uint32_t)W->group_root[g];
          __syncwarp();
          while (top > 0) {
            const int np = gather_objects<true>(S, W, R, lane, l, fbnd, -1.f, 0, top);
            for (int k = 0; k < np; ++k) {
              PairOut po;
              const int o = S.pobj[k];
              eval_pair(S, W, R, T64, fk64, lane, l, o, bnd, po, cnt, pair_seed(S, W, R, lane, l, o));
              if (!po.found) continue;
              const double e = exp(-(po.d - m) / A.tau);
              sum += e;
              add_wrench(S, lane, l, (float)e, po);
            }
          }
        }
      }
      if (lane == 0) A.wsum[b] = sum;
      pullback(S, R, lane, A.grad ? A.grad + (size_t)b * nl : nullptr);
    }
  }
  count_pairs(W, cnt, lane);
}

// ---- soft-min over a trajectory -----------------------------------------------
// The pairs of all waypoints go into one list, and every warp of the GPU
// takes pairs from it: one trajectory of 32 waypoints has a few thousand pairs
// within 30 tau of its minimum, and one waypoint's are up to a few hundred, so
// a warp per waypoint leaves the GPU idle or waiting for the last ones (one
// trajectory 33-72 -> 1.7 ms, 200 trajectories 98.5 -> 54 ms; 1.5 and 40 ms with
// the later work on the pair traversal).  Per chunk of waypoints:
//   k_soft_fk       FP32 and FP64 forward kinematics, kept for the chunk;
//   k_soft_bound    an upper bound of each trajectory's minimum, from the
//                   pairs nearest by their boxes at each waypoint;
//   k_soft_gather   pairs within reach -> list (pass 1: of that bound, pass
//                   2: of m + 30 tau);
//   k_soft_eval     one pair per warp: pass 1 lowers the trajectory's exact
//                   minimum, which prunes the pairs still to come; pass 2
//                   stores distance, point and direction;
//   k_soft_reduce   one warp per waypoint sums its pairs in the list order of
//                   the waypoint (links, then objects as gathered), so results
//                   do not depend on the scheduling.
// A waypoint whose pairs do not fit (list or segment table full) is flagged
// and done by one warp in k_dist<1> / k_dist<2>.
constexpr int kSoftSegs = 128;        // list segments per waypoint (of up to kDPairs pairs)
constexpr int kSoftPerWaypoint = 256; // list capacity per waypoint of a chunk, on average

struct SoftArgs {
  int robot, nl;
  const float* q;            // [waypoints, L]
  int first, n;              // the chunk: waypoints first .. first + n
  int W;                     // waypoints per trajectory
  double tau;
  // per waypoint of the chunk
  float* T;                  // [n, nl, 12]
  float* delta;              // [n, nl]
  double* T64;               // [n, nl, 12]
  int2* seg;                 // [n, kSoftSegs] (first pair, pairs)
  int* nseg;                 // [n]; -1: did not fit
  // per trajectory
  unsigned int* ub;          // FP32 bits of an upper bound of the minimum's magnitude
  unsigned long long* mkey;  // exact minimum (double_key)
  // the list
  uint2* item;               // (waypoint of the chunk or ~0, link << 27 | object)
  float* lb;                 // box lower bound
  double* d;                 // +inf: not below the bound
  float4* p;                 // point on the link; .w unused
  float4* u;                 // direction
  int cap;
  unsigned int* count;       // pairs in the list (may exceed cap)
  unsigned int* head;        // work queue of k_soft_eval
  double* wsum;              // [waypoints]
  float* grad;               // [waypoints, L] or null
};

__global__ void __launch_bounds__(kDW * 32) k_soft_fk(const KWorldDev* __restrict__ W, const SoftArgs A)
{
  __shared__ double q64[kDW][kMaxLinks];
  __shared__ double T64[kDW][kMaxLinks][12];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kDW + warp;
  if (w >= A.n) return;
  const KRobotDev& R = W->robots[A.robot];
  const int nl = A.nl;
  const float q = lane < nl ? __ldg(A.q + (size_t)(A.first + w) * nl + lane) : 0.f;
  const bool bad = __any_sync(0xffffffffu, lane < nl && !(fabsf(q) < 1.0e6f));
  if (bad && lane == 0) set_status(W->status, KGPU_ERR_NOT_FINITE);
  // (a bad waypoint goes on at q = 0: the query fails as a whole)
  const float qv = bad ? 0.f : q;
  float P[12], delta;
  warp_fk32(R, lane, qv, 0.f, P, &delta);
  if (lane < nl) {
    const size_t at = (size_t)w * nl + lane;
#pragma unroll
    for (int i = 0; i < 12; ++i) A.T[at * 12 + i] = P[i];
    A.delta[at] = delta;
    q64[warp][lane] = (double)qv;
  }
  __syncwarp();
  warp_fk64(R, q64[warp], T64[warp], lane);
  for (int i = lane; i < nl * 12; i += 32) A.T64[(size_t)w * nl * 12 + i] = T64[warp][i / 12][i % 12];
}

// the FP32 transforms of waypoint w of the chunk into S
__device__ __forceinline__ void soft_load(DistSmem& S, const SoftArgs& A, int w, int lane)
{
  __syncwarp();
  for (int i = lane; i < A.nl * 12; i += 32) S.T[i / 12][i % 12] = __ldg(A.T + (size_t)w * A.nl * 12 + i);
  if (lane < A.nl) S.delta[lane] = __ldg(A.delta + (size_t)w * A.nl + lane);
  __syncwarp();
}

// the trajectory's current upper bound: one read, broadcast (other warps lower
// it meanwhile, and the lanes have to agree)
__device__ __forceinline__ float soft_ub(const SoftArgs& A, int t, int lane)
{
  unsigned int u = 0;
  if (lane == 0) u = *((volatile unsigned int*)(A.ub + t));
  return __uint_as_float(__shfl_sync(0xffffffffu, u, 0));
}

__global__ void __launch_bounds__(kDW * 32, 2) k_soft_bound(const KWorldDev* __restrict__ W, const SoftArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  DistSmem& S = reinterpret_cast<DistSmem*>(smem_raw)[warp];
  const KRobotDev& R = W->robots[A.robot];
  DCnt cnt;
#pragma unroll 1
  for (int w = blockIdx.x * kDW + warp; w < A.n; w += gridDim.x * kDW) {
    soft_load(S, A, w, lane);
    const int t = (A.first + w) / A.W;
    // pairs nearest by their boxes: the search radius grows until some are there
    int np = 0;
    float radius = 0.05f;
#pragma unroll 1
    while (np == 0) {
      const float ub = soft_ub(A, t, lane);
      const float reach = fminf(radius, ub);
#pragma unroll 1
      for (int l = 0; l < A.nl && np <= kDPairs - 32; ++l) {
        if (R.link_root[l] < 0) continue;
#pragma unroll 1
        for (int g = 0; g < kMaxGroups && np <= kDPairs - 32; ++g) {
          if (!((R.env_mask[l] >> g) & 1u) || W->group_root[g] < 0) continue;
          int top = 1;
          if (lane == 0) S.gstack[0] = (uint32_t)W->group_root[g];
          __syncwarp();
          np = gather_objects<true>(S, W, R, lane, l, reach, -1.f, np, top);
        }
      }
      if (radius >= (float)kSoftCutoff || radius >= ub) break;
      radius *= 4.f;
    }
    // vertex-pair bounds of the three nearest; an object too large for one is
    // evaluated (any distance found is an upper bound)
#pragma unroll 1
    for (int k = 0; k < min(np, 3); ++k) {
      float v = FLT_MAX;
      int idx = 0;
      for (int i = lane; i < np; i += 32)
        if (S.plb[i] < v) { v = S.plb[i]; idx = i; }
      const float vm = warp_min(v);
      const int at = __shfl_sync(0xffffffffu, idx, __ffs(__ballot_sync(0xffffffffu, v == vm)) - 1);
      const int l = S.plink[at], o = S.pobj[at];
      __syncwarp();
      if (lane == 0) S.plb[at] = FLT_MAX;
      __syncwarp();
      const float ub = soft_ub(A, t, lane);
      if (vm > ub) break;
      float b = pair_seed(S, W, R, lane, l, o);
      if (!(b < FLT_MAX)) {
        PairOut po;
        int fk64 = 1;
        double(*T64)[12] = reinterpret_cast<double(*)[12]>(A.T64 + (size_t)w * A.nl * 12);
        eval_pair(S, W, R, T64, fk64, lane, l, o, ub < 1e3f ? (double)ub : kSoftCutoff, po, cnt);
        if (po.found) b = (float)fmax(po.d, 0.0) * 1.000001f + 1e-7f;
      }
      if (lane == 0 && b < ub) atomicMin(A.ub + t, __float_as_uint(b));
    }
  }
  count_pairs(W, cnt, lane);
}

// PASS 1: pairs within the bound of the trajectory's minimum; 2: within m + 30 tau
template <int PASS>
__global__ void __launch_bounds__(kDW * 32) k_soft_gather(const KWorldDev* __restrict__ W, const SoftArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  DistSmem& S = reinterpret_cast<DistSmem*>(smem_raw)[warp];
  const KRobotDev& R = W->robots[A.robot];
#pragma unroll 1
  for (int w = blockIdx.x * kDW + warp; w < A.n; w += gridDim.x * kDW) {
    soft_load(S, A, w, lane);
    const int t = (A.first + w) / A.W;
    float reach;
    if (PASS == 1) reach = fminf(__uint_as_float(A.ub[t]), (float)kSoftCutoff) * 1.00001f + 1e-6f;
    else reach = (float)fmax(key_min(A.mkey[t]) + kSoftK * A.tau, 0.0) * 1.000001f + 1e-6f;
    int ns = 0, np = 0;
    bool fits = true;
    auto put = [&] {
      unsigned int base = 0;
      if (lane == 0) base = atomicAdd(A.count, (unsigned)np);
      base = __shfl_sync(0xffffffffu, base, 0);
      fits = fits && ns < kSoftSegs && base + (unsigned)np <= (unsigned)A.cap;
      for (int k = lane; k < np; k += 32)
        if (base + (unsigned)k < (unsigned)A.cap) {
          A.item[base + k] = fits ? make_uint2((unsigned)w, ((unsigned)S.plink[k] << 27) | (unsigned)S.pobj[k])
                                  : make_uint2(~0u, 0u);
          A.lb[base + k] = S.plb[k];
        }
      if (fits && lane == 0) A.seg[(size_t)w * kSoftSegs + ns] = make_int2((int)base, np);
      ++ns;
      np = 0;
      __syncwarp();
    };
#pragma unroll 1
    for (int l = 0; l < A.nl && fits; ++l) {
      if (R.link_root[l] < 0) continue;
#pragma unroll 1
      for (int g = 0; g < kMaxGroups && fits; ++g) {
        if (!((R.env_mask[l] >> g) & 1u) || W->group_root[g] < 0) continue;
        int top = 1;
        if (lane == 0) S.gstack[0] = (uint32_t)W->group_root[g];
        __syncwarp();
        while (top > 0 && fits) {
          np = gather_objects<true>(S, W, R, lane, l, reach, -1.f, np, top);
          if (top > 0) put();
        }
      }
    }
    if (np > 0 && fits) put();
    if (lane == 0) A.nseg[w] = fits ? ns : -1;
  }
}

template <int PASS>
__global__ void __launch_bounds__(kDW * 32, 2) k_soft_eval(const KWorldDev* __restrict__ W, const SoftArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  DistSmem& S = *reinterpret_cast<DistSmem*>(smem_raw + kEvalSmem * warp);
  const KRobotDev& R = W->robots[A.robot];
  const unsigned total = min(*A.count, (unsigned)A.cap);
  DCnt cnt;
#pragma unroll 1
  for (;;) {
    unsigned int it = 0;
    if (lane == 0) it = atomicAdd(A.head, 1u);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it >= total) break;
    const uint2 e = A.item[it];
    if (e.x == ~0u) continue;
    const int w = (int)e.x, l = (int)(e.y >> 27), o = (int)(e.y & 0x7ffffffu);
    const int t = (A.first + w) / A.W;
    // (an increasing minimum is impossible: a stale value only prunes less)
    unsigned long long key = 0;
    if (lane == 0) key = PASS == 1 ? *((volatile unsigned long long*)(A.mkey + t)) : A.mkey[t];
    const double m = key_min(__shfl_sync(0xffffffffu, key, 0));
    __syncwarp();
    if (lane < 12) S.T[l][lane] = __ldg(A.T + ((size_t)w * A.nl + l) * 12 + lane);
    if (lane == 12) S.delta[l] = __ldg(A.delta + (size_t)w * A.nl + l);
    __syncwarp();
    double(*T64)[12] = reinterpret_cast<double(*)[12]>(A.T64 + (size_t)w * A.nl * 12);
    int fk64 = 1;
    PairOut po;
    if (PASS == 1) {
      if (A.lb[it] > (float)fmax(m, 0.0) * 1.00001f + 1e-6f) continue;
      if (m <= 0.0 && (!W->obj_convex[o] || !may_be_deeper(S, W, R, lane, l, o, (float)-m))) continue;
      const float ub = soft_ub(A, t, lane);
      eval_pair(S, W, R, T64, fk64, lane, l, o, nextafter(m, 1e300), po, cnt, ub);
      if (lane == 0 && po.found) {
        atomicMin(A.mkey + t, double_key(po.d));
        if (po.d < (double)ub) atomicMin(A.ub + t, __float_as_uint((float)fmax(po.d, 0.0) * 1.000001f + 1e-7f));
      }
    } else {
      eval_pair(S, W, R, T64, fk64, lane, l, o, m + kSoftK * A.tau, po, cnt, pair_seed(S, W, R, lane, l, o));
      if (lane == 0) {
        A.d[it] = po.found ? po.d : DBL_MAX;
        if (po.found) {
          A.p[it] = make_float4((float)po.cp[0], (float)po.cp[1], (float)po.cp[2], 0.f);
          A.u[it] = make_float4(po.dir[0], po.dir[1], po.dir[2], 0.f);
        }
      }
    }
    __syncwarp();
  }
  count_pairs(W, cnt, lane);
}

// One warp per waypoint: e_k = exp(-(d_k - m) / tau) of its pairs in list
// order, their sum and the weighted wrenches (lane l sums link l's), pulled
// back through the chain.
__global__ void __launch_bounds__(kDW * 32) k_soft_reduce(const KWorldDev* __restrict__ W, const SoftArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  DistSmem& S = reinterpret_cast<DistSmem*>(smem_raw)[warp];
  const KRobotDev& R = W->robots[A.robot];
  const int w = blockIdx.x * kDW + warp;
  if (w >= A.n) return;
  const int ns = A.nseg[w];
  if (ns < 0) return;  // done by k_dist<2>
  soft_load(S, A, w, lane);
  const double m = key_min(A.mkey[(A.first + w) / A.W]);
  double sum = 0.0;
  float F[3] = {0.f, 0.f, 0.f}, M[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
  for (int s = 0; s < ns; ++s) {
    const int2 sg = A.seg[(size_t)w * kSoftSegs + s];
#pragma unroll 1
    for (int base = 0; base < sg.y; base += 32) {
      const int k = sg.x + base + lane;
      const bool in = base + lane < sg.y;
      const double d = in ? A.d[k] : DBL_MAX;
      const bool found = d < DBL_MAX;
      double e = 0.0;
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f), u = p;
      int l = 0;
      if (found) {
        e = exp(-(d - m) / A.tau);
        p = A.p[k];
        u = A.u[k];
        l = (int)(A.item[k].y >> 27);
      }
      unsigned todo = __ballot_sync(0xffffffffu, found);
#pragma unroll 1
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const double es = __shfl_sync(0xffffffffu, e, src);
        sum += es;
        const float dx = __shfl_sync(0xffffffffu, u.x, src), dy = __shfl_sync(0xffffffffu, u.y, src),
                    dz = __shfl_sync(0xffffffffu, u.z, src);
        const float px = __shfl_sync(0xffffffffu, p.x, src), py = __shfl_sync(0xffffffffu, p.y, src),
                    pz = __shfl_sync(0xffffffffu, p.z, src);
        if (__shfl_sync(0xffffffffu, l, src) == lane) wrench_sum(F, M, (float)es, dx, dy, dz, px, py, pz);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    S.F[lane][c] = F[c];
    S.M[lane][c] = M[c];
  }
  __syncwarp();
  const size_t b = (size_t)A.first + w;
  if (lane == 0) A.wsum[b] = sum;
  pullback(S, R, lane, A.grad ? A.grad + b * A.nl : nullptr);
}

// L = m - tau log(sum) with the waypoints' sums in order, the gradient
// normalised by the sum; one warp per trajectory
__global__ void k_softmin_final(const double* wsum, const unsigned long long* mkey, int T, int Wn, int L, double tau,
                                double* out, float* grad)
{
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= T) return;
  double s = 0.0;
#pragma unroll 1
  for (int base = 0; base < Wn; base += 32) {
    const double v = base + lane < Wn ? wsum[(size_t)t * Wn + base + lane] : 0.0;
    for (int k = 0; k < min(32, Wn - base); ++k) s += __shfl_sync(0xffffffffu, v, k);
  }
  if (lane == 0) out[t] = key_min(mkey[t]) - tau * log(s);
  if (grad) {
    const float inv = (float)(1.0 / s);
    for (size_t k = lane; k < (size_t)Wn * L; k += 32) grad[(size_t)t * Wn * L + k] *= inv;
  }
}

// ---- self distance ----------------------------------------------------------
// Minimum distance between the robot's own links over its enabled self pairs
// (the link-link part of WorldPlannerSettings::DistanceLowerBound when a
// robot is checked against itself, Cpp/Planning/PlannerSettings.cpp:385-395,
// and of geometry_ad.MinDistance over link geometries).  Definition (the FP64
// oracle's, bit for bit on the value and the closest points):
//   d(i, j) = sqrt of the minimum canonical triangle distance (kx_tri_tri_dist2)
//             over the pair's triangles, ties to the smallest (triangle of i,
//             triangle of j) in mesh order; 0 when the surfaces meet;
//   d      = min over enabled pairs i < j with d(i, j) < cutoff; pairs are
//            visited in (i, j) order and a pair replaces the best so far
//            only if its squared minimum is below the square of the best
//            distance and its distance is strictly smaller (equal distances
//            keep the earlier pair, even when the squares differ in the last
//            bit); none: d = cutoff and pair (-1, -1).
// Gradient: dd/dq_k = u . (dcp/dq_k - dcq/dq_k), u = (cp - cq) / d at the
// closest points cp on link i and cq on link j (0 when d = 0), from FP64
// transforms.  One warp per configuration: FP32 traversal of each pair with
// conservative pruning against the running upper bound of the minimum,
// triangle pairs within the error band finalised in canonical FP64.
constexpr int kSW = 2;  // warps per block of k_self_dist

struct __align__(16) SelfDistSmem {
  float T[kMaxLinks][12];
  float delta[kMaxLinks];
  double T64[kMaxLinks][12];
  double q64[kMaxLinks];
  PairSmem P;                  // the current pair; P.b2 starts at the acceptance bound
  float plb[kMaxLinks * (kMaxLinks - 1) / 2];  // lower bounds of the pairs still to evaluate
  double b2, bcp[3], bcq[3];  // best over the pairs so far: squared distance, closest points
  double bd;                   // its distance (the cutoff before any pair is found)
  int bi, bj;
};

struct SelfDistArgs {
  int robot;
  const float* q;
  int B;
  double cutoff;
  double* d;       // [B]
  int* pair;       // [B, 2]
  double* cp;      // [B, 6] (point on link i, point on link j)
  float* grad;     // [B, L] or null
  double* dpair;   // per-pair mode: [B, L (L - 1) / 2], each pair's own minimum
  int all_pairs;   // per-pair mode: every pair i < j whose links have geometry, enabled or not
};

// An upper bound on the distance between the surfaces of links i and j:
// the vertex of i nearest the centre of j's root box and the vertex of j
// nearest that vertex (both surface points), widened by the links' FP32
// placement bounds and rounding.
__device__ __noinline__ float link_pair_seed(SelfDistSmem& S, const KWorldDev* __restrict__ W, const KRobotDev& R,
                                             int lane, int i, int j)
{
  const KNode nj = W->lnodes[R.link_root[j]];
  const float3 cj = xform32(S.T[j], make_float3(nj.a.x, nj.a.y, nj.a.z));
  float bd = FLT_MAX;
  float3 bv = cj;
  {
    const int vf = R.link_vert_first[i], vc = R.link_vert_count[i];
    for (int v = lane; v < vc; v += 32) {
      const float4 x = __ldg(W->lvert32 + vf + v);
      const float3 w = xform32(S.T[i], make_float3(x.x, x.y, x.z));
      const float dx = w.x - cj.x, dy = w.y - cj.y, dz = w.z - cj.z;
      const float d2 = dx * dx + dy * dy + dz * dz;
      if (d2 < bd) { bd = d2; bv = w; }
    }
  }
  const float m = warp_min(bd);
  if (!(m < FLT_MAX)) return FLT_MAX;  // no vertex: no surface point, no seed
  const unsigned mm = __ballot_sync(0xffffffffu, bd == m);
  const int src = __ffs(mm) - 1;
  bv = make_float3(__shfl_sync(0xffffffffu, bv.x, src), __shfl_sync(0xffffffffu, bv.y, src),
                   __shfl_sync(0xffffffffu, bv.z, src));
  float bo = FLT_MAX;
  {
    const int vf = R.link_vert_first[j], vc = R.link_vert_count[j];
    for (int v = lane; v < vc; v += 32) {
      const float4 x = __ldg(W->lvert32 + vf + v);
      const float3 w = xform32(S.T[j], make_float3(x.x, x.y, x.z));
      const float dx = w.x - bv.x, dy = w.y - bv.y, dz = w.z - bv.z;
      bo = fminf(bo, dx * dx + dy * dy + dz * dz);
    }
  }
  bo = warp_min(bo);
  if (!(bo < FLT_MAX)) return FLT_MAX;
  return sqrtf(bo) * (1.f + 1e-5f) + 2.f * (S.delta[i] + S.delta[j]) + 1e-6f;
}

// Per-pair mode: every queried pair's own minimum, in order.
__device__ __noinline__ void self_pairs(SelfDistSmem& S, const KWorldDev* __restrict__ W, const KRobotDev& R,
                                        const MeshView& M, const SelfDistArgs& A, int b, int lane, float fcut,
                                        PairCnt& cnt)
{
  const int nl = R.nlinks, npair = nl * (nl - 1) / 2;
  for (int k = lane; k < npair; k += 32) A.dpair[(size_t)b * npair + k] = -1.0;  // pairs not queried
  __syncwarp();
  const int nq = A.all_pairs ? npair : R.nqueries_self;
#pragma unroll 1
  for (int qi = 0; qi < nq; ++qi) {
    int i, j;
    if (A.all_pairs) {  // qi in upper-triangle order (0,1), (0,2), ..., (L-2, L-1)
      i = 0;
      int r = qi;
      while (r >= nl - 1 - i) { r -= nl - 1 - i; ++i; }
      j = i + 1 + r;
    } else {
      const uint32_t qw = __ldg(W->queries + R.query_off + R.nqueries_env + qi);
      i = qw & 0xff;
      j = (qw >> 8) & 0xff;
    }
    if (R.link_root[i] < 0 || R.link_root[j] < 0) continue;
    float m32 = fminf(fcut, link_pair_seed(S, W, R, lane, i, j));
    if (lane == 0) {
      const double bb = kx_mul(A.cutoff, A.cutoff);
      S.P.b2 = bb > 1e-300 ? bb : 1e-300;
      S.P.bA = S.P.bB = INT_MAX;
      S.P.have = 0;
    }
    int certA = -1;
    const int r = pair_distance<false, true>(S.P, M, M, R.link_root[i], R.link_root[j], S.T[i], S.T[j], S.T64[i],
                                             S.T64[j], S.delta[i] + S.delta[j], m32, certA, lane, cnt, [] {});
    if (lane == 0) {
      if (r == 2) set_status(W->status, KGPU_ERR_OVERFLOW);
      A.dpair[(size_t)b * npair + i * nl - i * (i + 1) / 2 + (j - i - 1)] =
          r == 1 ? 0.0 : (S.P.have ? kx_sqrt(S.P.b2) : A.cutoff);
    }
    __syncwarp();
  }
}

// Pairs nearest first by their root boxes (all bounded at once, one per
// lane): the first few set the bound that prunes the rest unseen, where the
// (i, j) order evaluated most of a humanoid's 435.  The result is the
// lexicographic minimum (distance, pair), whatever the order.  Blocks of two
// warps, so that a costly configuration holds up one other at most.  8,192
// humanoid configurations: 15.4 -> 5.96 ms by this order (4.3-8.3 ms by
// the drawn postures with the later work on the pair traversal).
__global__ void __launch_bounds__(kSW * 32, 16 / kSW) k_self_dist(const KWorldDev* __restrict__ W, const SelfDistArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SelfDistSmem& S = reinterpret_cast<SelfDistSmem*>(smem_raw)[warp];
  const MeshView M = {W->lnodes, W->lnode_r, W->ltri32, W->ltri64, W->ltri_orig};
  PairCnt cnt;
  const KRobotDev& R = W->robots[A.robot];
  const int nl = R.nlinks;
  const float fcut = A.cutoff < 1e30 ? (float)A.cutoff * 1.000001f + 1e-7f : FLT_MAX;
  const bool per_pair = A.dpair != nullptr;
  const int nwarps = gridDim.x * kSW;
#pragma unroll 1
  for (int b = blockIdx.x * kSW + warp; b < A.B; b += nwarps) {
    const float qv = lane < nl ? __ldg(A.q + (size_t)b * nl + lane) : 0.f;
    if (__any_sync(0xffffffffu, lane < nl && !(fabsf(qv) < 1.0e6f))) {
      if (lane == 0) set_status(W->status, KGPU_ERR_NOT_FINITE);
      continue;
    }
    float P32[12], delta;
    warp_fk32(R, lane, qv, 0.f, P32, &delta);
    if (lane < nl) {
#pragma unroll
      for (int k = 0; k < 12; ++k) S.T[lane][k] = P32[k];
      S.delta[lane] = delta + W->eps_extra;
      S.q64[lane] = (double)qv;
    }
    if (lane == 0) {
      S.b2 = DBL_MAX;
      S.bd = A.cutoff;
      S.bi = S.bj = -1;
    }
    __syncwarp();
    warp_fk64(R, S.q64, S.T64, lane);
    if (per_pair) {
      self_pairs(S, W, R, M, A, b, lane, fcut, cnt);
      continue;
    }
    // lower bounds of all pairs from their root boxes, one pair per lane
    const int nq = R.nqueries_self;
#pragma unroll 1
    for (int k = lane; k < nq; k += 32) {
      const uint32_t qw = __ldg(W->queries + R.query_off + R.nqueries_env + k);
      const int i = qw & 0xff, j = (qw >> 8) & 0xff;
      float lb = FLT_MAX;
      if (R.link_root[i] >= 0 && R.link_root[j] >= 0)
        lb = node_lb32<false>(M, M, S.T[i], S.T[j], W->lnodes[R.link_root[i]], W->lnodes[R.link_root[j]],
                              R.link_root[i], R.link_root[j], S.delta[i] + S.delta[j]);
      S.plb[k] = lb;
    }
    __syncwarp();
    float m32 = fcut;  // upper bound on the minimum so far (warp-uniform)
    int best = INT_MAX;  // position of the best pair in the (i, j) order
#pragma unroll 1
    for (;;) {
      // the nearest pair by its boxes that can still win; once a contact is
      // found, the first one in order before it (only an earlier contact can)
      const bool contact = S.bd == 0.0 && best < INT_MAX;
      const float lim = m32 * (1.f + 2e-5f);
      float v = FLT_MAX;
      int kq = INT_MAX;
#pragma unroll 1
      for (int k = lane; k < nq && !(contact && (k >= best || kq < INT_MAX)); k += 32) {
        const float lb = S.plb[k];
        if (lb <= lim && lb < v) {
          v = contact ? -FLT_MAX : lb;
          kq = k;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int ok = __shfl_xor_sync(0xffffffffu, kq, o);
        if (ov < v || (ov == v && ok < kq)) { v = ov; kq = ok; }
      }
      if (kq == INT_MAX) break;
      __syncwarp();
      if (lane == 0) S.plb[kq] = FLT_MAX;
      const uint32_t qw = __ldg(W->queries + R.query_off + R.nqueries_env + kq);
      const int i = qw & 0xff, j = (qw >> 8) & 0xff;
      // without a running bound to prune with, a vertex-pair bound of this pair
      if (m32 >= fcut) m32 = fminf(m32, link_pair_seed(S, W, R, lane, i, j));
      if (lane == 0) {
        // below the best distance, or (an earlier pair) equal to it: 1e-15
        // covers the squares whose root rounds to the same distance
        double bb = kx_mul(S.bd, S.bd);
        if (kq < best) bb = bb * (1.0 + 1e-15);
        S.P.b2 = bb > 1e-300 ? bb : 1e-300;
        S.P.bA = S.P.bB = INT_MAX;
        S.P.have = 0;
      }
      int certA = -1;
      const int r = pair_distance<false, true>(S.P, M, M, R.link_root[i], R.link_root[j], S.T[i], S.T[j], S.T64[i],
                                               S.T64[j], S.delta[i] + S.delta[j], m32, certA, lane, cnt, [] {});
      if (r == 2 && lane == 0) set_status(W->status, KGPU_ERR_OVERFLOW);
      const double dp = r == 1 ? 0.0 : (S.P.have ? kx_sqrt(S.P.b2) : DBL_MAX);
      const bool first = best == INT_MAX;
      if (r == 1 ? (first || S.bd > 0.0 || kq < best) : (dp < S.bd || (!first && dp == S.bd && kq < best))) {
        __syncwarp();
        if (lane == 0) {
          S.b2 = r == 1 ? 0.0 : S.P.b2;
          S.bd = dp;
          S.bi = i;
          S.bj = j;
          for (int c = 0; c < 3; ++c) { S.bcp[c] = S.P.bcp[c]; S.bcq[c] = S.P.bcq[c]; }
        }
        best = kq;
        if (dp == 0.0) m32 = 0.f;
      }
      __syncwarp();
    }
    // ---- outputs and the gradient (FP64 transforms)
    const bool found = S.b2 < DBL_MAX;
    const double d = found ? kx_sqrt(S.b2) : A.cutoff;
    if (lane == 0) {
      A.d[b] = d;
      A.pair[2 * (size_t)b] = found ? S.bi : -1;
      A.pair[2 * (size_t)b + 1] = found ? S.bj : -1;
    }
    if (lane < 6) A.cp[6 * (size_t)b + lane] = found && d > 0.0 ? (lane < 3 ? S.bcp[lane] : S.bcq[lane - 3]) : 0.0;
    if (A.grad && lane < nl) {
      double g = 0.0;
      if (found && d > 0.0 && R.jtype[lane] != KX_JOINT_WELD) {
        double u[3];
        for (int c = 0; c < 3; ++c) u[c] = (S.bcp[c] - S.bcq[c]) / d;
        const double* Tk = S.T64[lane];
        double w[3];
        for (int r = 0; r < 3; ++r) w[r] = Tk[3 * r] * R.axis64[lane][0] + Tk[3 * r + 1] * R.axis64[lane][1] +
                                          Tk[3 * r + 2] * R.axis64[lane][2];
        for (int side = 0; side < 2; ++side) {
          const int link = side == 0 ? S.bi : S.bj;
          bool anc = false;
          for (int a = link; a >= 0; a = R.parents[a])
            if (a == lane) { anc = true; break; }
          if (!anc) continue;
          const double* x = side == 0 ? S.bcp : S.bcq;
          double v[3];
          if (R.jtype[lane] == KX_JOINT_REVOLUTE) {
            const double rx = x[0] - Tk[9], ry = x[1] - Tk[10], rz = x[2] - Tk[11];
            v[0] = w[1] * rz - w[2] * ry;
            v[1] = w[2] * rx - w[0] * rz;
            v[2] = w[0] * ry - w[1] * rx;
          } else {
            v[0] = w[0]; v[1] = w[1]; v[2] = w[2];
          }
          const double t = u[0] * v[0] + u[1] * v[1] + u[2] * v[2];
          g += side == 0 ? t : -t;
        }
      }
      A.grad[(size_t)b * nl + lane] = (float)g;
    }
    __syncwarp();
  }
}

}  // namespace

cudaError_t dist_init()
{
  const int smem = (int)(sizeof(DistSmem) * kDW);
  const void* kernels[] = {(const void*)k_dist<0>,        (const void*)k_dist<1>,        (const void*)k_dist<2>,
                           (const void*)k_soft_bound,     (const void*)k_soft_gather<1>, (const void*)k_soft_gather<2>,
                           (const void*)k_soft_eval<1>,   (const void*)k_soft_eval<2>,   (const void*)k_soft_reduce};
  for (const void* k : kernels) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  return cudaFuncSetAttribute(k_self_dist, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(sizeof(SelfDistSmem) * kSW));
}

cudaError_t launch_distance(const KWorldDev* Wd, const Scratch& S, int robot, const float* q, int B, double cutoff,
                            double* d, int* pair, double* cp, float* grad, int num_sms, cudaStream_t s)
{
  if (B <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(S.counters + 8, 0, sizeof(unsigned int), s);
  if (e != cudaSuccess) return e;
  DistArgs A = {};
  A.robot = robot;
  A.q = q;
  A.B = B;
  A.cutoff = cutoff;
  A.d = d;
  A.pair = pair;
  A.cp = cp;
  A.grad = grad;
  A.head = S.counters + 8;
  A.scratch = S.spill;
  A.scratch_per_warp = (int)S.spill_per_warp;
  k_dist<0><<<num_sms * 2, kDW * 32, sizeof(DistSmem) * kDW, s>>>(Wd, A);
  return cudaGetLastError();
}

namespace {

// device scratch of a soft-min call, carved out of one block
struct SoftLayout {
  int chunk, cap;  // waypoints per chunk, list capacity
  size_t T, delta, T64, seg, nseg, ub, mkey, item, lb, d, p, u, wsum, count, bytes;
};

// level k: chunks and the smallest list 2^k times smaller (8 waypoints at the last)
SoftLayout soft_layout(int T, int Wn, int nl, int nobj, int level)
{
  SoftLayout L;
  const size_t B = (size_t)T * Wn;
  L.chunk = (int)std::min(B, (size_t)(kSoftChunk >> level));
  const size_t all = (size_t)L.chunk * nl * nobj, most = (size_t)L.chunk * kSoftPerWaypoint;
  const size_t cap = std::min(all, std::max(most, (size_t)65536 >> level));
  L.cap = (int)cap;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 255) / 256 * 256;
    return here;
  };
  L.T = take(sizeof(float) * 12 * nl * L.chunk);
  L.delta = take(sizeof(float) * nl * L.chunk);
  L.T64 = take(sizeof(double) * 12 * nl * L.chunk);
  L.seg = take(sizeof(int2) * kSoftSegs * L.chunk);
  L.nseg = take(sizeof(int) * L.chunk);
  L.item = take(sizeof(uint2) * cap);
  L.lb = take(sizeof(float) * cap);
  L.d = take(sizeof(double) * cap);
  L.p = take(sizeof(float4) * cap);
  L.u = take(sizeof(float4) * cap);
  L.wsum = take(sizeof(double) * B);
  L.ub = take(sizeof(unsigned int) * T);
  L.mkey = take(sizeof(unsigned long long) * T);
  L.count = take(4 * sizeof(unsigned int));
  L.bytes = at;
  return L;
}

}  // namespace

size_t softmin_work_bytes(int T, int Wn, int nl, int nobj, int level)
{
  return soft_layout(T, Wn, nl, nobj, level).bytes;
}

cudaError_t launch_softmin(const KWorldDev* Wd, const Scratch& S, int robot, const float* q, int T, int Wn,
                           double tau, double* L, float* dLdq, int nl, int nobj, void* work, int level, int num_sms,
                           cudaStream_t s)
{
  if (T <= 0) return cudaSuccess;
  const size_t smem = sizeof(DistSmem) * kDW;
  const int B = T * Wn;
  const SoftLayout lay = soft_layout(T, Wn, nl, nobj, level);
  char* w = (char*)work;
  SoftArgs A = {};
  A.robot = robot;
  A.nl = nl;
  A.q = q;
  A.W = Wn;
  A.tau = tau;
  A.T = (float*)(w + lay.T);
  A.delta = (float*)(w + lay.delta);
  A.T64 = (double*)(w + lay.T64);
  A.seg = (int2*)(w + lay.seg);
  A.nseg = (int*)(w + lay.nseg);
  A.ub = (unsigned int*)(w + lay.ub);
  A.mkey = (unsigned long long*)(w + lay.mkey);
  A.item = (uint2*)(w + lay.item);
  A.lb = (float*)(w + lay.lb);
  A.d = (double*)(w + lay.d);
  A.p = (float4*)(w + lay.p);
  A.u = (float4*)(w + lay.u);
  A.cap = lay.cap;
  A.count = (unsigned int*)(w + lay.count);
  A.head = A.count + 1;
  A.wsum = (double*)(w + lay.wsum);
  A.grad = dLdq;
  // the flagged waypoints of a chunk, one warp each
  DistArgs D = {};
  D.robot = robot;
  D.q = q;
  D.cutoff = kSoftCutoff;
  D.scratch = S.spill;
  D.scratch_per_warp = (int)S.spill_per_warp;
  D.nseg = A.nseg;
  D.T = A.T;
  D.delta = A.delta;
  D.mkey = A.mkey;
  D.wsum = A.wsum;
  D.W = Wn;
  D.tau = tau;
  D.grad = dLdq;
  D.head = A.count + 2;
  // bounds start above every distance (0x7f7f7f7f is 3.4e38), minima as "none"
  cudaError_t e = cudaMemsetAsync(A.ub, 0x7f, sizeof(unsigned int) * T, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(A.mkey, 0xff, sizeof(unsigned long long) * T, s);
  for (int pass = 1; pass <= 2 && e == cudaSuccess; ++pass) {
    for (int first = 0; first < B && e == cudaSuccess; first += lay.chunk) {
      A.first = D.first = first;
      A.n = D.B = B - first < lay.chunk ? B - first : lay.chunk;
      const int warps = (A.n + kDW - 1) / kDW, some = warps < 2 * num_sms ? warps : 2 * num_sms;
      if ((e = cudaMemsetAsync(A.count, 0, 4 * sizeof(unsigned int), s)) != cudaSuccess) return e;
      // (one chunk: the transforms of pass 1 are still there in pass 2)
      if (pass == 1 || lay.chunk < B) k_soft_fk<<<warps, kDW * 32, 0, s>>>(Wd, A);
      if (pass == 1) {
        k_soft_bound<<<some, kDW * 32, smem, s>>>(Wd, A);
        k_soft_gather<1><<<some, kDW * 32, smem, s>>>(Wd, A);
        k_soft_eval<1><<<2 * num_sms, kDW * 32, kEvalSmem * kDW, s>>>(Wd, A);
        k_dist<1><<<some, kDW * 32, smem, s>>>(Wd, D);
      } else {
        k_soft_gather<2><<<some, kDW * 32, smem, s>>>(Wd, A);
        k_soft_eval<2><<<2 * num_sms, kDW * 32, kEvalSmem * kDW, s>>>(Wd, A);
        k_dist<2><<<some, kDW * 32, smem, s>>>(Wd, D);
        k_soft_reduce<<<warps, kDW * 32, smem, s>>>(Wd, A);
      }
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) return e;
  k_softmin_final<<<(T + 3) / 4, 128, 0, s>>>(A.wsum, A.mkey, T, Wn, nl, tau, L, dLdq);
  return cudaGetLastError();
}

}  // namespace kgpu

namespace kgpu {

cudaError_t launch_self_distance(const KWorldDev* Wd, int robot, const float* q, int B, double cutoff, double* d,
                                 int* pair, double* cp, float* grad, double* dpair, int all_pairs, int num_sms,
                                 cudaStream_t s)
{
  if (B <= 0) return cudaSuccess;
  const size_t smem = sizeof(SelfDistSmem) * kSW;  // attribute set by dist_init()
  SelfDistArgs A;
  A.robot = robot;
  A.q = q;
  A.B = B;
  A.cutoff = cutoff;
  A.d = d;
  A.pair = pair;
  A.cp = cp;
  A.grad = grad;
  A.dpair = dpair;
  A.all_pairs = dpair != nullptr && all_pairs != 0;
  const int blocks = min((B + kSW - 1) / kSW, 64 * num_sms);
  k_self_dist<<<blocks, kSW * 32, smem, s>>>(Wd, A);
  return cudaGetLastError();
}

}  // namespace kgpu
