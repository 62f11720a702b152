// kgpu_pairdist.cuh — the minimum distance of two placed meshes by one warp,
// shared by the distance kernels (link against object, link against link, two
// free geometries).
//
// FP32 does the search, canonical FP64 the answer: a BVH-vs-BVH traversal with
// conservative pruning against m32, a running upper bound of the minimum;
// leaf pairs are expanded one triangle pair per lane; pairs whose lower bound
// does not exclude them are collected until a warp-full is there and then get
// the FP32 separation test and distance; those within the error band of m32
// become candidates, finalised in FP64 with a lexicographic reduction
// (squared distance, triangle of A, triangle of B).
//
// What bounds it: fetching its instructions (the soft-min's top stall, 41% of
// the samples; half the warps keep 91% of the speed), load latency, and in the
// soft-min the FP64 pipe (26% busy).  A triangle pair's separation test and distance are ~1,600
// instructions, and of the pairs whose bounds are computed 2-3% need them, so
// running them where they are found costs 15 warp-wide evaluations a mesh
// pair with 4-5 lanes active; collected they are 2-3 full ones.  Measured
// against testing them where they are found, with the FP64 code rolled and
// the node bound along the line of centres: 16,384 cylinder-icosphere
// distances 8.3 -> 4.0 ms, soft-min over 6,400 waypoints 140 -> 105 ms, 8,192
// humanoid self distances 20.0 -> 17.9 ms, 32,768 terrain clearances 43.7 ->
// 38.9 ms.  With one-instruction roots in the bounds, leaf-pair positions from
// a bit mask instead of a binary search and a division, and minima compared as
// integers, the same four went from 3.9, 45.2, 5.75 and 24.7 ms to 3.5, 39.2,
// 5.15 and 20.7 ms (mostly by the roots; the last two differ by the drawn
// configurations, 4.3-8.3 and 19-21 ms).
#pragma once

#include "kgpu_dist32.cuh"

namespace kgpu {

constexpr int kPStack = 384;  // node-pair stack entries per warp (512: soft-min +2.5%, L1; 256: terrain +20%, narrowed fronts)
constexpr int kPJobs = 64;    // leaf pairs
constexpr int kPFull = 64;    // triangle pairs for the full FP32 distance
constexpr int kPCand = 64;    // FP64 candidates

struct MeshView {
  const KNode* nodes;
  const float* node_r;  // radius per node about its FP32 centre, or null
  const float4* tri32;  // 3 per triangle, leaf order; .w of the first: flat_mark
  const double* tri64;  // 9 per triangle
  const int* orig;      // leaf order -> mesh order
};

struct __align__(16) PairSmem {
  uint2 stack[kPStack];
  uint32_t jobA[kPJobs], jobB[kPJobs], jobOff[kPJobs + 1];
  uint32_t fullA[kPFull], fullB[kPFull];
  float fullL[kPFull];                       // their lower bounds
  uint32_t candA[kPCand], candB[kPCand];
  float candD[kPCand];                       // lower end of their FP32 band
  uint8_t candS[kPCand];                     // FP32-separated: the canonical overlap test is not needed
  // running best in FP64: starts at the acceptance bound, have = 0
  double b2, bcp[3], bcq[3];
  int bA, bB, have;
};

// world placement of triangle t in FP32; ID: the mesh is in world coordinates
template <bool ID>
__device__ __forceinline__ void place32(const MeshView& M, const float* T, int t, float3* o)
{
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    const float4 x = __ldg(M.tri32 + 3 * (size_t)t + v);
    o[v] = ID ? make_float3(x.x, x.y, x.z) : xform32(T, make_float3(x.x, x.y, x.z));
  }
}

template <bool ID>
__device__ __forceinline__ void place64(const MeshView& M, const double* T, int t, double* o)
{
  const double* p = M.tri64 + 9 * (size_t)t;
  if (ID) {
    for (int i = 0; i < 9; ++i) o[i] = p[i];
  } else {
#pragma unroll 1
    for (int v = 0; v < 3; ++v) kx_xform_point(T, p + 3 * v, o + 3 * v);
  }
}

__device__ __forceinline__ float tri_span(const float3* P, const float3* Q)
{
  float3 lo = P[0], hi = P[0];
#pragma unroll
  for (int k = 1; k < 6; ++k) {
    const float3 v = k < 3 ? P[k] : Q[k - 3];
    lo = make_float3(fminf(lo.x, v.x), fminf(lo.y, v.y), fminf(lo.z, v.z));
    hi = make_float3(fmaxf(hi.x, v.x), fmaxf(hi.y, v.y), fmaxf(hi.z, v.z));
  }
  return fmaxf(fmaxf(hi.x - lo.x, hi.y - lo.y), hi.z - lo.z);
}

// Lower bound on the distance of two triangles: that of their boxes (the
// better one for large triangles that nearly touch)
__device__ __forceinline__ float tri_box_lb32(const float3* P, const float3* Q)
{
  float3 pl = P[0], ph = P[0], ql = Q[0], qh = Q[0];
#pragma unroll
  for (int k = 1; k < 3; ++k) {
    pl = make_float3(fminf(pl.x, P[k].x), fminf(pl.y, P[k].y), fminf(pl.z, P[k].z));
    ph = make_float3(fmaxf(ph.x, P[k].x), fmaxf(ph.y, P[k].y), fmaxf(ph.z, P[k].z));
    ql = make_float3(fminf(ql.x, Q[k].x), fminf(ql.y, Q[k].y), fminf(ql.z, Q[k].z));
    qh = make_float3(fmaxf(qh.x, Q[k].x), fmaxf(qh.y, Q[k].y), fmaxf(qh.z, Q[k].z));
  }
  const float gx = fmaxf(0.f, fmaxf(ql.x - ph.x, pl.x - qh.x));
  const float gy = fmaxf(0.f, fmaxf(ql.y - ph.y, pl.y - qh.y));
  const float gz = fmaxf(0.f, fmaxf(ql.z - ph.z, pl.z - qh.z));
  return root_below32(gx * gx + gy * gy + gz * gz);
}

// FP64 finalisation of the candidates still within the band of m32, merged
// into the running best.  dd: placement bound of both sides.  Returns the
// number of pairs this lane evaluated.
template <bool IDB>
__device__ __noinline__ int pair_flush(PairSmem& S, const MeshView& A, const MeshView& B, const float* TA,
                                       const float* TB, const double* TA64, const double* TB64, int lane, int ncand,
                                       float m32, float dd)
{
  const unsigned lt = lanemask_lt();
  const float lim = m32 * (1.f + 2e-5f) + 1e-6f;
  int keep = 0, done = 0;
#pragma unroll 1
  for (int base = 0; base < ncand; base += 32) {
    const int k = base + lane;
    bool ok = false;
    uint32_t a = 0, b = 0;
    uint8_t s = 0;
    if (k < ncand) {
      a = S.candA[k];
      b = S.candB[k];
      s = S.candS[k];
      ok = S.candD[k] <= lim;
    }
    __syncwarp();
    const unsigned mk = __ballot_sync(0xffffffffu, ok);
    if (ok) {
      const int r = keep + __popc(mk & lt);
      S.candA[r] = a;
      S.candB[r] = b;
      S.candS[r] = s;
    }
    keep += __popc(mk);
    __syncwarp();
  }
#pragma unroll 1
  for (int base = 0; base < keep; base += 32) {
    const int k = base + lane;
    double d2 = DBL_MAX;
    int oa = INT_MAX, ob = INT_MAX;
    double cp[3] = {0, 0, 0}, cq[3] = {0, 0, 0};
    if (k < keep) {
      const int tA = (int)S.candA[k], tB = (int)S.candB[k];
      double P[9], Q[9];
      place64<false>(A, TA64, tA, P);
      place64<IDB>(B, TB64, tB, Q);
      float3 P32[3], Q32[3];
      place32<false>(A, TA, tA, P32);
      place32<IDB>(B, TB, tB, Q32);
      const unsigned mask = tri_feature_mask32(P32[0], P32[1], P32[2], Q32[0], Q32[1], Q32[2],
                                               feature_thr2(P32, Q32, m32, dd));
      d2 = tri_dist2_masked64(P, Q, mask, S.candS[k] != 0, cp, cq);
      oa = A.orig[tA];
      ob = B.orig[tB];
      ++done;
    }
    int src;
    unsigned long long m2 = double_bits(d2);
    int ma = oa, mb = ob;
    warp_lexmin(m2, ma, mb, src, lane);
    // below the acceptance bound, or equal to the best with smaller triangles
    const unsigned long long b2 = double_bits(S.b2);
    const bool better = m2 < b2 || (S.have && m2 == b2 && (ma < S.bA || (ma == S.bA && mb < S.bB)));
    __syncwarp();
    if (m2 < double_bits(DBL_MAX) && better && lane == src) {
      S.b2 = d2;
      S.bA = oa;
      S.bB = ob;
      S.have = 1;
      for (int c = 0; c < 3; ++c) { S.bcp[c] = cp[c]; S.bcq[c] = cq[c]; }
    }
    __syncwarp();
  }
  return done;
}

// The FP32 separation test and distance of the last up to 32 collected
// triangle pairs: lowers m32, appends the pairs within its band to the
// candidates (room for 32 is the caller's).  Returns the number of candidates
// then held, or -1 - (link triangle of the contact) for a contact certified
// in FP32 (CERT).
template <bool IDB, bool CERT>
__device__ __noinline__ int pair_full(PairSmem& S, const MeshView& A, const MeshView& B, const float* TA,
                                      const float* TB, int lane, int nfull, int ncand, float dd, float& m32)
{
  const int n = min(nfull, 32);
  float d32 = FLT_MAX, e = 0.f;
  bool certain = false, flat = false;
  int tA = 0, tB = 0;
  if (lane < n) {
    const int k = nfull - 1 - lane;
    tA = (int)S.fullA[k];
    tB = (int)S.fullB[k];
    if (S.fullL[k] <= m32 * (1.f + 2e-5f)) {  // (m32 may have dropped since it was collected)
      float3 P[3], Q[3];
      place32<false>(A, TA, tA, P);
      place32<IDB>(B, TB, tB, Q);
      e = dd + 128.f * kU * tri_span(P, Q) + 1e-8f;
      flat = __ldg(&A.tri32[3 * (size_t)tA].w) + __ldg(&B.tri32[3 * (size_t)tB].w) > 0.f;
      // (a positive lower bound, bands included, has them apart already)
      if (!(S.fullL[k] > 0.f) && !tri_separated32(P, Q, dd, 0.f)) {
        d32 = 0.f;
        if (CERT) certain = tri_certain_hit32(P[0], P[1], P[2], Q[0], Q[1], Q[2], dd);
      } else {
        d32 = root_approx32(tri_dist2_32(P[0], P[1], P[2], Q[0], Q[1], Q[2]));
      }
    }
  }
  if (CERT) {
    const unsigned mc = __ballot_sync(0xffffffffu, certain);
    if (mc) return -1 - __shfl_sync(0xffffffffu, tA, __ffs(mc) - 1);
  }
  m32 = fminf(m32, warp_min(d32 < FLT_MAX ? d32 + e : FLT_MAX));
  // (a triangle without area: a contact for the canonical function, maybe)
  const bool cand = d32 < FLT_MAX && (flat || d32 - e <= m32 * (1.f + 2e-5f));
  const unsigned mk = __ballot_sync(0xffffffffu, cand);
  if (cand) {
    const int r = ncand + __popc(mk & lanemask_lt());
    S.candA[r] = (uint32_t)tA;
    S.candB[r] = (uint32_t)tB;
    S.candD[r] = flat ? 0.f : d32 - e;
    S.candS[r] = d32 > 0.f && !flat;
  }
  __syncwarp();
  return ncand + __popc(mk);
}

// Lower bound on the distance below two nodes of the trees, less every band a
// comparison with m32 (1 + 2e-5) needs: placement dd of both sides, rounding,
// and the width of the candidates' FP32 band.
template <bool IDB>
__device__ __forceinline__ float node_lb32(const MeshView& A, const MeshView& B, const float* TA, const float* TB,
                                           const KNode& na, const KNode& nb, int nodeA, int nodeB, float dd)
{
  const Box32 BA = xform_box(TA, na.a, na.b);
  Box32 BB;
  if (IDB) {
    BB.c = make_float3(nb.a.x, nb.a.y, nb.a.z);
    BB.h = make_float3(nb.b.x, nb.b.y, nb.b.z);
  } else {
    BB = xform_box(TB, nb.a, nb.b);
  }
  const float slack = 4.f * kU * (fabsf(BA.c.x) + fabsf(BA.c.y) + fabsf(BA.c.z) + fabsf(BB.c.x) + fabsf(BB.c.y) +
                                  fabsf(BB.c.z) + 1.f) +
                      dd * 4.7321f + 1e-5f;
  float lb = box_dist32(BA, BB.c, BB.h);
  const float3 d = sub3(BA.c, BB.c);
  const float n2 = dot3(d, d);
  if (IDB) {
    // the rotation-invariant sphere about A's node centre is tighter than the
    // world box of a rotated node in most directions
    const float gx = fmaxf(0.f, fabsf(d.x) - BB.h.x);
    const float gy = fmaxf(0.f, fabsf(d.y) - BB.h.y);
    const float gz = fmaxf(0.f, fabsf(d.z) - BB.h.z);
    lb = fmaxf(lb, root_below32(gx * gx + gy * gy + gz * gz) - __ldg(A.node_r + nodeA));
  } else {
    lb = fmaxf(lb, root_below32(n2) - __ldg(A.node_r + nodeA) - __ldg(B.node_r + nodeB));
  }
  // separation along the line of centres: both boxes projected onto it
  // (columns of T give the rotated box's half widths along d).  Boxes small
  // against their distance are bounded almost exactly; the soft-min tests 28%
  // fewer triangle pairs with it
  if (n2 > 1e-12f) {
    const float rn = rsqrtf(n2);
    float w = fabsf(TA[0] * d.x + TA[3] * d.y + TA[6] * d.z) * na.b.x +
              fabsf(TA[1] * d.x + TA[4] * d.y + TA[7] * d.z) * na.b.y +
              fabsf(TA[2] * d.x + TA[5] * d.y + TA[8] * d.z) * na.b.z;
    if (IDB)
      w += fabsf(d.x) * BB.h.x + fabsf(d.y) * BB.h.y + fabsf(d.z) * BB.h.z;
    else
      w += fabsf(TB[0] * d.x + TB[3] * d.y + TB[6] * d.z) * nb.b.x +
           fabsf(TB[1] * d.x + TB[4] * d.y + TB[7] * d.z) * nb.b.y +
           fabsf(TB[2] * d.x + TB[5] * d.y + TB[8] * d.z) * nb.b.z;
    // (the projections err by at most 4u |d| (|h| + |d|); 16u covers them
    // and the normalisation)
    lb = fmaxf(lb, (n2 - w) * rn - 16.f * kU * (n2 + w) * rn);
  }
  return lb - slack;
}

struct PairCnt {
  unsigned nodes = 0, tri = 0, fp64 = 0;  // per lane
};

// Minimum distance of A (under TA) and B (under TB, or in world coordinates),
// below m32 on entry: the caller has set S.b2 / S.have; `ready` makes the
// FP64 transforms available before the first finalisation.  Returns 0 (S.have
// tells whether something was found), 1 for a contact certified in FP32 (CERT;
// certA: the link triangle), 2 when the stack would overflow.  m32 is lowered
// to an upper bound of the minimum.
template <bool IDB, bool CERT, class Ready>
__device__ __forceinline__ int pair_distance(PairSmem& S, const MeshView& A, const MeshView& B, int rootA, int rootB,
                                             const float* TA, const float* TB, const double* TA64, const double* TB64,
                                             float dd, float& m32, int& certA, int lane, PairCnt& cnt, Ready&& ready)
{
  const unsigned lt = lanemask_lt();
  if (lane == 0) S.stack[0] = make_uint2((uint32_t)rootA, (uint32_t)rootB);
  __syncwarp();
  int top = 1, njobs = 0, nfull = 0, ncand = 0;
  uint32_t jpos = 0, jtotal = 0;  // expansion of the leaf pairs in progress
  int jbefore = 0;                // leaf pairs that start before jpos
  // collected pairs that may touch (lower bound <= 0) are tested at once: a
  // contact certified early ends the search
  bool touch = false;
#pragma unroll 1
  for (;;) {
    const bool drained = top == 0 && njobs == 0;
    if (nfull >= 32 || ((drained || touch) && nfull > 0)) {
      touch = false;
      if (ncand > kPCand - 32) {
        ready();
        cnt.fp64 += pair_flush<IDB>(S, A, B, TA, TB, TA64, TB64, lane, ncand, m32, dd);
        ncand = 0;
        if (S.have) m32 = fminf(m32, sqrtf((float)S.b2) * (1.f + 2e-6f));
      }
      const int r = pair_full<IDB, CERT>(S, A, B, TA, TB, lane, nfull, ncand, dd, m32);
      if (CERT && r < 0) {
        certA = -1 - r;
        return 1;
      }
      ncand = r;
      nfull -= min(nfull, 32);
      continue;
    }
    if (drained) break;
    if (jpos < jtotal) {
      // ---- triangle pairs of the leaf pairs, one per lane: lower bounds
      const uint32_t p = jpos + lane;
      bool go = false;
      float lb = 0.f;
      int tA = 0, tB = 0;
      const uint32_t starts = window_starts(S.jobOff, jbefore, njobs, jpos, lane);
      if (p < jtotal) {
        const int j = jbefore + __popc(starts & (lt | (1u << lane))) - 1;
        const uint32_t r = p - S.jobOff[j], cb = (S.jobB[j] >> 28) + 1, ra = leaf_quotient(r, cb);
        tA = (int)((S.jobA[j] & 0x0fffffffu) + ra);
        tB = (int)((S.jobB[j] & 0x0fffffffu) + r - ra * cb);
        float3 P[3], Q[3];
        place32<false>(A, TA, tA, P);
        place32<IDB>(B, TB, tB, Q);
        const float span = tri_span(P, Q);
        const float e = dd + 128.f * kU * span + 1e-8f;
        const float lim = m32 * (1.f + 2e-5f);
        lb = tri_axis_lb32(P, Q, span) - 2.f * e;
        if (lb <= lim) lb = fmaxf(lb, tri_box_lb32(P, Q) - 2.f * e);
        go = lb <= lim;
        cnt.tri++;
      }
      const unsigned mg = __ballot_sync(0xffffffffu, go);
      if (go) {
        const int r = nfull + __popc(mg & lt);
        S.fullA[r] = (uint32_t)tA;
        S.fullB[r] = (uint32_t)tB;
        S.fullL[r] = lb;
      }
      nfull += __popc(mg);
      if (CERT) touch = __any_sync(0xffffffffu, go && lb <= 0.f);
      jpos += 32;
      jbefore += __popc(starts);
      if (jpos >= jtotal) {
        jpos = jtotal = 0;
        njobs = 0;
      }
      __syncwarp();
      continue;
    }
    if (njobs >= 16 || top == 0) {
      uint32_t carry = 0;
#pragma unroll 1
      for (int b = 0; b < njobs; b += 32) {
        const int j = b + lane;
        const uint32_t c = j < njobs ? ((S.jobA[j] >> 28) + 1) * ((S.jobB[j] >> 28) + 1) : 0u;
        uint32_t incl = c;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += v;
        }
        if (j < njobs) S.jobOff[j] = carry + incl - c;
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      __syncwarp();
      jtotal = carry;
      jpos = 0;
      jbefore = 0;
      continue;
    }
    // ---- node pairs.  A batch of n pops grows the stack by at most n; near
    // the capacity the batch narrows down to plain depth-first order (one
    // pair), whose growth is bounded by the depth of the two trees, so a
    // wide front (a link deep inside an obstacle, where no box is pruned)
    // does not overflow the stack
    const int n = min(min(top, 32), max(1, kPStack - 64 - top));
    const bool have = lane < n;
    uint2 en = make_uint2(0, 0);
    if (have) en = S.stack[top - 1 - lane];
    __syncwarp();
    top -= n;
    const int nodeA = (int)en.x, nodeB = (int)en.y;
    int outcome = 0;
    uint2 c0 = make_uint2(0, 0), c1 = make_uint2(0, 0);
    uint32_t jA = 0, jB = 0;
    cnt.nodes += have ? 1 : 0;
    if (have) {
      const KNode na = A.nodes[nodeA];
      const KNode nb = B.nodes[nodeB];
      if (node_lb32<IDB>(A, B, TA, TB, na, nb, nodeA, nodeB, dd) <= m32 * (1.f + 2e-5f)) {
        const int cntA = f2i(na.b.w), cntB = f2i(nb.b.w);
        const int ia = f2i(na.a.w), ib = f2i(nb.a.w);
        if (cntA > 0 && cntB > 0) {
          outcome = 2;
          jA = (uint32_t)ia | ((uint32_t)(cntA - 1) << 28);
          jB = (uint32_t)ib | ((uint32_t)(cntB - 1) << 28);
        } else {
          outcome = 1;
          const bool splitB = cntA > 0 || (cntB == 0 && (nb.b.x + nb.b.y + nb.b.z) > (na.b.x + na.b.y + na.b.z));
          c0 = splitB ? make_uint2((uint32_t)nodeA, (uint32_t)ib) : make_uint2((uint32_t)ia, (uint32_t)nodeB);
          c1 = splitB ? make_uint2((uint32_t)nodeA, (uint32_t)ib + 1) : make_uint2((uint32_t)ia + 1, (uint32_t)nodeB);
        }
      }
    }
    const unsigned m1 = __ballot_sync(0xffffffffu, outcome == 1);
    const unsigned m2 = __ballot_sync(0xffffffffu, outcome == 2);
    if (top + 2 * __popc(m1) > kPStack) return 2;  // (not with the narrowing above; checked, not hidden)
    if (outcome == 1) {
      const int r = top + 2 * __popc(m1 & lt);
      S.stack[r] = c1;
      S.stack[r + 1] = c0;
    } else if (outcome == 2) {
      const int r = njobs + __popc(m2 & lt);
      S.jobA[r] = jA;
      S.jobB[r] = jB;
    }
    top += 2 * __popc(m1);
    njobs += __popc(m2);
    __syncwarp();
  }
  if (ncand > 0) {
    ready();
    cnt.fp64 += pair_flush<IDB>(S, A, B, TA, TB, TA64, TB64, lane, ncand, m32, dd);
    if (S.have) m32 = fminf(m32, sqrtf((float)S.b2) * (1.f + 2e-6f));
  }
  return 0;
}

}  // namespace kgpu
