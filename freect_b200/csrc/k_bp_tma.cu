// Helical Q-weighted backprojection, TMA-staged (sm_100a).
//
// Same algorithm as backproject_kernel (cuda_kernels.cuh:198-287) and
// k_bp (k_backproject.cu); this kernel is organised for throughput:
//
//  * Lanes are slices. A warp owns CPW (x, y) columns and the SL consecutive
//    native slices of a slab (SL = 32, or 16 with the warp's lanes 0-15 and
//    16-31 on two groups of CPW / 2 columns); lane l holds slice s0 + l % SL
//    of its group's columns. The geometry of a (column, view) pair -- p_hat,
//    l_hat, the asin term, the channel index and weight, and the row
//    coordinate as a linear function of z -- is computed once, by one lane,
//    and broadcast to the group's lanes through shared memory.
//  * Filtered rows are read in the backprojection layout [view][channel][row]
//    (rows contiguous), so the lanes of a column group, which sit at
//    consecutive rows of the same two channels, read consecutive shared-memory
//    words.
//  * A producer warp walks the half-turn angles theta~ and, for each, selects
//    the views j = theta~ + k P/2 whose table position can reach the CTA's
//    slab (the reference's z cull, cuda_kernels.cuh:232, and the detector's
//    cone), and TMA-loads the channel window each view needs for the CTA's
//    column tile (all rows) into a 2-stage mbarrier ring.
//  * For every column the NW consumer warps accumulate sum(W g) and sum(W)
//    over the staged views of theta~ and add (2 pi/P) sum(W g)/sum(W) to the
//    column's slice in registers (NaN when no view contributes, like the
//    reference). In wfbp_run the write-back also forms the requested slices
//    that lie inside the slab (fused thickening, bp_fused_thicken).
//
// Element types: float (FP32 rows) or uint32_t holding half2 pairs
// (row r, row r+1) of FP16 rows divided by one power of two for the whole
// scan, which the host folds into the write-back's 2 pi / P.
//
// Every mbarrier wait is bounded; on timeout the CTA records WFBP_ERR_TIMEOUT
// in the error word and stops. Window or slot overflows (which the host's
// sizing rules out) are recorded as well and the affected samples skipped.
#include "wfbp_internal.h"
#include "bp_math.cuh"
#include "wait.cuh"

#include <cuda.h>

#include <algorithm>
#include <cstring>

#include <type_traits>

namespace {


__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Bounded wait on phase parity (wait.cuh); false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) { return wfbp_mbar_wait(bar, parity); }

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// Clusters: barrier over all threads of the cluster's CTAs (release / acquire,
// which orders their shared-memory accesses), a word of another CTA's shared
// memory.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared(uint32_t saddr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(saddr), "f"(v) : "memory");
}

// Geometry of a pair of columns for one view, stored so that 16-byte
// shared-memory loads give both columns' fields as float2 operands of the
// packed FP32x2 instructions (FFMA2 / FADD2 / FMUL2). GeoP carries the row
// range the table-position cull leaves (cuda_kernels.cuh:232); when the
// host has shown that the cull never removes a sample whose row lies in
// [0, nr - 2] (the detector's cone is shorter than z_rot), that range is
// [0, nr - 2] for every record, GeoQ drops it and the test uses its centre
// and half width (nr - 2) / 2 as constants: the same compare on the same
// values, so both records give the same samples.
struct __align__(16) GeoP {
  float2 bq, cq;    // q(z) = bq z + cq
  float2 qmid, qhw;  // valid for |q - qmid| <= qhw (the row range [qlo, qhi] as centre and half width)
  int2 addr;        // shared-memory byte offset of (channel pf, row 0) of the view's slot
  float2 wp;        // FP32 rows: channel weight; half2 pairs: bits of the half2 (wp, wp)
};
struct __align__(16) GeoQ {
  float2 bq, cq;    // q(z) = bq z + cq (an invalid record: bq = 0, cq = -1e30)
  int2 addr;
  float2 wp;
};
// Record of the reference layout's form (REFQ): k_bp's own arithmetic per
// sample (an angle's quotient is the other forms'), q = (((z - zt) + zr2pi asn) inv + 1) hn with the roundings that
// kernel has, so that a sample at the edge of the detector falls the same way.
struct __align__(16) GeoR {
  float2 inv, asn;  // 1 / (l_hat tan(cone)), asin(p_hat / R) (an invalid record: 1, -1e30)
  int2 addr;
  float2 wp;
};
static_assert(sizeof(GeoR) == BP_GEO_BYTES, "record sizes of bp_smem_layout");
static_assert(sizeof(GeoP) == BP_GEO_BYTES_ZCULL && sizeof(GeoQ) == BP_GEO_BYTES, "record sizes of bp_smem_layout");

// a - b: fma(b, -1, a) rounds once, like the subtraction
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }

// Shared memory of a CTA: the mbarriers and small words at fixed offsets
// (they persist across the tiles of a persistent launch), then the regions
// of bp_smem_layout for the tile's scan.
// int [16]: [0..1] views per stage, [2..3] steps per stage, [8] failure flag, [9] next item
constexpr int BT_OFF_NVS = 64;

__device__ __forceinline__ void bp_init_barriers(uint8_t* smem, int nw) {
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  if (threadIdx.x == 0) {
    reinterpret_cast<int*>(smem + BT_OFF_NVS)[8] = 0;
    for (int s = 0; s < BT_STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&full[BT_STAGES + s], nw);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
}

// Fused thickening of one slab (ThickFuse) from its records (fz, nfz words).
// For every interior requested slice r each group of SL lanes (lane = slice
// s0 + lane % SL) gathers its native values with shuffles, in the CSR order
// and with the same FMA chain and division as k_thicken, so the result is
// bit-identical to thickening the written native volume. Lane c of a group
// writes column c of the group. All 32 lanes of the warp take part.
template <int CPW, int SL, int CPG>
__device__ __forceinline__ void bp_fused_thicken(const ThickFuse& tf, const float (&vals)[CPG], const int* fz,
                                                 int nfz, int warp, int lane, int ix0, int iy0, const BPTile& bt,
                                                 const BPParams& p) {
  const int grp = lane / SL, ll = lane % SL;
  const int tt = warp * CPW + grp * CPG + min(ll, CPG - 1);
  const int ix = ix0 + tt % bt.tx, iy = iy0 + tt / bt.tx;
  const bool wr = ll < CPG && ix < p.nx && iy < p.ny;
  const size_t plane = (size_t)p.nx * p.ny, vox = (size_t)iy * p.nx + ix;
  nfz = min(nfz, BT_FUSE_WORDS);
  for (int pos = 0; pos + 3 <= nfz;) {
    const int r = __ldg(fz + pos), n = __ldg(fz + pos + 1);
    const float ws = __int_as_float(__ldg(fz + pos + 2));
    if (n < 0 || pos + 3 + 2 * n > nfz) break;  // malformed records (host sizing guarantees otherwise)
    float acc[CPG];
#pragma unroll
    for (int c = 0; c < CPG; c++) acc[c] = 0.0f;
    for (int e = 0; e < n; e++) {
      const int src = grp * SL + (__ldg(fz + pos + 3 + 2 * e) & (SL - 1));
      const float wt = __int_as_float(__ldg(fz + pos + 4 + 2 * e));
#pragma unroll
      for (int c = 0; c < CPG; c++) acc[c] = fmaf(wt, __shfl_sync(0xffffffffu, vals[c], src), acc[c]);
    }
    float v = 0.0f;
#pragma unroll
    for (int c = 0; c < CPG; c++)
      if (c == ll) v = acc[c];
    if (wr && r >= 0 && r < tf.nzr) tf.out[(size_t)r * plane + vox] = v / ws;
    pos += 3 + 2 * n;
  }
}

// The same for a tile outside the FOV, whose native values are all +0:
// k_thicken gives +0 / sum of weights = +0 for every interior slice.
template <int CPW, int SL, int CPG>
__device__ __forceinline__ void bp_fused_zero(const ThickFuse& tf, int bz, int warp, int lane, int ix0, int iy0,
                                              const BPTile& bt, const BPParams& p) {
  const int2 rr = tf.slab_req[bz];
  const int grp = lane / SL, ll = lane % SL;
  const int tt = warp * CPW + grp * CPG + min(ll, CPG - 1);
  const int ix = ix0 + tt % bt.tx, iy = iy0 + tt / bt.tx;
  const bool wr = ll < CPG && ix < p.nx && iy < p.ny;
  const size_t plane = (size_t)p.nx * p.ny, vox = (size_t)iy * p.nx + ix;
  for (int k0 = rr.x; k0 < rr.y; k0 += 32) {
    const int mine = k0 + lane < rr.y ? __ldg(tf.req + k0 + lane) : -1;  // one load per lane
    const int cnt = min(32, rr.y - k0);
    for (int k = 0; k < cnt; k++) {
      const int r = __shfl_sync(0xffffffffu, mine, k);
      if (wr && r >= 0 && r < tf.nzr) tf.out[(size_t)r * plane + vox] = 0.0f;
    }
  }
}

// One column tile (bt.tx x bt.ty columns, SL slices from slab bz) of one scan.
// `ring` counts the theta~ steps this CTA has run through its two-stage
// ring before this tile (stage = ring & 1, phase = (ring >> 1) & 1), so a
// persistent CTA continues the barriers' phases from tile to tile. The tile
// sums the half-turn angles of chunk `chunk` of nc. With BP_CLUSTER the CTA is
// number `chunk` of a cluster of nc that share the tile's angles: the CTAs (if
// there are several) leave their sums in shared memory, and CTA r adds them in
// chunk order for its warps w = r mod nc and writes those columns. BP_ITEM with nc > 1 writes the
// plain sums (a batch's chunk).
// Returns the number of ring steps the tile used: te - tb, or 0 for a tile entirely
// outside the reconstruction FOV (whose voxels are written as 0, the value
// the reference leaves there). A bounded wait that gave up sets the failure
// word (the CTA must stop).
// The angles a tile sums: all of them, a chunk as a CTA of a cluster, or a
// chunk whose plain sums a persistent batch writes.
enum BpRange { BP_ALL, BP_CLUSTER, BP_ITEM };

template <typename T, int CPW, int CU, int NW, int SL, bool ZC, bool COUNT, bool FUSE, int RANGE, bool REFQ = false>
__device__ __forceinline__ int bp_tile(const CUtensorMap* map, float* __restrict__ vol,
                                        const float2* __restrict__ view_sc, const float* __restrict__ view_z,
                                        const float* __restrict__ zslices,
                                        const BPParams& p, const BPTile& bt, int bx, int by, int bz,
                                        unsigned long long* __restrict__ count, int* __restrict__ err, uint8_t* smem,
                                        uint32_t ring, const ThickFuse& tf, int chunk, int nc) {
  constexpr bool HALF = !std::is_same<T, float>::value;
  static_assert(!REFQ || (!HALF && !ZC), "the reference layout's form: FP32 rows, its own cull test");
  using Geo = typename std::conditional<REFQ, GeoR, typename std::conditional<ZC, GeoP, GeoQ>::type>::type;
  constexpr int NPW = CPW / 2;  // column pairs per warp
  // SL = 32: the warp's 32 lanes are 32 slices of each of its CPW columns.
  // SL = 16: lanes 0-15 and 16-31 are 16 slices of two column groups of
  // CPW / 2 columns each (a 16-slice slab: fewer lanes outside a view's cone).
  constexpr int NG = 32 / SL, CPG = CPW / NG;  // column groups per warp, columns per group
  static_assert(SL == 32 || SL == 16, "slab of 32 or 16 slices");
  static_assert(CU % 2 == 0 && CPG % CU == 0, "columns per step must be even and divide the columns per group");
  const BpSmem L = bp_smem_layout(bt, CPW);  // bt.zc == ZC (the launch picks the instantiation)
  uint8_t* slots = smem + L.slots;                            // [STAGES][nv_max][slot_bytes]
  int2* vinfo = reinterpret_cast<int2*>(smem + L.vinfo);      // [STAGES][nv_max] (view, first channel)
  BpViewGeo* vgeo = reinterpret_cast<BpViewGeo*>(smem + L.vgeo);  // [STAGES][nv_max] the views' angle and z
  float2* vwin = reinterpret_cast<float2*>(smem + L.vwin);    // [nv_max] slice range the tile can use of a view (producer)
  uint32_t* vlist = reinterpret_cast<uint32_t*>(smem + L.list);  // [STAGES][32] the lanes' views, 4 bits each
  int* nvs = reinterpret_cast<int*>(smem + BT_OFF_NVS);       // [STAGES] views, [2 + stage] steps, [8] failure flag
  // [warps][nv_max + 1] views of [NG][CPG / 2] records (bp_geo_view)
  constexpr unsigned GEO_G = bp_geo_group(CPW, SL, (int)sizeof(Geo)), GEO_V = bp_geo_view(CPW, SL, (int)sizeof(Geo));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + BT_STAGES;
  volatile int* s_fail = nvs + 8;

  const int tb = RANGE == BP_ALL ? 0 : bp_chunk_begin(chunk, nc, p.P2);
  const int te = RANGE == BP_ALL ? p.P2 : bp_chunk_begin(chunk + 1, nc, p.P2);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int ix0 = bx * bt.tx, iy0 = by * bt.ty;
  const int s0 = bz * SL;
  const int grp = lane / SL;  // column group of this lane

  // slab z range (all warps and groups compute the same values)
  const int my_s = s0 + lane % SL;
  const float zl = my_s < p.nz ? zslices[my_s] : __int_as_float(0x7fc00000);
  float zmn = my_s < p.nz ? zl : 3.0e38f, zmx = my_s < p.nz ? zl : -3.0e38f;
#pragma unroll
  for (int o = SL / 2; o > 0; o >>= 1) {
    zmn = fminf(zmn, __shfl_xor_sync(0xffffffffu, zmn, o));
    zmx = fmaxf(zmx, __shfl_xor_sync(0xffffffffu, zmx, o));
  }

  const float nxm = 0.5f * ((float)p.nx - 1.0f), nym = 0.5f * ((float)p.ny - 1.0f);
  auto xcoord = [&](int ix) { return ((float)ix - nxm) * p.fov / (float)p.nx + p.x0; };
  auto ycoord = [&](int iy) { return ((float)iy - nym) * p.fov / (float)p.ny + p.y0; };

  {
    // the voxel centre of the tile nearest the isocentre; with a margin for
    // rounding, a tile beyond the FOV circle holds no voxel the reference
    // backprojects (cuda_kernels.cuh:220)
    const float xa = xcoord(ix0), xb = xcoord(min(ix0 + bt.tx - 1, p.nx - 1));
    const float ya = ycoord(iy0), yb = ycoord(min(iy0 + bt.ty - 1, p.ny - 1));
    const float xn = fminf(fmaxf(0.0f, xa), xb), yn = fminf(fmaxf(0.0f, ya), yb);
    if (xn * xn + yn * yn > p.fov_half2 * 1.0001f + 1e-3f) {
      if (RANGE == BP_CLUSTER && chunk > 0) return 0;  // the cluster's first CTA writes
      if (warp < NW && my_s < p.nz) {
        const size_t plane = (size_t)p.nx * p.ny;
        for (int c = 0; c < CPG; c++) {
          const int tt = warp * CPW + grp * CPG + c;
          const int ix = ix0 + tt % bt.tx, iy = iy0 + tt / bt.tx;
          if (ix < p.nx && iy < p.ny) vol[(size_t)my_s * plane + (size_t)iy * p.nx + ix] = 0.0f;
        }
      }
      if (FUSE && tf.out && warp < NW) bp_fused_zero<CPW, SL, CPG>(tf, bz, warp, lane, ix0, iy0, bt, p);
      return 0;
    }
  }

  if (warp == NW) {
    // ---------------- producer ----------------
    // The 32 lanes test the half turns k of theta~ in parallel (lane = k
    // mod 32), the selected views are compacted in k order with a ballot, and
    // their copies are issued by as many lanes.
    const float zlo = zmn - bt.reach, zhi = zmx + bt.reach;
    const float xa = xcoord(ix0), xb = xcoord(min(ix0 + bt.tx - 1, p.nx - 1));
    const float ya = ycoord(iy0), yb = ycoord(min(iy0 + bt.ty - 1, p.ny - 1));
    const uint32_t view_bytes = (uint32_t)(bt.W * bt.nrp * sizeof(T));
    const unsigned below = (1u << lane) - 1u;
    // no lists where a slice range can be NaN: the tile has a corner beyond the
    // source's orbit (|p_hat| >= R for some angle)
    const bool lists = bt.nv_max <= BP_LIST_VIEWS &&
                       fmaxf(xa * xa, xb * xb) + fmaxf(ya * ya, yb * yb) < 0.999f * p.R2;
    int issued_upto = 0;
    bool failed = false;
    for (int t = tb; t < te; t++) {
      const uint32_t g = ring + (uint32_t)(t - tb);
      const int s = (int)(g & 1u);
      const uint32_t u = g >> 1;
      int ok = 1;
      if (lane == 0) ok = (u < 1 || mbar_wait(&empty[s], (u - 1) & 1)) && !*s_fail;
      if (!__shfl_sync(0xffffffffu, ok, 0)) {
        failed = true;
        break;
      }
      int nv = 0;
      for (int kb = 0; kb < p.K; kb += 32) {
        const int k = kb + lane;
        const int j = t + k * p.P2;
        bool sel = false;
        int c_lo = 0;
        float wlo = 0.0f, whi = 0.0f;
        float4 vf = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // FP32 form: the view's sin, cos, z for the records
        if (k < p.K) {
          const float zt = __ldg(view_z + j);
          const float2 sc = __ldg(view_sc + j);
          vf = make_float4(sc.x, sc.y, zt, 0.0f);
          if (!(zt < zlo || zt > zhi)) {
            const float p1 = xa * sc.x - ya * sc.y, p2 = xa * sc.x - yb * sc.y;
            const float p3 = xb * sc.x - ya * sc.y, p4 = xb * sc.x - yb * sc.y;
            const float pmax = fmaxf(fmaxf(p1, p2), fmaxf(p3, p4));
            const float pmin = fminf(fminf(p1, p2), fminf(p3, p4));
            // rows this tile can use: q in [0, nr-2] needs |z - zt + A| <= l_hat tan,
            // with l_hat <= R - min(t) over the tile and A monotonic in p_hat
            const float t1 = xa * sc.y + ya * sc.x, t2 = xa * sc.y + yb * sc.x;
            const float t3 = xb * sc.y + ya * sc.x, t4 = xb * sc.y + yb * sc.x;
            const float lhi = sqrtf(p.R2) - fminf(fminf(t1, t2), fminf(t3, t4));
            // (a bound is NaN at a corner beyond the source's orbit: then it excludes no view)
            const float amin = p.zr2pi * asinf(p.rR * pmin), amax = p.zr2pi * asinf(p.rR * pmax);
            const float eps = 1e-3f * (1.0f + fabsf(zt));
            wlo = zt - amax - lhi * p.tanc - eps;
            whi = zt - amin + lhi * p.tanc + eps;
            sel = !(whi < zmn || wlo > zmx);
            const float idx_min = p.kp - (pmax * p.ps + p.c0);  // p_idx decreases with p_hat
            c_lo = max(0, min((int)floorf(idx_min) - 1, p.nch - bt.W));
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, sel);
        const int pos = nv + __popc(m & below);
        if (sel) {
          if (pos < bt.nv_max) {
            vinfo[s * bt.nv_max + pos] = make_int2(j, c_lo);
            vwin[pos] = make_float2(wlo, whi);
            // the view's angle and z for the consumers' record pass (the
            // mixed form's FP64 tables; the FP32 form's values of the test)
            BpViewGeo* g = vgeo + s * bt.nv_max + pos;
            if constexpr (HALF) {
              const double2 sc64 = __ldg(p.sc64 + j);
              const double z64 = __ldg(p.z64 + j);
              g->s = sc64.x;
              g->c = sc64.y;
              g->z = z64;
            } else {
              *reinterpret_cast<float4*>(g) = vf;
            }
          } else {
            atomicOr(err, WFBP_ERRBIT_BP_SLOTS);  // more views than slots: host sizing violated
          }
        }
        nv = min(nv + __popc(m), bt.nv_max);
      }
      __syncwarp();
      {
        // lane = slice: the views, in order, whose slice range holds it
        uint32_t list = 0u;
        int n = 0;
        if (nv > 1 && lists)
          for (int v = 0; v < nv; v++) {
            const float2 w = vwin[v];
            if (zl >= w.x && zl <= w.y) {
              list |= n < 8 ? (uint32_t)v << (4 * n) : 0u;
              n++;
            }
          }
        const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
        // the idle record ends a list
        if (n < 8) list |= (uint32_t)(0x11111111u * (unsigned)bt.nv_max) << (4 * n);
        // Steps over lists cost more each (lanes on two views' samples meet in
        // the banks, more so with FP32 rows' eight loads per pair): every view
        // for every lane unless they save enough.
        const bool pays = nv > 1 && lists && most <= 8 &&
                          (HALF ? 6 * most < 5 * nv : 3 * most <= 2 * nv);
        vlist[s * 32 + lane] = pays ? list : 0x76543210u;
        if (lane == 0) nvs[2 + s] = pays ? most : nv;
      }
      __syncwarp();
      if (lane == 0) {
        nvs[s] = nv;
        mbar_arrive_tx(&full[s], (uint32_t)nv * view_bytes);
      }
      __syncwarp();
      for (int v = lane; v < nv; v += 32) {
        const int2 vi = vinfo[s * bt.nv_max + v];
        tma_load_3d(slots + ((size_t)s * bt.nv_max + v) * bt.slot_bytes, map, &full[s], 0, vi.y, vi.x);
      }
      issued_upto = t - tb + 1;
    }
    if (failed && lane == 0) {
      *s_fail = 1;
      atomicExch(err, WFBP_ERR_TIMEOUT);
      // let copies already issued land before the CTA's shared memory goes away
      for (int t = max(0, issued_upto - BT_STAGES); t < issued_upto; t++) {
        const uint32_t g = ring + (uint32_t)t;
        mbar_wait(&full[g & 1u], (g >> 1) & 1u);
      }
    }
    __syncwarp();
    if (RANGE == BP_CLUSTER && bp_exchanges(nc)) {  // the consumers' barriers below
      __syncthreads();
      cluster_sync();
      cluster_sync();
    }
    return te - tb;
  }

  // ---------------- consumers ----------------
  float2 vacc[CPG / 2];  // columns (2i, 2i + 1) of this lane's group
#pragma unroll
  for (int c = 0; c < CPG / 2; c++) vacc[c] = make_float2(0.0f, 0.0f);
  unsigned long long cnt = 0;
  const float k1 = 2.5f / p.hn;
  uint8_t* wgeo = smem + L.geo + (size_t)warp * (bt.nv_max + 1) * GEO_V;
  // the idle records: no lane valid, zeros to sample (those every warp writes, the same)
  for (int e = lane; e < 2 * bt.nrp; e += 32) reinterpret_cast<float*>(smem + L.zero)[e] = 0.0f;
  if (lane < NPW) {
    Geo* g = reinterpret_cast<Geo*>(wgeo + bt.nv_max * GEO_V + lane / (CPG / 2) * GEO_G) + lane % (CPG / 2);
    if constexpr (REFQ) {
      g->inv = make_float2(1.0f, 1.0f);
      g->asn = make_float2(-1.0e30f, -1.0e30f);
    } else {
      g->bq = make_float2(0.0f, 0.0f);
      g->cq = make_float2(-1.0e30f, -1.0e30f);
    }
    if constexpr (ZC) {
      g->qmid = make_float2(0.0f, 0.0f);
      g->qhw = make_float2(-1.0f, -1.0f);
    }
    g->addr = make_int2((int)L.zero, (int)L.zero);
    g->wp = make_float2(0.0f, 0.0f);
  }
  if (REFQ && lane == 0) reinterpret_cast<float4*>(vgeo + 2 * bt.nv_max)->z = 0.0f;
  __syncwarp();
  constexpr int VPP = 32 / CPW;  // views per geometry pass
  const int gc = lane % CPW, gv = lane / CPW;
  const int gt = warp * CPW + gc;  // tile column handled by this lane in geometry passes
  const int gix = ix0 + gt % bt.tx, giy = iy0 + gt / bt.tx;
  const float gx = xcoord(gix), gy = ycoord(giy);
  const bool gactive = gix < p.nx && giy < p.ny && !(gx * gx + gy * gy > p.fov_half2);
  unsigned active_mask = 0;  // bit c: column c of this warp is inside the grid and the FOV
#pragma unroll
  for (int c = 0; c < CPW; c++) active_mask |= (__shfl_sync(0xffffffffu, gactive ? 1u : 0u, c) & 1u) << c;
  const int nrpb = bt.nrp * 4;  // bytes between channels of a slot
  const float2 zl2 = make_float2(zl, zl);
  const float2 mhn2 = make_float2(-p.hn, -p.hn);
  const float2 pi2 = make_float2(3.14159265f, 3.14159265f);
  const float2 half2c = make_float2(0.5f, 0.5f);
  const unsigned nrm2u = (unsigned)(p.nr - 2);
  const unsigned nrm2b = __float_as_uint(p.nrm2);

  for (int t = tb; t < te; t++) {
    const uint32_t g = ring + (uint32_t)(t - tb);
    const int s = (int)(g & 1u);
    const uint32_t u = g >> 1;
    if (!mbar_wait(&full[s], u & 1u)) {
      *s_fail = 1;
      atomicExch(err, WFBP_ERR_TIMEOUT);
      break;
    }
    const int nv = nvs[s];
    // geometry of (column gc, view v) for v = gv, gv + VPP, ...
    for (int v = gv; v < nv; v += VPP) {
      const int2 vi = vinfo[s * bt.nv_max + v];
      const BpViewGeo& vg = vgeo[s * bt.nv_max + v];  // the view's angle and z, staged by the producer
      float p_hat, t_hat, zt;
      if constexpr (HALF) {
        // the mixed form's per-view geometry is FP64 (sin, cos and table
        // position of the view, from the FP64 tables of wfbp_set_views)
        const double2 sc = make_double2(vg.s, vg.c);
        const double gxd = (double)gx, gyd = (double)gy;
        p_hat = (float)fma(gxd, sc.x, -gyd * sc.y);
        t_hat = (float)fma(gxd, sc.y, gyd * sc.x);
        zt = (float)vg.z;
      } else {
        const float4 vf = *reinterpret_cast<const float4*>(&vg);
        // x sin - y cos and x cos + y sin (cuda_kernels.cuh:235-238) with one
        // rounding of the second product each, as the FP64 form's
        p_hat = fmaf(gx, vf.x, -(gy * vf.y));
        t_hat = fmaf(gx, vf.y, gy * vf.x);
        zt = vf.z;
      }
      float A, inv;  // REFQ: A is the arcsine itself
      if constexpr (REFQ) {
        const float4 vf = *reinterpret_cast<const float4*>(&vg);
        const float l_hat = fmaf(-gy, vf.x, fmaf(-gx, vf.y, sqrtf(fmaf(-p_hat, p_hat, p.R2))));
        A = asinf(p.rR * p_hat);
        inv = 1.0f / (l_hat * p.tanc);
      } else {
        const float l_hat = bp_sqrt(p.R2 - p_hat * p_hat) - t_hat;
        A = p.zr2pi * bp_asin(p.rR * p_hat);
        inv = bp_rcp(l_hat * p.tanc);
      }
      const float p_idx = p.kp - (p_hat * p.ps + p.c0);
      const float pf = floorf(p_idx);
      // floor(p_idx) >= 0 and ceil(p_idx) <= nch - 2 (cuda_kernels.cuh:259-263)
      bool valid = gactive && p_idx >= 0.0f && p_idx <= p.ncm2;
      const int cofs = (int)pf - vi.y;
      if (valid && (cofs < 0 || cofs > bt.W - 2)) {
        atomicOr(err, WFBP_ERRBIT_BP_WINDOW);  // channel window too narrow: host sizing violated
        valid = false;
      }
      const float bq = inv * p.hn;
      const float cq = p.hn * fmaf(A - zt, inv, 1.0f);
      const float wp = p_idx - pf;
      float* gf = reinterpret_cast<float*>(reinterpret_cast<Geo*>(wgeo + v * GEO_V + gc / CPG * GEO_G) +
                                           (gc % CPG >> 1)) +
                  (gc & 1);
      constexpr int O = ZC ? 4 : 0;  // float offset of addr / wp behind the row range
      if constexpr (REFQ) {
        gf[0] = valid ? inv : 1.0f;
        gf[2] = valid ? A : -1.0e30f;
      } else if constexpr (ZC) {
        gf[0] = bq;
        gf[2] = cq;
        // rows q in [0, nr - 2] (cuda_kernels.cuh:259-263) of views within z_rot (:232)
        const float qlo = fmaxf(0.0f, fmaf(zt - p.z_rot, bq, cq)), qhi = fminf(p.nrm2, fmaf(zt + p.z_rot, bq, cq));
        gf[4] = valid ? 0.5f * (qlo + qhi) : 0.0f;
        gf[6] = valid ? 0.5f * (qhi - qlo) : -1.0f;
      } else {
        // rows q in [0, nr - 2] (cuda_kernels.cuh:259-263); an invalid record
        // gives every lane q = -1e30, outside the rows, and finite row weights
        // (a NaN q would make 0 x NaN in the column's sums)
        gf[0] = valid ? bq : 0.0f;
        gf[2] = valid ? cq : -1.0e30f;
      }
      reinterpret_cast<int*>(gf)[4 + O] =
          (int)(L.slots + (size_t)(s * bt.nv_max + v) * bt.slot_bytes) + (valid ? cofs : 0) * nrpb;
      if constexpr (HALF) {
        const __half2 w2 = __float2half2_rn(wp);
        gf[6 + O] = __uint_as_float(*reinterpret_cast<const uint32_t*>(&w2));
      } else {
        gf[6 + O] = wp;
      }
    }
    __syncwarp();
    const uint32_t my_list = vlist[s * 32 + lane];
    const int steps = nvs[2 + s];
#pragma unroll
    for (int c0 = 0; c0 < CPG; c0 += CU) {
      unsigned any = 0u;  // warp-uniform: some group has an active column in this step
#pragma unroll
      for (int g2 = 0; g2 < NG; g2++) any |= (active_mask >> (g2 * CPG + c0)) & ((1u << CU) - 1u);
      if (!any) continue;
      float2 ag[CU / 2], aw[CU / 2];
#pragma unroll
      for (int u2 = 0; u2 < CU / 2; u2++) {
        ag[u2] = make_float2(0.0f, 0.0f);
        aw[u2] = make_float2(0.0f, 0.0f);
      }
      // Each lane takes the views whose cone can hold its slice, in order; the
      // views left out would add zeros. With every lane taking every view that
      // reaches the slab about half the lane slots of a 16-row scanner were
      // outside the cone (ms, every view / lists: 16 rows mixed 5.50 / 4.64,
      // FP32 5.45 / 4.84; 20 rows 17.8 / 15.4, 17.8 / 17.3; 64 rows 39.9 / 39.4,
      // 39.7 / 39.5; 8 x 16 / 8 / 16 slices).
      // (Eight views to a word; more only where every lane takes every view.)
      uint32_t list = my_list;
      const uint8_t* gb = wgeo + grp * GEO_G + c0 / 2 * sizeof(Geo);
      for (int i = 0; i < steps; i++) {
        unsigned v = list & 15u;
        list >>= 4;
        if (i >= 8) v = (unsigned)i;
        const Geo* gpv = reinterpret_cast<const Geo*>(gb + v * GEO_V);
        float dz = 0.0f;
        bool zok = true;
        if constexpr (REFQ) {
          dz = zl - reinterpret_cast<const float4*>(&vgeo[v < (unsigned)bt.nv_max ? s * bt.nv_max + v : 2 * bt.nv_max])->z;
          zok = fabsf(dz) <= p.z_rot;  // cuda_kernels.cuh:232
        }
#pragma unroll
        for (int u2 = 0; u2 < CU / 2; u2++) {
          const Geo g = gpv[u2];
          float2 q, qh = make_float2(0.0f, 0.0f);
          bool okx, oky;
          if constexpr (REFQ) {
            qh = __fmul2_rn(__ffma2_rn(make_float2(p.zr2pi, p.zr2pi), g.asn, make_float2(dz, dz)), g.inv);
            q = __fmul2_rn(__fadd2_rn(qh, make_float2(1.0f, 1.0f)), make_float2(p.hn, p.hn));
            okx = zok && q.x >= 0.0f && q.x <= p.nrm2;
            oky = zok && q.y >= 0.0f && q.y <= p.nrm2;
          } else {
            q = __ffma2_rn(zl2, g.bq, g.cq);
          }
          if constexpr (REFQ) {
          } else if constexpr (ZC) {
            const float2 dq = sub2(q, g.qmid);
            okx = fabsf(dq.x) <= g.qhw.x;
            oky = fabsf(dq.y) <= g.qhw.y;
          } else {
            // 0 <= q <= nr - 2 (cuda_kernels.cuh:259-263): order of the bits, negative q above all
            okx = __float_as_uint(q.x) <= nrm2b;
            oky = __float_as_uint(q.y) <= nrm2b;
          }
          // Row index and fraction through the FP32 pipe: for 0 <= q < 2^23,
          // q + 2^23 rounded down is 2^23 + floor(q), an integer held in the
          // low mantissa bits, and subtracting 2^23 again is exact. Invalid
          // lanes (weight 0; negative, huge or NaN q) read any in-range row:
          // the unsigned difference of the bit patterns is clamped to nr - 2.
          const float2 tq = __fadd2_rd(q, make_float2(8388608.0f, 8388608.0f));
          const float2 fq = __fadd2_rn(tq, make_float2(-8388608.0f, -8388608.0f));
          const unsigned rx = min(__float_as_uint(tq.x) - 0x4B000000u, nrm2u);
          const unsigned ry = min(__float_as_uint(tq.y) - 0x4B000000u, nrm2u);
          const float2 wq = sub2(q, fq);
          const uint8_t* ex = smem + g.addr.x + (rx << 2);
          const uint8_t* ey = smem + g.addr.y + (ry << 2);
          float2 top, bot;
          if constexpr (!HALF) {
            const float2 d00 = make_float2(*reinterpret_cast<const float*>(ex), *reinterpret_cast<const float*>(ey));
            const float2 d01 =
                make_float2(*reinterpret_cast<const float*>(ex + 4), *reinterpret_cast<const float*>(ey + 4));
            const float2 d10 = make_float2(*reinterpret_cast<const float*>(ex + nrpb),
                                           *reinterpret_cast<const float*>(ey + nrpb));
            const float2 d11 = make_float2(*reinterpret_cast<const float*>(ex + nrpb + 4),
                                           *reinterpret_cast<const float*>(ey + nrpb + 4));
            top = __ffma2_rn(g.wp, sub2(d10, d00), d00);
            bot = __ffma2_rn(g.wp, sub2(d11, d01), d01);
          } else {
            // (row r, row r+1) pairs of channels pf and pf+1, interpolated
            // across channels in half2 arithmetic
            const __half2 h0x = *reinterpret_cast<const __half2*>(ex);
            const __half2 h1x = *reinterpret_cast<const __half2*>(ex + nrpb);
            const __half2 h0y = *reinterpret_cast<const __half2*>(ey);
            const __half2 h1y = *reinterpret_cast<const __half2*>(ey + nrpb);
            const uint32_t wbx = __float_as_uint(g.wp.x), wby = __float_as_uint(g.wp.y);
            const __half2 wpx = *reinterpret_cast<const __half2*>(&wbx);
            const __half2 wpy = *reinterpret_cast<const __half2*>(&wby);
            const float2 fx = __half22float2(__hfma2(wpx, __hsub2(h1x, h0x), h0x));
            const float2 fy = __half22float2(__hfma2(wpy, __hsub2(h1y, h0y), h0y));
            top = make_float2(fx.x, fy.x);
            bot = make_float2(fx.y, fy.y);
          }
          const float2 gval = __ffma2_rn(wq, sub2(bot, top), top);
          // W(q) of cuda_kernels.cuh:79-93 with |q_hat| = |q - hn| / hn
          const float2 a = REFQ ? qh : __fadd2_rn(q, mhn2);
          const float ka = REFQ ? 2.5f : k1;
          const float2 tt = __fmul2_rn(make_float2(__saturatef(fmaf(fabsf(a.x), ka, -1.5f)),
                                                   __saturatef(fmaf(fabsf(a.y), ka, -1.5f))),
                                       pi2);
          float2 W = __ffma2_rn(half2c, make_float2(__cosf(tt.x), __cosf(tt.y)), half2c);
          if constexpr (REFQ) {
            // a sample that is not the voxel's stays out altogether: times a
            // weight of 0 one that is not finite would make the voxel NaN
            if (okx) {
              ag[u2].x = fmaf(W.x, gval.x, ag[u2].x);
              aw[u2].x += W.x;
            }
            if (oky) {
              ag[u2].y = fmaf(W.y, gval.y, ag[u2].y);
              aw[u2].y += W.y;
            }
          } else {
            W.x = okx ? W.x : 0.0f;
            W.y = oky ? W.y : 0.0f;
            ag[u2] = __ffma2_rn(W, gval, ag[u2]);
            aw[u2] = __fadd2_rn(aw[u2], W);
          }
          if (COUNT) cnt += (okx ? 1 : 0) + (oky ? 1 : 0);
        }
      }
      // cuda_kernels.cuh:283, vol += (2 pi / P) (sum W g) / (sum W): the
      // quotient through the hardware reciprocal (0 / 0 stays NaN), 2 pi / P
      // (times the FP16 rows' scale) applied once at the write-back
#pragma unroll
      for (int u2 = 0; u2 < CU / 2; u2++)
        vacc[c0 / 2 + u2] = __ffma2_rn(ag[u2], make_float2(bp_rcp(aw[u2].x), bp_rcp(aw[u2].y)), vacc[c0 / 2 + u2]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
  }

  bool mine = true;  // this CTA writes this warp's columns
  if (RANGE == BP_CLUSTER && bp_exchanges(nc)) {  // one chunk: its sums are complete, and the layout has no room for them
    // the chunks' sums of this warp's columns, added in chunk order
    const uint32_t part = smem_u32(smem + L.part) + (uint32_t)((warp * CPG * 32 + lane) * 4);
    __syncthreads();  // the ring is idle in this CTA
#pragma unroll
    for (int c = 0; c < CPG; c++) st_shared(part + c * 128, (c & 1) ? vacc[c / 2].y : vacc[c / 2].x);
    cluster_sync();
    mine = warp % nc == chunk;
    if (mine) {
#pragma unroll
      for (int c = 0; c < CPG; c++) {
        float v = ld_cluster(part + c * 128, 0);
        for (int r = 1; r < nc; r++) v += ld_cluster(part + c * 128, (uint32_t)r);
        if (c & 1) vacc[c / 2].y = v;
        else vacc[c / 2].x = v;
      }
    }
    cluster_sync();  // no CTA ends, or reuses its shared memory, while another reads it
  }

  // write the slab: columns outside the grid or the FOV keep the 0 the
  // reference leaves there
  const unsigned my_cols = (active_mask >> (grp * CPG)) & ((1u << CPG) - 1u);
  float vals[CPG];
  const float scale = RANGE == BP_ITEM && nc > 1 ? 1.0f : p.dtheta;
#pragma unroll
  for (int c = 0; c < CPG; c++)
    vals[c] = ((my_cols >> c) & 1u) ? scale * ((c & 1) ? vacc[c / 2].y : vacc[c / 2].x) : 0.0f;
  if (mine && my_s < p.nz) {
    const size_t plane = (size_t)p.nx * p.ny;
#pragma unroll
    for (int c = 0; c < CPG; c++) {
      const int tt = warp * CPW + grp * CPG + c;
      const int ix = ix0 + tt % bt.tx, iy = iy0 + tt / bt.tx;
      if (ix < p.nx && iy < p.ny) vol[(size_t)my_s * plane + (size_t)iy * p.nx + ix] = vals[c];
    }
  }
  if (FUSE && tf.out && mine) {
    const int2 fr = tf.slab_tab[bz];
    bp_fused_thicken<CPW, SL, CPG>(tf, vals, tf.tab + fr.x, fr.y - fr.x, warp, lane, ix0, iy0, bt, p);
  }
  if (COUNT) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(count, cnt);
  }
  return te - tb;
}

// CTAs per SM the launch bounds of the one-tile kernel ask for: three 9-warp
// CTAs (their registers, at most 75 per thread, and shared memory fit) for
// four columns per pass or 16-slice slabs, in both forms; eight columns per
// pass over 32-slice slabs would spill at that budget and keep two; the wider
// shapes one. (The persistent batch kernel holds more state per thread:
// three only for four columns per pass over 16-slice slabs.)
template <int NW, int CU, int SL, bool BATCH = false>
constexpr int bp_min_ctas() {
  return NW > 8 ? 1 : (BATCH ? (CU == 4 && SL == 16) : (CU == 4 || SL == 16)) ? 3 : 2;
}

// One tile per CTA: grid (tiles x, tiles y, SL-slice slabs x chunks of angles);
// the chunks of a tile are a cluster along z (RANGE = BP_CLUSTER; one chunk:
// BP_ALL, whose loop bounds need no registers).
template <typename T, int CPW, int CU, int NW, int SL, bool ZC, bool COUNT, int RANGE>
__global__ void __launch_bounds__((NW + 1) * 32, bp_min_ctas<NW, CU, SL>())
k_bp_tma(const __grid_constant__ CUtensorMap map, float* __restrict__ vol, const float2* __restrict__ view_sc,
         const float* __restrict__ view_z, const float* __restrict__ zslices, BPParams p, BPTile bt,
         unsigned long long* __restrict__ count, int* __restrict__ err, ThickFuse tf) {
  // the dynamic shared memory is the only shared memory of this kernel, so
  // it starts at the (128-byte aligned) base of the CTA's window
  extern __shared__ __align__(128) uint8_t smem[];
  bp_init_barriers(smem, NW);
  const int z = (int)blockIdx.z, nc = RANGE == BP_CLUSTER ? bt.nc : 1;
  bp_tile<T, CPW, CU, NW, SL, ZC, COUNT, true, RANGE>(&map, vol, view_sc, view_z, zslices, p, bt, blockIdx.x,
                                                      blockIdx.y, bt.zb0 + z / nc, count, err, smem, 0u, tf, z % nc, nc);
}

// The same on the reference layout's rows (transposed, rows_to_channels), with
// k_bp's arithmetic.
template <int CPW, int CU, int NW, int SL, bool COUNT>
__global__ void __launch_bounds__((NW + 1) * 32, bp_min_ctas<NW, CU, SL>())
k_bp_tma_refq(const __grid_constant__ CUtensorMap map, float* __restrict__ vol, const float2* __restrict__ view_sc,
              const float* __restrict__ view_z, const float* __restrict__ zslices, BPParams p, BPTile bt,
              unsigned long long* __restrict__ count, int* __restrict__ err) {
  extern __shared__ __align__(128) uint8_t smem[];
  bp_init_barriers(smem, NW);
  ThickFuse none;
  none.out = nullptr;
  bp_tile<float, CPW, CU, NW, SL, false, COUNT, true, BP_CLUSTER, true>(
      &map, vol, view_sc, view_z, zslices, p, bt, blockIdx.x, blockIdx.y, (int)blockIdx.z / bt.nc, count, err, smem, 0u,
      none, (int)blockIdx.z % bt.nc, bt.nc);
}

// out[view][channel][row] (rows padded to nrp, the padding not written) from
// FP32 rows in[view][row][channel], or FP16 rows times their power-of-two
// scales [view][row] (exact). One CTA per view and 32 channels, 64 rows at a
// time through shared memory: full lines on both sides.
template <typename T>
__global__ void __launch_bounds__(256)
k_rows_to_channels(const T* __restrict__ in, const float* __restrict__ scales, float* __restrict__ out, int nr, int nch,
                   int nrp) {
  __shared__ float tile[64][33];
  const size_t v = blockIdx.x;
  const int c0 = blockIdx.y * 32, nc = min(32, nch - c0);
  for (int r0 = 0; r0 < nr; r0 += 64) {
    const int n = min(64, nr - r0);
    for (int e = threadIdx.x; e < n * 32; e += 256) {
      const int r = e / 32, c = e % 32;
      if (c < nc) {
        const T x = in[(v * nr + r0 + r) * nch + c0 + c];
        if constexpr (std::is_same<T, float>::value) tile[r][c] = x;
        else tile[r][c] = __half2float(x) * __ldg(scales + v * nr + r0 + r);
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * nc; e += 256) {
      const int c = e / n, r = e % n;
      out[(v * nch + c0 + c) * nrp + r0 + r] = tile[r][c];
    }
    __syncthreads();
  }
}

// Persistent launch over the column tiles of several scans: each CTA takes
// the next work item (scan | chunk of angles << 24, tile x, tile y, slab) from
// a global counter until the list is exhausted.
template <typename T, int CPW, int CU, int NW, int SL, bool ZC>
__global__ void __launch_bounds__((NW + 1) * 32, bp_min_ctas<NW, CU, SL, true>())
k_bp_tma_batch(const BpScan* __restrict__ scans, const int4* __restrict__ items, int n_items,
               unsigned* __restrict__ next, int* __restrict__ err) {
  extern __shared__ __align__(128) uint8_t smem[];
  bp_init_barriers(smem, NW);
  volatile int* words = reinterpret_cast<volatile int*>(smem + BT_OFF_NVS);
  uint32_t ring = 0;
  for (;;) {
    if (threadIdx.x == 0) words[9] = (int)atomicAdd(next, 1u);
    __syncthreads();
    const int it = words[9];
    if (it >= n_items || words[8] != 0) break;
    const int4 w = items[it];
    const BpScan* sd = scans + (w.x & 0xffffff);
    const int chunk = w.x >> 24, nc = sd->nc;
    const BPParams p = sd->p;
    const BPTile bt = sd->bt;
    float* vol = sd->vol + (size_t)chunk * p.nz * p.ny * p.nx;
    ring += (uint32_t)bp_tile<T, CPW, CU, NW, SL, ZC, false, false, BP_ITEM>(
        &sd->map, vol, sd->view_sc, sd->view_z, sd->zslices, p, bt, w.y, w.z, w.w, nullptr, err, smem, ring, sd->tf,
        chunk, nc);
    // The next tile's layout may be another scan's: its TMA writes can land
    // where this tile had records, lists or sums.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // the tile's shared memory and words[9] are free again
  }
}

// Dynamic shared memory of `smem` bytes. Shapes meant to run two CTAs per SM
// (8 consumer warps) also ask for the whole unified L1 / shared memory as
// shared memory; the others leave the split to the driver, which keeps more
// L1 for the geometry and view-table loads.
template <int NW, typename K>
cudaError_t prepare_kernel(K* kern, int smem) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess && NW <= 8)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  return e;
}

template <typename... Args>
cudaError_t launch_cluster(void (*kern)(Args...), dim3 grid, int threads, int smem, int nc, cudaStream_t s,
                           Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = cluster.val.clusterDim.y = 1;
  cluster.val.clusterDim.z = (unsigned)nc;
  cfg.attrs = &cluster;
  cfg.numAttrs = nc > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <typename T, int CPW, int CU, int NW, int SL, bool ZC>
cudaError_t launch_one(const CUtensorMap& map, float* vol, const float2* sc,
                       const float* vz, const float* zs, const BPParams& p, const BPTile& bt,
                       unsigned long long* count, int* err, cudaStream_t s, const ThickFuse& tf) {
  const int nslab = (p.nz + SL - 1) / SL;
  if (bt.nc < 1 || bt.nc > BP_MAX_CHUNKS) return cudaErrorInvalidValue;
  if (bt.zb0 < 0 || bt.zb0 >= nslab || bt.nzb < 0 || bt.zb0 + bt.nzb > nslab) return cudaErrorInvalidValue;
  dim3 grid((unsigned)((p.nx + bt.tx - 1) / bt.tx), (unsigned)((p.ny + bt.ty - 1) / bt.ty),
            (unsigned)((bt.nzb ? bt.nzb : nslab - bt.zb0) * bt.nc));
  auto kern = count       ? k_bp_tma<T, CPW, CU, NW, SL, ZC, true, BP_CLUSTER>
              : bt.nc > 1 ? k_bp_tma<T, CPW, CU, NW, SL, ZC, false, BP_CLUSTER>
                          : k_bp_tma<T, CPW, CU, NW, SL, ZC, false, BP_ALL>;
  cudaError_t e = prepare_kernel<NW>(kern, bt.smem_bytes);
  if (e != cudaSuccess) return e;
  return launch_cluster(kern, grid, (NW + 1) * 32, bt.smem_bytes, bt.nc, s, map, vol, sc, vz, zs, p, bt, count, err, tf);
}

template <typename T, int CPW, int CU, int NW, int SL>
cudaError_t launch_batch_one(int zc, const BpScan* scans, const int4* items, int n_items, unsigned* next, int* err,
                             int smem_bytes, int grid, cudaStream_t s) {
  auto kern = zc ? k_bp_tma_batch<T, CPW, CU, NW, SL, true> : k_bp_tma_batch<T, CPW, CU, NW, SL, false>;
  cudaError_t e = prepare_kernel<NW>(kern, smem_bytes);
  if (e != cudaSuccess) return e;
  // grid = SMs; persistent CTAs: as many per SM as fit
  int per_sm = 1;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (NW + 1) * 32, smem_bytes);
  if (e != cudaSuccess) return e;
  grid = std::max(1, std::min(grid * std::max(per_sm, 1), n_items));
  kern<<<grid, (NW + 1) * 32, smem_bytes, s>>>(scans, items, n_items, next, err);
  return cudaGetLastError();
}

// The instantiated launch shapes: (columns per warp, columns per pass, consumer warps, slab slices).
// With 8 consumer warps two CTAs share an SM (registers and shared memory
// permitting), so one CTA's ring refills and tile tails overlap the other's
// updates.
#define WFBP_BP_SHAPES(X)                                                                                        \
  X(16, 4, 16, 32) X(16, 8, 16, 32) X(8, 4, 16, 32) X(8, 8, 16, 32) X(4, 4, 16, 32) X(8, 4, 20, 32) X(8, 8, 20, 32) \
  X(4, 4, 24, 32) X(16, 4, 16, 16) X(16, 8, 16, 16) X(8, 4, 20, 16) X(16, 4, 20, 16) X(16, 8, 20, 16)           \
  X(16, 4, 8, 32) X(16, 8, 8, 32) X(16, 4, 8, 16) X(16, 8, 8, 16)

template <typename T>
cudaError_t launch_elem(const CUtensorMap& map, float* vol, const float2* sc,
                        const float* vz, const float* zs, const BPParams& p, const BPTile& bt,
                        unsigned long long* count, int* err, cudaStream_t s, const ThickFuse& tf) {
  const int cpw = bt.tx * bt.ty / bt.nw;
#define WFBP_ONE(C, U, N, S) \
  if (cpw == C && bt.cu == U && bt.nw == N && bt.slab == S)                                                      \
    return bt.zc ? launch_one<T, C, U, N, S, true>(map, vol, sc, vz, zs, p, bt, count, err, s, tf)               \
                 : launch_one<T, C, U, N, S, false>(map, vol, sc, vz, zs, p, bt, count, err, s, tf);
  WFBP_BP_SHAPES(WFBP_ONE)
#undef WFBP_ONE
  return cudaErrorInvalidValue;
}

__global__ void k_sum_chunks(const float* __restrict__ part, float* __restrict__ vol, float scale, int nc, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float v = __ldg(part + i);
    for (int c = 1; c < nc; c++) v += __ldg(part + (size_t)c * n + i);
    vol[i] = scale * v;
  }
}

}  // namespace

cudaError_t launch_sum_chunks(const float* part, float* vol, float scale, int nc, size_t n, cudaStream_t s) {
  k_sum_chunks<<<(unsigned)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, s>>>(part, vol, scale, nc, n);
  return cudaGetLastError();
}

// Shared-memory bytes of one launch configuration.
size_t bp_tma_smem_bytes(const BPTile& bt, int elem_bytes) {
  (void)elem_bytes;
  return bp_smem_layout(bt, bt.tx * bt.ty / bt.nw).total;
}

bool bp_tma_supported(const BPTile& bt) {
  if (bt.nw < 1) return false;
  const int cpw = bt.tx * bt.ty / bt.nw;
  if (bt.tx * bt.ty != cpw * bt.nw) return false;
#define WFBP_SUP(C, U, N, S) \
  if (cpw == C && bt.cu == U && bt.nw == N && bt.slab == S) return true;
  WFBP_BP_SHAPES(WFBP_SUP)
#undef WFBP_SUP
  return false;
}

cudaError_t bp_tma_encode_map(const void* D, int elem_half2, const BPParams& p, const BPTile& bt, CUtensorMap* map) {
  // 3-D map over [V][nch][nrp] 4-byte elements, box {nrp, W, 1}
  EncodeTiledFn fn = wfbp_encode_tiled_fn();
  if (!fn) return cudaErrorNotSupported;
  cuuint64_t dims[3] = {(cuuint64_t)bt.nrp, (cuuint64_t)p.nch, (cuuint64_t)p.V};
  cuuint64_t strides[2] = {(cuuint64_t)bt.nrp * 4, (cuuint64_t)bt.nrp * 4 * p.nch};
  cuuint32_t box[3] = {(cuuint32_t)bt.nrp, (cuuint32_t)bt.W, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, elem_half2 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                  const_cast<void*>(D), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_backproject_tma(const void* D, int elem_half2, float row_scale, float* vol,
                                   const float2* sc, const float* vz, const float* zs, const BPParams& p0,
                                   const BPTile& bt, unsigned long long* count, int* err, cudaStream_t s,
                                   const ThickFuse* tf) {
  // half2 pairs hold the rows divided by row_scale (a power of two): the
  // write-back's 2 pi / P takes it back, exactly
  BPParams p = p0;
  if (elem_half2) p.dtheta *= row_scale;
  if (!bp_tma_supported(bt)) return cudaErrorInvalidValue;
  CUtensorMap map;
  cudaError_t e = bp_tma_encode_map(D, elem_half2, p, bt, &map);
  if (e != cudaSuccess) return e;
  ThickFuse none;
  memset(&none, 0, sizeof(none));
  const ThickFuse& f = tf ? *tf : none;
  if (elem_half2) return launch_elem<uint32_t>(map, vol, sc, vz, zs, p, bt, count, err, s, f);
  return launch_elem<float>(map, vol, sc, vz, zs, p, bt, count, err, s, f);
}

// The shapes of the reference layout's form: the default ones (default_bp_tile)
// and the smallest tile.
#define WFBP_REFQ_SHAPES(X) X(16, 8, 8, 16) X(16, 8, 20, 16) X(4, 4, 16, 32)

bool bp_refq_supported(const BPTile& bt) {
  const int cpw = bt.tx * bt.ty / bt.nw;
#define WFBP_SUP(C, U, N, S) \
  if (cpw == C && bt.cu == U && bt.nw == N && bt.slab == S) return true;
  WFBP_REFQ_SHAPES(WFBP_SUP)
#undef WFBP_SUP
  return false;
}

cudaError_t launch_rows_to_channels(const void* rows, const float* f16_scales, float* out, int V, int nr, int nch,
                                    int nrp, cudaStream_t s) {
  const dim3 g((unsigned)V, (unsigned)((nch + 31) / 32));
  if (f16_scales) k_rows_to_channels<<<g, 256, 0, s>>>((const __half*)rows, f16_scales, out, nr, nch, nrp);
  else k_rows_to_channels<<<g, 256, 0, s>>>((const float*)rows, f16_scales, out, nr, nch, nrp);
  return cudaGetLastError();
}

cudaError_t launch_backproject_refq(const float* D, float* vol, const float2* sc, const float* vz, const float* zs,
                                    const BPParams& p, const BPTile& bt, unsigned long long* count, int* err,
                                    cudaStream_t s) {
  CUtensorMap map;
  cudaError_t e = bp_tma_encode_map(D, 0, p, bt, &map);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((p.nx + bt.tx - 1) / bt.tx), (unsigned)((p.ny + bt.ty - 1) / bt.ty),
                  (unsigned)(((p.nz + bt.slab - 1) / bt.slab) * bt.nc));
  const int cpw = bt.tx * bt.ty / bt.nw;
#define WFBP_ONE(C, U, N, S)                                                                                       \
  if (cpw == C && bt.cu == U && bt.nw == N && bt.slab == S) {                                                      \
    auto kern = count ? k_bp_tma_refq<C, U, N, S, true> : k_bp_tma_refq<C, U, N, S, false>;                        \
    if ((e = prepare_kernel<N>(kern, bt.smem_bytes)) != cudaSuccess) return e;                                     \
    return launch_cluster(kern, grid, (N + 1) * 32, bt.smem_bytes, bt.nc, s, map, vol, sc, vz, zs, p, bt, count, err); \
  }
  WFBP_REFQ_SHAPES(WFBP_ONE)
#undef WFBP_ONE
  return cudaErrorInvalidValue;
}

cudaError_t launch_backproject_tma_batch(int elem_half2, int cpw, int cu, int nw, int slab, int zc, const BpScan* scans,
                                         const int4* items, int n_items, unsigned* next, int* err, int smem_bytes,
                                         int grid, cudaStream_t s) {
#define WFBP_B32(C, U, N, S) \
  if (cpw == C && cu == U && nw == N && slab == S) return launch_batch_one<uint32_t, C, U, N, S>(zc, scans, items, n_items, next, err, smem_bytes, grid, s);
#define WFBP_BF(C, U, N, S) \
  if (cpw == C && cu == U && nw == N && slab == S) return launch_batch_one<float, C, U, N, S>(zc, scans, items, n_items, next, err, smem_bytes, grid, s);
  if (elem_half2) {
    WFBP_BP_SHAPES(WFBP_B32)
  } else {
    WFBP_BP_SHAPES(WFBP_BF)
  }
#undef WFBP_B32
#undef WFBP_BF
  return cudaErrorInvalidValue;
}
