// pm_compat.cu -- the reference's own radius pipeline (PM_MODE_ZHOU_COMPAT).
//
// Restates KDTreePoint::PrecomputeQueryRadii / ComputeQueryRadii
// (KDTreePoint.cpp:187-248) and the kernels behind them
// (GPU/kdtree_point.cu:118-267, 295-546), then the range gather of
// dev_RangeSearch (GPU/photon_knn.cu:113-235):
//   1. node estimates: every tree slot (node) whose box radius (half
//      diagonal) is at most 0.5 R gets est = refine(centre, R); the others,
//      and all of them when the tree has fewer than 1000 slots, get +inf.
//      (The reference marks qualified nodes, unmarks their direct children
//      and re-marks two child levels, GPU/kdtree_point.cu:626-651; as child
//      boxes nest inside their parents, that is every qualified node.)
//   2. per query: est = min(R, min over the slots on the root-to-leaf path of
//      |q - centre| + est(slot)); the path follows the nearer child box (the
//      reference follows split planes; this tree has boxes);
//   3. refine(q, est): refine_iters rounds of a 32-bin histogram of the
//      distances d < r_max inside [r_min, r_max]; the first bin where the
//      cumulative count reaches k narrows [r_min, r_max] to that bin; counts
//      saturate at 0xfffe; the radius is the final r_max;
//   4. gather: every photon with d^2 < r^2 (strict), front test, filter;
//      r^2_used = max d^2 found when at least k were found, else r^2; fewer
//      than min_found photons -> 0.
// Arithmetic is FP32 with explicit roundings in a fixed order (the oracle
// restates the same steps on the exported tree); a histogram index that
// rounds to 32 (possible when d is just below r_max) goes to bin 31.
//
// Every range search is a warp's: one walk of the 32-wide tree, a child box
// per lane, a photon per lane in the leaves.  A leaf whose nearest and
// farthest possible distances fall into one histogram bin is counted as a
// whole (the bin is a monotone function of d^2, and both bounds are rounded as
// d^2 is), so a dense blob far from the centre costs a step per 32 leaves and
// not one per photon.  The root-to-leaf path of a query is a lane's: a warp
// takes several queries, descends for all of them at once and then refines and
// gathers one after the other.  With a thread per query and per slot instead
// the kernels ran at the pace of the slots beside the blob: 300,001 photons (20 %
// in a caustic of sigma 0.01), 307,200 queries, k = 50, R = 0.1, build included:
// 54.9 -> 3.37 ms; 1,500 photons and 4,000 radii: 350 -> 140 us.  Latency bounds
// what is left (dependent node loads; a quarter of the warps' slots is taken).
#include "pm_internal.h"

namespace pm {

namespace {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kHist = 32;             // one bin per lane
constexpr int kCompatWarps = 8;            // warps per block
// Wide nodes waiting in one walk: at most 31 per level and one more; codes and
// index ties give at most 71 binary levels, 15 wide ones.
constexpr uint32_t kCompatStack = 480;
constexpr uint32_t kCompatKeep = 256;      // photons of one gather kept for the second pass
constexpr uint32_t kCompatUnits = 128;     // half leaves (32 photons) listed by a walk

struct CompatSmem {                        // one warp's
    uint2 stack[kCompatStack];
    uint2 units[kCompatUnits];
    uint32_t hist[kHist];
    uint32_t keep[kCompatKeep];
};

__device__ __forceinline__ void slot_of(const Node* nodes, uint32_t sid, float* lo, float* hi, uint32_t& ref,
                                        uint32_t& cnt) {
    const ChildSlot& s = nodes[sid >> 1].c[sid & 1u];
    lo[0] = s.lo[0]; lo[1] = s.lo[1]; lo[2] = s.lo[2];
    hi[0] = s.hi[0]; hi[1] = s.hi[1]; hi[2] = s.hi[2];
    ref = s.ref; cnt = s.cnt;
}

// Box centre and radius (half the diagonal), FP32 in a fixed order.
__device__ __forceinline__ void extent_of(const float* lo, const float* hi, float* c, float& rad) {
    float d2 = 0.0f;
    for (int a = 0; a < 3; ++a) {
        c[a] = __fmul_rn(__fadd_rn(lo[a], hi[a]), 0.5f);
        const float e = __fsub_rn(hi[a], lo[a]);
        d2 = a == 0 ? __fmul_rn(e, e) : __fadd_rn(d2, __fmul_rn(e, e));
    }
    rad = __fmul_rn(__fsqrt_rn(d2), 0.5f);
}

// Upper bound of d2_rn(q, p) over every p inside [lo, hi], rounded as d2_rn is.
__device__ __forceinline__ float box_ub(float qx, float qy, float qz, const float* lo, const float* hi) {
    const float gx = fmaxf(fabsf(__fsub_rn(lo[0], qx)), fabsf(__fsub_rn(hi[0], qx)));
    const float gy = fmaxf(fabsf(__fsub_rn(lo[1], qy)), fabsf(__fsub_rn(hi[1], qy)));
    const float gz = fmaxf(fabsf(__fsub_rn(lo[2], qz)), fabsf(__fsub_rn(hi[2], qz)));
    return __fadd_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)), __fmul_rn(gz, gz));
}

// Warp-wide visit of every photon with d^2 < r2.  whole(pass, lb, ub, cnt),
// called with one leaf per lane, may take a passing leaf as a whole (true);
// each(in, t, d2) is called by all lanes with one photon per lane, `in` where
// it is one in range (tree position t).  Returns false on stack overflow.
// Leaves are listed first and their photons loaded four half leaves at a time:
// one leaf after the other the walks waited for their loads (3.81 -> 3.37 ms).
template <class Whole, class Each>
__device__ __forceinline__ bool warp_range(const MapView& m, float qx, float qy, float qz, float r2, CompatSmem& s,
                                           uint32_t lane, Whole&& whole, Each&& each) {
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t sp = 0, nu = 0;
    // the start slot as a node of one child
    const ChildSlot* first = m.wroot;
    uint32_t kids = 1;
    for (bool more = true; more;) {
#pragma unroll 1
        do {
            float lo[3], hi[3], lb = INFINITY;
            uint32_t ref = kInvalid, cnt = 0;
            if (lane < kids) {
                const float4* p = reinterpret_cast<const float4*>(first + lane);
                const float4 a = __ldg(p), b = __ldg(p + 1);
                lo[0] = a.x; lo[1] = a.y; lo[2] = a.z; hi[0] = a.w;
                hi[1] = b.x; hi[2] = b.y; ref = __float_as_uint(b.z); cnt = __float_as_uint(b.w);
                lb = box_lb(qx, qy, qz, lo, hi);
            }
            const bool pass = ref != kInvalid && lb < r2;
            const bool wide = pass && (cnt & kWideFlag);
            const bool leaf = pass && !wide && !whole(lb, box_ub(qx, qy, qz, lo, hi), cnt);
            const uint32_t intm = __ballot_sync(kFull, wide), leafm = __ballot_sync(kFull, leaf),
                           bigm = __ballot_sync(kFull, leaf && cnt > 32u);
            if (sp + __popc(intm) > kCompatStack) { __syncwarp(); return false; }
            if (wide) s.stack[sp + __popc(intm & lt)] = make_uint2(ref, cnt & kWideCount);
            if (leaf) {   // leaves hold up to 64 photons
                s.units[nu + __popc(leafm & lt)] = make_uint2(ref, min(cnt, 32u));
                if (cnt > 32u) s.units[nu + __popc(leafm) + __popc(bigm & lt)] = make_uint2(ref + 32u, cnt - 32u);
            }
            sp += __popc(intm);
            nu += __popc(leafm) + __popc(bigm);
            __syncwarp();
            more = sp > 0;
            if (more) {
                const uint2 e = s.stack[--sp];
                first = m.wchild + e.x;
                kids = e.y;
            }
            __syncwarp();   // read before a push reuses the entry
        } while (more && nu <= kCompatUnits - 64u);
#pragma unroll 1
        for (uint32_t u = 0; u < nu; u += 4) {
            float4 p[4];
            uint2 e[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                e[i] = u + i < nu ? s.units[u + i] : make_uint2(0u, 0u);
                p[i] = lane < e[i].y ? __ldg(m.pos + e[i].x + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float d2 = d2_rn(qx, qy, qz, p[i].x, p[i].y, p[i].z);
                each(lane < e[i].y && d2 < r2, e[i].x + lane, d2);
            }
        }
        nu = 0;
        __syncwarp();
    }
    return true;
}

// Zhou et al. 2008 histogram refinement of a query radius, by a warp.
__device__ float refine_radius(const MapView& m, float qx, float qy, float qz, float radius_max, uint32_t k,
                               uint32_t iters, CompatSmem& s, uint32_t lane, bool& ok) {
    float r_min = 0.0f, r_max = radius_max;
    // A photon without a finite position is in range of nothing, and a leaf's box
    // need not show it (the minima of a box drop a NaN): such a map's photons are
    // tested one by one.
    const bool one_by_one = m.hdr->nonfinite != 0;
    for (uint32_t it = 0; it < iters; ++it) {
        const float r = r_max, lo = r_min;
        const float delta = __fsub_rn(r_max, r_min);
        if (!(delta > 0.0f)) break;
        s.hist[lane] = 0;
        __syncwarp();
        auto bin = [&](float d2) {   // monotone in d^2
            const float fi = __fdiv_rn(__fmul_rn(fmaxf(__fsub_rn(__fsqrt_rn(d2), lo), 0.0f), (float)kHist), delta);
            return min((uint32_t)fi, kHist - 1u);
        };
        const float r2 = __fmul_rn(r, r);
        ok = warp_range(m, qx, qy, qz, r2, s, lane,
                        [&](float lb, float ub, uint32_t cnt) {
                            if (one_by_one || !(ub < r2)) return false;
                            const uint32_t b = bin(lb);
                            if (b != bin(ub)) return false;
                            atomicAdd(&s.hist[b], cnt);
                            return true;
                        },
                        [&](bool in, uint32_t, float d2) {
                            if (in) atomicAdd(&s.hist[bin(d2)], 1u);
                        }) && ok;
        uint32_t sum = min(s.hist[lane], 0xfffeu);   // the reference's counters saturate
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, sum, o);
            if (lane >= (uint32_t)o) sum += y;
        }
        const uint32_t reach = __ballot_sync(kFull, sum >= k);
        const uint32_t mb = reach ? (uint32_t)__ffs(reach) - 1u : kHist - 1u;
        const float inv = 1.0f / (float)kHist;
        r_min = __fadd_rn(lo, __fmul_rn(__fmul_rn((float)mb, delta), inv));
        r_max = __fadd_rn(lo, __fmul_rn(__fmul_rn((float)(mb + 1), delta), inv));
        __syncwarp();
    }
    return r_max;
}

// One warp per slot, taken from a counter (a slot in a dense blob walks a
// hundred nodes more than one beside it); the slot count comes from the map
// header (2 per internal node plus the super-root's two).
__global__ void __launch_bounds__(32 * kCompatWarps) k_compat_nodes(MapView m, uint32_t max_slots, float rmax, uint32_t k,
                                                                    uint32_t iters, float* est, uint32_t* next) {
    __shared__ CompatSmem s_warp[kCompatWarps];
    const uint32_t lane = lane_id();
    CompatSmem& s = s_warp[threadIdx.x >> 5];
    const uint32_t internal = m.hdr->num_nodes;
    const uint32_t nslots = min(2u * (internal + 1u), max_slots);
    const bool enabled = 2 * internal + 1 >= 1000;   // node estimates are skipped for small trees
    for (;;) {
        uint32_t sid = 0;
        if (lane == 0) sid = atomicAdd(next, 1u);
        sid = __shfl_sync(kFull, sid, 0);
        if (sid >= nslots) break;
        float e = INFINITY;
        float lo[3], hi[3];
        uint32_t ref, cnt;
        slot_of(m.nodes, sid, lo, hi, ref, cnt);
        if (enabled && ref != kInvalid) {
            float c[3], rad;
            extent_of(lo, hi, c, rad);
            if (rad <= __fmul_rn(0.5f, rmax)) {
                bool ok = true;
                e = refine_radius(m, c[0], c[1], c[2], rmax, k, iters, s, lane, ok);
                if (!ok && lane == 0) atomicOr(&m.hdr->errors, kErrStack);
            }
        }
        if (lane == 0) est[sid] = e;
    }
}

// The radius a query starts from (one lane's descent).
__device__ float path_radius(const Node* nodes, const float* est, float qx, float qy, float qz, float rmax) {
    float e = rmax;
    uint32_t sid = 0;
    float lo[3], hi[3];
    uint32_t ref, cnt;
    slot_of(nodes, 0, lo, hi, ref, cnt);
    for (int depth = 0; depth < 4096; ++depth) {
        if (ref == kInvalid) break;
        float c[3], rad;
        extent_of(lo, hi, c, rad);
        const float len = __fsqrt_rn(d2_rn(qx, qy, qz, c[0], c[1], c[2]));
        e = fminf(e, __fadd_rn(len, est[sid]));
        if (cnt > 0) break;
        float l1[3], h1[3];
        uint32_t r1, c1;
        const uint32_t kid = ref << 1;
        slot_of(nodes, kid, lo, hi, ref, cnt);
        slot_of(nodes, kid | 1u, l1, h1, r1, c1);
        const float b0 = ref == kInvalid ? INFINITY : box_lb(qx, qy, qz, lo, hi);
        const float b1 = r1 == kInvalid ? INFINITY : box_lb(qx, qy, qz, l1, h1);
        sid = kid;
        if (b1 < b0) {
            ++sid;
            ref = r1; cnt = c1;
            for (int a = 0; a < 3; ++a) { lo[a] = l1[a]; hi[a] = h1[a]; }
        }
    }
    return e;
}

struct CompatArgs {
    MapView m;
    const float* est;
    const float4* qpos;
    const float4* qnrm;
    uint32_t nq, k, iters, min_found;
    uint32_t per_warp;   // queries a warp takes, 1 to 32
    float rmax;
    int filter;
    float cone_k;
    float* out_radius;   // pm_compute_query_radii
    float4* out_rad;     // gather
    float* out_r2;
    uint32_t* out_count;
};

__global__ void __launch_bounds__(32 * kCompatWarps, 4) k_compat_query(CompatArgs a) {
    __shared__ CompatSmem s_warp[kCompatWarps];
    const uint32_t lane = lane_id(), lt = (1u << lane) - 1u;
    CompatSmem& s = s_warp[threadIdx.x >> 5];
    const uint64_t q0 = (uint64_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * a.per_warp;
    if (q0 >= a.nq) return;
    const uint32_t nw = (uint32_t)min((uint64_t)a.per_warp, (uint64_t)a.nq - q0);
    float4 qp = make_float4(0.f, 0.f, 0.f, 0.f);
    float e0 = a.rmax;
    bool fin = false;
    if (lane < nw) {   // a query per lane: its start radius
        qp = a.qpos[q0 + lane];
        fin = isfinite(qp.x) && isfinite(qp.y) && isfinite(qp.z);
        if (fin) e0 = path_radius(a.m.nodes, a.est, qp.x, qp.y, qp.z, a.rmax);
        else atomicOr(&a.m.hdr->errors, kErrQueryNonFinite);
    }
    bool ok = true;
    for (uint32_t i = 0; i < nw; ++i) {
        const uint32_t q = (uint32_t)q0 + i;
        const float qx = __shfl_sync(kFull, qp.x, i), qy = __shfl_sync(kFull, qp.y, i), qz = __shfl_sync(kFull, qp.z, i);
        const bool finite = __shfl_sync(kFull, fin ? 1 : 0, i);
        float r = __shfl_sync(kFull, e0, i);
        if (finite) r = refine_radius(a.m, qx, qy, qz, r, a.k, a.iters, s, lane, ok);
        if (a.out_radius && lane == 0) a.out_radius[q] = r;
        if (!a.out_rad) continue;
        const float r2 = __fmul_rn(r, r);
        uint32_t count = 0;   // photons in range; the first kCompatKeep are kept
        float maxd2 = 0.0f;
        auto none = [](float, float, uint32_t) { return false; };
        if (finite) {
            ok = warp_range(a.m, qx, qy, qz, r2, s, lane, none,
                            [&](bool in, uint32_t t, float d2) {
                                const uint32_t bal = __ballot_sync(kFull, in);
                                const uint32_t at = count + __popc(bal & lt);
                                if (in) {
                                    maxd2 = fmaxf(maxd2, d2);
                                    if (at < kCompatKeep) s.keep[at] = t;
                                }
                                count += __popc(bal);
                            }) && ok;
            maxd2 = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(maxd2)));
        }
        const float r2u = count >= a.k ? maxd2 : r2;
        float4 rad = make_float4(0.0f, 0.0f, 0.0f, (float)count);
        if (finite && count > 0 && count >= a.min_found && r2u > 0.0f) {
            const float4 qn = a.qnrm[q];
            const double r2d = (double)r2u;
            const double kc = (double)a.cone_k;
            // 2^40 / max flux: a range may hold far more than 128 photons
            const float scale = __fmul_rn(a.m.hdr->fix_scale, 1.220703125e-4f);
            long long c0 = 0, c1 = 0, c2 = 0;
            auto add = [&](uint32_t t) {
                const float4 w = __ldg(a.m.pow + t);
                if (!front_rn(qn.x, qn.y, qn.z, __float_as_uint(w.w))) return;
                const float4 p = __ldg(a.m.pos + t);
                const double dx = (double)p.x - (double)qx, dy = (double)p.y - (double)qy, dz = (double)p.z - (double)qz;
                const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                double wt = 1.0;
                if (a.filter == 1) wt = 1.0 - __dsqrt_rn(d2) / (kc * __dsqrt_rn(r2d));
                else if (a.filter == 2) wt = 1.0 - d2 / r2d;
                c0 += __double2ll_rn(wt * (double)w.x * (double)scale);
                c1 += __double2ll_rn(wt * (double)w.y * (double)scale);
                c2 += __double2ll_rn(wt * (double)w.z * (double)scale);
            };
            if (count <= kCompatKeep) {
                for (uint32_t e = lane; e < count; e += 32) add(s.keep[e]);
            } else {
                warp_range(a.m, qx, qy, qz, r2, s, lane, none, [&](bool in, uint32_t t, float) {
                    if (in) add(t);
                });
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                c0 += __shfl_xor_sync(kFull, c0, o);
                c1 += __shfl_xor_sync(kFull, c1, o);
                c2 += __shfl_xor_sync(kFull, c2, o);
            }
            if (scale > 0.0f) {
                const double pi = 3.14159265358979323846;
                double norm = 1.0 / (pi * r2d);
                if (a.filter == 1) norm = 1.0 / ((1.0 - 2.0 / (3.0 * kc)) * pi * r2d);
                else if (a.filter == 2) norm = 2.0 / (pi * r2d);
                const double f = norm / (double)scale;
                rad.x = __double2float_rn((double)c0 * f);
                rad.y = __double2float_rn((double)c1 * f);
                rad.z = __double2float_rn((double)c2 * f);
            }
        }
        if (lane == 0) {
            a.out_rad[q] = rad;
            if (a.out_r2) a.out_r2[q] = r2u;
            if (a.out_count) a.out_count[q] = count;
        }
        __syncwarp();   // keep is reused
    }
    if (!ok && lane == 0) atomicOr(&a.m.hdr->errors, kErrStack);
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

// est holds max_slots floats, max_slots >= 2 * (internal nodes + 1), and one word more.
int compat_node_estimates(const MapView& m, uint32_t max_slots, float rmax, uint32_t k, uint32_t iters, float* est,
                          cudaStream_t st) {
    const uint32_t need = (max_slots + kCompatWarps - 1) / kCompatWarps, most = (uint32_t)sm_count() * 4u;
    uint32_t* next = reinterpret_cast<uint32_t*>(est + max_slots);
    cudaMemsetAsync(next, 0, sizeof(uint32_t), st);
    k_compat_nodes<<<need < most ? need : most, 32 * kCompatWarps, 0, st>>>(m, max_slots, rmax, k, iters, est, next);
    return 1;
}

int compat_query(const MapView& m, const float* est, const QueryParams& p, uint32_t iters, const float4* qpos,
                 const float4* qnrm, uint32_t nq, float* out_radius, const QueryOutputs& out, cudaStream_t st) {
    if (!nq) return 0;
    CompatArgs a;
    a.m = m; a.est = est;
    a.qpos = qpos; a.qnrm = qnrm; a.nq = nq; a.k = p.k; a.iters = iters; a.min_found = p.min_found;
    a.rmax = p.r; a.filter = p.filter; a.cone_k = p.cone_k;
    a.out_radius = out_radius; a.out_rad = out.rad; a.out_r2 = out.r2; a.out_count = out.count;
    // as many queries per warp as leave about four waves of warps (56 per SM)
    const uint32_t warps = 4u * 56u * (uint32_t)sm_count();
    a.per_warp = 1;
    while (a.per_warp < 32 && nq / (a.per_warp * 2u) >= warps) a.per_warp *= 2u;
    const uint32_t per_block = a.per_warp * kCompatWarps;
    k_compat_query<<<(nq + per_block - 1) / per_block, 32 * kCompatWarps, 0, st>>>(a);
    return 1;
}

}  // namespace pm
