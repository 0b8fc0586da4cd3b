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
// not one per photon.  The root-to-leaf path of a query is a thread's.  With a
// thread per query and per slot throughout the kernels ran at the pace of the
// slots beside the blob: 300,001 photons (20 % in a caustic of sigma 0.01),
// 307,200 queries, k = 50, R = 0.1, build included: 54.7 -> 2.81 ms; 1,500 photons
// and 4,000 radii: 343 -> 78 us.  Latency bounds what is left (dependent node
// loads; a quarter of the warps' slots is taken).
//
// Ranges of no more than two leaves are the exception: a warp has 30 lanes too
// many for them, and where there are many queries a thread each answers more
// (k_compat_start).
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

// The histogram's bin of a squared distance in [lo, lo + delta]: monotone in d^2.
__device__ __forceinline__ uint32_t hist_bin(float d2, float lo, float delta) {
    const float fi = __fdiv_rn(__fmul_rn(fmaxf(__fsub_rn(__fsqrt_rn(d2), lo), 0.0f), (float)kHist), delta);
    return min((uint32_t)fi, kHist - 1u);
}
// Narrows [r_min, r_max] to bin mb.
__device__ __forceinline__ void narrow(float& r_min, float& r_max, float delta, uint32_t mb) {
    const float lo = r_min, inv = 1.0f / (float)kHist;
    r_min = __fadd_rn(lo, __fmul_rn(__fmul_rn((float)mb, delta), inv));
    r_max = __fadd_rn(lo, __fmul_rn(__fmul_rn((float)(mb + 1), delta), inv));
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
        const float lo = r_min, delta = __fsub_rn(r_max, r_min);
        if (!(delta > 0.0f)) break;
        s.hist[lane] = 0;
        __syncwarp();
        const float r2 = __fmul_rn(r_max, r_max);
        ok = warp_range(m, qx, qy, qz, r2, s, lane,
                        [&](float lb, float ub, uint32_t cnt) {
                            if (one_by_one || !(ub < r2)) return false;
                            const uint32_t b = hist_bin(lb, lo, delta);
                            if (b != hist_bin(ub, lo, delta)) return false;
                            atomicAdd(&s.hist[b], cnt);
                            return true;
                        },
                        [&](bool in, uint32_t, float d2) {
                            if (in) atomicAdd(&s.hist[hist_bin(d2, lo, delta)], 1u);
                        }) && ok;
        uint32_t sum = min(s.hist[lane], 0xfffeu);   // the reference's counters saturate
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, sum, o);
            if (lane >= (uint32_t)o) sum += y;
        }
        const uint32_t reach = __ballot_sync(kFull, sum >= k);
        narrow(r_min, r_max, delta, reach ? (uint32_t)__ffs(reach) - 1u : kHist - 1u);
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

// The radius a query starts from (a thread's descent), and the radius of the box
// the descent ends in.
__device__ float path_radius(const Node* nodes, const float* est, float qx, float qy, float qz, float rmax,
                             float& leaf_rad) {
    float e = rmax;
    leaf_rad = 0.0f;
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
        leaf_rad = rad;
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

struct CompatArgs {   // out_rad and what goes with it, or out_radius alone
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

// The scaled integer sums of one estimate: their order does not matter.
struct CompatFlux {
    double qx, qy, qz, r2, kc;
    float scale;   // 2^40 / max flux: a range may hold far more than 128 photons
    float4 qn;
    long long c0 = 0, c1 = 0, c2 = 0;
    __device__ __forceinline__ void begin(const CompatArgs& a, float x, float y, float z, const float4& n, float r2u) {
        qx = x; qy = y; qz = z; r2 = r2u; kc = a.cone_k; qn = n;
        scale = __fmul_rn(a.m.hdr->fix_scale, 1.220703125e-4f);
    }
    __device__ __forceinline__ void add(const CompatArgs& a, uint32_t t) {
        const float4 w = __ldg(a.m.pow + t);
        if (!front_rn(qn.x, qn.y, qn.z, __float_as_uint(w.w))) return;
        const float4 p = __ldg(a.m.pos + t);
        const double dx = (double)p.x - qx, dy = (double)p.y - qy, dz = (double)p.z - qz;
        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        double wt = 1.0;
        if (a.filter == 1) wt = 1.0 - __dsqrt_rn(d2) / (kc * __dsqrt_rn(r2));
        else if (a.filter == 2) wt = 1.0 - d2 / r2;
        c0 += __double2ll_rn(wt * (double)w.x * (double)scale);
        c1 += __double2ll_rn(wt * (double)w.y * (double)scale);
        c2 += __double2ll_rn(wt * (double)w.z * (double)scale);
    }
    __device__ __forceinline__ void result(const CompatArgs& a, float4& rad) const {
        if (!(scale > 0.0f)) return;
        const double pi = 3.14159265358979323846;
        double norm = 1.0 / (pi * r2);
        if (a.filter == 1) norm = 1.0 / ((1.0 - 2.0 / (3.0 * kc)) * pi * r2);
        else if (a.filter == 2) norm = 2.0 / (pi * r2);
        const double f = norm / (double)scale;
        rad.x = __double2float_rn((double)c0 * f);
        rad.y = __double2float_rn((double)c1 * f);
        rad.z = __double2float_rn((double)c2 * f);
    }
};

__device__ __forceinline__ void compat_store(const CompatArgs& a, uint32_t q, float r, const float4& rad, float r2u,
                                             uint32_t count) {
    if (a.out_radius) a.out_radius[q] = r;
    if (!a.out_rad) return;
    a.out_rad[q] = rad;
    if (a.out_r2) a.out_r2[q] = r2u;
    if (a.out_count) a.out_count[q] = count;
}

// A query that k_compat_start leaves to its warp: its start radius r > 0 waits where
// its result will be.
__device__ __forceinline__ void compat_defer(const CompatArgs& a, uint32_t q, float r) {
    if (a.out_rad) a.out_rad[q] = make_float4(r, 0.0f, 0.0f, -1.0f);
    else a.out_radius[q] = -r;
}
__device__ __forceinline__ bool compat_deferred(const CompatArgs& a, uint32_t q, float& r) {
    if (a.out_rad) {
        const float4 v = a.out_rad[q];
        r = v.x;
        return v.w < 0.0f;
    }
    r = -a.out_radius[q];
    return r > 0.0f;
}

// Leaves a thread lists for its own range, and their photons at most (a bit each).
constexpr uint32_t kOwnLeaves = 2, kOwnPhotons = 64, kOwnStack = 24, kOwnSteps = 64;
constexpr int kOwnThreads = 128;
// Queries from which threads answer first: below, a launch's warps are not all taken,
// and a warp answers one query sooner (maps of no more than a leaf: 20,000 queries,
// 64 photons, R = 0.1, a warp each 23 us, a thread each 11).
constexpr uint32_t kOwnMin = 65536, kOwnMinFew = 16384;

// A query's position and start radius; false where it is answered (a position that
// is not finite, a radius of zero).
__device__ __forceinline__ bool compat_begin(const CompatArgs& a, uint32_t q, float4& qp, float& r0, float& leaf_rad) {
    qp = a.qpos[q];
    r0 = a.rmax;
    const bool fin = isfinite(qp.x) && isfinite(qp.y) && isfinite(qp.z);
    if (fin) r0 = path_radius(a.m.nodes, a.est, qp.x, qp.y, qp.z, a.rmax, leaf_rad);
    else atomicOr(&a.m.hdr->errors, kErrQueryNonFinite);
    if (fin && r0 > 0.0f) return true;
    compat_store(a, q, r0, make_float4(0.0f, 0.0f, 0.0f, 0.0f), __fmul_rn(r0, r0), 0u);
    return false;
}

// Thread per query: the start radius, and the whole answer where the range is a
// leaf or two (start radius a quarter of the query's own leaf's, or a map of no more
// than a leaf): the leaves are listed by one descent, as every later radius is
// smaller, and their photons tested in place.  The other queries are left to
// k_compat_query.  1M queries, a warp for each / this, us: 64 photons, R = 0.1 512 / 70;
// 1,500 photons, R = 0.02 672 / 180; 20,000 photons, R = 0.003 795 / 291.  Ranges of
// more photons are slower by a thread's chain of tests (500 queries, 100,000 photons,
// R = 0.02, up to 160 photons: 17 / 130 us), so few queries take a warp each.
__global__ void __launch_bounds__(kOwnThreads) k_compat_start(CompatArgs a) {
    __shared__ uint32_t s_hist[kHist / 4][kOwnThreads];   // byte counters, a column per thread
    const uint64_t q64 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q64 >= a.nq) return;
    const uint32_t q = (uint32_t)q64, me = threadIdx.x;
    float4 qp;
    float r0, leaf_rad;
    if (!compat_begin(a, q, qp, r0, leaf_rad)) return;
    uint32_t ref[kOwnLeaves], cnt[kOwnLeaves], leaves = 0, photons = 0;
    bool own = a.m.n <= kLeafMax || 4.0f * r0 <= leaf_rad;
    if (a.m.n <= kLeafMax) {
        ref[0] = 0;
        cnt[0] = a.m.n;
        leaves = 1;
    } else if (own) {
        const float r2 = __fmul_rn(r0, r0);
        uint32_t stack[kOwnStack], sp = 1, steps = 0;
        stack[0] = 0u;
        while (sp > 0 && own) {
            float lo[3], hi[3];
            uint32_t kid, c;
            slot_of(a.m.nodes, stack[--sp], lo, hi, kid, c);
            if (kid != kInvalid && box_lb(qp.x, qp.y, qp.z, lo, hi) < r2) {
                if (c > 0) {
                    photons += c;
                    own = leaves < kOwnLeaves && photons <= kOwnPhotons;
                    if (own) { ref[leaves] = kid; cnt[leaves] = c; ++leaves; }
                } else {
                    own = sp + 2 <= kOwnStack;
                    if (own) { stack[sp++] = kid << 1 | 1u; stack[sp++] = kid << 1; }
                }
            }
            own = own && ++steps < kOwnSteps;
        }
    }
    if (!own) {
        compat_defer(a, q, r0);
        return;
    }
    auto each = [&](float r2, auto&& f) {   // the listed photons with d^2 < r2, four loads in flight
        uint32_t first = 0;
#pragma unroll 1
        for (uint32_t l = 0; l < leaves; ++l) {
#pragma unroll 1
            for (uint32_t j = 0; j < cnt[l]; j += 4) {
                float4 p[4];
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) p[u] = __ldg(a.m.pos + ref[l] + min(j + u, cnt[l] - 1u));
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const float d2 = d2_rn(qp.x, qp.y, qp.z, p[u].x, p[u].y, p[u].z);
                    if (j + u < cnt[l] && d2 < r2) f(first + j + u, d2);
                }
            }
            first += cnt[l];
        }
    };
    float r_min = 0.0f, r_max = r0;
    for (uint32_t it = 0; it < a.iters; ++it) {
        const float lo = r_min, delta = __fsub_rn(r_max, r_min);
        if (!(delta > 0.0f)) break;
        for (uint32_t b = 0; b < kHist / 4; ++b) s_hist[b][me] = 0;
        each(__fmul_rn(r_max, r_max), [&](uint32_t, float d2) {
            const uint32_t b = hist_bin(d2, lo, delta);
            s_hist[b >> 2][me] += 1u << ((b & 3u) * 8u);
        });
        uint32_t mb = 0, sum = 0;
        for (; mb < kHist - 1u; ++mb) {
            sum += (s_hist[mb >> 2][me] >> ((mb & 3u) * 8u)) & 255u;
            if (sum >= a.k) break;
        }
        narrow(r_min, r_max, delta, mb);
    }
    if (!a.out_rad) {
        a.out_radius[q] = r_max;
        return;
    }
    const float r2 = __fmul_rn(r_max, r_max);
    uint64_t found = 0;   // a bit per listed photon
    float maxd2 = 0.0f;
    each(r2, [&](uint32_t i, float d2) { found |= 1ull << i; maxd2 = fmaxf(maxd2, d2); });
    const uint32_t count = (uint32_t)__popcll(found);
    const float r2u = count >= a.k ? maxd2 : r2;
    float4 rad = make_float4(0.0f, 0.0f, 0.0f, (float)count);
    if (count > 0 && count >= a.min_found && r2u > 0.0f) {
        CompatFlux flux;
        flux.begin(a, qp.x, qp.y, qp.z, a.qnrm[q], r2u);
#pragma unroll 1
        for (; found; found &= found - 1) {
            const uint32_t i = (uint32_t)__ffsll((long long)found) - 1u;
            flux.add(a, i < cnt[0] ? ref[0] + i : ref[1] + (i - cnt[0]));
        }
        flux.result(a, rad);
    }
    compat_store(a, q, r_max, rad, r2u, count);
}

// A warp per query, per_warp queries after one another: those that k_compat_start
// left (kStarted), or all of them, each lane descending for one first.
template <bool kStarted>
__global__ void __launch_bounds__(32 * kCompatWarps, 4) k_compat_query(CompatArgs a) {
    __shared__ CompatSmem s_warp[kCompatWarps];
    const uint32_t lane = lane_id(), lt = (1u << lane) - 1u;
    CompatSmem& s = s_warp[threadIdx.x >> 5];
    const uint64_t q0 = (uint64_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * a.per_warp;
    if (q0 >= a.nq) return;
    const uint32_t nw = (uint32_t)min((uint64_t)a.per_warp, (uint64_t)a.nq - q0);
    float4 qp = make_float4(0.f, 0.f, 0.f, 0.f);
    float e0 = 0.0f;
    bool mine = false;
    if (lane < nw) {
        if constexpr (kStarted) {
            mine = compat_deferred(a, (uint32_t)q0 + lane, e0);
            if (mine) qp = a.qpos[q0 + lane];
        } else {
            float leaf_rad;
            mine = compat_begin(a, (uint32_t)q0 + lane, qp, e0, leaf_rad);
        }
    }
    uint32_t todo = __ballot_sync(kFull, mine);
    bool ok = true;
    for (; todo; todo &= todo - 1u) {
        const int i = __ffs(todo) - 1;
        const uint32_t q = (uint32_t)q0 + (uint32_t)i;
        const float qx = __shfl_sync(kFull, qp.x, i), qy = __shfl_sync(kFull, qp.y, i), qz = __shfl_sync(kFull, qp.z, i);
        const float r = refine_radius(a.m, qx, qy, qz, __shfl_sync(kFull, e0, i), a.k, a.iters, s, lane, ok);
        if (!a.out_rad) {
            if (lane == 0) a.out_radius[q] = r;
            continue;
        }
        const float r2 = __fmul_rn(r, r);
        uint32_t count = 0;   // photons in range; the first kCompatKeep are kept
        float maxd2 = 0.0f;
        auto none = [](float, float, uint32_t) { return false; };
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
        const float r2u = count >= a.k ? maxd2 : r2;
        float4 rad = make_float4(0.0f, 0.0f, 0.0f, (float)count);
        if (count > 0 && count >= a.min_found && r2u > 0.0f) {
            CompatFlux flux;
            flux.begin(a, qx, qy, qz, a.qnrm[q], r2u);
            if (count <= kCompatKeep) {
                for (uint32_t e = lane; e < count; e += 32) flux.add(a, s.keep[e]);
            } else {
                warp_range(a.m, qx, qy, qz, r2, s, lane, none, [&](bool in, uint32_t t, float) {
                    if (in) flux.add(a, t);
                });
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                flux.c0 += __shfl_xor_sync(kFull, flux.c0, o);
                flux.c1 += __shfl_xor_sync(kFull, flux.c1, o);
                flux.c2 += __shfl_xor_sync(kFull, flux.c2, o);
            }
            flux.result(a, rad);
        }
        if (lane == 0) compat_store(a, q, r, rad, r2u, count);
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
    // as many queries per warp as leave about seven waves of the 32 warps that shared
    // memory lets an SM hold
    const uint32_t warps = 7u * 32u * (uint32_t)sm_count();
    a.per_warp = 1;
    while (a.per_warp < 32 && nq / (a.per_warp * 2u) >= warps) a.per_warp *= 2u;
    const uint32_t per_block = a.per_warp * kCompatWarps;
    const uint32_t grid = (nq + per_block - 1) / per_block;
    if (nq < (m.n <= kLeafMax ? kOwnMinFew : kOwnMin)) {
        k_compat_query<false><<<grid, 32 * kCompatWarps, 0, st>>>(a);
        return 1;
    }
    k_compat_start<<<(nq + kOwnThreads - 1) / kOwnThreads, kOwnThreads, 0, st>>>(a);
    if (m.n <= kLeafMax) return 1;   // answered whole
    k_compat_query<true><<<grid, 32 * kCompatWarps, 0, st>>>(a);
    return 2;
}

}  // namespace pm
