// pm_knn_shared.cuh -- the exact-kNN estimate for dense query sets: eight
// consecutive queries of the processing order share one walk of the tree.
// Included by pm_query.cu.
//
// A warp-per-query search (k_knn_group<32, *, *, true>) is bound by
// instruction issue: of its 2,600 warp instructions per query (plain
// workload, k = 100) over half walk the tree and test leaves, and the
// selection and the flux sums pay for warp-wide reductions per query.  Where
// queries are dense against the photons (consecutive Hilbert neighbours lie
// much closer than their search radii), the photons within reach of eight
// neighbours are few more than those within reach of one.  So a warp takes
// eight queries, four lanes each:
//   1. every query's radius bound from the previous group's queries
//      (r_k(q) <= r_k(q') + |q - q'|), the box around the eight queries and
//      the largest bound B;
//   2. one walk of the 32-wide tree lists the leaves within B of the box, and
//      one pass over their photons (four loads in flight) stages those within
//      B of the box in shared memory: about 230 for k = 100;
//   3. a query's four lanes test the staged photons against its own bound:
//      a histogram of 64 buckets over [0, bound) (byte counters in a column
//      per lane, so no two lanes share a word) and a list of (bucket, photon);
//   4. the bucket of the k-th distance follows from the column sums; the list
//      entries below it are neighbours, those in it (two or three) are ranked
//      by their exact (d^2, caller index) keys;
//   5. the four lanes sum the filtered flux of a quarter of the neighbours
//      each; two shuffle steps finish the sums.
// The fixed-point sums do not depend on the order of the terms, so the bits
// are those of every other layout.
//
// A group whose photons do not fit is retried with half its queries.  Where
// the bounds are loose (a chunk's first query, a jump of the Hilbert curve) the
// same walk is tried around one query, at radii near the last neighbours', for
// one that holds k photons: the group then takes its bounds from it.  What this
// kernel cannot decide (queries apart by more than their radii, more ties in the
// boundary bucket than its row holds, a bound without a finite bucket scale)
// goes to the list of the fix pass, which searches any query.

constexpr uint32_t kShQ = 8;         // queries per group, 4 lanes each
constexpr uint32_t kShCand = 448;    // photons staged per group
constexpr uint32_t kShStack = 96;    // wide nodes waiting in the walk
constexpr uint32_t kShUnits = 192;   // half leaves (32 photons) listed by the walk
constexpr uint32_t kShTies = 16;     // boundary entries a query's neighbour row holds beyond k

// Shared memory of a warp: the staged photons (x, y, z and tree position, an
// array each), then one area that holds in turn the walk's stack and units,
// the histogram, and the neighbour rows with the ranked boundary entries.
// 9.3 KB at k = 100, so that 24 warps fit an SM.  Rows of (d^2, tree position)
// saved the estimate 12 instructions a neighbour but left 16 warps: 4.99
// against 4.23 ms on the plain workload.  Room for 512 photons in place of 448
// (22 warps): 3.22 against 3.12 ms.
__host__ __device__ inline uint32_t shared_row(uint32_t k) { return (k + kShTies + 1u) & ~1u; }
constexpr uint32_t kShCandBytes = kShCand * 4u * (uint32_t)sizeof(float);
constexpr uint32_t kShWalkBytes = (kShStack + kShUnits) * 8u;
constexpr uint32_t kShHistBytes = 16u * 32u * 4u;
inline int shared_smem_bytes_per_warp(uint32_t kmax) {
    const uint32_t rows = (kShQ * (shared_row(kmax) + kShTies) * (uint32_t)sizeof(uint16_t) + 15u) & ~15u;
    const uint32_t least = kShWalkBytes > kShHistBytes ? kShWalkBytes : kShHistBytes;
    return (int)(kShCandBytes + (rows > least ? rows : least));
}

// Two FP32 operations per instruction (sm_100), each rounded to nearest as the
// scalar ones are.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// A product that stays one: the assembler fuses mul.f32x2 into a following
// add.f32x2 (one ulp off d2_rn), so it is written as a sum with nz, -0 twice,
// which only the launch knows.
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b, uint64_t nz) { return fma2(a, b, nz); }

struct ShCand {   // the staged photons
    float* x;
    float* y;
    float* z;
    uint32_t* t;
    __device__ __forceinline__ void put(uint32_t i, const float4& p, uint32_t tree) const {
        x[i] = p.x; y[i] = p.y; z[i] = p.z; t[i] = tree;
    }
};

// Four staged photons' d2_rn to the query (nq: the negated position, twice)
// and their buckets: d^2 * 63 / bound rounded to nearest, 0 to 63 for a
// distance below the bound (the low bits of the sum with 2^23; monotone in
// d^2).
struct ShFour {
    float d[4];
    uint32_t b[4];
};
__device__ __forceinline__ void sh_four(const ShCand& c, uint32_t j, uint64_t nqx, uint64_t nqy, uint64_t nqz,
                                        uint64_t scale, uint64_t nz, ShFour& f) {
    const float4 X = *reinterpret_cast<const float4*>(c.x + j), Y = *reinterpret_cast<const float4*>(c.y + j),
                 Z = *reinterpret_cast<const float4*>(c.z + j);
    const uint64_t magic = pack2(8388608.0f, 8388608.0f);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint64_t dx = add2(h ? pack2(X.z, X.w) : pack2(X.x, X.y), nqx);
        const uint64_t dy = add2(h ? pack2(Y.z, Y.w) : pack2(Y.x, Y.y), nqy);
        const uint64_t dz = add2(h ? pack2(Z.z, Z.w) : pack2(Z.x, Z.y), nqz);
        const uint64_t d2 = add2(add2(mul2(dx, dx, nz), mul2(dy, dy, nz)), mul2(dz, dz, nz));
        float u, v;
        unpack2(d2, f.d[2 * h], f.d[2 * h + 1]);
        unpack2(fma2(d2, scale, magic), u, v);
        f.b[2 * h] = __float_as_uint(u);
        f.b[2 * h + 1] = __float_as_uint(v);
    }
}

// Lower bound of d2_rn(q, p) over q in [lo, hi] (p a point) or, with a box
// for p, over both: gaps per axis, squared and summed in d2_rn's order, so it
// never exceeds the FP32 distance of any pair.
__device__ __forceinline__ float gap2(float gx, float gy, float gz) {
    gx = fmaxf(gx, 0.0f); gy = fmaxf(gy, 0.0f); gz = fmaxf(gz, 0.0f);
    return __fadd_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)), __fmul_rn(gz, gz));
}

struct ShBox { float lx, ly, lz, hx, hy, hz, b2; };   // the group's box and largest bound (exclusive)

// Whether a photon may lie within the bound of the box: |x - c| - h per axis,
// with half-widths and bound widened far beyond the rounding of these steps
// and of d2_rn (2^-20 of every magnitude in them).  A photon too many is
// dropped by its exact distance later; none within the bound is missed.
struct ShNear {
    float cx, cy, cz, hx, hy, hz, b2;
    __device__ __forceinline__ explicit ShNear(const ShBox& b) {
        cx = 0.5f * (b.lx + b.hx); cy = 0.5f * (b.ly + b.hy); cz = 0.5f * (b.lz + b.hz);
        const float r = sqrtf(b.b2);
        hx = half_width(b.lx, b.hx, cx, r); hy = half_width(b.ly, b.hy, cy, r); hz = half_width(b.lz, b.hz, cz, r);
        b2 = b.b2 * 1.000002f;
    }
    static __device__ __forceinline__ float half_width(float lo, float hi, float c, float r) {
        const float h = fmaxf(hi - c, c - lo);
        return h + 9.5367431640625e-07f * (fabsf(c) + h + r);
    }
    __device__ __forceinline__ bool operator()(float x, float y, float z) const {
        const float gx = fmaxf(fabsf(x - cx) - hx, 0.0f), gy = fmaxf(fabsf(y - cy) - hy, 0.0f),
                    gz = fmaxf(fabsf(z - cz) - hz, 0.0f);
        return gx * gx + gy * gy + gz * gz < b2;
    }
};
__device__ __forceinline__ float sh_slot_lb(const ShBox& b, const float* lo, const float* hi) {
    return gap2(fmaxf(__fsub_rn(b.lx, hi[0]), __fsub_rn(lo[0], b.hx)),
                fmaxf(__fsub_rn(b.ly, hi[1]), __fsub_rn(lo[1], b.hy)),
                fmaxf(__fsub_rn(b.lz, hi[2]), __fsub_rn(lo[2], b.hz)));
}

// One walk of the 32-wide tree, a child slot per lane: every leaf within the
// bound of the box goes to the unit list as half leaves, and the listed
// photons are staged.  The next node's slots load while this one's are tested.
// One copy of each step: the group's code has to stay small (a warp runs
// through all of it per group, and instruction fetches were its largest
// stall).  Returns false when the staged photons (or the stack) do not fit.
__device__ __forceinline__ bool sh_collect(const KnnArgs& a, const ShBox& box, const ShCand& cand, uint32_t& n, uint2* stack,
                                           uint2* units, uint32_t lane, uint32_t lt) {
    const ShNear near(box);
    uint32_t sp = 0, nu = 0;
    n = 0;
    const ChildSlot* next = a.root;   // the start slot, as a node of one child
    uint32_t kids = 1;
    float4 ca = make_float4(0.f, 0.f, 0.f, 0.f), cb = ca;
    if (lane < kids) {
        ca = __ldg(reinterpret_cast<const float4*>(next));
        cb = __ldg(reinterpret_cast<const float4*>(next) + 1);
    }
    bool more = true;
    while (more) {
#pragma unroll 1
        for (;;) {
            const float lo[3] = {ca.x, ca.y, ca.z}, hi[3] = {ca.w, cb.x, cb.y};
            const uint32_t ref = __float_as_uint(cb.z), cnt = __float_as_uint(cb.w);
            const bool pass = lane < kids && ref != kInvalid && sh_slot_lb(box, lo, hi) < box.b2;
            const bool is_wide = (cnt & kWideFlag) != 0;
            const uint32_t had = sp;
            // the stack's top is the next node, unless this one pushes: then any of its children
            const uint32_t intm = __ballot_sync(kFull, pass && is_wide);
            const uint32_t leafm = __ballot_sync(kFull, pass && !is_wide);
            const uint32_t bigm = __ballot_sync(kFull, pass && !is_wide && cnt > 32u);
            if (had + __popc(intm) > kShStack) return false;
            if (pass) {
                if (is_wide) {
                    stack[had + __popc(intm & lt)] = make_uint2(ref, cnt & kWideCount);
                } else {
                    units[nu + __popc(leafm & lt)] = make_uint2(ref, min(cnt, 32u));
                    if (cnt > 32u) units[nu + __popc(leafm) + __popc(bigm & lt)] = make_uint2(ref + 32u, cnt - 32u);
                }
            }
            sp = had + __popc(intm);
            nu += __popc(leafm) + __popc(bigm);
            __syncwarp();
            more = sp > 0;
            if (more) {
                const uint2 e = stack[--sp];
                kids = e.y;
                if (lane < kids) {
                    const float4* p = reinterpret_cast<const float4*>(a.wchild + e.x + lane);
                    ca = __ldg(p);
                    cb = __ldg(p + 1);
                }
                __syncwarp();   // read before a push reuses the entry
            }
            if (!more || nu > kShUnits - 64u) break;   // room for one more visit's half leaves
        }
        // the units' photons, four loads in flight
#pragma unroll 1
        for (uint32_t u = 0; u < nu; u += 4) {
            float4 p[4];
            uint32_t t[4];
            bool have[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint2 e = u + i < nu ? units[u + i] : make_uint2(0u, 0u);
                have[i] = lane < e.y;
                t[i] = e.x + lane;
                p[i] = have[i] ? __ldg(a.pos + t[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool in = have[i] && near(p[i].x, p[i].y, p[i].z);
                const uint32_t bal = __ballot_sync(kFull, in);
                const uint32_t c = __popc(bal);
                if (n + c > kShCand) return false;
                if (in) cand.put(n + __popc(bal & lt), p[i], t[i]);
                n += c;
            }
        }
        nu = 0;
        __syncwarp();
    }
    return true;
}

// Ascending bitonic sort of the 32 R keys of a warp (R = 1, 2 or 4), slot
// lane R + r in v[r] (the all-ascending form: the first step of a merge pairs a
// slot with its mirror in the block).  The steps across lanes are one loop.
__device__ __forceinline__ void sh_order(uint64_t& x, uint64_t& y) {
    const uint64_t lo = x < y ? x : y, hi = x < y ? y : x;
    x = lo;
    y = hi;
}
template <int R>
__device__ __forceinline__ void sh_merge_lane(uint64_t (&v)[R]) {
    if constexpr (R == 4) { sh_order(v[0], v[2]); sh_order(v[1], v[3]); sh_order(v[2], v[3]); }
    if constexpr (R >= 2) sh_order(v[0], v[1]);
}
template <int R>
__device__ __forceinline__ void sh_sort_keys(uint64_t (&v)[R], uint32_t lane) {
    if constexpr (R == 2) sh_order(v[0], v[1]);
    if constexpr (R == 4) {
        sh_order(v[0], v[1]); sh_order(v[2], v[3]);
        sh_order(v[0], v[3]); sh_order(v[1], v[2]);
        sh_order(v[0], v[1]); sh_order(v[2], v[3]);
    }
#pragma unroll 1
    for (int block = 2; block <= 32; block <<= 1) {   // lanes merged
#pragma unroll 1
        for (int j = block >> 1; j > 0; j >>= 1) {
            const bool flip = j == block >> 1;
            const int mask = flip ? block - 1 : j;
            const bool lower = (lane & (uint32_t)j) == 0;
            uint64_t w[R];
#pragma unroll
            for (int r = 0; r < R; ++r) w[r] = __shfl_xor_sync(kFull, flip ? v[R - 1 - r] : v[r], mask);
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = ((w[r] < v[r]) == lower) ? w[r] : v[r];
        }
        sh_merge_lane<R>(v);
    }
}

// The sorted neighbour row of one query (warp-wide): the exact keys of its n
// listed photons, sorted in registers.
template <int R>
__device__ __forceinline__ void sh_write_row(const KnnArgs& a, const ShCand& cand, const uint16_t* row, uint32_t n, float qx, float qy, float qz, uint32_t* out, uint32_t lane) {
    uint64_t v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t e = lane * R + r;
        v[r] = ~0ull;
        if (e < n) {
            const uint32_t j = row[e];
            v[r] = ((uint64_t)__float_as_uint(d2_rn(qx, qy, qz, cand.x[j], cand.y[j], cand.z[j])) << 32) | __float_as_uint(__ldg(&a.pos[cand.t[j]].w));
        }
    }
    sh_sort_keys<R>(v, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t e = lane * R + r;
        if (e < a.k) out[e] = e < n ? (uint32_t)v[r] - a.ph_off : kInvalid;
    }
}

// One neighbour's terms, est_add32w without branches: a photon that faces
// away adds zeros.  kBox: every weight is 1, and the unweighted sums are not
// needed (est_needs_fp64).
template <bool kBox>
__device__ __forceinline__ void sh_add(int filter, const float4& w, float d2, float inv, float nx, float ny, float nz,
                                       float scale, uint64_t neg_zero2, EstAcc& acc) {
    const bool f = front_rn(nx, ny, nz, __float_as_uint(w.w));
    const float x = f ? w.x : 0.0f, y = f ? w.y : 0.0f, z = f ? w.z : 0.0f;
    const uint64_t xy = pack2(x, y);
    float wt = 1.0f, cx, cy;
    if constexpr (!kBox) {
        // the filters' one form, 1 - u inv: u = d (cone) or d^2 (Epanechnikov)
        const float d = d2 > 0.0f ? __fmul_rn(d2, rsqrtf(d2)) : 0.0f;
        wt = fmaxf(__fsub_rn(1.0f, __fmul_rn(filter == 1 ? d : d2, inv)), 0.0f);
        const float s32 = __fmul_rn(scale, 1.862645149230957e-09f);   // 2^-29
        float fx, fy;
        unpack2(mul2(xy, pack2(s32, s32), neg_zero2), fx, fy);
        acc.f0 += __float2uint_ru(fabsf(fx));
        acc.f1 += __float2uint_ru(fabsf(fy));
        acc.f2 += __float2uint_ru(__fmul_rn(fabsf(z), s32));
        unpack2(mul2(mul2(pack2(wt, wt), xy, neg_zero2), pack2(scale, scale), neg_zero2), cx, cy);
    } else {
        unpack2(mul2(xy, pack2(scale, scale), neg_zero2), cx, cy);
    }
    acc.c0 += __float2ll_rn(cx);
    acc.c1 += __float2ll_rn(cy);
    acc.c2 += fixed_term(wt, z, scale);
}

template <bool kBatch, bool kNbr>
__global__ void __launch_bounds__(256, 3) k_knn_shared(KnnArgs a0) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t lane = lane_id();
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t qi = lane >> 2, sub = lane & 3u;   // this lane's query of the group, and its share
    const uint32_t q4 = lane & ~3u;                   // first lane of the query
    unsigned char* wb = smem + (size_t)warp * a0.smem_per_warp;
    ShCand cand;
    cand.x = reinterpret_cast<float*>(wb);
    cand.y = cand.x + kShCand;
    cand.z = cand.y + kShCand;
    cand.t = reinterpret_cast<uint32_t*>(cand.z + kShCand);
    unsigned char* area = wb + kShCandBytes;
    uint2* stack = reinterpret_cast<uint2*>(area);
    uint2* units = stack + kShStack;
    uint32_t* hist = reinterpret_cast<uint32_t*>(area);   // [16][32]: row b / 4, byte b % 4 of a lane's column
    uint16_t* rows = reinterpret_cast<uint16_t*>(area);   // [kShQ][row_len]: staged photons
    uint16_t* tmp = rows + kShQ * a0.cap;                 // [kShQ][kShTies]: the ranked boundary entries
    const uint32_t row_len = a0.cap;
    const uint32_t nq = a0.nq;
    const uint32_t total_rounds = (nq + kShQ - 1) / kShQ;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    float guess = INFINITY;   // radius^2 that the next search without a bound tries first

    for (;;) {
        uint32_t chunk = 0;
        if (lane == 0) chunk = atomicAdd(a0.work_counter, 1u);
        chunk = __shfl_sync(kFull, chunk, 0);
        uint32_t rbegin = 0, rlen = 0;
        if (!guided_chunk(chunk, total_rounds, nwarps, a0.rounds_per_chunk,
                          a0.rounds_max, rbegin, rlen))
            break;
        uint32_t at = rbegin * kShQ;
        const uint32_t end = min(at + rlen * kShQ, nq);
        // this lane's entry of the bounds' source: an earlier query and its r_k (negative: none)
        float pqx = 0.f, pqy = 0.f, pqz = 0.f, pr = -1.0f;
        uint32_t pmap = kInvalid;
        uint32_t want = kShQ;    // queries the next group tries
        bool search = true;      // find a bound for the next query first
        bool fresh = false;      // the last step did
        uint32_t tries = 0;      // radii that search has tried
        bool sparse = false;     // the last search found fewer than k within R: R is the bound here
        uint32_t walks = 0;      // walks since the chunk began
        const uint32_t begin = at;
        uint32_t defers = 0;     // queries left to the fix pass since the last search or group
        while (at < end) {
            uint32_t len = min(want, end - at);
            const uint32_t slot = at + qi;
            KnnArgs a = a0;
            if constexpr (kBatch) {   // a group lies within one map
                const uint32_t map = (uint32_t)(a0.qkeys[min(slot, nq - 1u)] >> kBatchQueryMapShift);
                const uint32_t m0 = __shfl_sync(kFull, map, 0);
                const uint32_t other = __ballot_sync(kFull, qi < len && map != m0);
                if (other) len = (uint32_t)(__ffs(other) - 1) >> 2;
                const BatchQuery bq = a0.bq[m0];
                a.k = bq.k; a.r2max = bq.r2max; a.rmax = bq.rmax; a.filter = bq.filter; a.cone_k = bq.cone_k;
                a.min_found = bq.min_found; a.nbr_off = bq.nbr_off; a.q_off = bq.q_off; a.ph_off = bq.ph_off;
                a.norm_c = bq.norm_c;
                a.scale_ptr = &a0.bgeom[m0].fix_scale;
                a.root = &a0.bgeom[m0].wroot;
                if (m0 != pmap) {   // bounds only carry over within one map
                    pmap = m0;
                    pr = -1.0f;
                    want = kShQ;
                    if (!search) { search = true; fresh = false; tries = 0; continue; }
                }
            }
            const uint32_t k = a.k;
            const float r2max = a.r2max;
            bool inq = qi < len;
            uint32_t qo = 0;
            float qx = 0.f, qy = 0.f, qz = 0.f, nx = 0.f, ny = 0.f, nz = 0.f;
            bool active = false;
            if (inq) {
                float4 q, nn;
                if (a.qsorted) {
                    q = a.qsorted[2 * (size_t)slot];
                    nn = a.qsorted[2 * (size_t)slot + 1];
                    qo = __float_as_uint(q.w);
                } else {
                    qo = a.order ? a.order[slot] : slot;
                    q = a.qpos[qo];
                    nn = a.qnrm[qo];
                }
                qx = q.x; qy = q.y; qz = q.z;
                nx = nn.x; ny = nn.y; nz = nn.z;
                active = isfinite(qx) && isfinite(qy) && isfinite(qz);
            }
            // the query's bound: its lanes take two earlier queries each
            float tau = r2max;
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int src = (int)((2u * sub + (uint32_t)h) << 2);
                const float sx = __shfl_sync(kFull, pqx, src), sy = __shfl_sync(kFull, pqy, src);
                const float sz = __shfl_sync(kFull, pqz, src), sr = __shfl_sync(kFull, pr, src);
                if (sr >= 0.0f) {
                    const float dq = __fsqrt_rn(d2_rn(qx, qy, qz, sx, sy, sz));
                    const float b = __fmul_rn(__fadd_rn(sr, dq), 1.000244140625f);
                    tau = fminf(tau, __fmul_rn(__fmul_rn(b, b), 1.000244140625f));
                }
            }
            tau = fminf(tau, __shfl_xor_sync(kFull, tau, 1));
            tau = fminf(tau, __shfl_xor_sync(kFull, tau, 2));
            const float tau0 = tau;
            bool bounded = tau < r2max;   // fewer than k below tau means a failed bound
            float prmax = pr;
#pragma unroll 1
            for (int o = 4; o < 32; o <<= 1) prmax = fmaxf(prmax, __shfl_xor_sync(kFull, prmax, o));
            if (!search) {
                // A jump of the curve (two queries apart by more than the radii) ends the
                // group before it, and asks for a search at its far side: the walk that
                // would not fit is not taken.
                const float px = __shfl_up_sync(kFull, qx, 4), py = __shfl_up_sync(kFull, qy, 4),
                            pz = __shfl_up_sync(kFull, qz, 4);
                const uint32_t jumps = __ballot_sync(kFull, inq && qi > 0 && d2_rn(qx, qy, qz, px, py, pz) > prmax * prmax);
                if (jumps) len = (uint32_t)(__ffs(jumps) - 1) >> 2;
                inq = qi < len;
                active = active && inq;
                const float t0 = __shfl_sync(kFull, active ? tau : 0.0f, 0);
                if (!fresh && !sparse && defers == 0 && !(prmax >= 0.0f && t0 <= 4.0f * prmax * prmax) && t0 > 0.0f) {
                    search = true;
                    __syncwarp();
                    continue;
                }
            }
            uint32_t nc = 0;              // staged photons
            __syncwarp();
            // A search takes the first query alone: a radius that holds k photons, but
            // not more than fit, bounds its k-th distance and so every neighbour's.
            const bool probe = search && __shfl_sync(kFull, active ? 1 : 0, 0);
            ShBox box;
            {
                const bool in = active && (!probe || qi == 0);
                box.lx = in ? qx : INFINITY; box.ly = in ? qy : INFINITY; box.lz = in ? qz : INFINITY;
                box.hx = in ? qx : -INFINITY; box.hy = in ? qy : -INFINITY; box.hz = in ? qz : -INFINITY;
                box.b2 = in ? tau : 0.0f;
#pragma unroll 1
                for (int o = 4; o < 32; o <<= 1) {
                    box.lx = fminf(box.lx, __shfl_xor_sync(kFull, box.lx, o));
                    box.ly = fminf(box.ly, __shfl_xor_sync(kFull, box.ly, o));
                    box.lz = fminf(box.lz, __shfl_xor_sync(kFull, box.lz, o));
                    box.hx = fmaxf(box.hx, __shfl_xor_sync(kFull, box.hx, o));
                    box.hy = fmaxf(box.hy, __shfl_xor_sync(kFull, box.hy, o));
                    box.hz = fmaxf(box.hz, __shfl_xor_sync(kFull, box.hz, o));
                    box.b2 = fmaxf(box.b2, __shfl_xor_sync(kFull, box.b2, o));
                }
            }
            if (probe) box.b2 = fminf(box.b2, guess);
            const bool any = __any_sync(kFull, active);
            // far queries against their bounds' source: a jump, or queries apart by more than their radii
            const bool loose = any && !(prmax >= 0.0f && box.b2 <= 4.0f * prmax * prmax);
            const bool skip = !probe && loose && defers > 0;   // nothing but a search would help
            // a blob denser than the queries: the fix pass takes the rest of a chunk whose
            // walks outnumber three per eight queries by eight
            ++walks;
            const bool spent = walks > 8u + ((3u * (at - begin)) >> 3);
            const bool fits = !any || (!skip && sh_collect(a, box, cand, nc, stack, units, lane, lt));
            __syncwarp();
            if (probe) {
                ++tries;
                const bool few = fits && nc < k && box.b2 < r2max;
                if ((!fits || few) && tries < 12u && !spent) {
                    guess = box.b2 * (few ? fminf(fmaxf(1.5f * (float)k / (float)(nc + 1u), 2.0f), 8.0f)
                                          : (tries < 3u ? 0.5f : 0.25f));
                    continue;
                }
                if (fits && nc >= k) {   // the bound takes the place of the oldest source
                    if (qi == kShQ - 1) {
                        pqx = box.lx; pqy = box.ly; pqz = box.lz;
                        const float r = __fsqrt_ru(box.b2);   // and the staging test's margins
                        pr = r * 1.00001f + 2e-6f * (fabsf(box.lx) + fabsf(box.ly) + fabsf(box.lz) + r);
                    }
                    guess = box.b2 * fmaxf(0.5f, 1.3f * (float)k / (float)nc);
                }
                sparse = fits && nc < k;
                search = false;
                fresh = true;
                tries = 0;
                if (defers == 0) want = kShQ;
                defers = defers ? 1u : 0u;
                continue;
            }
            if (!fits) {
                if (spent) {
                    for (uint32_t i = at + lane; i < end; i += 32) fix_push(a0, i, kBatch ? INFINITY : r2max);
                    break;
                }
                if (loose && !fresh && !sparse && (defers == 0 || defers >= 32) && __shfl_sync(kFull, active ? 1 : 0, 0)) {
                    search = true;
                } else if (len > 1 && !skip) {   // a wide group: half of it
                    want = len >> 1;
                } else {   // the fix pass takes the first query
                    if (lane == 0) fix_push(a, slot, tau);
                    ++defers;
                    ++at;
                    fresh = false;
                }
                continue;
            }
            search = false;
            // pad to whole steps of the candidate loops with photons at no distance
            const uint32_t nc16 = (nc + 15u) & ~15u;
            if (nc + lane < nc16) cand.x[nc + lane] = INFINITY;
            __syncwarp();   // staged photons visible; the walk's area becomes the histogram

            // ---- histogram of the query's candidates, and the k-th distance's bucket
            uint32_t total, B, below, nb;
            float scale_b, lim;
            bool full;
            const uint64_t nqx = pack2(-qx, -qx), nqy = pack2(-qy, -qy), nqz = pack2(-qz, -qz);
#pragma unroll 1
            for (int pass = 0;; ++pass) {
#pragma unroll
                for (int i = 0; i < 16; ++i) hist[i * 32 + lane] = 0u;
                scale_b = __fdiv_rn(63.0f, tau);
                lim = active ? tau : 0.0f;
                const uint64_t scale2 = pack2(scale_b, scale_b);
#pragma unroll 1
                for (uint32_t j = 4u * sub; j < nc16; j += 16) {
                    ShFour f;
                    sh_four(cand, j, nqx, nqy, nqz, scale2, a0.neg_zero2, f);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (f.d[i] < lim) atomicAdd(&hist[((f.b[i] & 60u) << 3) + lane], 1u << ((f.b[i] & 3u) * 8u));
                }
                __syncwarp();
                // lane `sub` sums rows [4 sub, 4 sub + 4) = buckets [16 sub, 16 sub + 16) over the query's
                // columns: even and odd bytes as 16-bit pairs
                uint32_t ev[4], od[4], rowsum[4], tot = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 w = *reinterpret_cast<const uint4*>(hist + (4u * sub + i) * 32u + q4);
                    ev[i] = (w.x & 0xff00ffu) + (w.y & 0xff00ffu) + (w.z & 0xff00ffu) + (w.w & 0xff00ffu);
                    od[i] = ((w.x >> 8) & 0xff00ffu) + ((w.y >> 8) & 0xff00ffu) + ((w.z >> 8) & 0xff00ffu) +
                            ((w.w >> 8) & 0xff00ffu);
                    const uint32_t t = ev[i] + od[i];
                    rowsum[i] = (t & 0xffffu) + (t >> 16);
                    tot += rowsum[i];
                }
                uint32_t before = 0;   // entries in lower lanes' buckets
                {
                    const uint32_t u1 = __shfl_up_sync(kFull, tot, 1, 4), u2 = __shfl_up_sync(kFull, tot, 2, 4),
                                   u3 = __shfl_up_sync(kFull, tot, 3, 4);
                    if (sub >= 1) before += u1;
                    if (sub >= 2) before += u2;
                    if (sub >= 3) before += u3;
                }
                total = __shfl_sync(kFull, before + tot, (int)(q4 + 3u));
                full = total >= k;
                const bool mine = full && before < k && k <= before + tot;
                uint32_t run = before, e = 0, o = 0, mb = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {   // the row that holds the k-th
                    const bool here = run < k && k <= run + rowsum[i];
                    if (here) { mb = 16u * sub + 4u * i; e = ev[i]; o = od[i]; before = run; }
                    run += rowsum[i];
                }
                // its bucket: counts in order are e.lo, o.lo, e.hi, o.hi
                const uint32_t c0 = e & 0xffffu, c1 = o & 0xffffu, c2 = e >> 16, c3 = o >> 16;
                uint32_t mbelow = before, mnb = c0;
                if (mbelow + mnb < k) { mbelow += c0; mnb = c1; ++mb; }
                if (mbelow + mnb < k) { mbelow += c1; mnb = c2; ++mb; }
                if (mbelow + mnb < k) { mbelow += c2; mnb = c3; ++mb; }
                const uint32_t who = __ballot_sync(kFull, mine) >> q4 & 15u;
                const int src = (int)(q4 + (who ? (uint32_t)__ffs(who) - 1u : 0u));
                const uint32_t m = __shfl_sync(kFull, mb | (mbelow << 8) | (mnb << 20), src);
                B = full ? m & 255u : 64u;
                below = full ? (m >> 8) & 4095u : total;
                nb = full ? m >> 20 : 0u;
                // a loose bound puts many entries in the k-th's bucket: cut the bound at its upper edge
                const bool again = active && full && nb > 12u && B < 32u && scale_b < INFINITY;
                if (pass == 3 || !__any_sync(kFull, again)) break;
                if (again) tau = __fmul_ru(__fdiv_ru((float)B + 0.5f, scale_b), 1.00001f);
                bounded = bounded || again;
                __syncwarp();
            }
            // ---- this lane's own entries below B and in B, and where they go in the query's row
            uint32_t pos_a = 0, pos_b = below;
            {
                const uint32_t rB = B >> 2, sh = (B & 3u) * 8u, mlo = ((1u << sh) - 1u) & 0x01010101u;
                uint32_t own_below = 0, own_nb = 0;
#pragma unroll
                for (uint32_t i = 0; i < 16; ++i) {
                    const uint32_t w = hist[i * 32 + lane];
                    own_below = __dp4a(w, i < rB ? 0x01010101u : (i == rB ? mlo : 0u), own_below);
                    if (i == rB) own_nb = (w >> sh) & 255u;
                }
                const uint32_t v = own_below | (own_nb << 16);
                const uint32_t u1 = __shfl_up_sync(kFull, v, 1, 4), u2 = __shfl_up_sync(kFull, v, 2, 4),
                               u3 = __shfl_up_sync(kFull, v, 3, 4);
                uint32_t s = 0;
                if (sub >= 1) s += u1;
                if (sub >= 2) s += u2;
                if (sub >= 3) s += u3;
                pos_a += s & 0xffffu;
                pos_b += s >> 16;
            }
            // not decided here: left to the fix pass
            const bool hard = active && (nb > kShTies || (bounded && !full) || !(scale_b < INFINITY));
            __syncwarp();   // the histogram area becomes the rows
            uint16_t* row = rows + qi * row_len;
            {
                const float take = hard ? 0.0f : lim;
                const uint64_t scale2 = pack2(scale_b, scale_b);
#pragma unroll 1
                for (uint32_t j = 4u * sub; j < nc16; j += 16) {
                    ShFour f;
                    sh_four(cand, j, nqx, nqy, nqz, scale2, a0.neg_zero2, f);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t b = f.b[i] & 63u;
                        const bool in = f.d[i] < take && b < B, at = f.d[i] < take && b == B;
                        if (in || at) row[in ? pos_a : pos_b] = (uint16_t)(j + i);
                        pos_a += in ? 1u : 0u;
                        pos_b += at ? 1u : 0u;
                    }
                }
            }
            __syncwarp();
            // ---- rank the boundary bucket's exact keys; the first k - below are neighbours
            const uint32_t need = full && !hard ? k - below : 0u;
            float kd2 = 0.0f;
            {
                const uint32_t nbx = hard ? 0u : nb;
                const uint16_t* bnd = row + below;
#pragma unroll 1
                for (uint32_t i = sub; i < nbx; i += 4) {
                    const uint32_t jp = bnd[i];
                    const uint2 p = make_uint2(__float_as_uint(d2_rn(qx, qy, qz, cand.x[jp], cand.y[jp], cand.z[jp])), cand.t[jp]);
                    uint32_t rank = 0;
#pragma unroll 1
                    for (uint32_t o = 0; o < nbx; ++o) {
                        const uint32_t js = bnd[o];
                        const uint2 s = make_uint2(__float_as_uint(d2_rn(qx, qy, qz, cand.x[js], cand.y[js], cand.z[js])), cand.t[js]);   // the bits of non-negative distances order as they do
                        bool less = s.x < p.x;
                        if (s.x == p.x && o != i)
                            less = __float_as_uint(__ldg(&a.pos[s.y].w)) < __float_as_uint(__ldg(&a.pos[p.y].w));
                        rank += less ? 1u : 0u;
                    }
                    if (rank < need) tmp[qi * kShTies + rank] = (uint16_t)jp;
                    if (rank + 1 == need) kd2 = __uint_as_float(p.x);
                }
                __syncwarp();
                for (uint32_t i = sub; i < need; i += 4) row[below + i] = tmp[qi * kShTies + i];
            }
            kd2 = fmaxf(kd2, __shfl_xor_sync(kFull, kd2, 1));
            kd2 = fmaxf(kd2, __shfl_xor_sync(kFull, kd2, 2));
            __syncwarp();

            // ---- the estimate: a quarter of the neighbours per lane
            const uint32_t n = full ? k : total;
            const float r2 = full ? kd2 : r2max;
            float4 rad = make_float4(0.f, 0.f, 0.f, (float)n);
            const bool est = active && !hard && n > 0 && n >= a.min_found && r2 > 0.0f;
            const float scale = *a.scale_ptr;
            EstAcc acc = {0, 0, 0, 0, 0, 0};
            {
                const float inv = filter_inv32(a.filter, r2, a.cone_k);
                const uint32_t m = est ? n : 0u;
                uint32_t j = 0, jn = 0;
                float4 wn = make_float4(0.f, 0.f, 0.f, 0.f);
                if (sub < m) {
                    jn = row[sub];
                    wn = __ldg(a.pow + cand.t[jn]);
                }
#pragma unroll 1
                for (uint32_t e = sub; e < m; e += 4) {   // the next flux record loads while this one is summed
                    j = jn;
                    const float4 w = wn;
                    if (e + 4 < m) {
                        jn = row[e + 4];
                        wn = __ldg(a.pow + cand.t[jn]);
                    }
                    if (a.filter == 0) sh_add<true>(0, w, 0.0f, inv, nx, ny, nz, scale, a0.neg_zero2, acc);
                    else sh_add<false>(a.filter, w, d2_rn(qx, qy, qz, cand.x[j], cand.y[j], cand.z[j]), inv, nx, ny, nz,
                                       scale, a0.neg_zero2, acc);
                }
            }
#pragma unroll 1
            for (int o = 1; o < 4; o <<= 1) {
                acc.c0 += __shfl_xor_sync(kFull, acc.c0, o);
                acc.c1 += __shfl_xor_sync(kFull, acc.c1, o);
                acc.c2 += __shfl_xor_sync(kFull, acc.c2, o);
                acc.f0 += __shfl_xor_sync(kFull, acc.f0, o);
                acc.f1 += __shfl_xor_sync(kFull, acc.f1, o);
                acc.f2 += __shfl_xor_sync(kFull, acc.f2, o);
            }
            if (inq && sub == 0) {
                bool fix = hard;
                if (est) {
                    if (est_needs_fp64(a.filter, acc)) fix = true;   // the result below is replaced by the fix pass
                    rad = est_result(acc, (double)r2, scale, n, a.norm_c);
                }
                if (fix) fix_push(a, slot, hard ? (bounded && !full ? r2max : tau0) : full ? excl_bound(r2, true) : r2max);
                if (!active) {
                    atomicOr(&a.hdr->errors, kErrQueryNonFinite);
                    rad = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                a.out_rad[qo] = rad;
                if (a.out_r2) a.out_r2[qo] = active ? r2 : r2max;
                if (a.out_count) a.out_count[qo] = active ? n : 0u;
            }
            if constexpr (kNbr) {
                for (uint32_t i = 0; i < len; ++i) {
                    const int src = (int)(i << 2);
                    if (__shfl_sync(kFull, hard ? 1 : 0, src)) continue;   // the fix pass writes the row
                    const uint32_t m = __shfl_sync(kFull, active ? n : 0u, src), o = __shfl_sync(kFull, qo, src);
                    uint32_t* dst = a.out_nbr + a.nbr_off + (size_t)(o - a.q_off) * k;
                    const uint16_t* r = rows + i * row_len;
                    const float x = __shfl_sync(kFull, qx, src), y = __shfl_sync(kFull, qy, src), z = __shfl_sync(kFull, qz, src);
                    if (k <= 32) sh_write_row<1>(a, cand, r, m, x, y, z, dst, lane);
                    else if (k <= 64) sh_write_row<2>(a, cand, r, m, x, y, z, dst, lane);
                    else sh_write_row<4>(a, cand, r, m, x, y, z, dst, lane);
                }
            }
            if (active && full && !hard) {   // an earlier entry stays where this query gives no bound
                pqx = qx; pqy = qy; pqz = qz;
                pr = __fsqrt_rn(r2);
            }
            {
                const float g = __shfl_sync(kFull, full && !hard ? kd2 : 0.0f, 0);
                if (g > 0.0f) guess = 1.4f * g;
            }
            fresh = false;
            if (__any_sync(kFull, full && active)) sparse = false;
            if (len > 1) defers = 0;
            if (nc * 3u <= kShCand * 2u) want = min(2u * want, kShQ);   // twice the queries stage less than half more
            at += len;
            __syncwarp();   // the next group reuses every area
        }
    }
}
