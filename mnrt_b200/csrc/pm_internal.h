// pm_internal.h -- declarations shared by the engine's translation units.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "pm_common.cuh"

namespace pm {

// ------------------------------------------------ device-side helpers --

// Exclusive scan of one value per thread over the block (blockDim.x a
// multiple of 32, at most 1024); total = the block's sum.  s_warp: 32 words
// of shared memory.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = (lane < nwarps) ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nwarps) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[nwarps - 1];
    const uint32_t warp_prefix = warp ? s_warp[warp - 1] : 0u;
    __syncthreads();
    return warp_prefix + x - v;
}

// One 32-byte load (sm_100: 256 bits a lane) from a 32-byte aligned address of
// memory that no running kernel writes.  A gather's cost in L1 is the lines it
// touches, once per load: a record read in one load instead of two pays half.
__device__ __forceinline__ void ld_record32(const void* p, uint32_t (&v)[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// pm_sort.cu
size_t scan_scratch_words(uint32_t n);
int exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* scratch, uint32_t* total_out,
                   cudaStream_t st);
size_t sort_scratch_words(uint32_t n);
// Up to this many photons the last pass moves them.  Before it the order is by
// the low bits only, so its reads are scattered over the whole input: above, they
// miss L2 (20.5M photons in 64 maps: 1.37 ms for that pass, 0.16 for the others),
// and a pass over the sorted order, whose reads are near one another, follows
// instead.
constexpr uint32_t kGatherInSortMax = 1u << 21;
struct SortGather {   // the last pass moves the photons, not the values (n >= 2 only)
    const float4* in_pos;
    const float4* in_pow;
    int format;           // PM_PHOTONS_*: 0 = reference angles, converted to the packed direction
    float4* out_pos;      // tree order: xyz, w = caller index bits
    float4* out_pow;      // tree order: rgb, w = packed direction
    uint32_t* inv;        // caller index -> tree position
};
int radix_sort_pairs(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, int key_bits, uint32_t* scratch,
                     cudaStream_t st, int* launches = nullptr, const SortGather* gather = nullptr);
int radix_sort_pairs32(uint32_t* keys[2], uint32_t* vals[2], uint32_t n, int key_bits, uint32_t* scratch,
                       cudaStream_t st, int* launches = nullptr);

// One photon map of a batch: geometry written by the batch build, query
// parameters uploaded by the host.
struct __align__(16) BatchGeom {
    ChildSlot root;        // slot of the map's subtree (empty slot for an empty map)
    ChildSlot wroot;       // the same subtree in the 32-wide tree
    float lo[3];           // photon bounds, lower corner
    float mscale;          // Morton scale of the map's cubic cell
    float fix_scale;       // fix_scale_of(largest flux channel)
    float max_power;
    uint32_t pad[2];
};
struct __align__(16) BatchQuery {
    uint32_t q_off, q_n;   // queries [q_off, q_off + q_n) of the batch
    uint32_t ph_off, ph_n; // photons [ph_off, ph_off + ph_n) of the batch
    uint64_t nbr_off;      // first neighbour slot of the map's rows (rows hold k entries)
    uint32_t k, min_found;
    float r2max, rmax, cone_k;
    int filter;
    double norm_c;         // filter normalisation constant (the estimate's factor is norm_c / r^2)
};

// Device buffers describing one built map (the build writes them, the
// query reads them).  Pointers are device addresses.
struct MapView {
    const float4* pos;      // tree order: xyz, w = caller index bits
    const float4* pow;      // tree order: rgb, w = octahedral direction bits
    const uint32_t* inv;    // caller index -> tree position
    const Node* nodes;      // [0] = super-root, internal nodes from 1
    const ChildSlot* wchild;   // 32-wide tree: child slots
    const ChildSlot* wroot;    // 32-wide tree: start slot
    MapHeader* hdr;
    uint32_t n;             // photon count (host copy)
};

// Which sizes of a cluster sort (pm_sort_small.cuh) a handle has asked for, and
// which of them fit; one for each kernel.
struct SmallSortFits {
    uint32_t size[8] = {}, count = 0;   // size << 1 | fits (a kernel has seven sizes)
    bool find(uint32_t s, bool& fit) const {
        for (uint32_t i = 0; i < count; ++i)
            if (size[i] >> 1 == s) { fit = size[i] & 1u; return true; }
        return false;
    }
    bool asked(uint32_t s) const { bool f; return find(s, f); }
    bool holds(uint32_t s) const { bool f; return find(s, f) && f; }
    void keep(uint32_t s, bool fit) { if (count < 8) size[count++] = s << 1 | (fit ? 1u : 0u); }
};

struct BuildBuffers {
    SmallSortFits* fits;    // of k_small_build
    uint64_t* keys[2];
    uint32_t* vals[2];
    uint32_t* scratch;      // sort / scan scratch
    uint32_t* kfirst;       // Karras internal nodes: first, last, split
    uint32_t* klast;
    uint32_t* ksplit;
    uint32_t* kkeep;        // keep flag (node holds more than leaf_size photons)
    uint32_t* krank;        // exclusive scan of kkeep = compacted index - 1
    uint32_t* parent;       // compacted node -> parent (node << 1 | side)
    uint32_t* arrive;       // refit arrival counters per compacted node
    uint32_t* nleaf;        // leaf children per compacted node
    uint32_t* partials;     // bounds reduction partials (block count * 8 floats) + counter
    uint32_t num_partials;
};

struct WideBuffers {
    uint32_t* wcnt;        // per wide node: child count
    uint32_t* wfirst;      // per wide node: first child slot
    uint32_t* wslot;       // per child slot of a wide node: binary slot << 1 | wide
    ChildSlot* wchild;     // child slots of all wide nodes
    ChildSlot* wroot;      // start slot of the wide traversal
    uint32_t* scratch;     // one word: child slots taken
};

// pm_build.cu
size_t build_bytes_needed(uint32_t n);
// Returns the number of kernels launched; sort_done (if set) is recorded on
// the stream right after the radix sort.
// The whole single-map build, binary and 32-wide tree.
int build_map(const float4* in_pos, const float4* in_pow, uint32_t n, int format, uint32_t leaf_size,
              float4* out_pos, float4* out_pow, uint32_t* inv, Node* nodes, MapHeader* hdr, const BuildBuffers& bb,
              const WideBuffers& wide, cudaStream_t st, cudaEvent_t sort_done = nullptr);
void scale_flux(float4* pow, uint32_t n, float scale, MapHeader* hdr, cudaStream_t st);
int build_wide(uint32_t n, const Node* nodes, const uint32_t* parent, const uint32_t* rootmark, MapHeader* hdr,
               const WideBuffers& wb, cudaStream_t st);
int build_from_sorted(const float4* in_pos, const float4* in_pow, uint32_t n, int format, uint32_t leaf_size,
                      const uint64_t* keys, const uint32_t* vals, float4* out_pos, float4* out_pow, uint32_t* inv,
                      Node* nodes, MapHeader* hdr, const BuildBuffers& bb, cudaStream_t st, bool gathered = false,
                      const WideBuffers* wide = nullptr);   // wide: also the 32-wide tree (single map, n >= 2)

// pm_query.cu
struct QueryParams {
    uint32_t k;
    float r;             // R
    float r2;            // R^2 rounded in FP32
    int filter;
    float cone_k;
    uint32_t min_found;
};

struct QueryOutputs {
    float4* rad;         // required
    uint32_t* nbr;       // optional
    float* r2;           // optional
    uint32_t* count;     // optional
};

// Processing order of the queries (Hilbert, or Morton); with recs also their
// records in that order (needs the normals).  keys and vals: two buffers of nq
// words each, scratch: sort_scratch_words(nq), fits: of the Hilbert and the Morton sort.
const uint32_t* query_order(const float4* qpos, uint32_t nq, const MapHeader* hdr, uint32_t* const keys[2],
                            uint32_t* const vals[2], uint32_t* scratch, SmallSortFits* fits, cudaStream_t st, int* launches,
                            bool hilbert, const float4* qnrm = nullptr, float4* recs = nullptr);
constexpr int kQueryKeyBits = 30;         // bits of the query Hilbert keys (sorted as uint32)
constexpr int kBatchQueryMapShift = 30;   // batch query keys: (map id << 30) | 30-bit Hilbert index in the map's cell
constexpr uint32_t kSharedShapes = 2 * (kMaxK + 1);   // by k, without and with neighbour lists
struct QueryTuning {
    int layout;             // 0: lane per query with a shared-memory heap; 1: group buffers
    int queries_per_warp;   // group layout: 1, 2, 4 or 8 (32, 16, 8 or 4 lanes per query)
    int warps_per_block;
    int rounds_per_chunk;
    unsigned long long* stats;   // 8 traversal counters (group layout), nullptr = off
    const char** kernel;         // set to the search kernel's name
    uint32_t* shared_shapes;     // the handle's launch shapes of the shared walk (kSharedShapes words, 0: not asked yet)
    const float4* qsorted = nullptr;   // query records in sorted order (pos.xyz | caller index, normal), or nullptr
                                       // (a batch: set where it shares walks)
};
// Whether sorted queries in the wide layout share walks (k_knn_shared): nq of them in
// all, the sum of what their maps gain (in queries, negative where one by one is
// faster) and the largest of what their longest warps cost.
double shared_gain(uint32_t n, uint32_t nq, uint32_t k, bool lists);
double shared_tail(uint32_t n, uint32_t k);
bool shared_walk(uint64_t nq, double gain, double tail);
int gather_queries(const uint32_t* order, const float4* qpos, const float4* qnrm, uint32_t nq, float4* out, cudaStream_t st);
int query_knn(const MapView& m, const QueryParams& p, const float4* qpos, const float4* qnrm,
              const uint32_t* order, uint32_t nq, const QueryOutputs& out, uint32_t* work_counter, uint32_t* fix_list, float* fix_bound,
              const QueryTuning& t, cudaStream_t st);
int query_bruteforce(const MapView& m, const QueryParams& p, const float4* qpos, const float4* qnrm,
                      uint32_t nq, const QueryOutputs& out, cudaStream_t st);
int query_smem_bytes_per_warp(uint32_t k);
double filter_norm_const(int filter, float cone_k);

int query_knn_batch(const MapView& m, const BatchQuery* bq, const BatchGeom* bg, uint32_t kmax, const float4* qpos,
                    const float4* qnrm, const uint32_t* order, const uint64_t* qkeys, uint32_t nq,
                    const QueryOutputs& out, uint32_t* work_counter, uint32_t* fix_list, float* fix_bound, const QueryTuning& t,
                    cudaStream_t st);

// pm_batch.cu
int batch_bounds_and_keys(const float4* pos, const float4* pw, const uint32_t* ph_off, uint32_t m, uint32_t n,
                          uint32_t* acc, BatchGeom* geom, MapHeader* hdr, uint64_t* keys, uint32_t* vals,
                          cudaStream_t st);
int batch_query_keys(const float4* qpos, const uint32_t* q_off, uint32_t m, uint32_t nq, const BatchGeom* geom,
                     uint64_t* keys, uint32_t* vals, cudaStream_t st);
int batch_roots(const uint32_t* ph_off, uint32_t m, uint32_t n, uint32_t leaf_size, const float4* pos,
                const Node* nodes, const BuildBuffers& bb, BatchGeom* geom, cudaStream_t st);
int map_id_bits(uint32_t m);
int batch_wide(uint32_t n, uint32_t m, const Node* nodes, const uint32_t* parent, MapHeader* hdr, uint32_t* rootmark,
               const WideBuffers& wb, BatchGeom* geom, cudaStream_t st);

// pm_compat.cu
int compat_node_estimates(const MapView& m, uint32_t max_slots, float rmax, uint32_t k, uint32_t iters, float* est,
                          cudaStream_t st);
int compat_query(const MapView& m, const float* est, const QueryParams& p, uint32_t iters, const float4* qpos,
                 const float4* qnrm, uint32_t nq, float* out_radius, const QueryOutputs& out, cudaStream_t st);

// pm_icut.cu: illumination cuts.  Per-slot arrays hold 2 (num_nodes + 1)
// entries (slot 2j + side of node j, slot 0 = root); pslot holds one entry
// per node.
struct IcutParams {
    bool use_leafs;
    uint32_t level_emin;
    uint32_t refine_iters;
    float accuracy;
};
struct IcutBuffers {
    uint32_t* pslot;             // node -> slot referencing it
    uint32_t* level;             // slot depth (root 0), kInvalid for empty slots
    uint2* range;                // slot photons [x, y) in tree order
    float4* center;              // box centre xyz, largest box side w
    float4* normal;              // normal xyz (zero: none)
    float4* est;                 // photon-sum estimate E~ (rgb)
    float4* exact;               // estimate at the centre (rgb, w = photons used)
    uint32_t* coarse;            // coarse cut marks
    uint32_t* fin;               // final cut marks
    uint32_t* work[2];           // work flags (refinement), mark scratch (coarse cut)
    unsigned long long* acc;     // level statistics: max bits [0..2], fixed sums [3..5], count [6]
    float4* ibox;                // per slot, 2 entries: influence box lo (w = 1: interpolation stops here), hi
};
int icut_prepare(const MapView& m, uint32_t num_nodes, const IcutBuffers& b, cudaStream_t st);
int icut_normals(const MapView& m, uint32_t nslots, const float4* caller, const IcutBuffers& b, cudaStream_t st);
int icut_coarse(const MapView& m, uint32_t nslots, const IcutParams& p, const IcutBuffers& b, cudaStream_t st);
int icut_final(const MapView& m, uint32_t nslots, const IcutParams& p, const IcutBuffers& b, cudaStream_t st);
int icut_interpolate(const MapView& m, const IcutBuffers& b, const float4* qpos, const float4* qnrm,
                     const uint32_t* order, uint32_t nq, float r2, float4* out, cudaStream_t st);

// pm_gather.cu
int gather_normals(const float4* hit_nrm, const float4* ray_dir, uint32_t n, float4* out_nrm, cudaStream_t st);
int gather_accumulate(const float4* est, const float4* hit_pos, const float4* ray_origin, const float4* influence,
                      const float4* clr_diffuse, const uint32_t* idx_shading, uint32_t n, float4* io_rad,
                      float* io_recip, cudaStream_t st);

int merge_ranks(const uint32_t* is_valid, uint32_t n, uint32_t* flags, uint32_t* rank, uint32_t* scan_scratch,
                uint32_t* total, cudaStream_t st);
int merge_scatter(const float4* pos, const float4* pw, const uint32_t* flags, const uint32_t* rank, uint32_t n,
                  float4* dst_pos, float4* dst_pow, cudaStream_t st);
int scale_rgb(float4* pw, uint32_t n, float scale, cudaStream_t st);

// pm_backward.cu
// Per-query record of the adjoint, 64 bytes: everything the per-photon pass
// needs about one query in one aligned load.
struct __align__(32) BwdQuery {
    double gx, gy, gz;        // dL/dE * norm per channel
    double G;                 // the k-th neighbour's r^2 path (0 unless k were found)
    double rinv;              // the filter's reciprocal: 1 / (k_c r) cone, 1 / r^2 Epanechnikov, 1 box;
                              // 0 = the query carries no gradient
    float qx, qy, qz;         // position
    float nx, ny, nz;         // normal
};
static_assert(sizeof(BwdQuery) == 64, "one 64-byte record per query");

// A photon as the adjoint's per-query pass gathers it, in caller order (the
// order the neighbour lists name): one aligned 32-byte load gives all of it.
struct __align__(32) BwdPhoton {
    float x, y, z;
    uint32_t tree;            // tree position
    float r, g, b;
    uint32_t dir;
};
static_assert(sizeof(BwdPhoton) == 32, "one 32-byte record per photon");

struct BwdArgs {
    const BwdPhoton* photon;  // caller order (bwd_pack), or nullptr: too few pairs to pay for them
    const float4* pos;        // tree order
    const float4* pow;
    const uint32_t* inv;      // caller index -> tree position
    const float4* qpos;       // all queries (indexed by global query id)
    const float4* qnrm;
    const float4* grad;       // dL/dE per query (rgb)
    const uint32_t* nbr;      // this chunk's neighbour rows (caller indices, sorted by (d^2, index))
    const uint32_t* count_in; // this chunk's counts, or nullptr (derived from the rows)
    uint32_t n, k;
    float r_max;
    int filter;
    float cone_k;
    uint32_t min_found;
    BwdQuery* qrec;           // per chunk query: the record the per-photon pass reads
    uint32_t* keys;           // sort path: one photon key per neighbour slot (set by backward_chunk)
    uint32_t* vals;           // pair values: grouped by photon (placement), or per slot (sort)
    uint32_t* cursor;         // per photon: pair count, then the next free slot of its segment
    uint64_t pair_cap;        // slots in vals
    const uint32_t* order;    // the chunk's queries in Hilbert order (chunk-local ids), or nullptr
};
struct BwdBuffers {
    uint32_t* vals[2];        // one slot per neighbour pair of a chunk ([1]: sort path only)
    uint32_t* keys[2];        // sort path only
    uint32_t* scratch;        // the scan of the per-photon counts, or the sort's
    uint32_t* seg_start;
    uint32_t* seg_end;
    uint32_t* long_list;      // photons whose segments a block sorts (n entries)
    uint32_t* long_count;
    double* acc;              // 6 doubles per photon, carried between chunks
};
// Mean pairs per photon above which a chunk groups its pairs by a stable
// radix sort instead of counts, atomic placement and segment sorts.
constexpr uint64_t kBwdPlaceMaxFanIn = 256;
inline bool bwd_sort_path(uint64_t pairs, uint32_t n) { return pairs > kBwdPlaceMaxFanIn * (uint64_t)n; }
// Pairs per photon from which the photons' records are laid out first (bwd_pack): the
// layout costs every photon 64 bytes, and saves a pair two of its gathers.  Adjoint
// without / with records, us: 1M photons, 0.1 pairs each 144 / 179, 8 each (k = 64)
// 539 / 540, 32 each 1,398 / 1,363, 64 each 2,677 / 2,602; 8M photons, 0.1 each 1,366 /
// 1,556, 8 each 3,910 / 3,987; 65,536 photons, 16 each 102 / 105, 250 each 1,905 / 1,890.
constexpr uint64_t kBwdPackMin = 32;
inline bool bwd_packs(uint64_t pairs, uint32_t n) { return pairs >= kBwdPackMin * (uint64_t)n; }
size_t bwd_scratch_words(uint32_t n, uint64_t pairs, bool sort_path);
int bwd_pack(const float4* pos, const float4* pow, uint32_t n, BwdPhoton* out, cudaStream_t st);
int backward_chunk(const BwdArgs& a, uint32_t q0, uint32_t nq_chunk, bool first, bool last, const BwdBuffers& b,
                   float4* grad_pow, float4* grad_pos, cudaStream_t st);

}  // namespace pm
