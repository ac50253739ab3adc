// BVH traversal by warp ray pools: the walk of k_trace, k_occlude and the standalone queries.
//
// A ray's walk is a sequence of four unlike operations -- a node visit, an instance entry, a leaf test
// and the end of the ray -- whose order differs from ray to ray. With one ray per lane, lanes at
// different operations run one after another (measured: 5 to 9 of 32 lanes per issued instruction).
// Here every lane holds kPoolRays rays whose walk state lives in shared memory, the warp runs one
// operation at a time, and it picks the operation that most lanes have a ray for; a lane joins with
// whichever of its rays is due for it. BVH-stress frame, 1920 x 1080 x 16: k_trace 158 -> 91 ms with
// k_hits, k_occlude 66 -> 35 ms; Cornell box with spheres, 256 x 256 x 256: 55 -> 31 and 22 -> 13.5 ms.
// What bounds it now is latency at 16 warps per SM: the fixed latency of a visit's instructions and
// the L2 round trips of its node, with 16 (closest hits) and 18 (shadow rays) of 32 lanes per instruction.
#pragma once

namespace bf200 {

// Rays per lane, threads per block, resident blocks per SM (the registers a walk needs allow four; more
// blocks spill and leave less L1). BVH-stress frame, 16 samples, trace + occlude: 174 ms with 1 ray, 130
// with 2, 126 with 3. Shadow rays deal their leaves' triangles over the warp, and 2 rays suffice then
// (occlude 34.6 -> 32.7 ms).
constexpr int kPoolThreads = 128, kPoolBlocks = 4;
template <bool ANY>
constexpr int kPoolRays = ANY ? 2 : 3;
// Stack entries of a ray in shared memory; deeper ones, which few walks reach, are local.
constexpr int kPoolStack = 15;
// A node visit is repeated in registers while at least this many sixteenths of the lanes that began
// it still have a node to visit (6, 10 and 13 sixteenths measured within 1 % of one another).
constexpr uint32_t kPoolStay = 10;

// Words of one ray's state, in thread-interleaved columns of shared memory (every lane on its own bank).
enum PoolWord : int {
    kPoolO = 0,         // origin in the current frame (the world's, or the current instance's)
    kPoolInv = 3,       // reciprocal direction
    kPoolD = 6,         // direction
    kPoolLimit = 9,     // closest hit's t, or t_max
    kPoolTMin = 10,
    kPoolInst = 11,     // current instance
    kPoolBestInst = 12,
    kPoolBestLeaf = 13,
    kPoolId = 14,       // the job's ray id
    kPoolFlags = 15,    // stack size | axis-parallel bits | outcome bits
    kPoolFrames = 16    // first stack entry
};
constexpr int kPoolWords = kPoolFrames + kPoolStack;
constexpr uint32_t kPoolSpMask = 0xFFU, kPoolAxes = 0x700U, kPoolFound = 0x800U, kPoolFailed = 0x1000U;
constexpr int kPoolAxesShift = 8;
static_assert(kTraversalStack <= static_cast<int>(kPoolSpMask), "a stack size fits its bits");
// One operation's leaf triangles, per warp: the tests of all its lanes, and the lane and
// ray that asked for each.
constexpr uint32_t kPoolTests = 32U * kMaxLeafTriangles;
static_assert(kMaxLeafTriangles < 8 && kPoolRays<true> <= 8,
              "leaf sizes are dealt by three ballots, and a test's lane and ray fit one byte");
template <bool ANY>
constexpr int kPoolRayWords = kPoolWords * kPoolRays<ANY> * kPoolThreads;
template <bool ANY>
constexpr size_t kPoolSharedBytes =
    sizeof(uint32_t) * kPoolRayWords<ANY> +
    (ANY ? (sizeof(uint32_t) + sizeof(uint8_t)) * kPoolTests * (kPoolThreads / 32) : 0U);
constexpr uint32_t kPoolMiss = 0xFFFFFFFFU, kPoolFailure = 0xFFFFFFFEU;  // a test's answer

// The entry of a ray whose walk has ended (no stack code).
constexpr int kPoolDone = INT_MAX;

__device__ __forceinline__ RayInv pool_ray(F3 o, F3 inv, uint32_t flags) {
    return RayInv{o, inv, (flags & kPoolAxes) >> kPoolAxesShift};
}

// One lane's view of the pool: the shared column of ray k, and its stack.
struct PoolRay {
    uint32_t* w;  // the ray's first word
    int* deep;    // the ray's stack entries beyond kPoolStack
    __device__ __forceinline__ uint32_t& word(int i) const { return w[i * kPoolThreads]; }
    __device__ __forceinline__ float real(int i) const { return __uint_as_float(w[i * kPoolThreads]); }
    __device__ __forceinline__ void set(int i, float v) const { w[i * kPoolThreads] = __float_as_uint(v); }
    __device__ __forceinline__ F3 vec(int i) const { return F3{real(i), real(i + 1), real(i + 2)}; }
    __device__ __forceinline__ void set(int i, F3 v) const {
        set(i, v.x);
        set(i + 1, v.y);
        set(i + 2, v.z);
    }
    __device__ __forceinline__ void push(uint32_t& sp, int entry) const {
        if (sp < static_cast<uint32_t>(kPoolStack)) {
            w[(kPoolFrames + sp) * kPoolThreads] = static_cast<uint32_t>(entry);
        } else {
            deep[sp - kPoolStack] = entry;
        }
        ++sp;
    }
    __device__ __forceinline__ int pop(uint32_t& sp) const {
        if (sp == 0U) {
            return kPoolDone;
        }
        --sp;
        return sp < static_cast<uint32_t>(kPoolStack) ? static_cast<int>(w[(kPoolFrames + sp) * kPoolThreads])
                                                      : deep[sp - kPoolStack];
    }
    // moves the ray into a frame; returns its axis-parallel flags
    __device__ __forceinline__ uint32_t frame(F3 o, F3 d) const {
        const RayInv r = make_ray_inv(o, d);
        set(kPoolO, o);
        set(kPoolInv, r.inv);
        set(kPoolD, d);
        return r.axes << kPoolAxesShift;
    }
};

enum PoolOp : uint32_t { kPoolNode = 0U, kPoolInstance, kPoolLeaf, kPoolEnd, kPoolFetch, kPoolSphere };

// The operation an entry is due for. `world`: the ray is in the world's frame.
template <bool SPH>
__device__ __forceinline__ uint32_t pool_op(int entry, bool world) {
    if (entry >= 0) {
        return entry == kPoolDone ? kPoolEnd : kPoolNode;
    }
    if (entry >= kLeafEntryMin) {
        return SPH && (static_cast<uint32_t>(~entry) & (kMaxLeafSize - 1)) + 1U == kSphereLeafCount ? kPoolSphere
                                                                                                   : kPoolLeaf;
    }
    return world && ((static_cast<uint32_t>(entry) ^ 0x80000000U) & kTlasFlag) != 0U ? kPoolNode : kPoolInstance;
}

// Walks every ray of `job`. ANY: any hit in [t_min, t_max] ends the ray; otherwise its closest hit is
// found, ties going to the first (instance, primitive) as in the analytic accel's in-order scan. A
// ray meets its nodes and leaves in the order of its own stack whatever the warp runs between, so
// the result does not depend on the pool. The job hands out rays (fetch), reads them again where the
// walk changes frames (ray) and takes the outcome (finish).
template <bool ANY, bool SPH, class Job>
__device__ __forceinline__ void pool_walk(const SceneView& s, Job& job, uint32_t* shared) {
    uint32_t* const column = shared + threadIdx.x;
    constexpr int kRays = kPoolRays<ANY>;
    int deep[kRays][kTraversalStack - kPoolStack];
    int entry[kRays];  // each ray's next entry, popped
    uint32_t due_op[kRays];
    uint32_t world = 0U;  // bit k: ray k is in the world's frame
#pragma unroll
    for (int k = 0; k < kRays; ++k) {
        entry[k] = kPoolDone;
        due_op[k] = kPoolFetch;
    }
    while (true) {
        // the operation most lanes can run
        uint32_t mine = 0U;
#pragma unroll
        for (int k = 0; k < kRays; ++k) {
            mine |= 1U << due_op[k];
        }
        if (job.drained()) {
            mine &= ~(1U << kPoolFetch);
        }
        uint32_t best = 0U;  // lanes << 3 | operation
#pragma unroll
        for (uint32_t c = 0; c < (SPH ? 6U : 5U); ++c) {
            const uint32_t n = __popc(__ballot_sync(0xFFFFFFFFU, (mine >> c & 1U) != 0U));
            best = max(best, n << 3 | c);
        }
        if (best < 8U) {
            break;  // nothing in flight and nothing left to fetch
        }
        const uint32_t op = best & 7U;
        bool due = (mine >> op & 1U) != 0U;
        int k = 0, next = entry[0];
#pragma unroll
        for (int j = 1; j < kRays; ++j) {
            if (due_op[j] == op) {
                k = j;
                next = entry[j];
            }
        }
        const PoolRay ray{column + k * (kPoolWords * kPoolThreads), deep[k]};
        bool in_world = (world >> k & 1U) != 0U;
        uint32_t after = kPoolFetch;  // the ray's next operation
        if (op == kPoolNode) {
            uint32_t flags = 0U, sp = 0U;
            F3 o{}, inv{};
            float limit = 0.0F, t_min = 0.0F;
            if (due) {
                flags = ray.word(kPoolFlags);
                sp = flags & kPoolSpMask;
                o = ray.vec(kPoolO);
                inv = ray.vec(kPoolInv);
                limit = ray.real(kPoolLimit);
                t_min = ray.real(kPoolTMin);
            }
            const RayInv r = pool_ray(o, inv, flags);
            bool visit = due;
            do {
                if (visit) {
                    const bool tlas = next < 0;
                    const int node = tlas ? static_cast<int>((static_cast<uint32_t>(next) ^ 0x80000000U) & (kTlasFlag - 1U))
                                          : next;
                    int kids[4];
                    const int count = hit_children(r, s.nodes[node], t_min, limit, kids);
#pragma unroll
                    for (int c = 3; c >= 0; --c) {
                        if (tlas) {
                            kids[c] = kids[c] >= 0 ? tlas_entry(kids[c])
                                                   : instance_entry(static_cast<uint32_t>(~kids[c]));
                        }
                        if (c > 0 && c < count) {
                            ray.push(sp, kids[c]);
                        }
                    }
                    next = count > 0 ? kids[0] : ray.pop(sp);
                    after = pool_op<SPH>(next, in_world);
                    visit = after == kPoolNode;
                }
            } while (16U * __popc(__ballot_sync(0xFFFFFFFFU, visit)) >= kPoolStay * (best >> 3));
            if (due) {
                ray.word(kPoolFlags) = (flags & ~kPoolSpMask) | sp;
            }
        } else if (op == kPoolInstance) {
            if (due) {
                uint32_t flags = ray.word(kPoolFlags);
                uint32_t sp = flags & kPoolSpMask;
                F3 o, d;
                uint32_t mask;
                job.ray(ray.word(kPoolId), o, d, mask);
                const uint32_t code = static_cast<uint32_t>(next) ^ 0x80000000U;
                if ((code & kTlasFlag) != 0U) {  // back from an instance to the instance level
                    flags = (flags & ~kPoolAxes) | ray.frame(o, d);
                    in_world = true;
                } else {
                    // an instance (code = its index) is entered unless the ray's visibility mask excludes
                    // it or its world box is not met
                    const uint32_t inst = code;
                    const float4 blo = s.inst_world_box[2ULL * inst], bhi = s.inst_world_box[2ULL * inst + 1];
                    float near;
                    const RayInv r = make_ray_inv(o, d);
                    if ((mask & __float_as_uint(blo.w)) != 0U &&
                        slab(r, blo.x, bhi.x, blo.y, bhi.y, blo.z, bhi.z, ray.real(kPoolTMin), ray.real(kPoolLimit),
                             near)) {
                        const float4* m = s.inst_to_object + 3ULL * inst;
                        flags = (flags & ~kPoolAxes) | ray.frame(xform_point(m, o), xform_vector(m, d));
                        in_world = false;
                        ray.word(kPoolInst) = inst;
                        next = __float_as_int(bhi.w);  // the BLAS root
                    } else {
                        next = ray.pop(sp);
                    }
                }
                ray.word(kPoolFlags) = (flags & ~kPoolSpMask) | sp;
                after = pool_op<SPH>(next, in_world);
            }
        } else if (ANY && op == kPoolLeaf) {
            // the leaves' triangles, dealt evenly over the warp's lanes
            const uint32_t packed = static_cast<uint32_t>(~next);
            const uint32_t first = packed >> kLeafCountBits;
            const uint32_t n = due ? (packed & (kMaxLeafSize - 1)) + 1U : 0U;
            const uint32_t lane = threadIdx.x & 31U, below = (1U << lane) - 1U;
            const unsigned ones = __ballot_sync(0xFFFFFFFFU, (n & 1U) != 0U);
            const unsigned twos = __ballot_sync(0xFFFFFFFFU, (n & 2U) != 0U);
            const unsigned fours = __ballot_sync(0xFFFFFFFFU, (n & 4U) != 0U);
            const uint32_t from = __popc(ones & below) + 2U * __popc(twos & below) + 4U * __popc(fours & below);
            const uint32_t total = __popc(ones) + 2U * __popc(twos) + 4U * __popc(fours);
            uint32_t* const tests = shared + kPoolRayWords<ANY> + (threadIdx.x >> 5) * kPoolTests;
            uint8_t* const owners =
                reinterpret_cast<uint8_t*>(shared + kPoolRayWords<ANY> + (kPoolThreads / 32) * kPoolTests) +
                (threadIdx.x >> 5) * kPoolTests;
            for (uint32_t j = 0; j < n; ++j) {
                tests[from + j] = first + j;
                owners[from + j] = static_cast<uint8_t>(lane | static_cast<uint32_t>(k) << 5);
            }
            __syncwarp();
            for (uint32_t q = lane; q < total; q += 32U) {
                const uint32_t owner = owners[q];
                const PoolRay asked{shared + (threadIdx.x & ~31U) + (owner & 31U) +
                                        (owner >> 5) * (kPoolWords * kPoolThreads),
                                    nullptr};
                const float4* record = s.leaf_tris + 3ULL * tests[q];
                TriangleHit th;
                const int res = triangle_test(record[0], record[1], record[2], asked.vec(kPoolO), asked.vec(kPoolD),
                                              asked.real(kPoolTMin), asked.real(kPoolLimit), false, th);
                tests[q] = res == kTriHit ? 0U : (res == kTriFailure ? kPoolFailure : kPoolMiss);
            }
            __syncwarp();
            if (due) {
                uint32_t flags = ray.word(kPoolFlags);
                uint32_t sp = flags & kPoolSpMask;
                for (uint32_t j = 0; j < n; ++j) {
                    const uint32_t answer = tests[from + j];
                    flags |= answer == 0U ? kPoolFound : (answer == kPoolFailure ? kPoolFailed : 0U);
                }
                next = (flags & kPoolFound) != 0U ? kPoolDone : ray.pop(sp);
                ray.word(kPoolFlags) = (flags & ~kPoolSpMask) | sp;
                after = pool_op<SPH>(next, in_world);
            }
        } else if (op == kPoolLeaf || (SPH && op == kPoolSphere)) {
            if (due) {
                uint32_t flags = ray.word(kPoolFlags);
                uint32_t sp = flags & kPoolSpMask;
                const F3 o = ray.vec(kPoolO), d = ray.vec(kPoolD);
                const float t_min = ray.real(kPoolTMin);
                float limit = ray.real(kPoolLimit);
                const uint32_t packed = static_cast<uint32_t>(~next);
                const uint32_t first = packed >> kLeafCountBits;
                const uint32_t n = SPH && op == kPoolSphere ? 1U : (packed & (kMaxLeafSize - 1)) + 1U;
                const float4* record = s.leaf_tris + 3ULL * first;
                // most triangles of a leaf are certain misses; the double test then runs for the rest,
                // one per round, instead of for every triangle with whichever lanes still need it (trace and
                // k_hits, BVH stress 16 spp: 79.4 ms and 74.4 ms with the filter; Cornell box with spheres,
                // 256 spp: 29.3 and 27.1)
                uint32_t candidates = 1U;
                if constexpr (!ANY) {
                    if (!SPH || op == kPoolLeaf) {
                        const float d_sum = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
                        candidates = 0U;
                        for (uint32_t j = 0; j < n; ++j) {
                            candidates |= certain_miss(record[3U * j], record[3U * j + 1U], record[3U * j + 2U], o, d,
                                                       d_sum)
                                              ? 0U
                                              : 1U << j;
                        }
                    }
                }
                while (candidates != 0U) {
                    const uint32_t j = static_cast<uint32_t>(__ffs(static_cast<int>(candidates))) - 1U;
                    candidates &= candidates - 1U;
                    const uint32_t leaf = first + j;
                    const float4 v0 = record[3U * j], v1 = record[3U * j + 1U], v2 = record[3U * j + 2U];
                    int res = kTriMiss;
                    float t = 0.0F;
                    if (SPH && op == kPoolSphere) {
                        const SphereHit h = sphere_intersect(v0, v1.x, o, d, t_min, limit);
                        res = static_cast<int>(h.outcome);
                        t = h.t;
                    } else if constexpr (!ANY) {
                        TriangleHit th;
                        res = triangle_test(v0, v1, v2, o, d, t_min, limit, false, th);
                        t = th.t;
                    }
                    if (res == kTriFailure) {
                        flags |= kPoolFailed;
                        continue;
                    }
                    if (res != kTriHit) {
                        continue;
                    }
                    if (ANY) {
                        flags |= kPoolFound;
                        break;
                    }
                    const uint32_t inst = ray.word(kPoolInst);
                    bool closer = (flags & kPoolFound) == 0U || t < limit;
                    if (!closer && t == limit) {
                        const uint32_t best_inst = ray.word(kPoolBestInst);
                        closer = inst != best_inst
                                     ? inst < best_inst
                                     : __float_as_uint(v0.w) <
                                           __float_as_uint(s.leaf_tris[3ULL * ray.word(kPoolBestLeaf)].w);
                    }
                    if (closer) {
                        limit = t;
                        ray.word(kPoolBestInst) = inst;
                        ray.word(kPoolBestLeaf) = leaf;
                        flags |= kPoolFound;
                    }
                }
                if (!ANY) {
                    ray.set(kPoolLimit, limit);
                }
                next = ANY && (flags & kPoolFound) != 0U ? kPoolDone : ray.pop(sp);
                ray.word(kPoolFlags) = (flags & ~kPoolSpMask) | sp;
                after = pool_op<SPH>(next, in_world);
            }
        } else if (op == kPoolEnd) {
            if (due) {
                const uint32_t flags = ray.word(kPoolFlags);
                if constexpr (ANY) {
                    job.finish(s, ray.word(kPoolId), (flags & kPoolFound) != 0U ? 1 : ((flags & kPoolFailed) != 0U ? -1 : 0));
                } else {
                    ClosestResult c;
                    c.t = ray.real(kPoolLimit);
                    c.instance = (flags & kPoolFound) != 0U ? ray.word(kPoolBestInst) : 0xFFFFFFFFU;
                    c.leaf = (flags & kPoolFound) != 0U ? ray.word(kPoolBestLeaf) : 0xFFFFFFFFU;
                    c.failed = (flags & kPoolFailed) != 0U;
                    job.finish(s, ray.word(kPoolId), c);
                }
            }
        } else {
            uint32_t id = 0U, mask = 0U;
            F3 o{}, d{};
            float t_min = 0.0F, t_max = 0.0F;
            due = job.fetch(due, id, o, d, t_min, t_max, mask);
            if (due) {
                ray.word(kPoolId) = id;
                ray.set(kPoolTMin, t_min);
                ray.set(kPoolLimit, t_max);
                const uint32_t axes = ray.frame(o, d);
                in_world = true;
                uint32_t sp = 0U;
                if (s.tlas_root >= 0) {
                    next = tlas_entry(s.tlas_root);
                } else {
                    // few instances: every visible one whose world box the ray meets within
                    // [t_min, t_max], the lowest index on top
                    const RayInv r = pool_ray(o, ray.vec(kPoolInv), axes);
                    for (int inst = static_cast<int>(s.instance_count) - 1; inst >= 0; --inst) {
                        const float4 blo = s.inst_world_box[2 * inst], bhi = s.inst_world_box[2 * inst + 1];
                        float near;
                        if ((mask & __float_as_uint(blo.w)) != 0U &&
                            slab(r, blo.x, bhi.x, blo.y, bhi.y, blo.z, bhi.z, t_min, t_max, near)) {
                            ray.push(sp, instance_entry(static_cast<uint32_t>(inst)));
                        }
                    }
                    next = ray.pop(sp);
                }
                ray.word(kPoolFlags) = axes | sp;
                after = pool_op<SPH>(next, true);
            }
        }
        if (due) {
#pragma unroll
            for (int j = 0; j < kRays; ++j) {
                entry[j] = k == j ? next : entry[j];
                due_op[j] = k == j ? after : due_op[j];
            }
            world = (world & ~(1U << k)) | (in_world ? 1U << k : 0U);
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------------------
// k_trace: closest hit of every active slot's ray; writes the hit and the slot's shading route
// ------------------------------------------------------------------------------------------------

// The traced slots' hits: the barycentrics of each winning triangle (the trace leaves its t and leaf
// record) and the slot's shading route. A kernel of its own: inside k_trace this code, run once per ray
// between the walks of others, cost 12,400 cycles a pass and pushed the walk out of the instruction
// cache (no_instruction 3.2 stalls per issue).
template <bool SPH>
__global__ void __launch_bounds__(256) k_hits(SceneView s, Wavefront w) {
    chain_begin();
    const uint32_t count = static_cast<uint32_t>(w.counters[kCounterTraced]);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t slot = w.trace_queue[i];
        if (w.state[slot] != kSlotActive) {  // the walk failed
            w.route[slot] = kRouteNone;
            continue;
        }
        const uint2 id = w.hit_id[slot];
        if (id.x == 0xFFFFFFFFU) {
            w.route[slot] = static_cast<uint8_t>(kRouteMiss);
            continue;
        }
        const float4 o4 = w.ray_o[slot], d4 = w.ray_d[slot];
        const ClosestResult c{w.hit_tb[slot].x, id.x, id.y, false};
        TriangleHit th;
        if (!hit_barycentrics<SPH>(s, c, ld3(o4), ld3(d4), d4.w, o4.w, th)) {
            w.status[slot] = (w.status[slot] & ~0xFFU) | kLaneNumerical;
            w.state[slot] = kSlotDone;
            w.route[slot] = kRouteNone;
            continue;
        }
        w.hit_tb[slot] = make_float4(c.t, th.b0, th.b1, th.b2);
        w.route[slot] = s.inst_route[id.x];
    }
}

// The rays of the trace queue, handed out from a cursor with one atomic per warp for all of the
// warp's idle lanes.
struct TraceJob {
    const Wavefront& w;
    uint32_t count;
    bool done;

    __device__ __forceinline__ bool drained() const { return done; }
    __device__ __forceinline__ bool fetch(bool want, uint32_t& id, F3& o, F3& d, float& t_min, float& t_max,
                                          uint32_t& mask) {
        const uint32_t lane = threadIdx.x & 31U;
        const unsigned wanting = __ballot_sync(0xFFFFFFFFU, want);
        const int leader = __ffs(wanting) - 1;
        unsigned long long base = 0;
        if (static_cast<int>(lane) == leader) {
            base = atomicAdd(&w.counters[kCounterTraceCursor], static_cast<unsigned long long>(__popc(wanting)));
        }
        base = __shfl_sync(0xFFFFFFFFU, base, leader);
        done = base + __popc(wanting) >= count;
        const unsigned long long index = base + __popc(wanting & ((1U << lane) - 1U));
        if (!want || index >= count) {
            return false;
        }
        id = w.trace_queue[index];
        const float4 o4 = w.ray_o[id], d4 = w.ray_d[id];
        o = ld3(o4);
        d = ld3(d4);
        t_min = d4.w;
        t_max = o4.w;
        mask = w.mask[id];
        w.status[id] += 1U << 8;  // one extension segment
        return true;
    }
    __device__ __forceinline__ void ray(uint32_t id, F3& o, F3& d, uint32_t& mask) const {
        o = ld3(w.ray_o[id]);
        d = ld3(w.ray_d[id]);
        mask = w.mask[id];
    }
    __device__ __forceinline__ void finish(const SceneView&, uint32_t slot, const ClosestResult& c) const {
        if (c.failed) {
            w.status[slot] = (w.status[slot] & ~0xFFU) | kLaneTraversal;
            w.state[slot] = kSlotDone;
            return;
        }
        w.hit_id[slot] = make_uint2(c.instance, c.leaf);
        w.hit_tb[slot].x = c.t;
    }
};

template <bool SPH>
__global__ void __launch_bounds__(kPoolThreads, kPoolBlocks) k_trace(SceneView s, Wavefront w) {
    extern __shared__ uint32_t pool[];
    chain_begin();
    const uint32_t count = static_cast<uint32_t>(w.counters[kCounterTraced]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        w.counters[3] += count;  // extension segments
    }
    TraceJob job{w, count, count == 0U};
    pool_walk<false, SPH>(s, job, pool);
}

// ------------------------------------------------------------------------------------------------
// k_occlude: shadow rays of the compacted queue; unoccluded contributions join the path radiance
// ------------------------------------------------------------------------------------------------

template <bool ADJ>
struct OccludeJob {
    const Wavefront& w;
    const AdjointView& a;
    double* adjoint_sum;
    uint32_t count;
    bool done;

    __device__ __forceinline__ bool drained() const { return done; }
    __device__ __forceinline__ bool fetch(bool want, uint32_t& id, F3& o, F3& d, float& t_min, float& t_max,
                                          uint32_t& mask) {
        const uint32_t lane = threadIdx.x & 31U;
        const unsigned wanting = __ballot_sync(0xFFFFFFFFU, want);
        const int leader = __ffs(wanting) - 1;
        unsigned long long base = 0;
        if (static_cast<int>(lane) == leader) {
            base = atomicAdd(&w.counters[kCounterOccludeCursor], static_cast<unsigned long long>(__popc(wanting)));
        }
        base = __shfl_sync(0xFFFFFFFFU, base, leader);
        done = base + __popc(wanting) >= count;
        const unsigned long long index = base + __popc(wanting & ((1U << lane) - 1U));
        if (!want || index >= count) {
            return false;
        }
        id = w.shadow_queue[index];
        const float4 o4 = w.shadow_o[id];
        o = ld3(o4);
        d = ld3(w.shadow_d[id]);
        t_min = 0.0F;
        t_max = o4.w;
        mask = w.mask[id];
        return true;
    }
    __device__ __forceinline__ void ray(uint32_t id, F3& o, F3& d, uint32_t& mask) const {
        o = ld3(w.shadow_o[id]);
        d = ld3(w.shadow_d[id]);
        mask = w.mask[id];
    }
    __device__ __forceinline__ void finish(const SceneView&, uint32_t slot, int occluded) const {
        if (occluded < 0) {
            w.status[slot] = (w.status[slot] & ~0xFFU) | kLaneTraversal;
            w.state[slot] = kSlotDone;
            return;
        }
        if (occluded != 0) {
            return;
        }
        const float4 c = w.shadow_c[slot];
        float4 r = w.radiance[slot];
        r.x = r.x + c.x;
        r.y = r.y + c.y;
        r.z = r.z + c.z;
        r.w = r.w + c.w;
        w.radiance[slot] = r;
        if constexpr (ADJ) {
            const AdjointLane al = adjoint_lane(a, w.path_id[slot]);
            if (al.on) {  // the light's radiance scales this contribution; so may the roughness
                const float added[4] = {c.x, c.y, c.z, c.w};
                const double e = adjoint_dot(al, added);
                atomicAdd(&adjoint_sum[kAdjointEmission], e);
                const uint4 score = a.shadow_score[slot];
                if (score.w != 0U) {
                    atomicAdd(&adjoint_sum[score.z * kAdjointStride + 4U], e * __uint_as_float(score.x));
                    atomicAdd(&adjoint_sum[score.z * kAdjointStride + 5U], e * __uint_as_float(score.y));
                }
            }
        }
    }
};

template <bool ADJ, bool SPH>
__global__ void __launch_bounds__(kPoolThreads, kPoolBlocks) k_occlude(SceneView s, Wavefront w, AdjointView a) {
    extern __shared__ uint32_t pool[];
    chain_begin();
    __shared__ double adjoint_sum[ADJ ? kAdjointWords : 1];
    if constexpr (ADJ) {
        adjoint_zero(adjoint_sum);
    }
    const uint32_t count = w.shadow_offsets[1];
    OccludeJob<ADJ> job{w, a, adjoint_sum, count, count == 0U};
    pool_walk<true, SPH>(s, job, pool);
    if constexpr (ADJ) {
        adjoint_flush(adjoint_sum, a.gradients);
    }
}

// ------------------------------------------------------------------------------------------------
// Standalone closest-hit / occlusion queries (ClosestHit.hpp:21-28, Occlusion.hpp:19-26)
// ------------------------------------------------------------------------------------------------

// The rays of an array: every warp takes its own groups of 32, one in each round of all warps.
struct QueryRays {
    const bf200_ray_v1* rays;
    uint64_t n;
    uint64_t first, stride;  // the warp's next group, and the distance to the one after it
    uint32_t taken = 0U;     // rays of that group handed out

    __device__ __forceinline__ QueryRays(const bf200_ray_v1* r, uint64_t count) : rays(r), n(count) {
        first = (static_cast<uint64_t>(blockIdx.x) * (kPoolThreads / 32) + (threadIdx.x >> 5)) * 32U;
        stride = static_cast<uint64_t>(gridDim.x) * kPoolThreads;
    }
    __device__ __forceinline__ bool drained() const { return first >= n; }
    __device__ __forceinline__ bool fetch(bool want, uint32_t& id, F3& o, F3& d, float& t_min, float& t_max,
                                          uint32_t& mask) {
        const unsigned wanting = __ballot_sync(0xFFFFFFFFU, want);
        const uint32_t place = taken + __popc(wanting & ((1U << (threadIdx.x & 31U)) - 1U));
        const uint64_t index = place < 32U ? first + place : first + stride + (place - 32U);
        taken += __popc(wanting);
        if (taken >= 32U) {
            taken -= 32U;
            first += stride;
        }
        if (!want || index >= n) {
            return false;
        }
        id = static_cast<uint32_t>(index);
        const bf200_ray_v1& r = rays[index];
        o = F3{r.origin[0], r.origin[1], r.origin[2]};
        d = F3{r.direction[0], r.direction[1], r.direction[2]};
        t_min = r.t_min;
        t_max = r.t_max;
        mask = r.mask;
        return true;
    }
    __device__ __forceinline__ void ray(uint32_t id, F3& o, F3& d, uint32_t& mask) const {
        const bf200_ray_v1& r = rays[id];
        o = F3{r.origin[0], r.origin[1], r.origin[2]};
        d = F3{r.direction[0], r.direction[1], r.direction[2]};
        mask = r.mask;
    }
};

struct ClosestQuery : QueryRays {
    bf200_hit_v1* hits;
    __device__ __forceinline__ ClosestQuery(const bf200_ray_v1* r, uint64_t count, bf200_hit_v1* out)
        : QueryRays(r, count), hits(out) {}
    // the hit's t, instance and leaf record (as its primitive); k_query_hits completes it
    __device__ __forceinline__ void finish(const SceneView&, uint32_t id, const ClosestResult& c) const {
        bf200_hit_v1 h{};
        h.t = c.t;
        h.instance_index = c.failed ? 0xFFFFFFFFU : c.instance;
        h.primitive_index = c.leaf;
        h.status = c.failed ? kLaneTraversal : 0U;
        hits[id] = h;
    }
};

template <bool SPH>
__global__ void __launch_bounds__(128) k_query_hits(SceneView s, const bf200_ray_v1* rays, uint64_t n,
                                                    bf200_hit_v1* hits) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const bf200_hit_v1 walked = hits[i];
        bf200_hit_v1 h{};
        h.instance_index = 0xFFFFFFFFU;
        h.primitive_index = 0xFFFFFFFFU;
        h.status = walked.status;
        if (walked.instance_index != 0xFFFFFFFFU) {
            const bf200_ray_v1 r = rays[i];
            const ClosestResult c{walked.t, walked.instance_index, walked.primitive_index, false};
            TriangleHit th;
            if (hit_barycentrics<SPH>(s, c, F3{r.origin[0], r.origin[1], r.origin[2]},
                                      F3{r.direction[0], r.direction[1], r.direction[2]}, r.t_min, r.t_max, th)) {
                h.t = c.t;
                h.barycentrics[0] = th.b0;
                h.barycentrics[1] = th.b1;
                h.barycentrics[2] = th.b2;
                h.instance_index = c.instance;
                h.primitive_index = __float_as_uint(s.leaf_tris[3ULL * c.leaf].w);
            } else {
                h.status = kLaneNumerical;
            }
        }
        hits[i] = h;
    }
}

struct OcclusionQuery : QueryRays {
    uint32_t* out;
    __device__ __forceinline__ OcclusionQuery(const bf200_ray_v1* r, uint64_t count, uint32_t* o)
        : QueryRays(r, count), out(o) {}
    __device__ __forceinline__ void finish(const SceneView&, uint32_t id, int occluded) const {
        out[id] = occluded < 0 ? 2U : static_cast<uint32_t>(occluded);
    }
};

template <bool SPH>
__global__ void __launch_bounds__(kPoolThreads, kPoolBlocks) k_query_closest(SceneView s, const bf200_ray_v1* rays,
                                                                             uint64_t n, bf200_hit_v1* hits) {
    extern __shared__ uint32_t pool[];
    ClosestQuery job(rays, n, hits);
    pool_walk<false, SPH>(s, job, pool);
}

template <bool SPH>
__global__ void __launch_bounds__(kPoolThreads, kPoolBlocks) k_query_occlusion(SceneView s, const bf200_ray_v1* rays,
                                                                               uint64_t n, uint32_t* out) {
    extern __shared__ uint32_t pool[];
    OcclusionQuery job(rays, n, out);
    pool_walk<true, SPH>(s, job, pool);
}

// Launches a pool kernel over `rays` rays at most: one resident wave of blocks, or as many as give
// every lane a ray.
template <bool ANY, class... Params, class... Args>
cudaError_t launch_pool(void (*kernel)(Params...), uint64_t rays, cudaStream_t stream, bool chained, Args... args) {
    int device = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    }
    if (e == cudaSuccess) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kPoolSharedBytes<ANY>));
    }
    if (e != cudaSuccess) {
        return e;
    }
    const uint64_t wave = static_cast<uint64_t>(sms) * kPoolBlocks;
    const uint64_t need = (rays + kPoolThreads - 1U) / kPoolThreads;
    const uint32_t blocks = static_cast<uint32_t>(need < wave ? (need == 0U ? 1U : need) : wave);
    return launch_chained(kernel, blocks, static_cast<uint32_t>(kPoolThreads), kPoolSharedBytes<ANY>, stream, chained,
                          args...);
}

}  // namespace bf200
