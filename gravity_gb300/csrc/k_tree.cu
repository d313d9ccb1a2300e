// k_tree.cu — Karras LBVH build and single-pass bottom-up fill.
//
// Build: treeBuildBinaryRadixTreeKernel (SH/compute/tree/bh_tree.comp:43-133),
//   one thread per internal node, integer-exact.  It writes the topology into
//   compact arrays (children, counts, first slots, parents, arrival counters)
//   instead of the 80-byte nodes; the fill then writes every node whole, all
//   its words including the topology ones, so no sector of the node arrays is
//   written in part.  The stage entry point gbh_stage_build also writes the
//   reference's intermediate topology words into the nodes (k_build_nodes).
// Fill: treeInitLeafNodesKernel (bh_tree.comp:140-175) + 64 launches of
//   treePropagateNodesKernel (bh_tree.comp:183-259) become two kernels or three:
//   one warp per body group (a subtree of at most 96 bodies) initialises its
//   leaves and finishes its nodes; above the groups small trees are finished by
//   a block per subtree and one for the rest, larger ones by a thread per group
//   that climbs, where an atomic on an arrival counter lets the second child
//   finish a node (Karras 2012 / Apetrei 2014).  There is no pass limit, so trees taller
//   than 64 levels are filled completely, and the queue-reset race of the
//   reference (bh_tree.comp:188-193) does not exist.
#include "gbh_common.cuh"

// safeLCP, bh_tree.comp:20-37
__device__ __forceinline__ int safe_lcp(const uint64_t* __restrict__ keys, int n, int i, int j) {
    if (i < 0 || j < 0 || i >= n || j >= n) return -1;
    const uint64_t a = __ldg(keys + i), c = __ldg(keys + j);
    if (a == c) {
        const uint32_t x = (uint32_t)i ^ (uint32_t)j;
        return x == 0 ? 64 : 64 + __clz(x);
    }
    return __clzll(a ^ c);
}

// Body groups of the group walks: the subtrees of at most GBH_GROUP_MAX
// bodies whose parent holds more (every leaf lies in exactly one), as (first
// sorted slot, body count).  A group is a contiguous range of sorted slots,
// spatially compact because it is one tree node.  The build lists them: node
// i knows its children's ranges, so an internal node with more than
// GBH_GROUP_MAX bodies emits each child that holds at most that many; one
// counter update per warp.
__device__ __forceinline__ void emit_groups(const StepBuffers& b, uint32_t k, const uint2 (&mine)[2],
                                            const uint32_t (&node)[2]) {
    const uint32_t one = __ballot_sync(0xffffffffu, k > 0), two = __ballot_sync(0xffffffffu, k > 1);
    if (!one) return;
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(&b.st->num_groups, (uint32_t)(__popc(one) + __popc(two)));
    base = __shfl_sync(0xffffffffu, base, 0);
    const uint32_t first = base + __popc(one & lanemask_lt()) + __popc(two & lanemask_lt());
    for (uint32_t q = 0; q < k; ++q) {
        b.groups[first + q] = mine[q];
        b.group_node[first + q] = node[q];
    }
}

// bodies in a subtree that one block of k_fill_above fills above its groups;
// the largest capacity filled that way
#define FILL_SUBTREE 4096u
#define FILL_ABOVE_MAX 131072u

__global__ __launch_bounds__(256) void k_build(StepBuffers b) {
    const uint32_t n = b.st->n_new;
    const uint32_t N = b.N;
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t* keys = b.keys_in;
    if (gid == 0) b.st->group_next = 0;  // the group walk's ticket
    if (n <= 1) {
        if (n == 1 && gid == 0) {
            // single body, bh_tree.comp:46-62: root with one child, bodiesContained 0,
            // readyChildren 1
            b.topo_kids[0] = make_uint2(0u, GBH_NONE);
            b.topo_cnt[0] = 0;
            b.node_lo[0] = 0;
            b.fill_ready[0] = 1;
            b.parent_int[0] = GBH_NONE;
            b.parent_leaf[0] = N;
            b.groups[0] = make_uint2(0u, 1u);
            b.group_node[0] = N;
            b.st->num_groups = 1;
        }
        return;
    }
    // every lane of a warp reaches the group list below
    uint2 mine[2];
    uint32_t mine_node[2] = {0u, 0u};
    uint32_t k = 0;
    uint32_t bodies = 0, kid[2] = {0u, 0u}, kid_bodies[2] = {0u, 0u};
    if (gid < n - 1) {
    const int i = (int)gid, ni = (int)n;
    const uint64_t ki = keys[i];
    const int lcp_r = safe_lcp(keys, ni, i, i + 1);
    const int lcp_l = safe_lcp(keys, ni, i, i - 1);
    const int d = (lcp_l > lcp_r) ? -1 : 1;
    // The searches ask whether lcp(i, j) > delta for a fixed delta: j lies in
    // the range and the first delta + 1 bits of (key, index) agree with i's.
    // As a mask that is 4 instructions where the prefix length itself takes a
    // dozen; a warp runs as long as its longest search, about 40 probes.
    // Build stage at 16.8M bodies (with the start lists, 0.07): 0.53 -> 0.42 ms;
    // 4.2M bodies without them 0.128 -> 0.096.
    auto longer_than = [&](int delta) {
        const int bits = delta + 1;
        const uint64_t key_mask = bits >= 64 ? ~0ull : bits <= 0 ? 0ull : ~0ull << (64 - bits);
        const uint32_t idx_mask = bits <= 64 ? 0u : bits >= 96 ? ~0u : ~0u << (96 - bits);
        return [=](int j) {
            return (uint32_t)j < (uint32_t)ni && ((ki ^ keys[j]) & key_mask) == 0ull && (((uint32_t)i ^ (uint32_t)j) & idx_mask) == 0u;
        };
    };
    const auto beyond = longer_than(min(lcp_r, lcp_l));
    int lmax = 2;
    while (beyond(i + d * lmax)) lmax *= 2;
    int l = 0;
    for (int t = lmax >> 1; t > 0; t >>= 1)
        if (beyond(i + d * (l + t))) l += t;
    const int j = i + l * d;
    const auto within = longer_than(safe_lcp(keys, ni, i, j));
    int s = 0;
    int t = l;
    while (t > 1) {
        t = (t + 1) >> 1;
        if (within(i + (s + t) * d)) s += t;
    }
    const int gamma = i + s * d + min(d, 0);
    const int mn = min(i, j), mx = max(i, j);
    const uint32_t left = (mn == gamma) ? (uint32_t)gamma : (uint32_t)gamma + N;
    const uint32_t right = (mx == gamma + 1) ? (uint32_t)(gamma + 1) : (uint32_t)(gamma + 1) + N;
    b.topo_kids[i] = make_uint2(left, right);
    b.node_lo[i] = (uint32_t)mn;
    b.topo_cnt[i] = (uint32_t)(mx - mn + 1);
    b.fill_ready[i] = 0;
    const uint32_t self = (uint32_t)i + N;
    if (left < N) b.parent_leaf[left] = self; else b.parent_int[left - N] = self;
    if (right < N) b.parent_leaf[right] = self; else b.parent_int[right - N] = self;
    if (i == 0) b.parent_int[0] = GBH_NONE;
    const uint32_t cnt = (uint32_t)(mx - mn + 1);
    if (cnt > GBH_GROUP_MAX) {
        const uint32_t cl = (uint32_t)(gamma - mn + 1), cr = (uint32_t)(mx - gamma);
        bodies = cnt;
        kid[0] = left - N;
        kid[1] = right - N;
        kid_bodies[0] = cl;
        kid_bodies[1] = cr;
        if (cl <= GBH_GROUP_MAX) {
            mine_node[k] = left;
            mine[k++] = make_uint2((uint32_t)mn, cl);
        }
        if (cr <= GBH_GROUP_MAX) {
            mine_node[k] = right;
            mine[k++] = make_uint2((uint32_t)gamma + 1u, cr);
        }
    } else if (i == 0) {
        mine_node[k] = N;
        mine[k++] = make_uint2(0u, cnt);  // the whole tree is one group
    }
    }
    emit_groups(b, k, mine, mine_node);
    // the subtrees whose nodes above the groups a block fills, and the nodes
    // above the subtrees (k_fill_above): rare
    if (N <= FILL_ABOVE_MAX) {
        if (bodies > FILL_SUBTREE) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (kid_bodies[q] > GBH_GROUP_MAX && kid_bodies[q] <= FILL_SUBTREE)
                    b.fill_subtrees[0][atomicAdd(&b.st->num_subtrees[0], 1u)] = kid[q];
            b.fill_subtrees[1][atomicAdd(&b.st->num_subtrees[1], 1u)] = gid;
        } else if (gid == 0 && bodies > 0) {
            b.fill_subtrees[0][atomicAdd(&b.st->num_subtrees[0], 1u)] = 0u;  // the whole tree
        }
    }
}

// The reference's Node topology words after buildBinaryRadixTree (childA/B,
// nodeDepth = min(i, j), bodiesContained, readyChildren = 0, parentId; leaves:
// parentId), for the stage-level API.
__global__ void k_build_nodes(StepBuffers b) {
    const uint32_t n = b.st->n_new;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (n == 0) return;
    const uint32_t ni = n > 1 ? n - 1 : 1;
    if (t < ni) {
        gbh_node* nd = &b.internal[t];
        const uint2 k = b.topo_kids[t];
        nd->child_a = k.x;
        nd->child_b = k.y;
        nd->node_depth = b.node_lo[t];
        nd->bodies_contained = b.topo_cnt[t];
        nd->ready_children = b.fill_ready[t];
        nd->parent_id = b.parent_int[t];
    }
    if (t < n) b.leaf[t].parent_id = b.parent_leaf[t];
}

void launch_build_nodes(const StepBuffers& b, cudaStream_t s) {
    k_build_nodes<<<(b.N + 255) / 256, 256, 0, s>>>(b);
}

#define PATHS_THREADS 128  // one block fits on an SM beside k_fill's five (4,096 registers left)

// Where each group's walk starts: the group's own subtree and the sibling of
// every ancestor of it, which together hold every body once.  A walk from the
// root opens each ancestor of the group anyway (its box holds the group's
// bodies), one level per round of candidates; starting from this list gives
// the same accepted and listed nodes without those rounds.  One thread per
// group climbs the parent links; a group deeper than GBH_PATH_WORDS - 2
// levels, or past the list's capacity, starts from the root (count 0).
__global__ __launch_bounds__(PATHS_THREADS) void k_group_paths(StepBuffers b) {
    const uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t ng = min(b.st->num_groups, b.group_path_cap);
    if (gi >= ng) return;
    const uint32_t N = b.N, root = N;
    uint32_t* out = b.group_path + (size_t)gi * GBH_PATH_WORDS;
    uint32_t node = b.group_node[gi];
    uint32_t len = 0;
    out[1 + len++] = node;
    while (node != root && len < GBH_PATH_WORDS - 1) {
        const uint32_t p = node < N ? b.parent_leaf[node] : b.parent_int[node - N];
        if (p < N || p - N >= N) {  // not an internal node: leave the group to the root start
            len = 0;
            break;
        }
        const uint2 kids = b.topo_kids[p - N];
        out[1 + len++] = kids.x == node ? kids.y : kids.x;
        node = p;
    }
    if (node != root) len = 0;
    out[0] = len;
}

void launch_group_paths(const StepBuffers& b, cudaStream_t s) {
    // the groups of the step are counted on the device: enough threads for
    // the list's capacity, the surplus returns at once
    const uint32_t threads = min(b.N, b.group_path_cap);
    k_group_paths<<<(threads + PATHS_THREADS - 1) / PATHS_THREADS, PATHS_THREADS, 0, s>>>(b);
}

void launch_build(const StepBuffers& b, cudaStream_t s) {
    const uint32_t nodes = b.N > 1 ? b.N - 1 : 1;
    k_build<<<(nodes + 255) / 256, 256, 0, s>>>(b);
}

// ---------------------------------------------------------------------------
// getStarColor, common.glsl:232-276
__device__ __noinline__ float3 star_color_hot(float mass, float density) {
    const float e = 0.875f - 1.0f / 6.0f;
    float t = 5.95589e-19f * powf(mass, e);
    t = t * powf(density, 1.0f / 6.0f);
    const float temp = t / 100.0f;
    float r, g, bl;
    if (temp <= 66.0f) {
        r = 255.0f;
    } else {
        r = 329.698727446f * powf(temp - 60.0f, -0.1332047592f);
    }
    if (temp <= 66.0f) {
        g = 99.4708025861f * logf(gmax(temp, 1e-3f)) - 161.1195681661f;
    } else {
        g = 288.1221695283f * powf(temp, -0.0755148492f);
    }
    if (temp >= 66.0f) {
        bl = 255.0f;
    } else {
        bl = 138.5177312231f * logf(gmax(temp - 10.0f, 1e-3f)) - 305.0447927307f;
    }
    return make_float3(gclamp(r, 0.0f, 255.0f) / 255.0f, gclamp(g, 0.0f, 255.0f) / 255.0f,
                       gclamp(bl, 0.0f, 255.0f) / 255.0f);
}

__device__ __forceinline__ float3 star_color(float mass, float density) {
    // below these bounds the temperature is at most 0.23: red saturates and
    // both logarithms are negative before their clamps, so the colour is
    // exactly (1, 0, 0)
    if (mass <= 1e22f && density <= 1e24f) return make_float3(1.0f, 0.0f, 0.0f);
    return star_color_hot(mass, density);
}

// out of line: the fill's code has to stay in the instruction cache
__device__ __noinline__ float fill_radius(float body_len_const, float m, float rho) {
    return body_radius(body_len_const, m, rho);
}

struct NodeVals {
    float4 cm;
    float box[6];
    float4 col;
    uint32_t depth;
};

// L2-coherent read of the fields of a node written by another thread of this kernel
__device__ __forceinline__ NodeVals load_node_cg(const gbh_node* nd) {
    NodeVals v;
    const float4* p = reinterpret_cast<const float4*>(nd);
    v.cm = __ldcg(p + 0);
    const float4 a = __ldcg(p + 1);
    const float2 c = __ldcg(reinterpret_cast<const float2*>(p + 2));  // aabb4, aabb5
    v.depth = __ldcg(reinterpret_cast<const uint32_t*>(p + 3));
    v.col = __ldcg(p + 4);
    v.box[0] = a.x;
    v.box[1] = a.y;
    v.box[2] = a.z;
    v.box[3] = a.w;
    v.box[4] = c.x;
    v.box[5] = c.y;
    return v;
}

// the fields of a finished node
__device__ __forceinline__ NodeVals load_node(const gbh_node* nd) {
    NodeVals v;
    const float4* p = reinterpret_cast<const float4*>(nd);
    v.cm = p[0];
    const float4 a = p[1];
    const float2 c = *reinterpret_cast<const float2*>(p + 2);  // aabb4, aabb5
    v.depth = *reinterpret_cast<const uint32_t*>(p + 3);
    v.col = p[4];
    v.box[0] = a.x;
    v.box[1] = a.y;
    v.box[2] = a.z;
    v.box[3] = a.w;
    v.box[4] = c.x;
    v.box[5] = c.y;
    return v;
}

__device__ __forceinline__ float half_side(const float box[6]) {
    const float ex = box[3] - box[0], ey = box[4] - box[1], ez = box[5] - box[2];
    return gmax(ex, gmax(ey, ez)) / 2.0f;
}

__device__ __forceinline__ WalkRec make_rec(const NodeVals& v, uint32_t id, uint32_t count, bool leaf) {
    WalkRec r;
    r.cm = v.cm;
    r.half_side = leaf ? 0.0f : half_side(v.box);
    r.id = id;
    r.count = count;
    r.pad = 0;
    return r;
}

// a / m, correctly rounded, from inv = 1 / m correctly rounded (Markstein 1990):
// a quotient within one unit in the last place, corrected by its exact
// remainder times the correctly rounded reciprocal, rounds as a / m does.  The
// first correction brings the product a inv within that unit, the second
// applies the theorem.  Holds where the quotient is a normal number away from
// the largest and no remainder underflows: see div3.
__device__ __forceinline__ float div_by(float a, float m, float inv) {
    float q = a * inv;
    q = __fmaf_rn(__fmaf_rn(-q, m, a), inv, q);
    return __fmaf_rn(__fmaf_rn(-q, m, a), inv, q);
}

__device__ __noinline__ float3 div3_slow(float x, float y, float z, float m) {
    return make_float3(x / m, y / m, z / m);
}

// (x, y, z) / m as IEEE divisions.  One reciprocal serves the three: a node's
// centre of mass is a link of the fill's dependent chain, and three separate
// divisions take most of its instructions.
__device__ __forceinline__ void div3(float x, float y, float z, float m, float inv, float4& out) {
    const float lo = fminf(fabsf(x), fminf(fabsf(y), fabsf(z))), hi = fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z)));
    // numerators in [2^-80, 2^80] and m in [2^-60, 2^60]: remainders (above
    // 2^-128) stay normal; quotients in [2^-125, 2^126] by the bounds with m,
    // which are exact where they decide (a subnormal quotient is rounded twice,
    // and beside the largest number a inv overflows first).  NaN and zeros
    // divide below.
    if (lo >= 8.2718061e-25f && hi <= 1.2089258e24f && m >= 8.6736174e-19f && m <= 1.1529215e18f &&
        lo >= m * 2.3509887e-38f && hi <= m * 8.5070592e37f) {
        out.x = div_by(x, m, inv);
        out.y = div_by(y, m, inv);
        out.z = div_by(z, m, inv);
    } else {
        const float3 v = div3_slow(x, y, z, m);
        out.x = v.x;
        out.y = v.y;
        out.z = v.z;
    }
}

// One internal node from its two children (bh_tree.comp:223-246); L is
// childA's values, R childB's.
__device__ __forceinline__ NodeVals combine(const NodeVals& L, const NodeVals& R) {
    const float lw = L.cm.w, rw = R.cm.w;
    const float M = lw + rw;
    NodeVals out;
    if (M > 0.0f) {
        const float inv_m = 1.0f / M;
        div3(lw * L.cm.x + rw * R.cm.x, lw * L.cm.y + rw * R.cm.y, lw * L.cm.z + rw * R.cm.z, M, inv_m, out.cm);
        // the colour (render-only, compared with a tolerance) by the reciprocal
        out.col.x = (lw * L.col.x + rw * R.col.x) * inv_m;
        out.col.y = (lw * L.col.y + rw * R.col.y) * inv_m;
        out.col.z = (lw * L.col.z + rw * R.col.z) * inv_m;
    } else {
        out.cm.x = (L.cm.x + R.cm.x) * 0.5f;
        out.cm.y = (L.cm.y + R.cm.y) * 0.5f;
        out.cm.z = (L.cm.z + R.cm.z) * 0.5f;
        out.col.x = (L.col.x + R.col.x) * 0.5f;
        out.col.y = (L.col.y + R.col.y) * 0.5f;
        out.col.z = (L.col.z + R.col.z) * 0.5f;
    }
    out.cm.w = M;
    out.col.w = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        out.box[k] = gmin(L.box[k], R.box[k]);
        out.box[3 + k] = gmax(L.box[3 + k], R.box[3 + k]);
    }
    out.depth = 1u + max(L.depth, R.depth);
    return out;
}

// Write a finished internal node whole: its Node words (reference layout,
// common.glsl:40-58) including the topology ones, readyChildren claimed
// (0xFFFFFFFF, bh_tree.comp:200), and, for the plain walk, the walk records
// of its two children.
__device__ __forceinline__ void store_internal(const StepBuffers& b, uint32_t i, const NodeVals& out, const NodeVals& L,
                                               const NodeVals& R, uint32_t a_id, uint32_t b_id, uint32_t a_count,
                                               uint32_t b_count, uint32_t bodies, uint32_t parent) {
    float4* np = reinterpret_cast<float4*>(&b.internal[i]);
    __stcg(np + 0, out.cm);
    __stcg(np + 1, make_float4(out.box[0], out.box[1], out.box[2], out.box[3]));
    __stcg(reinterpret_cast<uint4*>(np + 2), make_uint4(__float_as_uint(out.box[4]), __float_as_uint(out.box[5]), a_id, b_id));
    __stcg(reinterpret_cast<uint4*>(np + 3), make_uint4(out.depth, bodies, GBH_NONE, parent));
    __stcg(np + 4, out.col);
    // the children's walk records feed the plain walk only
    if (b.params->mac_mode == GBH_MAC_PLAIN) {
        ChildPair pr;
        pr.a = make_rec(L, a_id, a_count, a_id < b.N);
        pr.b = make_rec(R, b_id, b_count, b_id < b.N);
        b.pairs[i] = pr;
    }
}

// Values of a group's leaves and finished nodes in shared memory.
struct FillSmem {
    float4 leaf_cm[GBH_GROUP_MAX];
    float4 leaf_col[GBH_GROUP_MAX];     // rgb; w: the parent's id
    float4 node_cm[GBH_GROUP_MAX];
    float4 node_box03[GBH_GROUP_MAX];
    float4 node_box45[GBH_GROUP_MAX];   // aabb[4..5], height, bodies
    float4 node_col[GBH_GROUP_MAX];     // rgb; w: the parent's id
    uint8_t kid_a[GBH_GROUP_MAX];       // children: slot in the group, + FILL_NODE for a node
    uint8_t kid_b[GBH_GROUP_MAX];
    uint8_t list[GBH_GROUP_MAX];        // nodes to finish in this round
};
#define FILL_NODE 128u
#define FILL_WARPS 4
#define FILL_THREADS (32 * FILL_WARPS)
#define FILL_SLOTS (GBH_GROUP_MAX / 32)
#define FILL_BLOCKS 5  // resident blocks per SM
static_assert(GBH_GROUP_MAX == 96, "the masks of a group's nodes below are three words");

__device__ __forceinline__ NodeVals fill_vals(const FillSmem& S, uint32_t kid) {
    NodeVals v;
    if (kid < FILL_NODE) {
        v.cm = S.leaf_cm[kid];
        v.col = S.leaf_col[kid];
        v.box[0] = v.box[3] = v.cm.x;
        v.box[1] = v.box[4] = v.cm.y;
        v.box[2] = v.box[5] = v.cm.z;
        v.depth = 0;
    } else {
        const uint32_t t = kid - FILL_NODE;
        v.cm = S.node_cm[t];
        v.col = S.node_col[t];
        const float4 a = S.node_box03[t], c = S.node_box45[t];
        v.box[0] = a.x;
        v.box[1] = a.y;
        v.box[2] = a.z;
        v.box[3] = a.w;
        v.box[4] = c.x;
        v.box[5] = c.y;
        v.depth = __float_as_uint(c.z);
    }
    return v;
}

// Fill of the body groups, one warp each (persistent: each warp takes every
// W-th group).  A group is a subtree, so no node of it depends on another
// warp, and the nodes above the groups (one per group) are left to k_fill_above
// or k_fill_top.
//   1. Every lane initialises its leaves and keeps their values in shared
//      memory, beside its nodes' children.
//   2. Rounds: the nodes whose children are finished (masks of finished
//      nodes, held by every lane) are listed and finished by consecutive lanes.
//   3. The warp writes the group's leaf and internal nodes, consecutive lanes
//      consecutive 16-byte words.
// The arithmetic of a node depends only on its two children, so the result is
// the same in any schedule.
//
// What bounds it: each round is a dependent chain (children's words, three
// divisions by one mass, store) of a few lanes, about 10 rounds per group, and
// before them a gather of the bodies through the index.  So the work of
// different groups has to overlap: 20 warps per SM (5 blocks of 4 warps at 96
// registers and 40 KB; 4 or 3 blocks: 2.14 and 2.63 ms), all loads of a group
// issued together and the next group's ids loaded during the rounds (1.84 ->
// 1.43 ms).  A subtree per warp needs no block barrier and leaves 1.7% of the
// nodes to k_fill_top, where tiles of 64 or 512 consecutive slots leave 9% or
// 2%, in chains as long as the tree is high.  Unrolling the output loops
// overflows the instruction cache (1.58 ms); so do the star colour and the
// plain divisions inlined.
// Fill stage, ms, before (512-slot tiles, threads climbing from their leaves)
// and after: 16,777,216-body mixture 1.99 -> 1.43; 8,388,608 bodies in clusters 1.12 -> 0.78; 4,194,301
// bodies with the plain walk's records 0.63 -> 0.46; 65,536 bodies 0.094 -> 0.070 (0.059 with
// k_fill_above).
__global__ __launch_bounds__(FILL_THREADS, FILL_BLOCKS) void k_fill(StepBuffers b) {
    extern __shared__ __align__(16) unsigned char fill_smem[];
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    FillSmem& S = reinterpret_cast<FillSmem*>(fill_smem)[w];
    const uint32_t n = b.st->n_new;
    const uint32_t N = b.N;
    if (n == 0) return;
    const gbh_sim_values* sim = b.sim;
    const uint32_t groups = b.st->num_groups;
    const bool radii = b.params->merging_collision_or_neither != GBH_MODE_NEITHER;
    const bool pairs = b.params->mac_mode == GBH_MAC_PLAIN;
    const uint32_t stride = gridDim.x * FILL_WARPS;
    uint32_t gi = blockIdx.x * FILL_WARPS + w;
    // one group ahead: its range, and (from the rounds on) its body ids
    uint2 grp = gi < groups ? b.groups[gi] : make_uint2(0u, 0u);
    uint32_t bi[FILL_SLOTS];
#pragma unroll
    for (int q = 0; q < FILL_SLOTS; ++q) bi[q] = lane + 32 * q < grp.y ? b.idx_in[grp.x + lane + 32 * q] : 0u;
    for (; gi < groups; gi += stride) {
        const uint32_t base = grp.x, count = grp.y;
        // every load of the group at once: bodies, topology (written by the build)
        float4 pm[FILL_SLOTS];
        float density[FILL_SLOTS];
        uint2 kids[FILL_SLOTS];
        uint32_t first[FILL_SLOTS], bodies[FILL_SLOTS], parent[FILL_SLOTS], leaf_parent[FILL_SLOTS];
#pragma unroll
        for (int q = 0; q < FILL_SLOTS; ++q) {
            const uint32_t t = lane + 32 * q, g = base + t;
            pm[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            density[q] = 0.0f;
            kids[q] = make_uint2(0u, 0u);
            first[q] = bodies[q] = parent[q] = leaf_parent[q] = 0u;
            if (t < count) {
                pm[q] = ld_pos_mass(b.bodies_in, bi[q]);
                density[q] = b.bodies_in[bi[q]].vel_density[3];
                leaf_parent[q] = b.parent_leaf[g];
                if (g + 1 < n) {
                    kids[q] = b.topo_kids[g];
                    first[q] = b.node_lo[g];
                    bodies[q] = b.topo_cnt[g];
                    parent[q] = b.parent_int[g];
                }
            }
        }
        grp = gi + stride < groups ? b.groups[gi + stride] : make_uint2(0u, 0u);
        uint32_t in_mask[FILL_SLOTS], done[FILL_SLOTS], need[FILL_SLOTS][FILL_SLOTS];
        __syncwarp();  // the last group's words are written out
#pragma unroll
        for (int q = 0; q < FILL_SLOTS; ++q) {
            // internal node g is inside the group, or (at most one index) an
            // ancestor of it
            const uint32_t t = lane + 32 * q;
            in_mask[q] = done[q] = 0u;
            if (32u * q >= count) continue;  // (uniform) no bodies in this slot
            const bool inside = t < count && base + t + 1 < n && first[q] >= base && first[q] + bodies[q] <= base + count;
#pragma unroll
            for (int k = 0; k < FILL_SLOTS; ++k) need[q][k] = 0u;
            if (inside) {
                const bool a_leaf = kids[q].x < N, c_leaf = kids[q].y < N;
                const uint32_t a = kids[q].x - base - (a_leaf ? 0u : N), c = kids[q].y - base - (c_leaf ? 0u : N);
                S.kid_a[t] = (uint8_t)(a_leaf ? a : a + FILL_NODE);
                S.kid_b[t] = (uint8_t)(c_leaf ? c : c + FILL_NODE);
                S.node_box45[t].w = __uint_as_float(bodies[q]);
                S.node_col[t].w = __uint_as_float(parent[q]);
#pragma unroll
                for (int k = 0; k < FILL_SLOTS; ++k) {
                    if (!a_leaf && a / 32 == k) need[q][k] |= 1u << (a & 31u);
                    if (!c_leaf && c / 32 == k) need[q][k] |= 1u << (c & 31u);
                }
            }
            in_mask[q] = __ballot_sync(0xffffffffu, inside);
            if (t >= count) continue;
            // leaf init, bh_tree.comp:153-166
            const uint32_t g = base + t;
            float3 rgb = make_float3(0.0f, 0.0f, 0.0f);
            if (pm[q].w > 0.0f && density[q] > 0.0f)
                rgb = star_color(pm[q].w * sim->unit_mass, density[q] * sim->unit_density);
            S.leaf_cm[t] = pm[q];
            S.leaf_col[t] = make_float4(rgb.x, rgb.y, rgb.z, __uint_as_float(leaf_parent[q]));
            b.leaf_pm[g] = pm[q];
            if (radii) b.leaf_rad[g] = fill_radius(sim->body_length_constant, pm[q].w, density[q]);
            if (b.prec) {
                // precision form: the FP32 residual of the FP64 position
                const double2 xy = reinterpret_cast<const double2*>(b.pos64_in)[2 * (size_t)bi[q]];
                const double z = b.pos64_in[4 * (size_t)bi[q] + 2];
                b.leaf_lo[g] = make_float4((float)(xy.x - (double)pm[q].x), (float)(xy.y - (double)pm[q].y),
                                           (float)(z - (double)pm[q].z), 0.0f);
            }
        }
#pragma unroll
        for (int q = 0; q < FILL_SLOTS; ++q) bi[q] = lane + 32 * q < grp.y ? b.idx_in[grp.x + lane + 32 * q] : 0u;
        for (;;) {
            uint32_t m[FILL_SLOTS], c = 0;
#pragma unroll
            for (int q = 0; q < FILL_SLOTS; ++q) {
                m[q] = 0u;
                if (in_mask[q] == done[q]) continue;  // (uniform) nothing left in this slot
                bool ready = ((in_mask[q] & ~done[q]) >> lane) & 1u;
#pragma unroll
                for (int k = 0; k < FILL_SLOTS; ++k) ready = ready && (done[k] & need[q][k]) == need[q][k];
                m[q] = __ballot_sync(0xffffffffu, ready);
                if (ready) S.list[c + __popc(m[q] & lanemask_lt())] = (uint8_t)(lane + 32 * q);
                c += __popc(m[q]);
            }
            __syncwarp();
            if (!c) break;
            for (uint32_t k = lane; k < c; k += 32) {
                const uint32_t i = S.list[k];
                const NodeVals out = combine(fill_vals(S, S.kid_a[i]), fill_vals(S, S.kid_b[i]));
                S.node_cm[i] = out.cm;
                S.node_box03[i] = make_float4(out.box[0], out.box[1], out.box[2], out.box[3]);
                S.node_box45[i].x = out.box[4];
                S.node_box45[i].y = out.box[5];
                S.node_box45[i].z = __uint_as_float(out.depth);
                S.node_col[i].x = out.col.x;
                S.node_col[i].y = out.col.y;
                S.node_col[i].z = out.col.z;
            }
#pragma unroll
            for (int q = 0; q < FILL_SLOTS; ++q) done[q] |= m[q];
            __syncwarp();
        }
        // the whole tree is one group: its root is finished here
        if (n > 1 && count == n) {
            for (uint32_t i = lane; i < n - 1; i += 32)
                if (__float_as_uint(S.node_col[i].w) == GBH_NONE) {
                    const NodeVals out = fill_vals(S, i + FILL_NODE);
                    b.st->tree_height = out.depth;
                    *b.root_rec = make_rec(out, base + i + N, n, false);
                }
        }

        // the group's nodes, whole: Node words (reference layout,
        // common.glsl:40-58) including the topology ones, readyChildren claimed
        // (0xFFFFFFFF, bh_tree.comp:200)
        float4* leaf_words = reinterpret_cast<float4*>(b.leaf + base);
        float4* node_words = reinterpret_cast<float4*>(b.internal + base);
        const float none = __uint_as_float(GBH_NONE);
        auto id_of = [&](uint32_t kid) { return kid < FILL_NODE ? base + kid : base + kid - FILL_NODE + N; };
        const uint32_t in0 = in_mask[0], in1 = in_mask[1], in2 = in_mask[2];
        auto is_in = [=](uint32_t i) { return ((i < 32 ? in0 : i < 64 ? in1 : in2) >> (i & 31u)) & 1u; };
#pragma unroll 1
        for (uint32_t q = lane; q < 5 * count; q += 32) {
            const uint32_t i = q / 5, part = q - 5 * i;
            float4 v = (part < 3 ? S.leaf_cm : S.leaf_col)[i];
            if (part == 1) v.w = v.x;
            if (part == 2) v = make_float4(v.y, v.z, none, none);
            if (part == 3) v = make_float4(0.0f, 0.0f, none, v.w);
            if (part == 4) v.w = 0.0f;
            leaf_words[q] = v;
            if (is_in(i)) {
                const float4* words = part == 0 ? S.node_cm : part == 1 ? S.node_box03 : part == 4 ? S.node_col : S.node_box45;
                float4 x = words[i];
                if (part == 2) x = make_float4(x.x, x.y, __uint_as_float(id_of(S.kid_a[i])), __uint_as_float(id_of(S.kid_b[i])));
                if (part == 3) x = make_float4(x.z, x.w, none, S.node_col[i].w);
                if (part == 4) x.w = 0.0f;
                node_words[q] = x;
            }
        }
        // the children's walk records feed the plain walk only
        if (pairs) {
            float4* pair_words = reinterpret_cast<float4*>(b.pairs + base);
#pragma unroll 1
            for (uint32_t q = lane; q < 4 * count; q += 32) {
                const uint32_t i = q >> 2;
                if (!is_in(i)) continue;
                const uint32_t kid = (q & 2u) ? S.kid_b[i] : S.kid_a[i];
                const bool leaf = kid < FILL_NODE;
                float4 v = leaf ? S.leaf_cm[kid] : S.node_cm[kid - FILL_NODE];
                if (q & 1u) {
                    float half = 0.0f, bodies = __uint_as_float(1u);
                    if (!leaf) {
                        const float4 b03 = S.node_box03[kid - FILL_NODE], b45 = S.node_box45[kid - FILL_NODE];
                        const float box[6] = {b03.x, b03.y, b03.z, b03.w, b45.x, b45.y};
                        half = half_side(box);
                        bodies = b45.w;
                    }
                    v = make_float4(half, __uint_as_float(id_of(kid)), bodies, 0.0f);
                }
                pair_words[q] = v;
            }
        }
    }
}

// Climb from node `self` (values `own`, `self_count` bodies) through the
// global counters readyChildren (release/acquire at GPU scope): the second
// arriving child reads its sibling from L2 and finishes the node.
__device__ void climb_global(const StepBuffers& b, uint32_t self, uint32_t self_count, NodeVals own,
                             uint32_t node) {
    const uint32_t N = b.N;
    while (node != GBH_NONE) {
        const uint32_t i = node - N;
        // the topology does not depend on the count: loaded beside it
        const uint2 kids = b.topo_kids[i];
        const uint32_t bodies = b.topo_cnt[i];
        const uint32_t parent = b.parent_int[i];
        // release: own node's writes before the count; acquire: the sibling's writes after it
        const uint32_t old = atomic_add_acq_rel(&b.fill_ready[i], 1u);
        if (old == 0u) return;
        const bool self_is_a = kids.x == self;
        const uint32_t sib = self_is_a ? kids.y : kids.x;
        NodeVals S;
        uint32_t sib_count = bodies - self_count;
        if (sib == GBH_NONE) {  // single-body tree: the missing child contributes nothing
            S.cm = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            S.col = S.cm;
            S.box[0] = S.box[1] = S.box[2] = 1e38f;
            S.box[3] = S.box[4] = S.box[5] = -1e38f;
            S.depth = 0;
            sib_count = 0;
        } else {
            S = load_node_cg(sib < N ? &b.leaf[sib] : &b.internal[sib - N]);
        }
        const NodeVals& L = self_is_a ? own : S;
        const NodeVals& R = self_is_a ? S : own;
        const NodeVals out = combine(L, R);
        const uint32_t a_id = self_is_a ? self : sib, b_id = self_is_a ? sib : self;
        store_internal(b, i, out, L, R, a_id, b_id, self_is_a ? self_count : sib_count,
                       self_is_a ? sib_count : self_count, bodies, parent);
        self = node;
        self_count = self_count + sib_count;
        own = out;
        if (parent == GBH_NONE) {
            b.st->tree_height = out.depth;
            *b.root_rec = make_rec(out, node, self_count, false);
            return;
        }
        node = parent;
    }
}

// Fill of the nodes above the body groups, capacities above FILL_ABOVE_MAX: one
// thread per group climbs from its subtree's root.
__global__ __launch_bounds__(256) void k_fill_top(StepBuffers b) {
    const uint32_t groups = b.st->num_groups;
    const uint32_t N = b.N;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < groups; e += gridDim.x * blockDim.x) {
        const uint32_t id = b.group_node[e];
        const gbh_node* nd = id < N ? &b.leaf[id] : &b.internal[id - N];
        const uint32_t parent = id < N ? b.parent_leaf[id] : b.parent_int[id - N];
        // a single body's group is named by the root, whose one child it is
        if (b.st->n_new == 1)
            climb_global(b, 0u, 1u, load_node_cg(&b.leaf[0]), N);
        else if (parent != GBH_NONE)
            climb_global(b, id, b.groups[e].y, load_node_cg(nd), parent);
    }
}

// An internal node above the groups, with what its finishing needs.
struct AboveNode {
    uint32_t id, first, bodies, parent, left, right;  // left, right: the children's bodies
    uint2 kids;
};

__device__ __forceinline__ AboveNode above_node(const StepBuffers& b, uint32_t i) {
    AboveNode a;
    a.id = i;
    a.kids = b.topo_kids[i];
    a.first = b.node_lo[i];
    a.bodies = b.topo_cnt[i];
    a.parent = b.parent_int[i];
    // the left child ends at the split, where its index lies too
    a.left = (a.kids.x < b.N ? a.kids.x : a.kids.x - b.N) - a.first + 1;
    a.right = a.bodies - a.left;
    return a;
}

__device__ __forceinline__ NodeVals load_child(const StepBuffers& b, uint32_t id) {
    return load_node(id < b.N ? &b.leaf[id] : &b.internal[id - b.N]);
}

__device__ __forceinline__ void store_above(const StepBuffers& b, const AboveNode& a, const NodeVals& out,
                                            const NodeVals& L, const NodeVals& R) {
    store_internal(b, a.id, out, L, R, a.kids.x, a.kids.y, a.left, a.right, a.bodies, a.parent);
    if (a.parent == GBH_NONE) {
        b.st->tree_height = out.depth;
        *b.root_rec = make_rec(out, a.id + b.N, a.bodies, false);
    }
}

template <int THREADS>
struct AboveSmem {
    float4 cm[THREADS], box03[THREADS], box45[THREADS], col[THREADS];  // finished nodes' values
    uint32_t ids[THREADS];
    uint32_t round[THREADS];  // the round that finished the node, 0 before
    uint32_t count;
};

// A list longer than the block has threads (trees far from the usual shapes: long
// chains).  A thread starts at every node with no child in the list and climbs, up
// to the last node of at most `most` bodies: where the other child is not in the
// list its words are there already, and the climb goes straight on; where it is,
// the second to arrive goes on (`fill_ready`, as in climb_global).  The starts hold
// more than `floor` bodies each and are disjoint, so there are fewer than THREADS.
// A level takes one round trip to L2, the next node's words loaded beside the
// arithmetic.  Steps of 56,800 and 113,600 bodies in clumps with chains along the
// axes (46 nodes above the groups per 142 bodies), us: a climb from every group of
// the state 296 and 318, rounds over the list 418 and 446, this 221 and 245.
template <int THREADS>
__device__ __noinline__ void fill_long_list(const StepBuffers& b, AboveSmem<THREADS>& S, const uint32_t* list,
                                            uint32_t m, uint32_t floor, uint32_t most) {
    const uint32_t t = threadIdx.x;
    __syncthreads();  // every thread has read the count
    if (t == 0) S.count = 0;
    __syncthreads();
    for (uint32_t k = t; k < m; k += THREADS) {
        const AboveNode a = above_node(b, list[k]);
        b.fill_ready[a.id] = 0u;
        if (a.left > floor || a.right > floor) continue;
        const uint32_t at = atomicAdd(&S.count, 1u);
        if (at < THREADS) S.ids[at] = a.id;
    }
    __syncthreads();
    const uint32_t start = t % 32 * (THREADS / 32) + t / 32;  // over all warps
    if (start >= S.count) return;
    AboveNode a = above_node(b, S.ids[start]);
    NodeVals L = load_child(b, a.kids.x), R = load_child(b, a.kids.y);
    for (;;) {
        // the next node, and its other child's words if they are there, beside this one
        const bool top = a.parent == GBH_NONE;
        const AboveNode up = top ? a : above_node(b, a.parent - b.N);
        const bool is_left = up.kids.x == a.id + b.N;
        const uint32_t other = is_left ? up.kids.y : up.kids.x;
        const gbh_node* words = other < b.N ? &b.leaf[other] : &b.internal[other - b.N];
        const bool last = top || up.bodies > most, meets = (is_left ? up.right : up.left) > floor;
        NodeVals v;
        if (!last && !meets) v = load_node_cg(words);
        const NodeVals out = combine(L, R);
        store_above(b, a, out, L, R);
        if (last || (meets && atomic_add_acq_rel(&b.fill_ready[up.id], 1u) == 0u)) return;
        if (meets) v = load_node_cg(words);
        L = is_left ? out : v;
        R = is_left ? v : out;
        a = up;
    }
}

// The nodes of one list (more than `floor` bodies each, their smaller children
// finished), a thread each.
template <int THREADS>
__device__ void fill_list(const StepBuffers& b, AboveSmem<THREADS>& S, uint32_t m, uint32_t floor) {
    const uint32_t t = threadIdx.x;
    AboveNode a;
    a.left = a.right = 0;
    if (t < m) {
        a = above_node(b, S.ids[t]);
        b.fill_ready[a.id] = t;  // its place, for its parent
    }
    S.round[t] = 0;
    __syncthreads();
    // children in the list by their place, the others' values now
    uint32_t at_l = GBH_NONE, at_r = GBH_NONE;
    NodeVals L, R, out;
    if (t < m) {
        if (a.left > floor) at_l = *(volatile uint32_t*)&b.fill_ready[a.kids.x - b.N]; else L = load_child(b, a.kids.x);
        if (a.right > floor) at_r = *(volatile uint32_t*)&b.fill_ready[a.kids.y - b.N]; else R = load_child(b, a.kids.y);
    }
    auto get = [&](uint32_t k) {
        NodeVals v;
        v.cm = S.cm[k];
        const float4 p = S.box03[k], q = S.box45[k];
        v.col = S.col[k];
        v.box[0] = p.x;
        v.box[1] = p.y;
        v.box[2] = p.z;
        v.box[3] = p.w;
        v.box[4] = q.x;
        v.box[5] = q.y;
        v.depth = __float_as_uint(q.z);
        return v;
    };
    bool pending = t < m;
    for (uint32_t round = 1;; ++round) {
        // only what an earlier round finished: its values are behind a barrier
        auto finished = [&](uint32_t at) {
            if (at == GBH_NONE) return true;
            const uint32_t f = *(volatile uint32_t*)&S.round[at];
            return f != 0u && f < round;
        };
        const bool ready = pending && finished(at_l) && finished(at_r);
        if (ready) {
            if (at_l != GBH_NONE) L = get(at_l);
            if (at_r != GBH_NONE) R = get(at_r);
            out = combine(L, R);
            S.cm[t] = out.cm;
            S.box03[t] = make_float4(out.box[0], out.box[1], out.box[2], out.box[3]);
            S.box45[t] = make_float4(out.box[4], out.box[5], __uint_as_float(out.depth), 0.0f);
            S.col[t] = out.col;
            S.round[t] = round;
            pending = false;
        }
        if (!__syncthreads_or(ready)) break;
    }
    if (t < m) store_above(b, a, out, L, R);
}

// Fill of the nodes above the body groups for capacities up to FILL_ABOVE_MAX:
// first a block per subtree of at most FILL_SUBTREE bodies (it finds its nodes,
// those with more bodies than a group, by their indices, which lie in the
// subtree's slots), then (LISTED) one block for the nodes above the subtrees, as
// the build listed them.
//
// What bounds it: the chain of heights.  A climb from every group with an
// atomic per node (release its words, meet the sibling, read its words from L2)
// takes 2.2 us per height, 45 us for the 20 heights above the groups of 65,536
// bodies.  Here a round takes the children's values from shared memory or
// registers and has one barrier; the nodes are written after the last one.
// At larger capacities the climbs (k_fill_top) hide each other's latency.  Fill
// stage, us, climb -> subtrees: 1,024 bodies 45 -> 35, 65,536 68 -> 59, 100,000
// 51 -> 49, 300,000 84 -> 76, 1,048,576 150 -> 158, 4,194,304 463 -> 586; with
// three contexts' steps in flight the chain is partly hidden, a step: 1,024
// bodies 44.5 -> 41.7, 65,536 99.9 -> 95.1, 100,000 the same, 300,000 266.8 ->
// 268.9.  A level between with subtrees of 131,072 bodies costs 35 us for the
// scan that finds its nodes.
template <int THREADS, bool LISTED>
__global__ __launch_bounds__(THREADS, LISTED ? 1 : 4) void k_fill_above(StepBuffers b) {
    extern __shared__ __align__(16) unsigned char fill_smem[];
    AboveSmem<THREADS>& S = *reinterpret_cast<AboveSmem<THREADS>*>(fill_smem);
    const uint32_t n = b.st->n_new;
    if (LISTED) {
        const uint32_t m = b.st->num_subtrees[1];
        if (m > THREADS) {
            fill_long_list(b, S, b.fill_subtrees[1], m, FILL_SUBTREE, ~0u);
        } else {
            if (threadIdx.x < m) S.ids[threadIdx.x] = b.fill_subtrees[1][threadIdx.x];
            fill_list<THREADS>(b, S, m, FILL_SUBTREE);
        }
        return;
    }
    if (n == 1 && blockIdx.x == 0 && threadIdx.x == 0)
        climb_global(b, 0u, 1u, load_node_cg(&b.leaf[0]), b.N);  // the root's one child
    const uint32_t subtrees = b.st->num_subtrees[0];
    for (uint32_t s = blockIdx.x; s < subtrees; s += gridDim.x) {
        const uint32_t root = b.fill_subtrees[0][s];
        const uint32_t lo = b.node_lo[root], bodies = b.topo_cnt[root];
        uint32_t* list = b.idx_out + lo;  // the spare index buffer: free until the next compaction
        __syncthreads();
        if (threadIdx.x == 0) S.count = 0;
        __syncthreads();
#pragma unroll 8
        for (uint32_t k = threadIdx.x; k < bodies; k += THREADS) {
            const uint32_t i = lo + k;
            // at most one index of the range belongs to an ancestor (more bodies)
            const uint32_t c = i + 1 < n ? b.topo_cnt[i] : 0u;
            if (c > GBH_GROUP_MAX && c <= bodies) {
                const uint32_t at = atomicAdd(&S.count, 1u);
                list[at] = i;
                if (at < THREADS) S.ids[at] = i;
            }
        }
        __syncthreads();
        const uint32_t m = S.count;
        if (m > THREADS)
            fill_long_list(b, S, list, m, GBH_GROUP_MAX, bodies);
        else
            fill_list<THREADS>(b, S, m, GBH_GROUP_MAX);
    }
}

#define ABOVE_THREADS 128  // a subtree: about 40 nodes
#define TOPS_THREADS 512   // the nodes above: one per 2,700 bodies

void fill_setup() {
    cudaFuncSetAttribute(k_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(FILL_WARPS * sizeof(FillSmem)));
    static_assert(sizeof(AboveSmem<TOPS_THREADS>) <= 48 * 1024, "above the default limit");
}

void launch_fill(const StepBuffers& b, cudaStream_t s) {
    // persistent: the blocks that fit at once, no more than the groups need
    const uint32_t blocks = min(b.num_sms * FILL_BLOCKS, (b.N + FILL_WARPS - 1) / FILL_WARPS);
    k_fill<<<blocks, FILL_THREADS, FILL_WARPS * sizeof(FillSmem), s>>>(b);
    if (b.N > FILL_ABOVE_MAX) {
        k_fill_top<<<b.num_sms * 4, 256, 0, s>>>(b);
        return;
    }
    k_fill_above<ABOVE_THREADS, false>
        <<<min(b.num_sms * 4, b.N / GBH_GROUP_MAX + 1), ABOVE_THREADS, sizeof(AboveSmem<ABOVE_THREADS>), s>>>(b);
    if (b.N > FILL_SUBTREE)
        k_fill_above<TOPS_THREADS, true><<<1, TOPS_THREADS, sizeof(AboveSmem<TOPS_THREADS>), s>>>(b);
}
