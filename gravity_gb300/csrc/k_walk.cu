// k_walk.cu — plain theta walk with leaf collisions, merge-task emission and
// the symplectic update.
//
// Replaces forceComputeKernel (SH/compute/force/bh_force.comp:6-142): one
// thread per body with a private 64-entry stack, a full 80-byte node gather per
// visit and a global atomic per opened node.
//
// Both kernels here give a warp 32 consecutive bodies of the Morton order
// (spatial neighbours; 4, 8 or 16 in small states) and ONE shared stack
// of (node, mask of the lanes whose own walk opened the node), so every lane
// interacts with exactly the nodes that its own reference walk would interact
// with.  The children of an opened
// node come as one 64-byte ChildPair record.
//
//   k_walk_plain     gravity and merges, FP32 and the precision form.  Up to 16
//                    opened nodes are popped at once and their children, one
//                    per lane, classified against the box of the
//                    warp's bodies; only the children whose acceptance differs
//                    inside the box get the per-body test.
//   k_walk_collide   collision mode, where a contact changes the body (position
//                    and velocity) in the reference's depth-first order, which
//                    the next tests and forces use: one node at a time in that
//                    order (childB before childA).
//
// Arithmetic: the MAC is the reference's (half side * invDist < theta, with
// invDist from the softened distance); the force sum uses fused multiply-adds
// (G m inv^3 r accumulated with FMA), which is within 1e-7 relative of the
// reference's operation order.
#include "gbh_common.cuh"

// ---- gravity and merges ----------------------------------------------------------
//
// What bounds it: instruction issue.  A walk of one node at a time per warp
// (the collision kernel below) spends about 46 instructions on every node that
// any of its 32 bodies meets, with the 20-30% of the lanes active whose own
// walk meets it: 66,600 instructions per warp on a 4,194,304-body mixture.  Of
// the nodes that a warp meets (976 on a 1,048,576-body mixture at theta 0.5)
// two thirds are accepted or opened by all of the warp's bodies alike, which
// one lane can tell from the box of the 32 bodies.  So a round pops up to 16
// opened nodes and classifies their 32 children, one per lane (about 60
// instructions for all of them); the force of a node on the bodies of its mask
// and the test of a node that the box leaves undecided, force included, take
// two nodes per packed FP32 instruction (17 and 23 instructions per node one
// by one, about 9 and 14 in pairs).  A finer box (per 16, 8 or 4 bodies) leaves 309, 290 or
// 267 of the 327 undecided nodes of a warp and was not worth its tests; 64
// bodies per warp leave more undecided tests per body (485 against 654 for two
// warps of 32, at twice the work each).
// Walk stage, ms, one node at a time -> classified in batches -> in pairs:
// 4,194,301-body mixture at theta 0.5 8.04 -> 3.14 -> 2.88; 2,097,152-body
// galaxy pair, precision form, 6.43 -> 2.50 -> 2.08; 1,048,576-body merge state
// at theta 0.7 0.457 -> 0.352 -> 0.338; 65,536-body Plummer sphere 0.289 ->
// 0.092 -> 0.080; 1,024 bodies 0.131 -> 0.045 -> 0.041 (0.035 with 4 bodies per
// warp).  Popping 32 nodes and
// classifying both children of each in turn: 4.12 ms on the mixture.

#define PW_THREADS 128
#define PW_WARPS (PW_THREADS / 32)
#define PW_LIST 64     // below 32 entries wait, one append adds up to 32
#define PW_STACK 288
#define PW_BATCH 64    // what one batch can add: 16 opened nodes and the undecided ones that wait (31)
#define PW_LEVELS 96   // the tallest tree: 63 key and 32 tie-break levels

enum PlainForm { PF_FP32 = 0, PF_PREC = 1, PF_MERGE = 2 };

// Resident blocks per SM: seven (72 registers, 28 warps) where 8 and 6 take
// 2.91 and 3.00 ms (4.2M mixture), 2.20 and 2.17 against 2.08 ms in the
// precision form; eight in the merge form (0.338 against 0.346 ms).
template <int FORM>
struct PlainBlocks {
    static constexpr int value = FORM == PF_MERGE ? 8 : 7;
};

// per-warp shared memory
template <int FORM>
struct PlainSmem {
    // entries every lane of the mask interacts with, by component (the force
    // loop takes two per packed instruction): centre of mass, G x mass
    alignas(16) float a_x[PW_LIST], a_y[PW_LIST], a_z[PW_LIST], a_w[PW_LIST];
    uint32_t a_mask[PW_LIST];
    // nodes to test body by body, with their half sides; the lanes of the mask
    // that accepted an entry
    float x_x[PW_LIST], x_y[PW_LIST], x_z[PW_LIST], x_w[PW_LIST], x_half[PW_LIST];
    uint32_t x_mask[PW_LIST];
    uint32_t x_id[PW_LIST];
    uint32_t x_accept[32];
    uint2 stack[PW_STACK];    // (opened node's internal index, lanes that opened it)
    // merge and precision forms: leaves apart (mask; radius and slot, or residual)
    float4 l_cm[FORM == PF_FP32 ? 1 : PW_LIST];
    float4 l_lo[FORM == PF_PREC ? PW_LIST : 1];
    uint32_t l_mask[FORM == PF_FP32 ? 1 : PW_LIST];
    float l_rad[FORM == PF_MERGE ? PW_LIST : 1];
    uint32_t l_id[FORM == PF_MERGE ? PW_LIST : 1];
};

// PREC: the precision form.  Offsets are formed from the FP32 position and
// its FP32 residual (leaf_lo), r = (x_j - x_b) + (lo_j - lo_b) for a leaf and
// (com - x_b) - lo_b for a node, and the leaf terms are summed with Kahan
// compensation apart from the node terms.  Gravity only.
template <int FORM>
__global__ __launch_bounds__(PW_THREADS, PlainBlocks<FORM>::value) void k_walk_plain(StepBuffers b, uint32_t per_warp) {
    constexpr bool PREC = FORM == PF_PREC;
    constexpr bool MERGE = FORM == PF_MERGE;
    __shared__ PlainSmem<FORM> s_warp[PW_WARPS];
    __shared__ unsigned long long s_inter, s_opened;
    __shared__ uint32_t s_depth;
    const uint32_t n = b.st->n_new;
    const uint32_t N = b.N;
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    const uint32_t base = (blockIdx.x * PW_WARPS + w) * per_warp;
    const uint32_t g = base + lane;
    if (blockIdx.x == 0 && threadIdx.x == 0) b.st->sorted_valid = 1u;  // the update below fills sorted_pm
    uint32_t s_lo, s_hi;
    shard_slots(b, n, s_lo, s_hi);
    const uint32_t per_block = PW_WARPS * per_warp, block_first = blockIdx.x * per_block;
    if (block_first >= n || block_first + per_block <= s_lo || block_first >= s_hi) return;
    if (threadIdx.x == 0) {
        s_inter = s_opened = 0ull;
        s_depth = 0u;
    }
    __syncthreads();
    // every live body of the warp walks, so that a body's sums do not depend on
    // the sharding; only the shard's own bodies count, merge and are updated
    const bool active = lane < per_warp && g < n;
    const bool owned = active && g >= s_lo && g < s_hi;
    const uint32_t everyone = __ballot_sync(0xffffffffu, active);
    const uint32_t owners = __ballot_sync(0xffffffffu, owned);
    const gbh_step_params* P = b.params;
    const gbh_sim_values* sim = b.sim;
    const float G = sim->gravitational_constant;
    const float soft = P->softening, theta = P->theta;
    PlainSmem<FORM>& S = s_warp[w];
    const uint32_t bit = 1u << lane;

    const uint32_t bi = active ? b.idx_in[g] : 0u;
    const float4 pm = active ? b.leaf_pm[g] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float my_rad = (MERGE && active) ? b.leaf_rad[g] : 0.0f;
    const float4 lo_b = (PREC && active) ? b.leaf_lo[g] : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool want_pot = (P->flags & GBH_FLAG_STORE_POTENTIAL) && b.potential;

    // box of the warp's bodies; `boxed` is false when it cannot speak for all
    // of them (positions that are not finite, parameters outside the range the
    // margins below are made for): then every node is tested body by body
    float mnx = active ? pm.x : 3.0e38f, mny = active ? pm.y : 3.0e38f, mnz = active ? pm.z : 3.0e38f;
    float mxx = active ? pm.x : -3.0e38f, mxy = active ? pm.y : -3.0e38f, mxz = active ? pm.z : -3.0e38f;
    float grp_rad = my_rad;
    float res = PREC ? fmaxf(fabsf(lo_b.x), fmaxf(fabsf(lo_b.y), fabsf(lo_b.z))) : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
        mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
        mnz = fminf(mnz, __shfl_xor_sync(0xffffffffu, mnz, o));
        mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
        mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
        mxz = fmaxf(mxz, __shfl_xor_sync(0xffffffffu, mxz, o));
        if (MERGE) grp_rad = fmaxf(grp_rad, __shfl_xor_sync(0xffffffffu, grp_rad, o));
        if (PREC) res = fmaxf(res, __shfl_xor_sync(0xffffffffu, res, o));
    }
    if (PREC) {
        // the bodies' residuals, and the rounding of the widened corners
        const float pad = 2.0f * res + 2.4e-7f * fmaxf(fmaxf(fmaxf(fabsf(mnx), fabsf(mxx)), fmaxf(fabsf(mny), fabsf(mxy))),
                                                       fmaxf(fabsf(mnz), fabsf(mxz)));
        mnx = mnx - pad;
        mny = mny - pad;
        mnz = mnz - pad;
        mxx = mxx + pad;
        mxy = mxy + pad;
        mxz = mxz + pad;
    }
    const bool boxed = !__any_sync(0xffffffffu, active && !(finite3(pm.x, pm.y, pm.z) && finite3(lo_b.x, lo_b.y, lo_b.z))) &&
                       (theta >= 1e-18f || theta == 0.0f) && theta <= 1e3f && soft >= 0.0f && soft <= 1e30f;
    // theta^2 with margins of 1e-5: the body's own test (a reciprocal square
    // root of at most 2 ulp error and six more roundings, together below 1e-6)
    // decides the same way wherever the box test decides.  Holds down to 1e-18,
    // where theta^2 is still a normal number; theta 0 (the exact sum) opens
    // everything.  With thetas below 1e-3 left to the tests body by body, theta 0
    // took 9.9 ms at 16,384 bodies and 43.2 at 65,536 (Plummer spheres), now 1.0 and
    // 6.6.
    const float t2_accept = theta * theta * 0.99999f, t2_open = theta * theta * 1.00001f;

    float ax = 0.0f, ay = 0.0f, az = 0.0f, pot = 0.0f;
    float nx_ = 0.0f, ny_ = 0.0f, nz_ = 0.0f, np_ = 0.0f;  // PREC: leaf terms (Kahan)
    float cx_ = 0.0f, cy_ = 0.0f, cz_ = 0.0f, cp_ = 0.0f;
    uint32_t inter = 0, opened = 0;  // this lane's share of the warp's counts
    uint32_t sp = 0, max_sp = 0, an = 0, xn = 0, ln = 0;
    bool overflow = false;
    // above this many stack entries the walk turns depth-first: what is left holds
    // one batch and then the descent through a tree of this height
    const uint32_t low_at = PW_STACK - PW_BATCH - min(b.st->tree_height + 1u, (uint32_t)PW_LEVELS);
    // a candidate of this lane was not finite (or far out of range), or the
    // softening does not keep the squared distances normal numbers
    bool wild = !boxed || soft < GBH_MIN_NORMAL;

    // push the opened nodes of the lanes with mask != 0 (warp-collective)
    auto push = [&](uint32_t id, uint32_t mask) {
        const uint32_t bo = __ballot_sync(0xffffffffu, mask != 0u);
        const uint32_t cnt = __popc(bo);
        if (sp + cnt > PW_STACK) {
            overflow = true;
            return;
        }
        if (mask) S.stack[sp + __popc(bo & lanemask_lt())] = make_uint2(id - N, mask);
        opened += __popc(mask & owners);
        sp += cnt;
    };
    // forces of list A's entries [0, cnt) on the lanes of each entry's mask, one
    // by one: with the potential, or where an entry's offset may not be finite
    // (times the zero of a masked lane it would not vanish)
    auto flush_a_single = [&](uint32_t cnt) {
        for (uint32_t j = 0; j < cnt; ++j) {
            float rx = S.a_x[j] - pm.x, ry = S.a_y[j] - pm.y, rz = S.a_z[j] - pm.z;
            const float m = S.a_w[j];
            if (PREC) rx = rx - lo_b.x, ry = ry - lo_b.y, rz = rz - lo_b.z;
            const float inv = rsqrtf(__fmaf_rn(rz, rz, __fmaf_rn(ry, ry, __fmaf_rn(rx, rx, soft))));
            const float f = m * (inv * inv * inv);
            if (S.a_mask[j] & bit) {
                ax = __fmaf_rn(f, rx, ax);
                ay = __fmaf_rn(f, ry, ay);
                az = __fmaf_rn(f, rz, az);
                if (want_pot) pot = __fmaf_rn(-m, inv, pot);
            }
        }
    };
    // the same, cnt a multiple of four, two entries per packed instruction
    auto flush_a = [&](uint32_t cnt) {
        const float2 px = make_float2(-pm.x, -pm.x), py = make_float2(-pm.y, -pm.y), pz = make_float2(-pm.z, -pm.z);
        const float2 lx = make_float2(-lo_b.x, -lo_b.x), ly = make_float2(-lo_b.y, -lo_b.y), lz = make_float2(-lo_b.z, -lo_b.z);
        const float2 soft2 = make_float2(soft, soft);
        float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx;
        auto two = [&](float2 x, float2 y, float2 z, float2 m, uint32_t m0, uint32_t m1) {
            float2 rx = __fadd2_rn(x, px), ry = __fadd2_rn(y, py), rz = __fadd2_rn(z, pz);
            if (PREC) rx = __fadd2_rn(rx, lx), ry = __fadd2_rn(ry, ly), rz = __fadd2_rn(rz, lz);
            const float2 rr = __ffma2_rn(rz, rz, __ffma2_rn(ry, ry, __ffma2_rn(rx, rx, soft2)));
            const float2 inv = make_float2(rsqrt_normal(rr.x), rsqrt_normal(rr.y));
            float2 f = __fmul2_rn(m, __fmul2_rn(__fmul2_rn(inv, inv), inv));
            f.x = (m0 & bit) ? f.x : 0.0f;
            f.y = (m1 & bit) ? f.y : 0.0f;
            sx = __ffma2_rn(f, rx, sx);
            sy = __ffma2_rn(f, ry, sy);
            sz = __ffma2_rn(f, rz, sz);
        };
#pragma unroll 2
        for (uint32_t j = 0; j < cnt; j += 4) {
            const float4 x = *reinterpret_cast<const float4*>(S.a_x + j), y = *reinterpret_cast<const float4*>(S.a_y + j),
                         z = *reinterpret_cast<const float4*>(S.a_z + j), m = *reinterpret_cast<const float4*>(S.a_w + j);
            const uint4 mk = *reinterpret_cast<const uint4*>(S.a_mask + j);
            two(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y), make_float2(m.x, m.y), mk.x, mk.y);
            two(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w), make_float2(m.z, m.w), mk.z, mk.w);
        }
        ax += sx.x + sx.y;
        ay += sy.x + sy.y;
        az += sz.x + sz.y;
    };
    // the same for the leaves of the merge and precision forms
    auto flush_l = [&](uint32_t cnt) {
        __syncwarp();
        ln -= cnt;
        for (uint32_t j = 0; j < cnt; ++j) {
            const float4 c = S.l_cm[ln + j];
            const bool me = S.l_mask[ln + j] & bit;
            float rx = c.x - pm.x, ry = c.y - pm.y, rz = c.z - pm.z;
            if (PREC) {
                const float4 lo_j = S.l_lo[ln + j];
                rx = rx + (lo_j.x - lo_b.x);
                ry = ry + (lo_j.y - lo_b.y);
                rz = rz + (lo_j.z - lo_b.z);
            }
            const float inv = rsqrtf(__fmaf_rn(rz, rz, __fmaf_rn(ry, ry, __fmaf_rn(rx, rx, soft))));
            const float f = c.w * (inv * inv * inv);
            if (me) {
                if (PREC) {
                    kahan_add(nx_, cx_, f * rx);
                    kahan_add(ny_, cy_, f * ry);
                    kahan_add(nz_, cz_, f * rz);
                    if (want_pot) kahan_add(np_, cp_, -c.w * inv);
                } else {
                    ax = __fmaf_rn(f, rx, ax);
                    ay = __fmaf_rn(f, ry, ay);
                    az = __fmaf_rn(f, rz, az);
                    if (want_pot) pot = __fmaf_rn(-c.w, inv, pot);
                }
            }
        }
        if (MERGE) {
            // lane j screens leaf j: within reach of the box (its radius plus
            // the warp's largest, a margin for rounding)?  Only those get the
            // per-body overlap test (bh_force.comp:109-112).
            bool near = false;
            if (lane < cnt) {
                const float4 c = S.l_cm[ln + lane];
                const float dx = fmaxf(fmaxf(mnx - c.x, c.x - mxx), 0.0f);
                const float dy = fmaxf(fmaxf(mny - c.y, c.y - mxy), 0.0f);
                const float dz = fmaxf(fmaxf(mnz - c.z, c.z - mxz), 0.0f);
                const float reach = S.l_rad[ln + lane] + grp_rad;
                near = dx * dx + dy * dy + dz * dz <= 1.001f * (reach * reach);
            }
            uint32_t m = __ballot_sync(0xffffffffu, near);
            while (m) {
                const uint32_t j = ln + __ffs(m) - 1;
                m &= m - 1;
                if (!(owned && (S.l_mask[j] & bit))) continue;
                const float4 c = S.l_cm[j];
                const uint32_t slot_j = S.l_id[j];
                const float rx = c.x - pm.x, ry = c.y - pm.y, rz = c.z - pm.z;
                const float dist = sqrtf(rx * rx + ry * ry + rz * rz);
                const float pen = my_rad + S.l_rad[j] - dist;
                if (pen > 0.0f) {
                    const uint32_t oi = b.idx_in[slot_j];
                    if (bi < oi) {
                        const uint32_t slot = atomicAdd(&b.mq->tail, 1u);
                        if (slot < N) {
                            // the reference's walk meets a body's leaves in
                            // descending slot order (childB before childA)
                            b.mq->pairs[slot] = make_uint2(bi, oi);
                            b.mkeys[slot] = ((unsigned long long)g << 32) | (N - 1u - slot_j);
                            b.mslots[slot] = slot_j;
                        }
                    }
                }
            }
        }
        __syncwarp();
    };
    // list X's entries [0, cnt), body by body: the accepting lanes take the
    // force, x_accept their mask; one by one as flush_a_single
    auto test_x_single = [&](uint32_t cnt) {
        for (uint32_t j = 0; j < cnt; ++j) {
            float rx = S.x_x[j] - pm.x, ry = S.x_y[j] - pm.y, rz = S.x_z[j] - pm.z;
            const float m = S.x_w[j];
            if (PREC) rx = rx - lo_b.x, ry = ry - lo_b.y, rz = rz - lo_b.z;
            const float inv = rsqrtf(__fmaf_rn(rz, rz, __fmaf_rn(ry, ry, rx * rx)) + soft);
            const bool accept = (S.x_mask[j] & bit) && S.x_half[j] * inv < theta;
            const float f = m * (inv * inv * inv);
            if (accept) {
                ax = __fmaf_rn(f, rx, ax);
                ay = __fmaf_rn(f, ry, ay);
                az = __fmaf_rn(f, rz, az);
                if (want_pot) pot = __fmaf_rn(-m, inv, pot);
            }
            const uint32_t am = __ballot_sync(0xffffffffu, accept);
            if (lane == 0) S.x_accept[j] = am;
        }
    };
    // the same, cnt a multiple of four, two entries per packed instruction
    auto test_x = [&](uint32_t cnt) {
        const float2 px = make_float2(-pm.x, -pm.x), py = make_float2(-pm.y, -pm.y), pz = make_float2(-pm.z, -pm.z);
        const float2 lx = make_float2(-lo_b.x, -lo_b.x), ly = make_float2(-lo_b.y, -lo_b.y), lz = make_float2(-lo_b.z, -lo_b.z);
        const float2 soft2 = make_float2(soft, soft);
        float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx;
        auto two = [&](uint32_t j, float2 x, float2 y, float2 z, float2 m, float2 half, uint32_t m0, uint32_t m1) {
            float2 rx = __fadd2_rn(x, px), ry = __fadd2_rn(y, py), rz = __fadd2_rn(z, pz);
            if (PREC) rx = __fadd2_rn(rx, lx), ry = __fadd2_rn(ry, ly), rz = __fadd2_rn(rz, lz);
            const float2 rr = __fadd2_rn(__ffma2_rn(rz, rz, __ffma2_rn(ry, ry, __fmul2_rn(rx, rx))), soft2);
            const float2 inv = make_float2(rsqrt_normal(rr.x), rsqrt_normal(rr.y));
            const float2 h = __fmul2_rn(half, inv);
            const bool a0 = (m0 & bit) && h.x < theta, a1 = (m1 & bit) && h.y < theta;
            float2 f = __fmul2_rn(m, __fmul2_rn(__fmul2_rn(inv, inv), inv));
            f.x = a0 ? f.x : 0.0f;
            f.y = a1 ? f.y : 0.0f;
            sx = __ffma2_rn(f, rx, sx);
            sy = __ffma2_rn(f, ry, sy);
            sz = __ffma2_rn(f, rz, sz);
            const uint32_t am0 = __ballot_sync(0xffffffffu, a0), am1 = __ballot_sync(0xffffffffu, a1);
            if (lane == 0) *reinterpret_cast<uint2*>(S.x_accept + j) = make_uint2(am0, am1);
        };
#pragma unroll 2
        for (uint32_t j = 0; j < cnt; j += 4) {
            const float4 x = *reinterpret_cast<const float4*>(S.x_x + j), y = *reinterpret_cast<const float4*>(S.x_y + j),
                         z = *reinterpret_cast<const float4*>(S.x_z + j), m = *reinterpret_cast<const float4*>(S.x_w + j),
                         h = *reinterpret_cast<const float4*>(S.x_half + j);
            const uint4 mk = *reinterpret_cast<const uint4*>(S.x_mask + j);
            two(j, make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y), make_float2(m.x, m.y),
                make_float2(h.x, h.y), mk.x, mk.y);
            two(j + 2, make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w), make_float2(m.z, m.w),
                make_float2(h.z, h.w), mk.z, mk.w);
        }
        ax += sx.x + sx.y;
        ay += sy.x + sy.y;
        az += sz.x + sz.y;
    };
    // one candidate per lane (`m`: the lanes whose walk reached it): leaves
    // and nodes that every body of the box accepts to list A (leaves to L in
    // the merge and precision forms), nodes that every body opens to the
    // stack, the others to list X (warp-collective)
    auto classify = [&](bool has, float4 cm, float half, uint32_t id, uint32_t m) {
        const bool leaf = has && id < N;
        bool accept = false, open = false;
        if (has) {
            const float ux = mnx - cm.x, uy = mny - cm.y, uz = mnz - cm.z;
            const float vx = cm.x - mxx, vy = cm.y - mxy, vz = cm.z - mxz;
            const float lx = fmaxf(fmaxf(ux, vx), 0.0f), ly = fmaxf(fmaxf(uy, vy), 0.0f), lz = fmaxf(fmaxf(uz, vz), 0.0f);
            const float hx = fminf(ux, vx), hy = fminf(uy, vy), hz = fminf(uz, vz);
            const float near2 = __fmaf_rn(lz, lz, __fmaf_rn(ly, ly, __fmaf_rn(lx, lx, soft)));
            const float far2 = __fmaf_rn(hz, hz, __fmaf_rn(hy, hy, __fmaf_rn(hx, hx, soft)));
            // a centre of mass that is not finite has no far2 below 1e30; the
            // small constants leave squares that lose bits to underflow to X
            const float h2 = half * half;
            const bool ok = !leaf && boxed && far2 < 1e30f;
            wild = wild || !(far2 < 1e30f);
            accept = ok && h2 < __fmaf_rn(t2_accept, near2, -1e-33f);
            open = ok && h2 >= __fmaf_rn(t2_open, far2, 1e-33f);
        }
        uint32_t take = m;
        if (leaf) {
            const uint32_t own = id - base;  // the body's own leaf, bh_force.comp:76-78
            if (own < 32u) take &= ~(1u << own);
        }
        if (leaf || accept) inter += __popc(take & owners);
        const bool to_a = accept || (FORM == PF_FP32 && leaf);
        const uint32_t ba = __ballot_sync(0xffffffffu, to_a);
        if (to_a) {
            const uint32_t pos = an + __popc(ba & lanemask_lt());
            S.a_x[pos] = cm.x;
            S.a_y[pos] = cm.y;
            S.a_z[pos] = cm.z;
            S.a_w[pos] = G * cm.w;
            S.a_mask[pos] = take;
        }
        an += __popc(ba);
        const bool to_x = has && !leaf && !accept && !open;
        const uint32_t bx = __ballot_sync(0xffffffffu, to_x);
        if (to_x) {
            const uint32_t pos = xn + __popc(bx & lanemask_lt());
            S.x_x[pos] = cm.x;
            S.x_y[pos] = cm.y;
            S.x_z[pos] = cm.z;
            S.x_w[pos] = G * cm.w;
            S.x_half[pos] = half;
            S.x_mask[pos] = m;
            S.x_id[pos] = id;
        }
        xn += __popc(bx);
        if (FORM != PF_FP32) {
            const uint32_t bl = __ballot_sync(0xffffffffu, leaf);
            if (leaf) {
                const uint32_t pos = ln + __popc(bl & lanemask_lt());
                S.l_cm[pos] = make_float4(cm.x, cm.y, cm.z, G * cm.w);
                S.l_mask[pos] = take;
                if (PREC) S.l_lo[pos] = b.leaf_lo[id];
                if (MERGE) {
                    S.l_rad[pos] = b.leaf_rad[id];
                    S.l_id[pos] = id;
                }
            }
            ln += __popc(bl);
        }
        push(id, open ? m : 0u);
    };

    // one site for each of the parts above, so that the code stays in the
    // instruction cache; every list holds fewer than 32 entries before an
    // append, which adds up to 32
    for (bool first = true; n > 1 && owners;) {
        const bool end = !first && sp == 0 && xn == 0;
        if (an >= 32 || (end && an)) {
            __syncwarp();
            const uint32_t cnt = min(an, 32u);
            if (want_pot || __any_sync(0xffffffffu, wild)) {
                flush_a_single(cnt);
            } else {
                // massless entries up to a multiple of four
                const uint32_t pad = (4u - (cnt & 3u)) & 3u;
                if (lane < pad) {
                    S.a_x[cnt + lane] = S.a_x[0];
                    S.a_y[cnt + lane] = S.a_y[0];
                    S.a_z[cnt + lane] = S.a_z[0];
                    S.a_w[cnt + lane] = 0.0f;
                    S.a_mask[cnt + lane] = 0u;
                }
                __syncwarp();
                flush_a(cnt + pad);
            }
            an -= cnt;
            __syncwarp();
            if (lane < an) {  // the remaining entries to the front
                S.a_x[lane] = S.a_x[32 + lane];
                S.a_y[lane] = S.a_y[32 + lane];
                S.a_z[lane] = S.a_z[32 + lane];
                S.a_w[lane] = S.a_w[32 + lane];
                S.a_mask[lane] = S.a_mask[32 + lane];
            }
            __syncwarp();
            continue;
        }
        if (FORM != PF_FP32 && (ln >= 32 || (end && ln))) {
            flush_l(min(ln, 32u));
            continue;
        }
        if (end) break;
        // the undecided nodes when a full batch waits, when the stack is empty
        // (the opened ones refill it) and, above low_at entries, always: the
        // walk then takes one node at a time, depth-first, so the stack holds
        // what the tree needs.  With one line for every tree, 120 entries, walks
        // at thetas from 0 to 0.05 ran depth-first most of the time (65,536-body
        // Plummer sphere at theta 0, 0.005 and 0.02: 13.0, 32.6 and 24.7 ms, now
        // 6.6, 15.1 and 10.0).  Testing them earlier, from 8 to 24
        // waiting ones at 8 to 48 stack entries, changed nothing (3.26 to 3.29
        // ms).
        const bool low = sp > low_at;
        if (xn && (xn >= 32 || sp == 0 || low)) {
            __syncwarp();
            const uint32_t cnt = min(xn, 32u);
            if (want_pot || __any_sync(0xffffffffu, wild)) {
                test_x_single(cnt);
            } else {
                const uint32_t pad = (4u - (cnt & 3u)) & 3u;
                if (lane < pad) {
                    S.x_x[cnt + lane] = S.x_x[0];
                    S.x_y[cnt + lane] = S.x_y[0];
                    S.x_z[cnt + lane] = S.x_z[0];
                    S.x_w[cnt + lane] = 0.0f;
                    S.x_half[cnt + lane] = 0.0f;
                    S.x_mask[cnt + lane] = 0u;
                }
                __syncwarp();
                test_x(cnt + pad);
            }
            __syncwarp();
            uint32_t id = 0u, opening = 0u;
            if (lane < cnt) {
                id = S.x_id[lane];
                const uint32_t mask = S.x_mask[lane], accept = S.x_accept[lane];
                opening = mask & ~accept;
                inter += __popc(accept & owners);
            }
            push(id, opening);
            xn -= cnt;
            __syncwarp();
            if (lane < xn) {  // the remaining entries to the front
                S.x_x[lane] = S.x_x[32 + lane];
                S.x_y[lane] = S.x_y[32 + lane];
                S.x_z[lane] = S.x_z[32 + lane];
                S.x_w[lane] = S.x_w[32 + lane];
                S.x_half[lane] = S.x_half[32 + lane];
                S.x_mask[lane] = S.x_mask[32 + lane];
                S.x_id[lane] = S.x_id[32 + lane];
            }
            __syncwarp();
            continue;
        }
        bool has;
        uint32_t m = 0u;
        float4 cm = make_float4(0.f, 0.f, 0.f, 0.f);
        uint2 meta = make_uint2(0u, 0u);
        if (first) {  // the root, bh_force.comp:53
            has = lane == 0;
            cm = b.root_rec->cm;
            meta = make_uint2(__float_as_uint(b.root_rec->half_side), N);
            m = everyone;
            first = false;
        } else {
            max_sp = max(max_sp, sp);
            const uint32_t k = low ? 1u : min(sp, 16u);
            sp -= k;
            has = lane < 2 * k;
            __syncwarp();
            if (has) {  // lane l: child l & 1 of popped node l / 2
                const uint2 e = S.stack[sp + (lane >> 1)];
                const float4* q = reinterpret_cast<const float4*>(b.pairs + e.x) + 2 * (lane & 1u);
                m = e.y;
                cm = __ldg(q);
                meta = __ldg(reinterpret_cast<const uint2*>(q + 1));
            }
            __syncwarp();
        }
        classify(has, cm, __uint_as_float(meta.x), meta.y, m);
    }
    if (overflow && lane == 0) set_error(b.st, GBH_DEVERR_WALK_STACK);

    // counters: one add per block (the whole grid adds to the same words)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        inter += __shfl_xor_sync(0xffffffffu, inter, o);
        opened += __shfl_xor_sync(0xffffffffu, opened, o);
    }
    if (lane == 0) {
        atomicAdd(&s_inter, (unsigned long long)inter);
        atomicAdd(&s_opened, (unsigned long long)opened);
        atomicMax(&s_depth, max_sp + 1);
    }
    if (owned) {
        if (PREC) {
            ax = ax + (nx_ - cx_);
            ay = ay + (ny_ - cy_);
            az = az + (nz_ - cz_);
            pot = pot + (np_ - cp_);
        }
        const float4 vd = ld_vel_density(b.bodies_in, bi);
        if (b.accel && (P->flags & GBH_FLAG_STORE_ACCEL)) b.accel[bi] = make_float4(ax, ay, az, 0.0f);
        if (b.accel_mag) b.accel_mag[bi] = sqrtf(ax * ax + ay * ay + az * az);
        if (want_pot) b.potential[bi] = pot;
        if (PREC)
            walk_update_fp64(b, P, sim, g, bi, pm, vd, ax, ay, az);
        else
            walk_update(b, P, sim, g, bi, pm, vd, ax, ay, az);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&b.st->interactions, s_inter);
        atomicAdd(&b.st->opened, s_opened);
        atomicAdd(&b.sim->uint_debug[0], (uint32_t)s_opened);
        atomicMax(&b.st->max_stack, s_depth);
    }
}

// ---- collision mode ----------------------------------------------------------------

#define WALK_THREADS 256
#define WALK_WARPS (WALK_THREADS / 32)
#define WALK_STACK 128

struct __align__(16) StackEntry {
    float4 cm;
    float half;
    uint32_t id;
    uint32_t mask;
    uint32_t pad;
};

__global__ __launch_bounds__(WALK_THREADS) void k_walk_collide(StepBuffers b, uint32_t per_warp) {
    __shared__ StackEntry s_stack[WALK_WARPS][WALK_STACK];
    const uint32_t n = b.st->n_new;
    const uint32_t N = b.N;
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    const uint32_t base = (blockIdx.x * WALK_WARPS + w) * per_warp;
    const uint32_t g = base + lane;
    if (blockIdx.x == 0 && threadIdx.x == 0) b.st->sorted_valid = 1u;  // the update below fills sorted_pm
    if (base >= n) return;
    uint32_t s_lo, s_hi;
    shard_slots(b, n, s_lo, s_hi);
    if (base + per_warp <= s_lo || base >= s_hi) return;
    const bool active = lane < per_warp && g < n && g >= s_lo && g < s_hi;
    const gbh_step_params* P = b.params;
    const gbh_sim_values* sim = b.sim;
    const float G = sim->gravitational_constant;
    const float soft = P->softening, theta = P->theta;
    const ChildPair* __restrict__ pairs = b.pairs;
    StackEntry* stk = s_stack[w];

    const uint32_t bi = active ? b.idx_in[g] : 0u;
    float4 pm = active ? b.leaf_pm[g] : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 vd = active ? ld_vel_density(b.bodies_in, bi) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float my_rad = active ? b.leaf_rad[g] : 0.0f;
    const bool want_pot = (P->flags & GBH_FLAG_STORE_POTENTIAL) && b.potential;
    float ax = 0.0f, ay = 0.0f, az = 0.0f, pot = 0.0f;
    uint32_t inter = 0;
    uint32_t opened = 0;
    uint32_t sp = 0, max_sp = 0;
    bool overflow = false;

    // current entry (warp-uniform): starts at the root, bh_force.comp:53
    float4 cur_cm;
    float cur_half;
    uint32_t cur_id, cur_mask;
    {
        const WalkRec root = *b.root_rec;
        cur_cm = root.cm;
        cur_half = root.half_side;
        cur_id = N;
        cur_mask = __ballot_sync(0xffffffffu, active);
    }
    const bool walk = n > 1;
    while (walk) {
        const bool me = (cur_mask >> lane) & 1u;
        const float rx = cur_cm.x - pm.x, ry = cur_cm.y - pm.y, rz = cur_cm.z - pm.z;
        const float rr = __fmaf_rn(rz, rz, __fmaf_rn(ry, ry, rx * rx));
        const float inv = rsqrtf(rr + soft);
        bool open = false, interact;
        if (cur_id >= N) {
            const bool accept = cur_half * inv < theta;
            interact = me && accept;
            open = me && !accept;
        } else {
            interact = me && cur_id != g;  // the body's own leaf, bh_force.comp:76-78
        }
        if (interact) {
            const float f = G * cur_cm.w * (inv * inv * inv);
            ax = __fmaf_rn(f, rx, ax);
            ay = __fmaf_rn(f, ry, ay);
            az = __fmaf_rn(f, rz, az);
            if (want_pot) pot = __fmaf_rn(-(G * cur_cm.w), inv, pot);
            ++inter;
            if (cur_id < N) {
                const uint32_t oi = b.idx_in[cur_id];
                const float orad = b.leaf_rad[cur_id];
                const float dist = sqrtf(rx * rx + ry * ry + rz * rz);
                const float pen = my_rad + orad - dist;
                if (pen > 0.0f) {
                    // bh_force.comp:93-107, in the reference's operation order
                    const float ow = cur_cm.w;
                    const float4 ov = ld_vel_density(b.bodies_in, oi);
                    const float vx = ov.x - vd.x, vy = ov.y - vd.y, vz = ov.z - vd.z;
                    const float nx = rx / dist, ny = ry / dist, nz = rz / dist;
                    const float vimp = vx * nx + vy * ny + vz * nz;
                    if (vimp < 0.0f) {
                        const float meff = 1.0f / (1.0f / pm.w + 1.0f / ow);
                        const float imp = (1.0f + P->elasticity) * meff * vimp;
                        vd.x += nx * imp / pm.w;
                        vd.y += ny * imp / pm.w;
                        vd.z += nz * imp / pm.w;
                    }
                    const float sc = pen / (pm.w + ow) * P->restitution;
                    pm.x -= sc * nx;
                    pm.y -= sc * ny;
                    pm.z -= sc * nz;
                }
            }
        }
        const uint32_t om = __ballot_sync(0xffffffffu, open);
        if (om) {
            opened += __popc(om);
            const float4* q = reinterpret_cast<const float4*>(pairs + (cur_id - N));
            const float4 a_cm = __ldg(q + 0);
            const uint4 a_meta = __ldg(reinterpret_cast<const uint4*>(q + 1));
            const float4 b_cm = __ldg(q + 2);
            const uint4 b_meta = __ldg(reinterpret_cast<const uint4*>(q + 3));
            if (sp >= WALK_STACK) {
                overflow = true;
                break;
            }
            if (lane == 0) {
                stk[sp].cm = a_cm;
                *reinterpret_cast<uint4*>(&stk[sp].half) = make_uint4(a_meta.x, a_meta.y, om, 0u);
            }
            ++sp;
            max_sp = max(max_sp, sp);
            cur_cm = b_cm;
            cur_half = __uint_as_float(b_meta.x);
            cur_id = b_meta.y;
            cur_mask = om;
        } else {
            if (sp == 0) break;
            --sp;
            __syncwarp();
            const float4 e_cm = stk[sp].cm;
            const uint4 e_meta = *reinterpret_cast<const uint4*>(&stk[sp].half);
            __syncwarp();
            cur_cm = e_cm;
            cur_half = __uint_as_float(e_meta.x);
            cur_id = e_meta.y;
            cur_mask = e_meta.z;
        }
    }
    if (overflow && lane == 0) set_error(b.st, GBH_DEVERR_WALK_STACK);

    // counters: one atomic per warp
    uint32_t tot = inter;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0) {
        atomicAdd(&b.st->interactions, (unsigned long long)tot);
        atomicAdd(&b.st->opened, (unsigned long long)opened);
        atomicAdd(&b.sim->uint_debug[0], opened);
        atomicMax(&b.st->max_stack, max_sp + 1);
    }
    if (!active) return;
    if (b.accel && (P->flags & GBH_FLAG_STORE_ACCEL)) b.accel[bi] = make_float4(ax, ay, az, 0.0f);
    if (b.accel_mag) b.accel_mag[bi] = sqrtf(ax * ax + ay * ay + az * az);
    if (want_pot) b.potential[bi] = pot;
    walk_update(b, P, sim, g, bi, pm, vd, ax, ay, az);
}

// Bodies per warp.  A small state leaves most of the GPU idle, and its walk is
// the longest warp's chain, shorter with fewer bodies (a smaller box opens fewer
// nodes), until the warps need each other's issue slots.  Walk stage, us, 32, 16,
// 8 and 4 bodies per warp, Plummer spheres at theta 0.5: 1,024 bodies 45, 41, 37,
// 35; 4,096 53, 45, 41, 39; 8,192 55, 51, 47, 47; 16,384 61, 57, 59, 70; 32,768
// 72, 66, 80, 119.  Steps with three contexts in flight: 1,024 bodies 34.1 ->
// 31.0 us, 4,096 50.5 -> 47.6, 8,192 58.3 -> 57.8, 6,000 in the precision form
// 66.1 -> 63.0, but 24,000 with 16 per warp 68.6 -> 69.9.
static uint32_t bodies_per_warp(uint32_t n) { return n <= 4096u ? 4u : n <= 8192u ? 8u : 32u; }

// The same for the collision kernel, where one node at a time makes the chain
// longer.  Walk stage, us, 32, 16, 8 and 4 bodies per warp, bodies in a box at
// theta 0.7: 1,024 bodies 39, 31, 27, 21; 8,192 51, 39, 35, 31; 16,384 55, 41, 35,
// 35; 32,768 59, 47, 47, 59; 65,536 68, 61, 78, 96; 100,003 72, 80, 98, 139.  Steps
// with three contexts in flight: 1,024 bodies 34.1 -> 26.9 us, 8,192 56.0 -> 48.3,
// 16,384 59.0 -> 53.6, 32,768 65.0 -> 62.2.  With 32 and 16 per warp, in flight
// (alone): 40,000 bodies 63.8 (181) and 62.4 us (172), 65,536 79.8 (201) and 81.2
// (193), 100,003 92.7 (214) and 109.2 (221): the two cross between 40,000 and
// 65,536 bodies in flight, and above 65,536 alone.
static uint32_t collide_per_warp(uint32_t n) {
    return n <= 8192u ? 4u : n <= 16384u ? 8u : n <= 32768u ? 16u : 32u;
}

void launch_walk_plain(const StepBuffers& b, cudaStream_t s) {
    const uint32_t per_warp = bodies_per_warp(b.N);
    const uint32_t blocks = (b.N + PW_WARPS * per_warp - 1) / (PW_WARPS * per_warp);
    const uint32_t per_block = WALK_WARPS * collide_per_warp(b.N);
    if (b.collide)
        k_walk_collide<<<(b.N + per_block - 1) / per_block, WALK_THREADS, 0, s>>>(b, collide_per_warp(b.N));
    else if (b.prec)
        k_walk_plain<PF_PREC><<<blocks, PW_THREADS, 0, s>>>(b, per_warp);
    else if (b.merge)
        k_walk_plain<PF_MERGE><<<blocks, PW_THREADS, 0, s>>>(b, per_warp);
    else
        k_walk_plain<PF_FP32><<<blocks, PW_THREADS, 0, s>>>(b, per_warp);
}
