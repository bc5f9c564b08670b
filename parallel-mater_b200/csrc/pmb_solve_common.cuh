// SPDX-License-Identifier: MIT
// Device helpers of the AVBD solve kernels: body displacements, contact
// rows, the group-per-body and body-per-thread primal, the dual updates and
// the residual reduction. Shared by the solve kernels' translation units.
#pragma once
#include <type_traits>

#include "pmb_joint.cuh"

namespace pmb {

struct Lite {  // what a contact row needs of a body during the solve: its displacement
    V6 dx;
};
__device__ __forceinline__ Lite load_lite(const Dev& d, uint32_t i) {
    const float4 l = d.dx[2 * i], a = d.dx[2 * i + 1];
    return {{{l.x, l.y, l.z, a.x, a.y, a.z}}};
}

// Contact jacobians (geometry_constraints.slang:508-532). They depend only on
// the contact geometry and the AVBD target poses, both fixed during a solve
// phase, so they are evaluated once per phase and stored in the contact's
// phase record (d.c_row).
__device__ __forceinline__ void contact_jacobians(V3 n, V3 pt, V3 anc_a, V3 anc_b, V3 xa, Q4 qa, V3 xb, Q4 qb,
                                                  V6 ja[3], V6 jb[3]) {
    V3 t0, t1;
    basis(n, t0, t1);
    const V3 axes[3] = {n, t0, t1};
    const V3 arm_a = sub(pt, xa), arm_b = sub(pt, xb);
    const V3 ra_t = rotate(qa, anc_a), rb_t = rotate(qb, anc_b);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        V3 ra = k == 0 ? arm_a : ra_t;
        V3 rb = k == 0 ? arm_b : rb_t;
        ja[k] = jac(mul(axes[k], -1.0f), mul(cross(ra, axes[k]), -1.0f));
        jb[k] = jac(axes[k], cross(rb, axes[k]));
    }
}
// A contact's phase record (d.c_row): the row values are those of
// contact_jacobians, with body a's linear parts (the negated axes) not kept.
struct ContactRow {
    V3 axis[3], ang_a[3], ang_b[3];
    float friction, beta;
    float e[3];
    __device__ __forceinline__ V6 ja(int k) const {
        return jac(V3{-axis[k].x, -axis[k].y, -axis[k].z}, ang_a[k]);
    }
    __device__ __forceinline__ V6 jb(int k) const { return jac(axis[k], ang_b[k]); }
};
__device__ __forceinline__ ContactRow load_row32(const Dev& d, uint32_t c) {
    const float4* p = d.c_row + size_t(c) * 8;
    float f[32];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float4 v = p[k];
        f[4 * k] = v.x;
        f[4 * k + 1] = v.y;
        f[4 * k + 2] = v.z;
        f[4 * k + 3] = v.w;
    }
    ContactRow r;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r.axis[k] = V3{f[3 * k], f[3 * k + 1], f[3 * k + 2]};
        r.ang_a[k] = V3{f[9 + 3 * k], f[10 + 3 * k], f[11 + 3 * k]};
        r.ang_b[k] = V3{f[18 + 3 * k], f[19 + 3 * k], f[20 + 3 * k]};
        r.e[k] = f[29 + k];
    }
    r.friction = f[27];
    r.beta = f[28];
    return r;
}
__device__ __forceinline__ void store_row32(const Dev& d, uint32_t c, const V6 ja[3], const V6 jb[3], float friction,
                                            float beta, float4 e) {
    float f[32];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            f[3 * k + q] = jb[k].v[q];
            f[9 + 3 * k + q] = ja[k].v[3 + q];
            f[18 + 3 * k + q] = jb[k].v[3 + q];
        }
    f[27] = friction;
    f[28] = beta;
    f[29] = e.x;
    f[30] = e.y;
    f[31] = e.z;
    float4* p = d.c_row + size_t(c) * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) p[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
}
// Contact c's values of a phase: its jacobians at the phase's target poses,
// its friction and penalty growth factor (its bodies' materials and masses).
__device__ __forceinline__ void contact_phase_row(const Dev& d, uint32_t c, uint32_t a, uint32_t b, float dt, V6 ja[3],
                                                  V6 jb[3], float& friction, float& beta) {
    contact_jacobians(v3(d.c_n[c]), v3(d.c_p[c]), v3(d.c_aa[c]), v3(d.c_ab[c]), v3(d.tx[a]), q4(d.tq[a]), v3(d.tx[b]),
                      q4(d.tq[b]), ja, jb);
    friction = sqrtf(d.p1[a].x * d.p1[b].x);
    beta = (1.0f / (fmx(d.p0[a].x + d.p0[b].x, 1.0e-6f) * dt * dt)) * 100.0f;
}
// The rows' errors at the bodies' displacements: e + J_a . dx_a + J_b . dx_b.
__device__ __forceinline__ void contact_errors(const ContactRow& r, const Lite& A, const Lite& B, float err[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) err[k] = r.e[k] + dot6(r.ja(k), A.dx) + dot6(r.jb(k), B.dx);
}

__device__ __forceinline__ void apply_pose_update(const Dev& d, uint32_t i, const V6& u, float4 l, float4 dq) {
    l.x += u.v[0];
    l.y += u.v[1];
    l.z += u.v[2];
    d.dx[2 * i] = l;
    V3 r{u.v[3], u.v[4], u.v[5]};
    if (r.x == 0.0f && r.y == 0.0f && r.z == 0.0f) return;
    Q4 rel = q4(dq);
    Q4 dd = qmul(Q4{r.x, r.y, r.z, 0.0f}, rel);
    rel = qnormalize(Q4{rel.x + 0.5f * dd.x, rel.y + 0.5f * dd.y, rel.z + 0.5f * dd.z, rel.w + 0.5f * dd.w});
    if (rel.w < 0.0f) rel = {-rel.x, -rel.y, -rel.z, -rel.w};
    d.dq[i] = f4(rel);
    d.dx[2 * i + 1] = make_float4(2.0f * rel.x, 2.0f * rel.y, 2.0f * rel.z, 0.0f);
}
__device__ __forceinline__ void apply_pose_update(const Dev& d, uint32_t i, const V6& u) {
    apply_pose_update(d, i, u, d.dx[2 * i], d.dq[i]);
}

// Group-per-body primal: G lanes (G = 8, 16 or 32) solve one body. Lanes
// evaluate the body's contact rows G at a time (coalesced SoA loads) and
// stage them in shared memory; each lane owns ceil(27/G) of the 27 entries of
// the packed 6x6 block (21 Hessian, 6 gradient) and adds the staged rows to
// them in list order. Every entry thus sees exactly the additions, in exactly
// the order, of the serial per-body loop of
// geometry_constraints_solve.slang:339-400, whatever G is, and the block is
// bit-identical to it; the LDL^T solve then runs in registers. The crossing
// safeguard reuses the staged normal rows: its error term is the same
// expression at the same displacements.
//
// G is chosen per colour: 8 lanes when the colour has more bodies than the
// grid has 16-lane groups, else 16, or 32 when even 32-lane groups cover it.
// The tail colours of a pile hold few but heavily loaded bodies (tens of
// rows), and a colour ends when its slowest body does, so wider groups
// there shorten the critical path.
//
// A staged contact holds its three rows side by side, one 16-byte word per
// jacobian component (its n, t0, t1 values): J[6], the forces, then stiffness
// x J[6], so an entry takes a contact's three products from two 128-bit loads
// (A and B of entry_words) where it took six of 32 bits. An 8-lane group at
// 11 contacts a body: 256 instead of about 400 instructions a chunk.
//
// Shared-memory banks: a 128-bit access goes eight lanes at a time, and a
// lane's slot of 52 words puts eight lanes' writes on distinct banks; a group
// reads distinct words of one slot. Normal rows (scalar accesses) are 9 words,
// and groups start 24 (8 lanes) or 16 (16 lanes) banks apart, so the groups of
// a warp do not collide on them either.
constexpr int kSlotWords = 52;   // a lane's contact: 13 float4
constexpr int kSlotForce = 24, kSlotScaled = 28;  // words of the forces and of stiffness x J
template <int G> struct GroupRowsData {
    // Normal rows kept for the crossing safeguard (rows past them are
    // evaluated again there): 32 for 8-lane groups, 64 for the 16- and
    // 32-lane groups of the heavy bodies (which fit the same staging area).
    static constexpr uint32_t kSlots = G >= 16 ? 64u : 32u;
    float r[G][kSlotWords];  // the chunk being accumulated; the body's block while it is factorised
    float nrow[kSlots][9];   // normal row: jacobian[6], raw penalty, trial force (and a pad word)
};
template <int G> struct __align__(16) GroupRows : GroupRowsData<G> {
    // Pads the group to 24 banks mod 32 (8 lanes: bases 0, 24, 16, 8) or 16
    // (16 lanes: bases 0, 16).
    static constexpr int kWords = int(sizeof(GroupRowsData<G>) / 4);
    static constexpr int kTarget = G == 8 ? 24 : G == 16 ? 16 : kWords % 32;
    static constexpr int kPad = (kTarget - kWords % 32 + 32) % 32;
    float pad[kPad == 0 ? 32 : kPad];
    __device__ __forceinline__ float4* slot(int s) { return reinterpret_cast<float4*>(&this->r[s][0]); }
    __device__ __forceinline__ float* block() { return &this->r[0][0]; }  // 27 entries
};
static_assert(sizeof(GroupRows<8>) / 4 % 32 == 24 && sizeof(GroupRows<16>) / 4 % 32 == 16, "group bank offsets");
// Per-warp staging area: four 8-lane groups, two 16-lane groups or one
// 32-lane group.
constexpr size_t kWarpStage = 4 * sizeof(GroupRows<8>);
static_assert(2 * sizeof(GroupRows<16>) <= kWarpStage && sizeof(GroupRows<32>) <= kWarpStage, "staging area");
// Per-thread slots of the body-per-thread sweep: a block and a joint's two
// body views, in shared memory so the joint visit (a call) reads them there
// rather than from local memory.
constexpr size_t kThreadViews = 32 * sizeof(Blk);
static_assert(kThreadViews + 64 * sizeof(BodyView) <= kWarpStage, "per-thread joint slots");

__device__ __forceinline__ void entry_ik(int e, int& i, int& k) {
    i = e >= 15 ? 5 : e >= 10 ? 4 : e >= 6 ? 3 : e >= 3 ? 2 : e >= 1 ? 1 : 0;
    k = e - i * (i + 1) / 2;
}

// Lane gl owns entries gl, gl+G, gl+2G, ... (those below 27).
template <int G> struct Owned {
    static constexpr int E = (27 + G - 1) / G;
};
// The lane's entries and the whole block through the group's shared memory.
template <int G>
__device__ __forceinline__ void publish_entries(const float* ent, GroupRows<G>& sm, int gl) {
#pragma unroll
    for (int m = 0; m < Owned<G>::E; ++m)
        if (gl + G * m < 27) sm.block()[gl + G * m] = ent[m];
}
template <int G> __device__ __forceinline__ void own_entries(GroupRows<G>& sm, int gl, float* ent) {
#pragma unroll
    for (int m = 0; m < Owned<G>::E; ++m) ent[m] = gl + G * m < 27 ? sm.block()[gl + G * m] : 0.0f;
}

// Word offsets in a staged contact of the two factors of entry e's products
// (three each: n, t0, t1): stiffness x J_i and J_k of the Hessian entry
// (i, k), J_r and the force of the gradient entry r.
__device__ __forceinline__ void entry_words(int e, int& a, int& b) {
    int i, k;
    entry_ik(e, i, k);
    a = e < 21 ? kSlotScaled + 4 * i : e < 27 ? 4 * (e - 21) : 0;
    b = e < 21 ? 4 * k : kSlotForce;
}
template <int G>
__device__ __forceinline__ void accumulate_chunk(float* ent, int gl, GroupRows<G>& sm, uint32_t m) {
    const float *pa[Owned<G>::E], *pb[Owned<G>::E];
#pragma unroll
    for (int q = 0; q < Owned<G>::E; ++q) {
        int a, b;
        entry_words(gl + G * q, a, b);
        pa[q] = &sm.r[0][a];
        pb[q] = &sm.r[0][b];
    }
    // A contact's products, then the ordered adds (contacts past m are formed
    // from the slot's stale values and dropped).
    auto contact = [&](int t, bool in) {
#pragma unroll
        for (int q = 0; q < Owned<G>::E; ++q) {
            const float4 a = *reinterpret_cast<const float4*>(pa[q] + kSlotWords * t);
            const float4 b = *reinterpret_cast<const float4*>(pb[q] + kSlotWords * t);
            const float p0 = a.x * b.x, p1 = a.y * b.y, p2 = a.z * b.z;
            if (in) {
                ent[q] += p0;
                ent[q] += p1;
                ent[q] += p2;
            }
        }
    };
    if (G <= 8) {
#pragma unroll 2  // (more contacts' loads in flight spill at 512 threads)
        for (int t = 0; t < G; ++t) contact(t, t < int(m));
    } else {
#pragma unroll 1
        for (int t0 = 0; t0 < int(m); t0 += 4)
#pragma unroll
            for (int u = 0; u < 4; ++u) contact(t0 + u, t0 + u < int(m));
    }
}

// The group's block in every lane's registers (seven 128-bit broadcasts
// where shuffles took 27). Every lane then factorises it: with a lane per row
// of the block, exchanging rows by shuffles, the solve took 4.0 us instead of
// 2.7 in the settled pile's first colour -- half the instructions, but each
// column waits for a shuffle of the one before.
template <int G> __device__ __forceinline__ void read_block(GroupRows<G>& sm, Blk& blk) {
    const float4* p = reinterpret_cast<const float4*>(sm.block());
    float f[28];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        const float4 v = p[k];
        f[4 * k] = v.x;
        f[4 * k + 1] = v.y;
        f[4 * k + 2] = v.z;
        f[4 * k + 3] = v.w;
    }
#pragma unroll
    for (int e = 0; e < 21; ++e) blk.h[e] = f[e];
#pragma unroll
    for (int r = 0; r < 6; ++r) blk.g[r] = f[21 + r];
}

// Whether a staged normal row's trial force crosses zero under the update
// (geometry_constraints_solve.slang:433-475).
__device__ __forceinline__ bool crosses(const float* row, const V6& upd) {
    V6 nr;
#pragma unroll
    for (int k = 0; k < 6; ++k) nr.v[k] = row[k];
    const float k0 = row[6], trial = row[7];
    return trial <= 0.0f && trial + k0 * dot6(nr, upd) > k0 * 1.0e-6f;
}
// Adds the crossing rows of a chunk (bit t of `mask`: row s0 + t) to the
// lane's entries, rows in list order.
template <int G>
__device__ __forceinline__ void accumulate_crossing(float* ent, int gl, const GroupRows<G>& sm, uint32_t s0,
                                                    uint32_t m, uint32_t mask) {
#pragma unroll
    for (int q = 0; q < Owned<G>::E; ++q) {
        const int e = gl + G * q;
        if (e >= 27) continue;
        int ei = 0, ek = 0;
        if (e < 21) entry_ik(e, ei, ek);
        for (uint32_t t = 0; t < m; ++t) {
            if (!((mask >> t) & 1u)) continue;
            const float* row = sm.nrow[(s0 + t) % GroupRows<G>::kSlots];
            if (e < 21) ent[q] += row[6] * row[ei] * row[ek];
            else ent[q] += row[e - 21] * row[7];
        }
    }
}

// What a body's solve reads of one of its contact rows: the contact (code:
// index, bit 31 set when the body is the contact's second body) and the other
// body. Loaded apart from the arithmetic so a body's first rows can be in
// flight while its own state arrives.
struct RawContact {
    uint32_t c;
    bool first;
    Lite other;
    float4 lam, pen;
    ContactRow row;
};
__device__ __forceinline__ RawContact load_contact(const Dev& d, uint32_t code, uint32_t other_body) {
    RawContact r;
    r.c = code & 0x7fffffffu;
    r.first = (code >> 31) == 0;
    r.other = load_lite(d, other_body);
    r.lam = d.c_lam[r.c];
    r.pen = d.c_pen[r.c];
    r.row = load_row32(d, r.c);
    return r;
}

// Rows of one contact for body i into chunk slot `slot`; its normal row,
// raw penalty and normal trial also go to nrow[nslot].
template <int G>
__device__ __forceinline__ void stage_loaded(const Dev& d, const Lite& me, const RawContact& rc,
                                             uint32_t phase, GroupRows<G>& sm, int slot, int nslot) {
    const bool first = rc.first;
    const Lite A = first ? me : rc.other;  // values, not run-time references (no local copies)
    const Lite B = first ? rc.other : me;
    const float4 lam = rc.lam, pen = rc.pen;
    float err[3];
    contact_errors(rc.row, A, B, err);
    const F3 trial{lam.x + pen.x * err[0], lam.y + pen.y * err[1], lam.z + pen.z * err[2]};
    // This body's jacobians: element by element (a reference chosen at run
    // time would give the arrays addresses, local memory).
    V6 j[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const V6 a = rc.row.ja(x), b = rc.row.jb(x);
#pragma unroll
        for (int k = 0; k < 6; ++k) j[x].v[k] = first ? a.v[k] : b.v[k];
    }
    if (nslot >= 0) {
#pragma unroll
        for (int k = 0; k < 6; ++k) sm.nrow[nslot][k] = j[0].v[k];
        sm.nrow[nslot][6] = pen.x;
        sm.nrow[nslot][7] = trial.n;
    }
    if (slot < 0) return;
    F3 f, sc;
    project_with_scales(trial, rc.row.friction, f, sc);
    if (phase != 0) {
        const float4 fo = d.c_foff[rc.c];
        f.n -= fo.x;
        f.t0 -= fo.y;
        f.t1 -= fo.z;
    }
    const float st[3] = {pen.x * sc.n, pen.y * sc.t0, pen.z * sc.t1};
    float4* out = sm.slot(slot);
#pragma unroll
    for (int k = 0; k < 6; ++k) out[k] = make_float4(j[0].v[k], j[1].v[k], j[2].v[k], 0.0f);
    out[kSlotForce / 4] = make_float4(f.n, f.t0, f.t1, 0.0f);
#pragma unroll
    for (int k = 0; k < 6; ++k)
        out[kSlotScaled / 4 + k] =
            make_float4(st[0] * j[0].v[k], st[1] * j[1].v[k], st[2] * j[2].v[k], 0.0f);  // (stiffness x J_i)
}
template <int G>
__device__ __forceinline__ void stage_contact(const Dev& d, const Lite& me, uint32_t code,
                                              uint32_t other_body, uint32_t phase, GroupRows<G>& sm, int slot,
                                              int nslot) {
    stage_loaded<G>(d, me, load_contact(d, code, other_body), phase, sm, slot, nslot);
}

// The body a lane group solves next in its colour, fetched while the current
// one solves (bodies of one colour share no contact, so nothing the current
// body writes is read here): its record and this lane's row codes of its
// first two chunks.
struct Ahead {
    uint32_t i, ro, rn;
    uint32_t code0, other0, code1, other1;
    uint32_t impact;  // the body's impact flag (the velocity phase solves impacted bodies only)
};
template <int G>
__device__ __forceinline__ void fetch_codes(const Dev& d, Ahead& a, int gl) {
    const uint32_t s0 = uint32_t(gl), s1 = uint32_t(gl) + uint32_t(G);
    a.code0 = s0 < a.rn ? d.blist[a.ro + s0] : 0u;
    a.other0 = s0 < a.rn ? d.bother[a.ro + s0] : 0u;
    a.code1 = s1 < a.rn ? d.blist[a.ro + s1] : 0u;
    a.other1 = s1 < a.rn ? d.bother[a.ro + s1] : 0u;
}
template <int G>
__device__ __forceinline__ Ahead fetch_ahead(const Dev& d, uint32_t k, int gl) {
    const uint4 r = d.crec[k];
    Ahead a{r.x, r.y, r.z, 0u, 0u, 0u, 0u, r.w};
    fetch_codes<G>(d, a, gl);
    return a;
}

// The two bodies of a joint as its rows read them during a sweep.
struct JointEnds {
    V6 dxa, dxb;
    V3 xa, xb;
    Q4 qa, qb;
};
__device__ __forceinline__ void load_end(const Dev& d, uint32_t i, V6& dx, V3& x, Q4& q) {
    const float4 tx = d.tx[i], tq = d.tq[i], l = d.dx[2 * i], a = d.dx[2 * i + 1], dq = d.dq[i];
    dx = {{l.x, l.y, l.z, a.x, a.y, a.z}};
    x = add(v3(tx), v3(l));
    q = q4(tq);
    if (dq.x != 0.0f || dq.y != 0.0f || dq.z != 0.0f) q = qnormalize(qmul(q4(dq), q));  // body_pose
}
__device__ __forceinline__ JointEnds load_ends(const Dev& d, uint32_t a, uint32_t b) {
    JointEnds e;
    load_end(d, a, e.dxa, e.xa, e.qa);
    load_end(d, b, e.dxb, e.xb, e.qb);
    return e;
}

// Joint rows of body i added to its block entries by the group's lanes, in
// the serial loop's order (joints in list order, then axes, then rows).
// A lane takes one axis of one joint -- two, five or ten joints at a time
// for 8, 16 and 32 lanes -- and stages its rows over the contact rows, which
// are in the entries by now: a lane's kSlotWords hold three rows, and only an
// axis of a generic or spring joint, or of a piston with linear and angular
// limits, has more; such a joint is taken alone, its lanes' rows spread over
// the group's slots.
constexpr int kJointWords = 12;  // jacobian[6], stiffness, force, curvature[3], whether it has one
constexpr int kJointRowsMost = 6;
template <int G>
__device__ __forceinline__ void joint_rows_lanes(const Dev& d, uint32_t i, uint32_t phase, float dt, float* ent,
                                                 GroupRows<G>& sm, uint32_t gmask, int gl, int gbase) {
    static_assert(3 * kJointWords <= kSlotWords && 3 * kJointRowsMost * kJointWords <= G * kSlotWords, "joint rows");
    constexpr uint32_t kJoints = uint32_t(G) / 3u;
    const uint32_t jcnt = d.jdeg[i], jlo = d.jinc_off[i];
    float* const stage = &sm.r[0][0];
    auto add_staged = [&](const float* row) {
#pragma unroll
        for (int q = 0; q < Owned<G>::E; ++q) {
            const int e = gl + G * q;
            if (e >= 27) continue;
            int ei = 0, ek = 0;
            if (e < 21) entry_ik(e, ei, ek);
            ent[q] += e < 21 ? row[6] * row[ei] * row[ek] : row[e - 21] * row[7];
            if (e < 21 && ei == ek && ei >= 3 && row[11] != 0.0f) ent[q] += row[8 + ei - 3];
        }
    };
    if (phase == 0) {
        const uint32_t mine = uint32_t(gl) / 3u, axis = uint32_t(gl) % 3u;
        for (uint32_t k = 0; k < jcnt;) {
            uint32_t j = 0, rows = 0;
            JointState js{};
            if (mine < kJoints && k + mine < jcnt) {
                j = d.jinc_list[jlo + k + mine];
                js = d.jstate[j];
                rows = js.enabled ? js.rows : 0u;
            }
            const uint32_t before = __popc(rows & ((1u << (axis * kAxisBits)) - 1u));
            uint32_t mask = (rows >> (axis * kAxisBits)) & kAxisMask;
            uint32_t count = __popc(mask), taken = min(kJoints, jcnt - k);
            uint32_t slot_words = kSlotWords;
            if (__any_sync(gmask, count > 3u)) {
                taken = 1;
                slot_words = kJointRowsMost * kJointWords;
                if (mine != 0) mask = count = 0;
            }
            if (mask) {
                const Joint& o = d.joints[j];
                const uint32_t type = o.type;
                const JointEnds en = load_ends(d, js.dense_a, js.dense_b);
                const JointOld old = load_joint_old(d.jold + size_t(j) * kOldWords, type);
                const JointPose pose = joint_pose(o, en.xa, en.qa, en.xb, en.qb);
                const V3 dir = rotate(pose.frame_a, unit_axis(axis));
                const bool first = i == js.dense_a;
                const JointRow* src = d.jrows + size_t(j) * 18 + before;
                float* out = stage + gl * slot_words;
                for (uint32_t m = mask; m; m &= m - 1u, ++src, out += kJointWords) {
                    const unsigned bit = __ffs(m) - 1;
                    const bool angular = bit >= kRowKinds;
                    const LaneRow r = lane_row(o, pose, old, dir, axis, angular, angular ? bit - kRowKinds : bit,
                                               en.dxa, en.dxb, Dual{src->lambda, src->penalty}, dt);
#pragma unroll
                    for (int c = 0; c < 6; ++c) out[c] = first ? r.ja.v[c] : r.jb.v[c];
                    out[6] = r.stiff;
                    out[7] = r.force;
                    out[11] = angular ? 0.0f : 1.0f;
                    if (!angular) {
                        const V3 curv = lane_curvature(dir, first ? add(pose.error, pose.arm_a) : pose.arm_b, r.force);
                        out[8] = curv.x;
                        out[9] = curv.y;
                        out[10] = curv.z;
                    }
                }
            }
            __syncwarp(gmask);
            for (uint32_t l = 0; l < 3u * taken; ++l) {
                const uint32_t n = __shfl_sync(gmask, count, gbase + int(l));
                for (uint32_t r = 0; r < n; ++r) add_staged(stage + l * slot_words + r * kJointWords);
            }
            __syncwarp(gmask);
            k += taken;
        }
    } else {
        // Velocity phase: the stored rows (formed by the phase's preparation).
        for (uint32_t k = 0; k < jcnt; ++k) {
            const uint32_t j = d.jinc_list[jlo + k];
            const JointState js = d.jstate[j];
            if (!js.enabled) continue;
            const bool first = i == js.dense_a;
            const Lite A = load_lite(d, js.dense_a), B = load_lite(d, js.dense_b);
            for (uint32_t base = 0; base < js.count; base += G) {
                const uint32_t r = base + uint32_t(gl);
                bool hard = false;
                if (r < js.count) {
                    const Row row = load_row(d.jrows[size_t(j) * 18 + r]);
                    hard = row.stiffness >= kMaxPenalty;
                    if (hard) {
                        // row_accumulate's terms
                        const float trial = row_trial(row, A.dx, B.dx, dt);
                        const bool two_sided = row.lower < 0.0f && row.upper > 0.0f;
                        float* out = stage + gl * kSlotWords;
#pragma unroll
                        for (int c = 0; c < 6; ++c) out[c] = first ? row.a.v[c] : row.b.v[c];
                        out[6] = two_sided || (trial > row.lower && trial < row.upper)
                                     ? row.dual.penalty + row.damping / dt
                                     : 0.0f;
                        out[7] = fclamp(trial, row.lower, row.upper) - row.reference_force;
                        out[11] = 0.0f;
                    }
                }
                constexpr uint32_t kLanes = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
                uint32_t m = (__ballot_sync(gmask, hard) >> gbase) & kLanes;
                __syncwarp(gmask);
                for (; m; m &= m - 1u) add_staged(stage + (__ffs(m) - 1) * kSlotWords);
                __syncwarp(gmask);
            }
        }
    }
}

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Joints: the world has joints (a world without them gets a build with no
// joint code, which needs fewer registers).
// ah: the body (its record and this lane's first row codes, fetched ahead);
// on return it holds the same for slot kn of the colour order (~0u: none).
template <int G, bool Joints>
__device__ void solve_body_group(const Dev& d, Ahead& ah, uint32_t kn, uint32_t phase, float dt, GroupRows<G>& sm,
                                 uint32_t gmask, int gl, int gbase, uint32_t trace = 0) {
    // trace 1: slowest body of the colour per stage; 2: stage times summed
    // over the colour's bodies (profiling only).
    const unsigned long long t0 = trace ? gtimer() : 0ull;
    auto mark = [&](int k) {
        if (trace == 1 && gl == 0) atomicMax(&d.ctr->dbg_body[k], gtimer() - t0);
        if (trace == 2 && gl == 0) atomicAdd(&d.ctr->dbg_sum[k], gtimer() - t0);
    };
    const uint32_t i = ah.i, ro = ah.ro, rn = ah.rn;
    const uint32_t code0 = ah.code0, other0 = ah.other0, code1 = ah.code1, other1 = ah.other1;
    uint4 nrec = make_uint4(0u, 0u, 0u, 0u);
    if (kn != ~0u) nrec = d.crec[kn];
    const Lite me = load_lite(d, i);
    float ent[Owned<G>::E];
    const float4 ia = d.inA[i], ib = d.inB[i];
    // The block's starting entries: inertia and its gradient. Formed after
    // the first chunk's rows are requested, so those loads and this body's
    // own state are in flight together.
    // The inertia block H is zero outside the linear diagonal and the
    // angular 3x3. Its gradient H dx is the serial sum over c = 0..5 from +0;
    // with dx finite, the sum's zero terms (0 x dx[c], exact zeros) leave
    // every partial sum unchanged (it is never -0), so each sum reduces to
    // its nonzero terms in order, bit for bit; a non-finite dx (0 x inf is
    // NaN) takes the full sums. All indices are compile-time (a lane's entry
    // picks its value by comparison), so nothing goes to local memory.
    auto init_entries = [&] {
        const V6& x = me.dx;
        bool finite = true;
#pragma unroll
        for (int c = 0; c < 6; ++c) finite = finite && fab(x.v[c]) < kFltMax;
        float gr[6];
        if (finite) {
            gr[0] = 0.0f + ia.x * x.v[0];
            gr[1] = 0.0f + ia.x * x.v[1];
            gr[2] = 0.0f + ia.x * x.v[2];
            gr[3] = ((0.0f + ia.y * x.v[3]) + ia.z * x.v[4]) + ib.x * x.v[5];
            gr[4] = ((0.0f + ia.z * x.v[3]) + ia.w * x.v[4]) + ib.y * x.v[5];
            gr[5] = ((0.0f + ib.x * x.v[3]) + ib.y * x.v[4]) + ib.z * x.v[5];
        } else {
            float H[21];
#pragma unroll
            for (int k = 0; k < 21; ++k) H[k] = 0.0f;
            H[bidx(0, 0)] = ia.x;
            H[bidx(1, 1)] = ia.x;
            H[bidx(2, 2)] = ia.x;
            H[bidx(3, 3)] = ia.y;
            H[bidx(4, 3)] = ia.z;
            H[bidx(5, 3)] = ib.x;
            H[bidx(4, 4)] = ia.w;
            H[bidx(5, 4)] = ib.y;
            H[bidx(5, 5)] = ib.z;
#pragma unroll
            for (int r = 0; r < 6; ++r) {
                float gs = 0.0f;
#pragma unroll
                for (int c = 0; c < 6; ++c) gs += H[bidx(r, c)] * x.v[c];
                gr[r] = gs;
            }
        }
#pragma unroll
        for (int q = 0; q < Owned<G>::E; ++q) {
            const int e = gl + G * q;
            float v = 0.0f;
            v = (e == int(bidx(0, 0)) || e == int(bidx(1, 1)) || e == int(bidx(2, 2))) ? ia.x : v;
            v = e == int(bidx(3, 3)) ? ia.y : v;
            v = e == int(bidx(4, 3)) ? ia.z : v;
            v = e == int(bidx(5, 3)) ? ib.x : v;
            v = e == int(bidx(4, 4)) ? ia.w : v;
            v = e == int(bidx(5, 4)) ? ib.y : v;
            v = e == int(bidx(5, 5)) ? ib.z : v;
#pragma unroll
            for (int r = 0; r < 6; ++r) v = e == 21 + r ? gr[r] : v;
            ent[q] = v;
        }
    };
    if (rn == 0) init_entries();
    for (uint32_t base = 0; base < rn; base += G) {
        const uint32_t sidx = base + gl;
        if (sidx < rn) {
            const int nslot = sidx < GroupRows<G>::kSlots ? int(sidx) : -1;
            const uint32_t code = base == 0 ? code0 : base == uint32_t(G) ? code1 : d.blist[ro + sidx];
            const uint32_t other = base == 0 ? other0 : base == uint32_t(G) ? other1 : d.bother[ro + sidx];
            stage_contact<G>(d, me, code, other, phase, sm, gl, nslot);
        }
        if (base == 0) init_entries();
        __syncwarp(gmask);
        accumulate_chunk<G>(ent, gl, sm, min(uint32_t(G), rn - base));
        __syncwarp(gmask);
    }
    // The next body's record and row codes, in flight while this one solves.
    if (kn != ~0u) {
        ah.i = nrec.x;
        ah.ro = nrec.y;
        ah.rn = nrec.z;
        ah.impact = nrec.w;
        fetch_codes<G>(d, ah, gl);
    }
    mark(0);
    if constexpr (Joints) joint_rows_lanes<G>(d, i, phase, dt, ent, sm, gmask, gl, gbase);
    mark(1);
    // The block's solution, then the crossing safeguard
    // (geometry_constraints_solve.slang:433-475) -- a ballot per chunk flags
    // the rows; rows past the kept normal rows are evaluated again into the
    // slots -- and, with the crossing rows added, the solution again. One loop
    // for both solutions: the factorisation is the longest code here.
    constexpr uint32_t kSlots = GroupRows<G>::kSlots;
    constexpr uint32_t kLanes = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
    V6 upd;
    float4 dq_start = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
#pragma unroll 1
    for (int pass = 0;; ++pass) {
        publish_entries<G>(ent, sm, gl);
        __syncwarp(gmask);
        Blk blk;
        read_block<G>(sm, blk);
        // Every lane has read the block before a lane writes its words again:
        // the second pass's entries, or the next body's rows.
        __syncwarp(gmask);
        V6 x;
        const bool solved = block_solve(blk, x);
        if (pass != 0) {
            if (solved) upd = x;
            break;
        }
        if (!solved) return;
        upd = x;
        mark(2);
        // The body's rotation offset, read while the safeguard runs (only
        // this group writes it in the colour), so the update at the end waits
        // on no load; its displacement is `me` (read at the start; both w
        // are 0).
        if (phase == 0) dq_start = d.dq[i];
        bool crossing = false;
        for (uint32_t base = 0; base < rn; base += G) {
            const uint32_t sidx = base + gl;
            if (base >= kSlots) {
                __syncwarp(gmask);  // the slots' previous rows are read
                if (sidx < rn)
                    stage_contact<G>(d, me, d.blist[ro + sidx], d.bother[ro + sidx], phase, sm, -1, int(sidx % kSlots));
                __syncwarp(gmask);
            }
            const bool f = sidx < rn && crosses(sm.nrow[sidx % kSlots], upd);
            const uint32_t m = (__ballot_sync(gmask, f) >> gbase) & kLanes;
            if (m) {
                if (!crossing) own_entries<G>(sm, gl, ent);
                crossing = true;
                accumulate_crossing<G>(ent, gl, sm, base % kSlots, min(uint32_t(G), rn - base), m);
            }
        }
        mark(3);
        if (!crossing) break;
    }
    mark(4);
    if (trace == 1 && gl == 0) atomicMax(&d.ctr->dbg_rn, rn);
    if (trace == 2 && gl == 0) {
        atomicAdd(&d.ctr->dbg_sum[6], 1ull);
        atomicAdd(&d.ctr->dbg_sum[7], (unsigned long long)rn);
    }
    if (gl == 0) {
        float4 l = make_float4(me.dx.v[0], me.dx.v[1], me.dx.v[2], 0.0f);
        if (phase == 0) {
            apply_pose_update(d, i, upd, l, dq_start);
        } else {
            float4 a = make_float4(me.dx.v[3], me.dx.v[4], me.dx.v[5], 0.0f);
            l.x += upd.v[0];
            l.y += upd.v[1];
            l.z += upd.v[2];
            a.x += upd.v[3];
            a.y += upd.v[4];
            a.z += upd.v[5];
            d.dx[2 * i] = l;
            d.dx[2 * i + 1] = a;
        }
    }
}

// One thread solves body i: the serial loop of geometry_constraints_solve.
// slang:339-475 as written -- add_row per contact row in list order, the
// joints' rows, LDL^T, then the crossing safeguard over the normal rows --
// for colours with far more bodies than the grid has lane groups, where a
// body per thread finishes the colour in fewer rounds than wider groups.
// `sb`: this thread's shared-memory block slot for the joint visit.
__device__ __forceinline__ float load_normal_rows(const Dev& d, uint32_t c, V6& ja, V6& jb) {
    const float* p = reinterpret_cast<const float*>(d.c_row + size_t(c) * 8);
    const V3 n{p[0], p[1], p[2]};
    ja = jac(V3{-n.x, -n.y, -n.z}, V3{p[9], p[10], p[11]});
    jb = jac(n, V3{p[18], p[19], p[20]});
    return p[29];  // the error at the phase's start
}
template <bool Joints>
__device__ void solve_body_thread(const Dev& d, uint32_t i, uint32_t phase, float dt, Blk* sb, BodyView* views) {
    const Lite me = load_lite(d, i);
    const uint32_t ro = d.roff[i], rn = d.rcount[i];
    Blk blk;
    {
        const float4 ia = d.inA[i], ib = d.inB[i];
#pragma unroll
        for (int k = 0; k < 21; ++k) blk.h[k] = 0.0f;
        blk.h[bidx(0, 0)] = ia.x;
        blk.h[bidx(1, 1)] = ia.x;
        blk.h[bidx(2, 2)] = ia.x;
        blk.h[bidx(3, 3)] = ia.y;
        blk.h[bidx(4, 3)] = ia.z;
        blk.h[bidx(5, 3)] = ib.x;
        blk.h[bidx(4, 4)] = ia.w;
        blk.h[bidx(5, 4)] = ib.y;
        blk.h[bidx(5, 5)] = ib.z;
#pragma unroll
        for (int r = 0; r < 6; ++r) {
            float gs = 0.0f;
#pragma unroll
            for (int c = 0; c < 6; ++c) gs += blk.h[bidx(r, c)] * me.dx.v[c];
            blk.g[r] = gs;
        }
    }
    for (uint32_t r = 0; r < rn; ++r) {
        const uint32_t code = d.blist[ro + r], other_body = d.bother[ro + r];
        const uint32_t c = code & 0x7fffffffu;
        const bool first = (code >> 31) == 0;
        const Lite other = load_lite(d, other_body);
        const Lite A = first ? me : other, B = first ? other : me;
        const float4 lam = d.c_lam[c], pen = d.c_pen[c];
        const ContactRow cr = load_row32(d, c);
        float err[3];
        contact_errors(cr, A, B, err);
        const F3 trial{lam.x + pen.x * err[0], lam.y + pen.y * err[1], lam.z + pen.z * err[2]};
        F3 f, sc;
        project_with_scales(trial, cr.friction, f, sc);
        float forces[3] = {f.n, f.t0, f.t1};
        if (phase != 0) {
            const float4 fo = d.c_foff[c];
            forces[0] = f.n - fo.x;
            forces[1] = f.t0 - fo.y;
            forces[2] = f.t1 - fo.z;
        }
        const float st[3] = {pen.x * sc.n, pen.y * sc.t0, pen.z * sc.t1};
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            V6 row;
            const V6 ja = cr.ja(x), jb = cr.jb(x);
#pragma unroll
            for (int k = 0; k < 6; ++k) row.v[k] = first ? ja.v[k] : jb.v[k];
            add_row(blk, row, st[x], forces[x]);
        }
    }
    if constexpr (Joints) {
        if (d.jdeg[i]) {
            // The joint visit takes the block's address: work on this thread's
            // shared-memory copy so the register block never needs one.
            *sb = blk;
            const uint32_t jcnt = d.jdeg[i], jlo = d.jinc_off[i];
            for (uint32_t k = 0; k < jcnt; ++k) {
                const uint32_t j = d.jinc_list[jlo + k];
                const JointState js = d.jstate[j];
                if (!js.enabled) continue;
                const uint32_t a = js.dense_a, b = js.dense_b;
                const bool first = i == a;
                if (phase == 0) {
                    views[0] = load_body(d, a);
                    views[1] = load_body(d, b);
                    visit_joint(d.joints[j], d.jrows + size_t(j) * 18, views[0], views[1], v3(d.x[a]), q4(d.q[a]),
                                v3(d.x[b]), q4(d.q[b]), d.p0[a], d.p0[b], dt, sb, first, kVisitAccumulate, nullptr);
                } else {
                    const Lite A = load_lite(d, a), B = load_lite(d, b);
                    for (uint32_t r = 0; r < js.count; ++r) {
                        Row row = load_row(d.jrows[size_t(j) * 18 + r]);
                        if (row.stiffness >= kMaxPenalty) row_accumulate(*sb, row, first, A.dx, B.dx, dt);
                    }
                }
            }
            blk = *sb;
        }
    }
    V6 upd;
    if (!block_solve(blk, upd)) return;
    // Crossing safeguard: the normal rows again, at the same displacements.
    bool crossing = false;
    for (uint32_t r = 0; r < rn; ++r) {
        const uint32_t code = d.blist[ro + r], other_body = d.bother[ro + r];
        const uint32_t c = code & 0x7fffffffu;
        const bool first = (code >> 31) == 0;
        const Lite other = load_lite(d, other_body);
        const Lite A = first ? me : other, B = first ? other : me;
        V6 ja, jb;
        const float e0 = load_normal_rows(d, c, ja, jb);
        const float err0 = e0 + dot6(ja, A.dx) + dot6(jb, B.dx);
        const float k0 = d.c_pen[c].x;
        const float trial = d.c_lam[c].x + k0 * err0;
        V6 nr;
#pragma unroll
        for (int k = 0; k < 6; ++k) nr.v[k] = first ? ja.v[k] : jb.v[k];
        if (trial <= 0.0f && trial + k0 * dot6(nr, upd) > k0 * 1.0e-6f) {
            add_row(blk, nr, k0, trial);
            crossing = true;
        }
    }
    if (crossing) {
        V6 safe;
        if (block_solve(blk, safe)) upd = safe;
    }
    if (phase == 0) {
        apply_pose_update(d, i, upd);
    } else {
        float4 l = d.dx[2 * i], a = d.dx[2 * i + 1];
        l.x += upd.v[0];
        l.y += upd.v[1];
        l.z += upd.v[2];
        a.x += upd.v[3];
        a.y += upd.v[4];
        a.z += upd.v[5];
        d.dx[2 * i] = l;
        d.dx[2 * i + 1] = a;
    }
}

// Residual accumulator of one dual pass (this build's addition): rows that
// carry force or penetrate contribute |C_n| (force > 0) or C_n (penetration
// only); hard joint rows contribute |C|. Reported as the RMS, the largest
// value, and the number of rows above the schedule's tolerance.
struct Res {
    double sq;
    uint32_t n;
    float mx;
    uint32_t over;
    float tol;
};
__device__ __forceinline__ void res_add(Res& r, float v) {
    r.sq += double(v) * double(v);
    r.n += 1;
    r.mx = fmx(r.mx, v);
    if (v > r.tol) r.over += 1;
}

// advance_duals for one contact point (geometry_constraints_solve.slang:
// 494-532; the last-iteration block runs in k_finish_contacts). ab: the
// contact's bodies (c_bodies[c]), loaded by the caller ahead of time.
static __device__ void dual_contact(const Dev& d, uint32_t c, uint2 ab, float dt, uint32_t phase, Res& res,
                                    uint32_t it) {
    const uint32_t a = ab.x, b = ab.y;
    if (phase != 0 && d.impact[a] == 0 && d.impact[b] == 0) return;
    // Batched worlds: a scene past its budget is finished; its last sweep
    // feeds the scene's residual.
    uint32_t scene = 0;
    bool scene_last = false;
    if (batched(d)) {
        scene = d.scene_of[a];
        const uint32_t budget = d.scene_budget[scene];
        if (it >= budget) return;
        scene_last = phase == 0 && it + 1 == budget;  // the tick's residual is the pose phase's
    }
    const Lite A = load_lite(d, a), B = load_lite(d, b);
    float4 lam = d.c_lam[c], pen = d.c_pen[c];
    const ContactRow cr = load_row32(d, c);
    const float friction = cr.friction, beta = cr.beta;
    float err[3];
    contact_errors(cr, A, B, err);
    F3 f = project_contact(F3{lam.x + pen.x * err[0], lam.y + pen.y * err[1], lam.z + pen.z * err[2]}, friction);
    const float tx = lam.y + pen.y * err[1];
    const float ty = lam.z + pen.z * err[2];
    const float bound = friction * f.n;
    const bool stick = tx * tx + ty * ty <= bound * bound;
    lam.x = f.n;
    lam.y = f.t0;
    lam.z = f.t1;
    if (f.n > 0.0f) pen.x = fmn(kMaxPenalty, pen.x + beta * fab(err[0]));
    if (stick) {
        pen.y = fmn(kMaxPenalty, pen.y + beta * fab(err[1]));
        pen.z = fmn(kMaxPenalty, pen.z + beta * fab(err[2]));
    }
    pen.w = stick ? 1.0f : 0.0f;
    d.c_lam[c] = lam;
    d.c_pen[c] = pen;
    if (f.n > 0.0f || err[0] > 0.0f) {
        const float v = f.n > 0.0f ? fab(err[0]) : err[0];
        res_add(res, v);
        if (scene_last) {
            atomicAdd(&d.scene_res_sq[scene], v * v);
            atomicAdd(&d.scene_res_n[scene], 1u);
            atomicMax(reinterpret_cast<int*>(&d.scene_res_mx[scene]), __float_as_int(v));
        }
    }
}

// One thread's dual update of a joint.
static __device__ void dual_joint(const Dev& d, uint32_t j, uint32_t phase, float dt, Res& res, uint32_t it) {
    JointState js = d.jstate[j];
    if (js.count == 0 || !js.enabled) return;
    const uint32_t a = js.dense_a, b = js.dense_b;
    if (phase != 0 && d.impact[a] == 0 && d.impact[b] == 0) return;
    uint32_t scene = 0;
    bool scene_last = false;
    if (batched(d)) {
        scene = d.scene_of[a];
        const uint32_t budget = d.scene_budget[scene];
        if (it >= budget) return;
        scene_last = it + 1 == budget;
    }
    float impulse = 0.0f;
    if (phase == 0) {
        const BodyView va = load_body(d, a), vb = load_body(d, b);
        JointRes jr{0.0, 0u, 0.0f, 0u};
        // An advance visit leaves the block alone (no block pointer).
        impulse = visit_joint(d.joints[j], d.jrows + size_t(j) * 18, va, vb, v3(d.x[a]), q4(d.q[a]), v3(d.x[b]),
                              q4(d.q[b]), d.p0[a], d.p0[b], dt, nullptr, true, kVisitAdvance, nullptr, &jr, res.tol);
        // The joint's own residual (a batched world also needs it per scene),
        // added in the same order as a running sum would.
        res.sq += jr.sq;
        res.n += jr.n;
        res.mx = fmx(res.mx, jr.mx);
        res.over += jr.over;
        if (scene_last && jr.n) {
            atomicAdd(&d.scene_res_sq[scene], float(jr.sq));
            atomicAdd(&d.scene_res_n[scene], jr.n);
            atomicMax(reinterpret_cast<int*>(&d.scene_res_mx[scene]), __float_as_int(fmx(jr.mx, 0.0f)));
        }
    } else {
        const Lite A = load_lite(d, a), B = load_lite(d, b);
        for (uint32_t r = 0; r < js.count; ++r) {
            JointRow& s = d.jrows[size_t(j) * 18 + r];
            Row row = load_row(s);
            impulse += fab(row.stiffness < kMaxPenalty ? row.reference_force : row_force(row, A.dx, B.dx, dt)) * dt;
            if (row.stiffness >= kMaxPenalty) store_row(s, row_advance(row, A.dx, B.dx));
        }
    }
    js.applied = impulse;
    const float thr = d.joints[j].breaking_threshold;
    if (thr > 0.0f && impulse > thr) {
        js.broken = 1;
        js.enabled = 0;
    }
    d.jstate[j] = js;
}

// dual_joint's position phase by four lanes: lane l < 3 of the quad takes
// axis l; the sums over the joint's rows (impulse, residual) run through the
// lanes in row order. Of a row, only its dual changes from sweep to sweep (the
// rest is formed anew by every visit), so only that is stored. All four lanes
// call it, with the same j.
static __device__ __forceinline__ void dual_joint_quad(const Dev& d, uint32_t j, float dt, Res& res, uint32_t it,
                                                       uint32_t axis, uint32_t qmask, int qbase) {
    JointState js = d.jstate[j];
    if (js.count == 0 || !js.enabled) return;
    const uint32_t a = js.dense_a, b = js.dense_b;
    uint32_t scene = 0;
    bool scene_last = false;
    if (batched(d)) {
        scene = d.scene_of[a];
        const uint32_t budget = d.scene_budget[scene];
        if (it >= budget) return;
        scene_last = it + 1 == budget;
    }
    const Joint& o = d.joints[j];
    float impulse[kJointRowsMost], viol[kJointRowsMost];
    uint32_t count = 0;
    {
        const uint32_t mask = axis < 3 ? (js.rows >> (axis * kAxisBits)) & kAxisMask : 0u;
        const uint32_t before = __popc(js.rows & ((1u << (axis * kAxisBits)) - 1u));
        count = __popc(mask);
        if (mask) {
            const JointEnds en = load_ends(d, a, b);
            const JointOld old = load_joint_old(d.jold + size_t(j) * kOldWords, o.type);
            const JointPose pose = joint_pose(o, en.xa, en.qa, en.xb, en.qb);
            const V3 dir = rotate(pose.frame_a, unit_axis(axis));
            uint32_t m = mask;
#pragma unroll
            for (int r = 0; r < kJointRowsMost; ++r) {
                impulse[r] = viol[r] = 0.0f;
                if (!m) continue;
                const unsigned bit = __ffs(m) - 1;
                m &= m - 1u;
                const bool angular = bit >= kRowKinds;
                JointRow& s = d.jrows[size_t(j) * 18 + before + r];
                const Dual dual{s.lambda, s.penalty};
                const LaneRow row = lane_row(o, pose, old, dir, axis, angular, angular ? bit - kRowKinds : bit, en.dxa,
                                             en.dxb, dual, dt);
                impulse[r] = fab(row.force) * dt;
                viol[r] = row.stiffness >= kMaxPenalty ? fab(row.error) : -1.0f;  // -1: no hard row
                const Dual next = update_dual(dual, row.error, s.beta, row.lower, row.upper, row.stiffness);
                s.lambda = next.lambda;
                s.penalty = next.penalty;
            }
        }
    }
    float sum = 0.0f;
    JointRes jr{0.0, 0u, 0.0f, 0u};
#pragma unroll
    for (uint32_t l = 0; l < 3; ++l) {
        if (axis == l)
#pragma unroll
            for (int r = 0; r < kJointRowsMost; ++r)
                if (r < int(count)) {
                    sum += impulse[r];
                    const float v = viol[r];
                    if (!(v < 0.0f)) {
                        jr.sq += double(v) * double(v);
                        jr.n += 1;
                        jr.mx = fmx(jr.mx, v);
                        if (v > res.tol) jr.over += 1;
                    }
                }
        sum = __shfl_sync(qmask, sum, qbase + int(l));
        jr.sq = __shfl_sync(qmask, jr.sq, qbase + int(l));
        jr.n = __shfl_sync(qmask, jr.n, qbase + int(l));
        jr.mx = __shfl_sync(qmask, jr.mx, qbase + int(l));
        jr.over = __shfl_sync(qmask, jr.over, qbase + int(l));
    }
    if (axis != 0) return;
    res.sq += jr.sq;
    res.n += jr.n;
    res.mx = fmx(res.mx, jr.mx);
    res.over += jr.over;
    if (scene_last && jr.n) {
        atomicAdd(&d.scene_res_sq[scene], float(jr.sq));
        atomicAdd(&d.scene_res_n[scene], jr.n);
        atomicMax(reinterpret_cast<int*>(&d.scene_res_mx[scene]), __float_as_int(fmx(jr.mx, 0.0f)));
    }
    js.applied = sum;
    const float thr = o.breaking_threshold;
    if (thr > 0.0f && sum > thr) {
        js.broken = 1;
        js.enabled = 0;
    }
    d.jstate[j] = js;
}

// One block's residual partials into slot `slot` of the counters: warp
// trees, then warps in order (deterministic).
template <int T>
__device__ __forceinline__ void block_residual(Res res, double* wsq, uint32_t* wn, float* wmx, uint32_t* wov,
                                               Counters* c, uint32_t slot) {
    for (int o = 16; o > 0; o >>= 1) {
        res.sq += __shfl_xor_sync(0xffffffffu, res.sq, o);
        res.n += __shfl_xor_sync(0xffffffffu, res.n, o);
        res.mx = fmx(res.mx, __shfl_xor_sync(0xffffffffu, res.mx, o));
        res.over += __shfl_xor_sync(0xffffffffu, res.over, o);
    }
    if ((threadIdx.x & 31) == 0) {
        wsq[threadIdx.x >> 5] = res.sq;
        wn[threadIdx.x >> 5] = res.n;
        wmx[threadIdx.x >> 5] = res.mx;
        wov[threadIdx.x >> 5] = res.over;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double bs = 0.0;
        uint32_t bn = 0, bo = 0;
        float bm = 0.0f;
        for (int k = 0; k < T / 32; ++k) {
            bs += wsq[k];
            bn += wn[k];
            bm = fmx(bm, wmx[k]);
            bo += wov[k];
        }
        c->res_sum[slot] = bs;
        c->res_cnt[slot] = bn;
        c->res_mx[slot] = bm;
        c->res_over[slot] = bo;
    }
}

// The sweep's residual from every block's partials (slots base .. base +
// gridDim.x): RMS, largest row violation, fraction of rows above the
// tolerance, and whether the schedule's measure meets the tolerance
// (residual_norm 0: every row within it; 1: the RMS; 2: at most one row in a
// thousand above it).
struct SweepResidual {
    float rms, mx, over, measure;
    bool met;
};
// Every block needs the same decision, so every block sums the partials in
// the same order. One warp per block reads them -- each lane the slots of its
// index modulo 32, all loads in flight at once -- and adds the lanes' sums in
// a tree (when every thread walked the slots itself, the whole grid's
// uncached reads of the same few L2 lines kept each sweep's start waiting
// tens of microseconds; the 148 slots one after another took 2 us a sweep).
__device__ __forceinline__ SweepResidual sweep_residual(Counters* c, uint32_t base, const StepParams& sp) {
    __shared__ SweepResidual shared_result;
    if (threadIdx.x < 32) {
        const uint32_t lane = threadIdx.x;
        double tsq = 0.0;
        uint32_t tn = 0, to = 0;
        float tmx = 0.0f;
        constexpr uint32_t kAhead = 5;  // slots per lane loaded together (160 blocks)
        for (uint32_t k0 = 0; k0 < gridDim.x; k0 += 32u * kAhead) {
            double sq[kAhead];
            uint32_t cn[kAhead], ov[kAhead];
            float mx[kAhead];
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j) {
                const uint32_t k = k0 + 32u * j + lane;
                const bool in = k < gridDim.x;
                sq[j] = in ? ((volatile double*)c->res_sum)[base + k] : 0.0;
                cn[j] = in ? ((volatile uint32_t*)c->res_cnt)[base + k] : 0u;
                mx[j] = in ? ((volatile float*)c->res_mx)[base + k] : 0.0f;
                ov[j] = in ? ((volatile uint32_t*)c->res_over)[base + k] : 0u;
            }
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j) {
                tsq += sq[j];
                tn += cn[j];
                tmx = fmx(tmx, mx[j]);
                to += ov[j];
            }
        }
        for (int o = 16; o > 0; o >>= 1) tsq += __shfl_xor_sync(0xffffffffu, tsq, o);
        for (int o = 16; o > 0; o >>= 1) tmx = fmx(tmx, __shfl_xor_sync(0xffffffffu, tmx, o));
        tn = __reduce_add_sync(0xffffffffu, tn);
        to = __reduce_add_sync(0xffffffffu, to);
        if (lane == 0) {
            SweepResidual r;
            r.rms = tn ? float(sqrt(tsq / double(tn))) : 0.0f;
            r.mx = tmx;
            r.over = tn ? float(to) / float(tn) : 0.0f;
            if (sp.residual_norm == 1) {
                r.measure = r.rms;
                r.met = r.rms <= sp.tolerance;
            } else if (sp.residual_norm == 2) {
                r.measure = r.over;
                r.met = uint64_t(to) * 1000u <= uint64_t(tn);
            } else {
                r.measure = tmx;
                r.met = tmx <= sp.tolerance;
            }
            shared_result = r;
        }
    }
    __syncthreads();
    return shared_result;
}

__device__ __forceinline__ void atomic_max_pos(float* addr, float v) {
    atomicMax(reinterpret_cast<int*>(addr), __float_as_int(fmx(v, 0.0f)));
}

}  // namespace pmb
