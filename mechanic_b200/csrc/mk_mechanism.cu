// mk_mechanism.cu — articulated passes of the tick.
//
// Stage map (reference kernel -> this file), in the dispatch order of
// device.rs:963-1155:
//   articulated.wgsl project_bearing_velocities :287-316
//   and apply_velocity_deltas :318-337                     -> k_bearing_pass
//   articulated.wgsl advance_coordinates :366-415          -> k_advance_coordinates
//   mechanism.wgsl prepare_links / jump_* :72-149          -> k_prepare_links / k_jump (list-restricted)
//   closure.wgsl evaluate / finalize / solve_closure_pcg   -> k_closure_block (systems that fit its shared memory, all
//                                                             12 Newton steps), else k_closure_loop (one block or grid)
//   mechanism.wgsl publish_* :151-185                      -> k_publish
//   articulated.wgsl reconstruct_body_velocities :431-456  -> k_reconstruct_level (one launch per depth), or
//                                                             k_reconstruct_rows / _walk / _store (deep, narrow trees)
//   articulated.wgsl capture_coordinates :417-429          -> k_capture_coordinates
//   articulated.wgsl validate_articulated_state :458-484   -> k_validate_state
//   bearings.wgsl validate_* :68-102                       -> k_validate_bearings
//   articulated.wgsl project_bearing_velocities_serial     -> k_project_bearings_serial
//
// The serial reconstruction becomes level-synchronous (every body of depth
// d after all of depth d-1: the same arithmetic per body, so the same bits).
// The closure accumulators are gathered per coordinate from per-joint slots
// in the serial accumulation order instead of float atomics.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <vector>

#include "mk_device.cuh"
#include "mk_mechanism.h"
#include "mk_mlp.h"

namespace mk {

constexpr uint32_t kMBlock = 256;
constexpr uint32_t kPassBlock = 128;       // threads of a bearing projection block
constexpr uint32_t kClosureThreads = 1024;
constexpr uint32_t kClosureSteps = 12;     // device.rs:974
constexpr uint32_t kClosureRounds = 8;     // closure.wgsl:356
constexpr uint32_t kMaxLoop = 8;           // coordinates of one per-loop preconditioner block (storage)
// A closure constrains 5 directions (3 of position, 2 of its hinge axis), so a
// loop's J^T J has rank at most 5: a block of more of its coordinates is
// singular (its Cholesky then hangs on the ridge alone, and the preconditioned
// iteration diverged on 16-body loops).  Loops are cut into pieces of 5.
constexpr uint32_t kLoopPiece = 5;
constexpr uint32_t kSideRows = 6;         // float4 per bearing side in the projection cache
constexpr uint32_t kWalkWidth = 4096;      // most bodies of a level of k_reconstruct_walk (two in shared memory)
constexpr uint32_t kLongList = 256;        // slot runs longer than this are summed in chunks of this many

// ----------------------------------------------------------------- host side
MechParams make_mech_params(const MkCreation* cr, const StepParams& p, uint32_t iterations, uint32_t closure_mode,
                            float closure_tol, uint32_t closure_max_it, uint32_t learned_precond) {
    MechParams m;
    m.body_count = cr->body_count;
    m.bearing_count = cr->bearing_count;
    m.coordinate_count = cr->coordinate_count;
    m.max_depth = cr->max_depth;
    m.closure_count = cr->closure_count;
    uint32_t covered = 1, rounds = 0;
    while (covered < cr->max_depth) { covered *= 2; ++rounds; }
    if (cr->max_depth > 0 && rounds == 0) rounds = 1;
    m.jump_rounds = rounds;
    m.final_is_a = (rounds % 2 == 0) ? 1u : 0u;
    m.iterations = iterations;
    m.closure_mode = closure_mode;
    m.has_dynamic_root = cr->has_dynamic_root;
    m.serial_contacts = (cr->max_depth > 0 && cr->has_dynamic_root && cr->bearing_count <= 64) ? 1u : 0u;
    m.dt = p.dt;
    m.ang_damp = p.ang_damp;
    m.closure_tol = closure_tol > 0.0f ? closure_tol : 1.0e-5f;
    m.closure_max_it = closure_max_it ? closure_max_it : 256u;
    m.learned_precond = (closure_mode == MK_CLOSURE_PCG_RESIDUAL && learned_precond == MK_PRECOND_LEARNED) ? 1u : 0u;
    m.precond = learned_precond;
    return m;
}

bool pcg_residual_mode(const MechParams& p) { return p.closure_mode == MK_CLOSURE_PCG_RESIDUAL && p.closures > 0; }

// Tables of the one-block closure solve (k_closure_block), for systems whose
// counts it can hold; p.block_solve stays 0 for the others and for topologies
// where a branch leaves its component or two joints share a coordinate.
constexpr uint32_t kClosureSmem = 220u * 1024u;   // its dynamic shared memory at most
constexpr uint32_t kBlockChunks = 2;              // 1,024-coordinate chunks that its registers hold
static void derive_block_solve(const MkCreation* cr, MechParams& p, MechTopology& t) {
    const GpuMechanismBody* mb = cr->mechanism_bodies;
    const uint32_t NC = p.closures, S = p.slots, B = cr->body_count;
    if (NC == 0 || p.long_coords || p.closure_coords > kBlockChunks * kClosureThreads || p.loops > kClosureThreads) return;
    if ((uint64_t)S * 40u > kClosureSmem || (uint64_t)NC * 28u > kClosureSmem) return;
    // closures by falling slot count, and the first entry of each place among their slots
    auto slots_of = [&](uint32_t k) { return t.cl_slot_off[k + 1] - t.cl_slot_off[k]; };
    t.cl_order.resize(NC);
    for (uint32_t k = 0; k < NC; ++k) t.cl_order[k] = k;
    std::stable_sort(t.cl_order.begin(), t.cl_order.end(),
                     [&](uint32_t x, uint32_t y) { return slots_of(x) > slots_of(y); });
    p.closure_depth = slots_of(t.cl_order[0]);
    t.cl_columns.assign(p.closure_depth + 1, 0u);
    for (uint32_t k : t.cl_order)
        for (uint32_t j = 0; j < slots_of(k); ++j) ++t.cl_columns[j + 1];
    for (uint32_t j = 0; j < p.closure_depth; ++j) t.cl_columns[j + 1] += t.cl_columns[j];
    // in that order: coordinate (position) | closure << 16, and place in the runs
    std::vector<uint32_t> q_of(S, 0u);
    for (uint32_t q = 0; q < p.closure_coords; ++q)
        for (uint32_t i = t.cq_off[q]; i < t.cq_off[q + 1]; ++i) q_of[t.cq_slots[i]] = q;
    t.col_coord.resize(S);
    t.col_pos.resize(S);
    for (uint32_t k = 0; k < NC; ++k) {
        const uint32_t s0 = t.cl_slot_off[t.cl_order[k]];
        for (uint32_t j = 0; j < slots_of(t.cl_order[k]); ++j) {
            t.col_coord[t.cl_columns[j] + k] = q_of[s0 + j] | (k << 16);
            t.col_pos[t.cl_columns[j] + k] = t.slot_pos[s0 + j];
        }
    }
    // places in cb_bodies: of the closures' bodies, each slot's parent, each coordinate's child body, the parents
    bool ok = true;
    std::vector<uint32_t> place(B, kInvalid);
    for (uint32_t i = 0; i < p.closure_bodies; ++i) place[t.cb_bodies[i]] = i;
    auto find = [&](uint32_t body) {
        const uint32_t at = body < B ? place[body] : kInvalid;
        ok = ok && at != kInvalid;
        return at == kInvalid ? 0u : at;
    };
    for (uint32_t j : t.cl_bearings)
        for (int side = 0; side < 2; ++side) t.cl_places.push_back(find(cr->bearings[j].metadata[side]));
    for (uint32_t body : t.slot_body) t.slot_parent.push_back(find(mb[body].metadata[0]));
    for (uint32_t q = 0; q < p.closure_coords; ++q) t.cq_child.push_back(find(t.slot_body[t.cq_slots[t.cq_off[q]]]));
    std::vector<uint8_t> driven(cr->coordinate_count, 0);
    for (uint32_t body : t.cb_bodies) {
        t.cb_parents.push_back(find(mb[body].metadata[3] ? body : mb[body].metadata[0]));
        if (mb[body].metadata[3]) continue;
        const uint32_t coord = cr->bearings[mb[body].metadata[1]].metadata[2];
        if (coord >= cr->coordinate_count || driven[coord]) ok = false;
        else driven[coord] = 1;
    }
    p.block_solve = ok ? 1u : 0u;
}

MechTopology derive_topology(const MkCreation* cr, MechParams& p) {
    MechTopology t;
    const uint32_t B = cr->body_count;
    if (cr->max_depth == 0 || !cr->mechanism_bodies) return t;
    const GpuMechanismBody* mb = cr->mechanism_bodies;
    // projection passes: bodies with bearings first; their bearing sides in lists of whole warps, a body's sides
    // inside one warp (bodies of more than 32 in a list of their own)
    {
        std::vector<uint32_t> off(B + 1ull, 0u);
        for (uint32_t j = 0; j < cr->bearing_count; ++j)
            for (int side = 0; side < 2; ++side)
                if (cr->bearings[j].metadata[side] < B) ++off[cr->bearings[j].metadata[side] + 1u];
        for (uint32_t i = 0; i < B; ++i)
            if (off[i + 1]) t.pass_bodies.push_back(i);
        p.bearing_bodies = (uint32_t)t.pass_bodies.size();
        for (uint32_t i = 0; i < B; ++i)
            if (!off[i + 1]) t.pass_bodies.push_back(i);
        for (uint32_t i = 0; i < B; ++i) off[i + 1] += off[i];
        std::vector<uint2> entries(off[B]);   // 2 bearing + side, the other body
        std::vector<uint32_t> at(off.begin(), off.end() - 1);
        for (uint32_t j = 0; j < cr->bearing_count; ++j)
            for (uint32_t side = 0; side < 2; ++side) {
                const uint32_t body = cr->bearings[j].metadata[side], other = cr->bearings[j].metadata[side ^ 1u];
                if (body < B) entries[at[body]++] = make_uint2(2u * j + side, std::min(other, B - 1u));
            }
        t.side_place.resize(cr->bearing_count, make_uint2(0u, 0u));
        auto put_side = [&](const uint2& en) {
            (en.x & 1u ? t.side_place[en.x >> 1].y : t.side_place[en.x >> 1].x) = (uint32_t)t.side_entries.size();
            t.side_entries.push_back(make_uint2(en.x & 1u, en.y));
        };
        auto pad_to = [&](size_t n) {
            t.side_body.resize(n, kInvalid);
            t.side_entries.resize(n, make_uint2(0u, 0u));
        };
        for (uint32_t i = 0; i < p.bearing_bodies; ++i) {
            const uint32_t body = t.pass_bodies[i], n = off[body + 1] - off[body];
            if (n > 32u) {
                t.hub_bodies.push_back(body);
                continue;
            }
            const size_t used = t.side_body.size() % 32u;
            if (used + n > 32u) pad_to(t.side_body.size() + 32u - used);
            t.side_body.insert(t.side_body.end(), n, body);
            for (uint32_t q = off[body]; q < off[body + 1]; ++q) put_side(entries[q]);
            p.most_sides = std::max(p.most_sides, n);
        }
        pad_to((t.side_body.size() + kPassBlock - 1) / kPassBlock * kPassBlock);
        p.padded_sides = (uint32_t)t.side_body.size();
        for (uint32_t h = 0; h < (uint32_t)t.hub_bodies.size(); ++h) {
            const uint32_t body = t.hub_bodies[h], n = off[body + 1] - off[body];
            for (uint32_t k = 0; k < n; k += kPassBlock)
                t.hub_chunks.push_back(make_uint4(body, (uint32_t)t.side_entries.size() + k,
                                                  std::min(n - k, kPassBlock) | h << 8, (n + kPassBlock - 1) / kPassBlock));
            for (uint32_t q = off[body]; q < off[body + 1]; ++q) put_side(entries[q]);
        }
        p.hub_bodies = (uint32_t)t.hub_bodies.size();
        p.hub_chunks = (uint32_t)t.hub_chunks.size();
        p.all_sides = (uint32_t)t.side_entries.size();
    }
    // depth levels 1..max_depth (roots are skipped by the reconstruction)
    t.level_offsets.assign(cr->max_depth + 2, 0);
    for (uint32_t i = 0; i < B; ++i)
        if (!mb[i].metadata[3] && mb[i].traversal[1] <= cr->max_depth) ++t.level_offsets[mb[i].traversal[1] + 1];
    for (size_t l = 1; l < t.level_offsets.size(); ++l) t.level_offsets[l] += t.level_offsets[l - 1];
    t.level_bodies.resize(t.level_offsets.back());
    std::vector<uint32_t> fill(t.level_offsets.begin(), t.level_offsets.end() - 1);
    for (uint32_t i = 0; i < B; ++i)
        if (!mb[i].metadata[3] && mb[i].traversal[1] <= cr->max_depth) t.level_bodies[fill[mb[i].traversal[1]]++] = i;
    // deep, narrow trees are walked by one block (k_reconstruct_walk): a launch per level costs about
    // as much as 8 rounds of 1,024 bodies there (5 us against 0.6 us), and the row kernel a few launches
    {
        const uint32_t levels = (uint32_t)t.level_offsets.size() - 1u;
        uint64_t rounds = 0;
        uint32_t widest = 0;
        bool filled = true;   // every level down to the deepest has its parents in the level before
        for (uint32_t l = 1; l < levels; ++l) {
            const uint32_t n = t.level_offsets[l + 1] - t.level_offsets[l];
            rounds += (n + 1023) / 1024;
            widest = std::max(widest, n);
        }
        std::vector<uint32_t> at(B, kInvalid);
        if (levels > 16 && widest <= kWalkWidth && rounds <= 8ull * levels) {
            for (uint32_t l = 0; l < levels; ++l)
                for (uint32_t i = t.level_offsets[l]; i < t.level_offsets[l + 1]; ++i)
                    at[t.level_bodies[i]] = i - t.level_offsets[l];
            t.level_parent.resize(t.level_bodies.size());
            for (uint32_t i = 0; i < (uint32_t)t.level_bodies.size(); ++i) {
                const GpuMechanismBody& r = mb[t.level_bodies[i]];
                const uint32_t up = r.metadata[0], depth = r.traversal[1];
                const bool root = up < B && mb[up].metadata[3] != 0u;
                filled = filled && up < B && depth >= 1 && (depth == 1 ? root : !root && mb[up].traversal[1] + 1 == depth);
                t.level_parent[i] = depth == 1 ? up : up < B ? at[up] : 0u;
            }
            if (filled) p.walk_levels = levels;
        }
    }
    // closure branches: walk each endpoint to its root (closure.wgsl:154-192)
    std::map<uint32_t, std::vector<uint32_t>> coord_slots;
    std::vector<uint8_t> closure_root(B, 0);
    t.cl_slot_off.push_back(0);
    for (uint32_t j = 0; j < cr->bearing_count; ++j) {
        const GpuBearing& br = cr->bearings[j];
        if (br.metadata[3] == 0) continue;
        t.cl_bearings.push_back(j);
        for (int side = 0; side < 2; ++side) {
            if (side == 1) t.cl_split.push_back((uint32_t)t.slot_body.size());
            uint32_t body = br.metadata[side];
            for (uint32_t guard = 0; guard <= B && body < B; ++guard) {
                if (mb[body].metadata[3] != 0) { closure_root[body] = 1; break; }
                const uint32_t coord = cr->bearings[mb[body].metadata[1]].metadata[2];
                coord_slots[coord].push_back((uint32_t)t.slot_body.size());
                t.slot_body.push_back(body);
                body = mb[body].metadata[0];
            }
        }
        t.cl_slot_off.push_back((uint32_t)t.slot_body.size());
    }
    t.cq_off.push_back(0);
    for (auto& kv : coord_slots) {
        t.cq_coords.push_back(kv.first);
        for (uint32_t sl : kv.second) t.cq_slots.push_back(sl);
        t.cq_off.push_back((uint32_t)t.cq_slots.size());
    }
    // bodies whose root carries a closure: the only links the closure loop changes
    if (!t.cl_bearings.empty()) {
        for (uint32_t i = 0; i < B; ++i) {
            uint32_t body = i;
            for (uint32_t guard = 0; guard <= B && mb[body].metadata[3] == 0; ++guard) body = mb[body].metadata[0];
            if (closure_root[body]) t.cb_bodies.push_back(i);
        }
    }
    // slot values are stored at their position in cq_slots, so each coordinate reads its
    // run contiguously; runs longer than kLongList (coordinates near the root of a large
    // loop lattice carry a slot of nearly every closure) are summed in chunks
    t.slot_pos.assign(t.slot_body.size(), 0u);
    for (uint32_t i = 0; i < (uint32_t)t.cq_slots.size(); ++i) t.slot_pos[t.cq_slots[i]] = i;
    t.long_chunk_off.push_back(0);
    for (uint32_t q = 0; q + 1 < (uint32_t)t.cq_off.size(); ++q) {
        const uint32_t n = t.cq_off[q + 1] - t.cq_off[q];
        if (n <= kLongList) continue;
        const uint32_t w = (uint32_t)t.long_q.size();
        t.long_q.push_back(q);
        for (uint32_t c = 0; c < (n + kLongList - 1) / kLongList; ++c) t.chunk_long.push_back(w);
        t.long_chunk_off.push_back((uint32_t)t.chunk_long.size());
    }
    p.long_coords = (uint32_t)t.long_q.size();
    p.wide_closures = (!t.cl_bearings.empty() && t.slot_body.size() >= 32ull * t.cl_bearings.size()) ? 1u : 0u;
    p.long_chunks = (uint32_t)t.chunk_long.size();
    t.slot_closure.resize(t.slot_body.size());
    for (size_t k = 0; k + 1 < t.cl_slot_off.size(); ++k)
        for (uint32_t sl = t.cl_slot_off[k]; sl < t.cl_slot_off[k + 1]; ++sl) t.slot_closure[sl] = (uint32_t)k;
    p.closures = (uint32_t)t.cl_bearings.size();
    p.slots = (uint32_t)t.slot_body.size();
    p.closure_coords = (uint32_t)t.cq_coords.size();
    p.closure_bodies = (uint32_t)t.cb_bodies.size();
    p.blocks = (p.closure_coords + 1) / 2;
    // per-loop blocks: each closure coordinate joins the block of the first closure that
    // contains it; loops longer than kLoopPiece are cut into consecutive pieces
    {
        std::map<uint32_t, uint32_t> position;
        for (uint32_t q = 0; q < t.cq_coords.size(); ++q) position[t.cq_coords[q]] = q;
        std::vector<uint8_t> taken(t.cq_coords.size(), 0);
        t.loop_off.push_back(0);
        for (size_t k = 0; k + 1 < t.cl_slot_off.size(); ++k) {
            std::vector<uint32_t> qs;
            for (uint32_t sl = t.cl_slot_off[k]; sl < t.cl_slot_off[k + 1]; ++sl) {
                const uint32_t coord = cr->bearings[mb[t.slot_body[sl]].metadata[1]].metadata[2];
                auto it = position.find(coord);
                if (it == position.end() || taken[it->second]) continue;
                taken[it->second] = 1;
                qs.push_back(it->second);
            }
            std::sort(qs.begin(), qs.end());
            for (size_t i = 0; i < qs.size(); i += kLoopPiece) {
                for (size_t j = i; j < std::min<size_t>(qs.size(), i + kLoopPiece); ++j) t.loop_q.push_back(qs[j]);
                t.loop_off.push_back((uint32_t)t.loop_q.size());
            }
        }
        p.loops = (uint32_t)t.loop_off.size() - 1;
    }
    derive_block_solve(cr, p, t);
    return t;
}

void carve_mechanism(MechBuffers& m, const MechParams& p, uint32_t B, uint32_t J, uint32_t Q,
                     const std::function<char*(uint64_t)>& take) {
    B = B ? B : 1;
    J = J ? J : 1;
    Q = Q ? Q : 1;
    auto u32 = [&](uint64_t n) { return reinterpret_cast<uint32_t*>(take(4ull * (n ? n : 1))); };
    auto f32 = [&](uint64_t n) { return reinterpret_cast<float*>(take(4ull * (n ? n : 1))); };
    m.bearings = reinterpret_cast<GpuBearing*>(take(sizeof(GpuBearing) * (uint64_t)J));
    m.bodies = reinterpret_cast<GpuMechanismBody*>(take(sizeof(GpuMechanismBody) * (uint64_t)B));
    m.coords = reinterpret_cast<GpuMechanismCoordinate*>(take(sizeof(GpuMechanismCoordinate) * (uint64_t)Q));
    m.drives = reinterpret_cast<GpuMechanismDrive*>(take(sizeof(GpuMechanismDrive) * (uint64_t)Q));
    m.preorder = u32(B);
    m.links_a = reinterpret_cast<GpuLinkState*>(take(sizeof(GpuLinkState) * (uint64_t)B));
    m.links_b = reinterpret_cast<GpuLinkState*>(take(sizeof(GpuLinkState) * (uint64_t)B));
    m.pass_bodies = u32(B);
    m.side_body = u32(p.padded_sides);
    m.side_entries = reinterpret_cast<uint2*>(take(8ull * std::max(1u, p.all_sides)));
    m.side_place = reinterpret_cast<uint2*>(take(8ull * J));
    m.side_cache = reinterpret_cast<float4*>(take(16ull * kSideRows * std::max(1u, p.all_sides)));
    m.hub_chunks = reinterpret_cast<uint4*>(take(16ull * p.hub_chunks));
    m.hub_sums = u32(8ull * p.hub_bodies);
    m.level_bodies = u32(B);
    if (p.walk_levels) {
        m.level_begin = u32(p.walk_levels + 1ull);
        m.level_parent = u32(B);
        m.level_rows = reinterpret_cast<float4*>(take(48ull * B));
    }
    m.cl_bearings = u32(p.closures);
    m.cl_slot_off = u32(p.closures + 1);
    m.cl_split = u32(p.closures);
    if (p.block_solve) {
        m.cl_order = u32(p.closures);
        m.cl_columns = u32(p.closure_depth + 1ull);
        m.col_coord = u32(p.slots);
        m.col_pos = u32(p.slots);
        m.cl_places = u32(2ull * p.closures);
        m.slot_parent = u32(p.slots);
        m.cq_child = u32(p.closure_coords);
        m.cb_parents = u32(p.closure_bodies);
    }
    m.slot_body = u32(p.slots);
    m.cq_coords = u32(p.closure_coords);
    m.cq_off = u32(p.closure_coords + 1);
    m.cq_slots = u32(p.slots);
    m.cb_bodies = u32(p.closure_bodies);
    m.slot_g = f32(p.slots);
    m.slot_d = f32(p.slots);
    m.slot_pos = u32(p.slots);
    m.long_q = u32(p.long_coords);
    m.long_chunk_off = u32(p.long_coords + 1);
    m.chunk_long = u32(p.long_chunks);
    m.chunk_g = f32(p.long_chunks);
    m.chunk_d = f32(p.long_chunks);
    m.grad = f32(Q);
    m.diag = f32(Q);
    m.pcg = f32(5ull * Q);
    m.grid_barrier = u32(64);   // its own 256-byte line
    m.loop_state = u32(2ull * kClosureSteps);
    m.columns_stale = u32(1);
    m.chunk_part = f32(2ull * ((p.closure_coords + kClosureThreads - 1) / kClosureThreads));
    m.chunk_part_d = reinterpret_cast<double*>(take(16ull * ((p.closure_coords + kClosureThreads - 1) / kClosureThreads + 1)));
    m.links_final = p.final_is_a ? m.links_a : m.links_b;
    m.slot_v = reinterpret_cast<float4*>(take(32ull * (p.slots ? p.slots : 1)));   // Jacobian columns
    if (pcg_residual_mode(p)) {
        m.slot_closure = u32(p.slots);
        m.blk_m = reinterpret_cast<float4*>(take(16ull * (p.blocks ? p.blocks : 1)));
        m.blk_feat = reinterpret_cast<float4*>(take(64ull * (p.blocks ? p.blocks : 1)));
        m.blk_out = f32(3ull * p.blocks);
        m.blk_hist = f32(3ull * kClosureSteps * p.blocks);
        m.probe = f32(2ull * Q);
        m.cstate = reinterpret_cast<ClosureState*>(take(sizeof(ClosureState)));
        if (p.learned_precond) m.precond_params = f32(mlp::kParams + 16);
        m.loop_off = u32(p.loops + 1);
        m.loop_q = u32(p.closure_coords);
        m.loop_l = f32(36ull * p.loops);
    }
}

template <class T>
static cudaError_t put(T* dst, const std::vector<T>& v, cudaStream_t s) {
    if (v.empty()) return cudaSuccess;
    return cudaMemcpyAsync(dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, s);
}

bool upload_mechanism(MechBuffers& m, const MechParams& p, const MechTopology& t, const MkCreation* cr,
                      cudaStream_t s, MkError* err) {
    cudaError_t e = cudaSuccess;
    if (cr->bearing_count)
        e = cudaMemcpyAsync(m.bearings, cr->bearings, sizeof(GpuBearing) * cr->bearing_count, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && cr->mechanism_bodies)
        e = cudaMemcpyAsync(m.bodies, cr->mechanism_bodies, sizeof(GpuMechanismBody) * cr->body_count,
                            cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && cr->preorder)
        e = cudaMemcpyAsync(m.preorder, cr->preorder, 4ull * cr->body_count, cudaMemcpyHostToDevice, s);
    std::vector<GpuMechanismDrive> d(cr->coordinate_count);
    if (cr->coordinate_count) {
        if (cr->drives) {
            std::memcpy(d.data(), cr->drives, sizeof(GpuMechanismDrive) * cr->coordinate_count);
        } else {
            for (auto& r : d) {   // GpuMechanismDrive::PASSIVE (abi.rs:266-275)
                std::memset(&r, 0, sizeof(r));
                r.min_angle = -INFINITY;
                r.max_angle = INFINITY;
            }
        }
        if (e == cudaSuccess) e = put(m.drives, d, s);
    }
    if (e == cudaSuccess) e = put(m.pass_bodies, t.pass_bodies, s);
    if (e == cudaSuccess) e = put(m.side_body, t.side_body, s);
    if (e == cudaSuccess) e = put(m.side_entries, t.side_entries, s);
    if (e == cudaSuccess) e = put(m.side_place, t.side_place, s);
    if (e == cudaSuccess) e = put(m.hub_chunks, t.hub_chunks, s);
    if (e == cudaSuccess) e = put(m.level_bodies, t.level_bodies, s);
    if (e == cudaSuccess && p.walk_levels) e = put(m.level_begin, t.level_offsets, s);
    if (e == cudaSuccess && p.walk_levels) e = put(m.level_parent, t.level_parent, s);
    if (e == cudaSuccess) e = put(m.cl_bearings, t.cl_bearings, s);
    if (e == cudaSuccess) e = put(m.cl_slot_off, t.cl_slot_off, s);
    if (e == cudaSuccess) e = put(m.cl_split, t.cl_split, s);
    if (p.block_solve) {
        if (e == cudaSuccess) e = put(m.cl_order, t.cl_order, s);
        if (e == cudaSuccess) e = put(m.cl_columns, t.cl_columns, s);
        if (e == cudaSuccess) e = put(m.col_coord, t.col_coord, s);
        if (e == cudaSuccess) e = put(m.col_pos, t.col_pos, s);
        if (e == cudaSuccess) e = put(m.cl_places, t.cl_places, s);
        if (e == cudaSuccess) e = put(m.slot_parent, t.slot_parent, s);
        if (e == cudaSuccess) e = put(m.cq_child, t.cq_child, s);
        if (e == cudaSuccess) e = put(m.cb_parents, t.cb_parents, s);
    }
    if (e == cudaSuccess && m.slot_closure) e = put(m.slot_closure, t.slot_closure, s);
    if (e == cudaSuccess && m.loop_off) e = put(m.loop_off, t.loop_off, s);
    if (e == cudaSuccess && m.loop_q) e = put(m.loop_q, t.loop_q, s);
    if (e == cudaSuccess) e = put(m.slot_body, t.slot_body, s);
    if (e == cudaSuccess) e = put(m.cq_coords, t.cq_coords, s);
    if (e == cudaSuccess) e = put(m.cq_off, t.cq_off, s);
    if (e == cudaSuccess) e = put(m.cq_slots, t.cq_slots, s);
    if (e == cudaSuccess) e = put(m.slot_pos, t.slot_pos, s);
    if (e == cudaSuccess && !t.long_q.empty()) e = put(m.long_q, t.long_q, s);
    if (e == cudaSuccess && !t.long_q.empty()) e = put(m.long_chunk_off, t.long_chunk_off, s);
    if (e == cudaSuccess && !t.chunk_long.empty()) e = put(m.chunk_long, t.chunk_long, s);
    if (e == cudaSuccess) e = put(m.cb_bodies, t.cb_bodies, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    (void)p;
    if (e != cudaSuccess) {
        if (err) {
            std::memset(err, 0, sizeof(*err));
            err->code = MK_ERR_DEVICE_FAILURE;
            std::snprintf(err->message, sizeof(err->message), "upload mechanism: %s", cudaGetErrorString(e));
        }
        return false;
    }
    return true;
}

// --------------------------------------------------------------- device math
__device__ __forceinline__ f3 r3(const float* v) { return mkf3(v[0], v[1], v[2]); }
__device__ __forceinline__ float4 r4(const float* v) { return make_float4(v[0], v[1], v[2], v[3]); }

// articulated.wgsl:94-102: world inverse inertia from the body-frame rows.
__device__ __forceinline__ f3 wii(const StepBuffers& b, uint32_t body, f3 v) {
    const float4 r = b.rot[body];
    const f3 l = quat_rotate(conjq(r), v);
    const float4* m = b.mass + 4ull * body;
    const f3 lr = xyz(m[1]) * l.x + xyz(m[2]) * l.y + xyz(m[3]) * l.z;
    return quat_rotate(r, lr);
}
__device__ __forceinline__ float inv_mass(const StepBuffers& b, uint32_t body) { return b.mass[4ull * body].x; }

__device__ __forceinline__ void hinge_tangents(const StepBuffers& b, uint32_t a, uint32_t c, const GpuBearing& br,
                                               f3& ta, f3& tb) {
    const f3 axa = normalize(quat_rotate(b.rot[a], r3(br.local_axis_a)));
    const f3 axb = normalize(quat_rotate(b.rot[c], r3(br.local_axis_b)));
    const f3 hinge = normalize(axa + axb);
    const f3 helper = fabsf(hinge.x) > 0.8f ? mkf3(0, 1, 0) : mkf3(1, 0, 0);
    ta = normalize(cross(hinge, helper));
    tb = cross(hinge, ta);
}

// The parts of a bearing's five rows that depend on the poses only: they stay
// fixed over a set of projection passes (the poses change at the forward
// kinematics, not between passes), so they are computed once per set, with the
// same expressions as the rows would compute them.  Each of its two sides gets
// its own copy, kSideRows float4 at the side's place in the passes' lists (an
// array per row, so the passes read them coalesced: with 9 float4 per bearing,
// 144 bytes apart, a pass of 198,009 bearings with contact deltas took a ninth
// longer, 37 us against 33 at the time):
// {arm_a, 1/m own} {arm_b, den0} {t_a, den3} {t_b, den4} {I t_a own, den1}
// {I t_b own, den2}: arms of the three linear rows (world axes), hinge tangents
// of the two angular rows, the side's world inverse inertia products and the
// rows' denominators.
__global__ void __launch_bounds__(kMBlock) k_bearing_cache(StepBuffers b, MechBuffers m, MechParams p) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= p.bearing_count) return;
    const GpuBearing br = m.bearings[j];
    const uint32_t a = br.metadata[0], c = br.metadata[1];
    const f3 arm_a = quat_rotate(b.rot[a], r3(br.local_anchor_a)), arm_b = quat_rotate(b.rot[c], r3(br.local_anchor_b));
    const float ima = inv_mass(b, a), imb = inv_mass(b, c);
    float den[5];
#pragma unroll
    for (uint32_t row = 0; row < 3; ++row) {
        const f3 d = row == 0 ? mkf3(1, 0, 0) : row == 1 ? mkf3(0, 1, 0) : mkf3(0, 0, 1);
        const f3 ang_a = cross(arm_a, d), ang_b = cross(arm_b, d);
        den[row] = ima + imb + dot(ang_a, wii(b, a, ang_a)) + dot(ang_b, wii(b, c, ang_b));
    }
    f3 ta, tb;
    hinge_tangents(b, a, c, br, ta, tb);
    const f3 ia3 = wii(b, a, ta), ib3 = wii(b, c, ta), ia4 = wii(b, a, tb), ib4 = wii(b, c, tb);
    den[3] = dot(ta, ia3 + ib3);
    den[4] = dot(tb, ia4 + ib4);
    const uint2 place = m.side_place[j];
#pragma unroll
    for (uint32_t side = 0; side < 2; ++side) {
        float4* o = m.side_cache + (side ? place.y : place.x);
        const uint64_t n = p.all_sides;
        o[0] = f4(arm_a, side ? imb : ima);
        o[n] = f4(arm_b, den[0]);
        o[2 * n] = f4(ta, den[3]);
        o[3 * n] = f4(tb, den[4]);
        o[4 * n] = f4(side ? ib3 : ia3, den[1]);
        o[5 * n] = f4(side ? ib4 : ia4, den[2]);
    }
}

// One projection pass (articulated.wgsl:114-155, 287-316 and the velocity apply
// :318-337), gathered by body: every body of a bearing sums its own side of its
// bearings' rows, so a pass is one launch that reads one pair of velocity
// buffers and writes the other (every row reads the velocities of before the
// pass, Jacobi).  The rows' impulses are converted to fixed point as the
// reference does, and integer sums are order-free, so the result is that of its
// atomics bit for bit.  A thread per bearing side computes the five rows (a
// lane per row left three eighths of the lanes idle and issued both kinds of
// row in every warp); a body's sides are neighbouring lanes of one warp and are
// added by a segmented scan.  A row's pose-only parts come from the set's
// bearing cache.  Bound: issue.  One B200, 198,009 bearings on 100,000 bodies: a
// bearing per eight lanes with twelve atomics, and an apply launch, 52 us; this
// 22 us (25 us against 60 with a contact iteration's apply).
//
// kContacts: the pass follows a contact iteration whose fixed-point deltas are
// still to be applied (collision.wgsl:1050-1069): each body it reads gets them
// on the way, and bodies without bearings are written too.  It then clears
// `clear`, the delta buffer of the next iteration.
struct VelocityPass {
    const float4 *lin, *ang;       // velocities before the pass
    float4 *lin_out, *ang_out;     // bodies with bearings
    float4 *lin_rest, *ang_rest;   // the others
    const int32_t* deltas;         // contact deltas of the iteration before (kContacts)
    int32_t* clear;                // contact deltas of the next one (kContacts)
};
// v + delta / 2^20 (an apply of zeros changes -0.0, NaN payloads and w only)
__device__ __forceinline__ void apply_fixed(const int32_t* v, float4& lin, float4& ang) {
    const float s = 1048576.0f;
    lin = f4(xyz(lin) + mkf3((float)v[0], (float)v[1], (float)v[2]) / s, 0.0f);
    ang = f4(xyz(ang) + mkf3((float)v[3], (float)v[4], (float)v[5]) / s, 0.0f);
}
// Blocks [0, side_blocks): padded bearing sides.  [side_blocks, side_blocks +
// hub_blocks): chunks of kPassBlock sides of bodies with more than 32 bearings; a body's
// last chunk finishes it (a warp per body walked 5,000 sides in 190 us a pass, this takes 6).
// Then the rest.  kHubs: there are such bodies (a kernel of its own: their part in the
// common one cost the lattice's pass 0.5 us of 24).
template <bool kContacts, bool kHubs>
__global__ void __launch_bounds__(kPassBlock) k_bearing_pass(StepBuffers b, MechBuffers m, MechParams p, VelocityPass f,
                                                            uint32_t side_blocks, uint32_t hub_blocks) {
    const bool contacts = kContacts && b.counts->active != 0u;   // collision.wgsl:744: no apply without active contacts
    auto velocity = [&](uint32_t body, float4& lin, float4& ang) {
        lin = __ldg(f.lin + body);
        ang = __ldg(f.ang + body);
        if (contacts) {
            const int2* d2 = reinterpret_cast<const int2*>(f.deltas + 6ull * body);   // 24-byte rows
            const int2 x0 = __ldg(d2), x1 = __ldg(d2 + 1), x2 = __ldg(d2 + 2);
            const int32_t v[6] = {x0.x, x0.y, x1.x, x1.y, x2.x, x2.y};
            apply_fixed(v, lin, ang);
        }
    };
    auto clear = [&](uint32_t body) {
        if (!kContacts) return;
        int2* d2 = reinterpret_cast<int2*>(f.clear + 6ull * body);
        d2[0] = d2[1] = d2[2] = make_int2(0, 0);
    };
    auto finish = [&](uint32_t body, const uint32_t* sum, float4 lin, float4 ang) {
        const int32_t total[6] = {(int32_t)sum[0], (int32_t)sum[1], (int32_t)sum[2],
                                  (int32_t)sum[3], (int32_t)sum[4], (int32_t)sum[5]};
        apply_fixed(total, lin, ang);
        f.lin_out[body] = lin;
        f.ang_out[body] = ang;
        clear(body);
    };
    // the fixed-point deltas of one side of a bearing's five rows, added to `sum`
    auto add_side = [&](uint32_t body, uint32_t at, const float4& lin, const float4& ang, uint32_t* sum) {
        const uint2 ent = __ldg(m.side_entries + at);
        const bool side_b = ent.x != 0u;
        const float4* cache = m.side_cache + at;
        const uint64_t n = p.all_sides;
        const float4 ca = __ldg(cache), cb = __ldg(cache + n), t3 = __ldg(cache + 2 * n), t4 = __ldg(cache + 3 * n);
        const float4 in3 = __ldg(cache + 4 * n), in4 = __ldg(cache + 5 * n);
        // the body's rotation and inertia rows before the branches that use them (the lattice's ticks 1% shorter)
        const float4 rot = __ldg(b.rot + body), *rows = b.mass + 4ull * body;
        const float4 i1 = __ldg(rows + 1), i2 = __ldg(rows + 2), i3 = __ldg(rows + 3);
        auto inertia_of = [&](f3 v) {   // wii
            const f3 l = quat_rotate(conjq(rot), v);
            return quat_rotate(rot, xyz(i1) * l.x + xyz(i2) * l.y + xyz(i3) * l.z);
        };
        float4 ol, oa;
        velocity(ent.y, ol, oa);
        auto add = [&](f3 l, f3 a) {
            const float s = 1048576.0f;
            sum[0] += (uint32_t)fixed_i32(l.x * s);
            sum[1] += (uint32_t)fixed_i32(l.y * s);
            sum[2] += (uint32_t)fixed_i32(l.z * s);
            sum[3] += (uint32_t)fixed_i32(a.x * s);
            sum[4] += (uint32_t)fixed_i32(a.y * s);
            sum[5] += (uint32_t)fixed_i32(a.z * s);
        };
        const f3 arm_a = xyz(ca), arm_b = xyz(cb);
        const f3 own = xyz(lin) + cross(xyz(ang), side_b ? arm_b : arm_a);
        const f3 other = xyz(ol) + cross(xyz(oa), side_b ? arm_a : arm_b);
        const f3 rel = side_b ? own - other : other - own;   // body b's minus body a's
#pragma unroll
        for (uint32_t row = 0; row < 3; ++row) {
            const f3 d = row == 0 ? mkf3(1, 0, 0) : row == 1 ? mkf3(0, 1, 0) : mkf3(0, 0, 1);
            const float den = row == 0 ? cb.w : row == 1 ? in3.w : in4.w;
            if (den <= 1.0e-12f) continue;
            const f3 imp = d * (0.5f * dot(rel, d) / den);
            if (side_b) add(-imp * ca.w, inertia_of(cross(arm_b, -imp)));
            else add(imp * ca.w, inertia_of(cross(arm_a, imp)));
        }
        const f3 rang = side_b ? xyz(ang) - xyz(oa) : xyz(oa) - xyz(ang);
#pragma unroll
        for (uint32_t row = 3; row < 5; ++row) {
            const float4 ax = row == 3 ? t3 : t4;   // hinge tangent, denominator
            const f3 inertia = xyz(row == 3 ? in3 : in4);
            if (ax.w <= 1.0e-12f) continue;
            const float imp = 0.5f * dot(rang, xyz(ax)) / ax.w;
            add(mkf3(0, 0, 0), side_b ? -inertia * imp : inertia * imp);
        }
    };
    const uint32_t lane = lane_id();
    if (blockIdx.x < side_blocks) {
        const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;   // the list is padded to whole blocks
        const uint32_t body = __ldg(m.side_body + t);
        uint32_t sum[6] = {0u, 0u, 0u, 0u, 0u, 0u};
        float4 lin = make_float4(0, 0, 0, 0), ang = lin;
        if (body != kInvalid) {
            velocity(body, lin, ang);
            add_side(body, t, lin, ang, sum);
        }
        // segmented sum over the body's lanes (a body never crosses a warp): its last lane finishes it
        const uint32_t before = __shfl_up_sync(0xffffffffu, body, 1);
        const uint32_t after = __shfl_down_sync(0xffffffffu, body, 1);
        const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0 || before != body);
        const uint32_t head = 31u - __clz(heads & ((2u << lane) - 1u));
        for (uint32_t o = 1; o < p.most_sides; o <<= 1)
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, sum[c], o);
                if (lane >= head + o) sum[c] += u;
            }
        if (body != kInvalid && (lane == 31u || after != body)) finish(body, sum, lin, ang);
        return;
    }
    if (kHubs && blockIdx.x < side_blocks + hub_blocks) {
        __shared__ uint32_t s_sum[kPassBlock / 32][6];
        const uint4 ch = __ldg(m.hub_chunks + (blockIdx.x - side_blocks));   // body, first side, sides | hub << 8, chunks
        const uint32_t body = ch.x;
        uint32_t sum[6] = {0u, 0u, 0u, 0u, 0u, 0u};
        float4 lin, ang;
        velocity(body, lin, ang);
        if (threadIdx.x < (ch.z & 0xffu)) add_side(body, ch.y + threadIdx.x, lin, ang, sum);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            sum[c] = __reduce_add_sync(0xffffffffu, sum[c]);
            if (lane == 0) s_sum[threadIdx.x >> 5][c] = sum[c];
        }
        __syncthreads();
        if (threadIdx.x != 0) return;
#pragma unroll
        for (int c = 0; c < 6; ++c)
#pragma unroll
            for (uint32_t w = 1; w < kPassBlock / 32; ++w) sum[c] += s_sum[w][c];
        if (ch.w > 1u) {
            uint32_t* all = m.hub_sums + 8ull * (ch.z >> 8);   // six sums and the arrivals, zero between passes
#pragma unroll
            for (int c = 0; c < 6; ++c)
                if (sum[c]) atomicAdd(all + c, sum[c]);
            __threadfence();
            if (atomicAdd(all + 6, 1u) != ch.w - 1u) return;
            __threadfence();
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                sum[c] = __ldcg(all + c);
                all[c] = 0u;
            }
            all[6] = 0u;
        }
        finish(body, sum, lin, ang);
        return;
    }
    // bodies without bearings: the apply of zero deltas
    const uint32_t i = (blockIdx.x - side_blocks - hub_blocks) * blockDim.x + threadIdx.x + p.bearing_bodies;
    if (i >= p.body_count) return;
    const uint32_t body = m.pass_bodies[i];
    const int32_t zeros[6] = {0, 0, 0, 0, 0, 0};
    float4 lin, ang;
    velocity(body, lin, ang);
    if (!kContacts && zero_apply_is_identity(lin) && zero_apply_is_identity(ang)) return;   // in place
    apply_fixed(zeros, lin, ang);
    f.lin_rest[body] = lin;
    f.ang_rest[body] = ang;
    clear(body);
}
// After an odd number of passes: the velocities of the listed bodies back into place.
__global__ void __launch_bounds__(kMBlock) k_pass_back(MechBuffers m, uint32_t count, VelocityPass f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint32_t body = m.pass_bodies[i];
    f.lin_out[body] = f.lin[body];
    f.ang_out[body] = f.ang[body];
}

// articulated.wgsl:157-285: forward then backward sweeps with immediate updates.
__device__ void project_row_immediate(const StepBuffers& b, const MechBuffers& m, uint32_t j) {
    const GpuBearing br = m.bearings[j];
    const uint32_t a = br.metadata[0], c = br.metadata[1];
    const f3 arm_a = quat_rotate(b.rot[a], r3(br.local_anchor_a)), arm_b = quat_rotate(b.rot[c], r3(br.local_anchor_b));
    const float ima = inv_mass(b, a), imb = inv_mass(b, c);
    const f3 dirs[3] = {mkf3(1, 0, 0), mkf3(0, 1, 0), mkf3(0, 0, 1)};
    for (int k = 0; k < 3; ++k) {
        const f3 va = xyz(b.lin[a]) + cross(xyz(b.ang[a]), arm_a);
        const f3 vb = xyz(b.lin[c]) + cross(xyz(b.ang[c]), arm_b);
        const f3 rel = vb - va, d = dirs[k];
        const f3 ang_a = cross(arm_a, d), ang_b = cross(arm_b, d);
        const float den = ima + imb + dot(ang_a, wii(b, a, ang_a)) + dot(ang_b, wii(b, c, ang_b));
        if (den <= 1.0e-12f) continue;
        const f3 imp = d * (dot(rel, d) / den);
        b.lin[a] = f4(xyz(b.lin[a]) + imp * ima, 0.0f);
        b.ang[a] = f4(xyz(b.ang[a]) + wii(b, a, cross(arm_a, imp)), 0.0f);
        b.lin[c] = f4(xyz(b.lin[c]) - imp * imb, 0.0f);
        b.ang[c] = f4(xyz(b.ang[c]) + wii(b, c, cross(arm_b, -imp)), 0.0f);
    }
    f3 ta, tb;
    hinge_tangents(b, a, c, br, ta, tb);
    const f3 tangents[2] = {ta, tb};
    for (int k = 0; k < 2; ++k) {
        const f3 rang = xyz(b.ang[c]) - xyz(b.ang[a]);
        const f3 axis = tangents[k];
        const f3 ia = wii(b, a, axis), ib = wii(b, c, axis);
        const float den = dot(axis, ia + ib);
        if (den <= 1.0e-12f) continue;
        const float imp = dot(rang, axis) / den;
        b.ang[a] = f4(xyz(b.ang[a]) + ia * imp, 0.0f);
        b.ang[c] = f4(xyz(b.ang[c]) - ib * imp, 0.0f);
    }
}

// Dispatched through indirect args that are zero without active contacts
// (collision.wgsl:747-749, device.rs:1101-1110).
__global__ void k_project_bearings_serial(StepBuffers b, MechBuffers m, MechParams p) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (b.counts->active == 0u) return;
    for (uint32_t j = 0; j < p.bearing_count; ++j) project_row_immediate(b, m, j);
    for (uint32_t j = p.bearing_count; j > 0; --j) project_row_immediate(b, m, j - 1);
}

// articulated.wgsl:339-364
__device__ __forceinline__ f3 permitted_axis(const StepBuffers& b, const MechBuffers& m, uint32_t body) {
    const GpuMechanismBody mb = m.bodies[body];
    const uint32_t parent = mb.metadata[0];
    const GpuBearing& br = m.bearings[mb.metadata[1]];
    f3 axis = normalize(quat_rotate(b.rot[parent], r3(br.local_axis_a)));
    if (mb.metadata[2] != 0u) axis = -normalize(quat_rotate(b.rot[parent], r3(br.local_axis_b)));
    return axis;
}
__device__ __forceinline__ float permitted_speed(const StepBuffers& b, const MechBuffers& m, uint32_t body) {
    const uint32_t parent = m.bodies[body].metadata[0];
    return dot(xyz(b.ang[body]) - xyz(b.ang[parent]), permitted_axis(b, m, body));
}
__device__ __forceinline__ float stabilized_speed(const StepBuffers& b, const MechBuffers& m, uint32_t body,
                                                  float speed) {
    const bool aligned = fabsf(permitted_axis(b, m, body).y) > 0.999f;
    return (aligned && fabsf(speed) < 0.005f) ? 0.0f : speed;
}

// articulated.wgsl:366-415
__global__ void __launch_bounds__(kMBlock) k_advance_coordinates(StepBuffers b, MechBuffers m, MechParams p) {
    const uint32_t body = blockIdx.x * blockDim.x + threadIdx.x;
    if (body >= p.body_count || m.bodies[body].metadata[3] != 0u) return;
    const uint32_t c = m.bearings[m.bodies[body].metadata[1]].metadata[2];
    if (c == kInvalid) return;
    const float measured = permitted_speed(b, m, body) * p.ang_damp;
    const GpuMechanismDrive dr = m.drives[c];
    float speed = 0.0f;
    if (dr.mode == MK_DRIVE_MODE_PASSIVE) {
        speed = stabilized_speed(b, m, body, measured);
    } else {
        float desired = clampf(dr.target_speed, -dr.max_speed, dr.max_speed);
        if (dr.mode == MK_DRIVE_MODE_ANGLE) {
            const float err = dr.target_angle - m.coords[c].angle;
            const float brake = sqrtf(2.0f * dr.max_acceleration * fabsf(err));
            desired = sgnf(err) * mnf(brake, dr.max_speed);
            if (fabsf(err) < 0.0005f) desired = 0.0f;
        }
        const float budget = dr.max_acceleration * p.dt;
        speed = measured + clampf(desired - measured, -budget, budget);
    }
    float angle = m.coords[c].angle + speed * p.dt;
    if (angle < dr.min_angle) {
        angle = dr.min_angle;
        speed = 0.0f;
    } else if (angle > dr.max_angle) {
        angle = dr.max_angle;
        speed = 0.0f;
    }
    m.coords[c].angular_velocity = speed;
    m.coords[c].angle = angle;
}

// articulated.wgsl:417-429
__global__ void __launch_bounds__(kMBlock) k_capture_coordinates(StepBuffers b, MechBuffers m, MechParams p) {
    const uint32_t body = blockIdx.x * blockDim.x + threadIdx.x;
    if (body >= p.body_count || m.bodies[body].metadata[3] != 0u) return;
    const uint32_t c = m.bearings[m.bodies[body].metadata[1]].metadata[2];
    if (c != kInvalid) m.coords[c].angular_velocity = stabilized_speed(b, m, body, permitted_speed(b, m, body));
}

// ------------------------------------------------------ forward kinematics
struct Link { float4 pos, rot; uint4 meta; };
__device__ __forceinline__ Link ld_link(const GpuLinkState* L, uint32_t i) {
    const float4* p = reinterpret_cast<const float4*>(L + i);
    const float4 m = p[2];
    return {p[0], p[1], make_uint4(__float_as_uint(m.x), __float_as_uint(m.y), __float_as_uint(m.z), __float_as_uint(m.w))};
}
__device__ __forceinline__ void st_link(GpuLinkState* L, uint32_t i, const Link& v) {
    float4* p = reinterpret_cast<float4*>(L + i);
    p[0] = v.pos;
    p[1] = v.rot;
    p[2] = make_float4(__uint_as_float(v.meta.x), __uint_as_float(v.meta.y), __uint_as_float(v.meta.z),
                       __uint_as_float(v.meta.w));
}

// mechanism.wgsl:67-70
__device__ __forceinline__ float4 axis_rotation(f3 axis, float angle) {
    const float h = angle * 0.5f;
    const f3 v = normalize(axis) * sin_cr(h);
    return make_float4(v.x, v.y, v.z, cos_cr(h));
}

// mechanism.wgsl:72-108
__device__ __forceinline__ void prepare_link(const MechBuffers& m, uint32_t body) {
    const GpuMechanismBody mb = m.bodies[body];
    if (mb.metadata[3] != 0u) {
        st_link(m.links_a, body, {make_float4(0, 0, 0, 0), make_float4(0, 0, 0, 1), make_uint4(body, 1, 0, 0)});
        return;
    }
    const GpuBearing& br = m.bearings[mb.metadata[1]];
    const float angle = m.coords[br.metadata[2]].angle;
    const float4 bind = r4(mb.bind_relative_rotation);
    float4 rr;
    f3 rp;
    if (mb.metadata[2] == 0u) {
        rr = quat_multiply(axis_rotation(r3(br.local_axis_a), angle), bind);
        rp = r3(br.local_anchor_a) - quat_rotate(rr, r3(br.local_anchor_b));
    } else {
        rr = quat_multiply(axis_rotation(r3(br.local_axis_b), -angle), bind);
        rp = r3(br.local_anchor_b) - quat_rotate(rr, r3(br.local_anchor_a));
    }
    st_link(m.links_a, body, {f4(rp, 0.0f), rr, make_uint4(mb.metadata[0], 0, 0, 0)});
}

// mechanism.wgsl:110-149
__device__ __forceinline__ void jump_link(const GpuLinkState* src, GpuLinkState* dst, uint32_t body) {
    const Link child = ld_link(src, body);
    if (child.meta.y != 0u) {
        st_link(dst, body, child);
        return;
    }
    const Link par = ld_link(src, child.meta.x);
    Link r;
    r.pos = f4(xyz(par.pos) + quat_rotate(par.rot, xyz(child.pos)), 0.0f);
    r.rot = normalize4(quat_multiply(par.rot, child.rot));
    r.meta = make_uint4(par.meta.x, par.meta.y, 0, 0);
    st_link(dst, body, r);
}

__global__ void __launch_bounds__(kMBlock) k_prepare_links(MechBuffers m, MechParams p) {
    const uint32_t body = blockIdx.x * blockDim.x + threadIdx.x;
    if (body < p.body_count) prepare_link(m, body);
}
__global__ void __launch_bounds__(kMBlock) k_jump(const GpuLinkState* src, GpuLinkState* dst, MechParams p) {
    const uint32_t body = blockIdx.x * blockDim.x + threadIdx.x;
    if (body < p.body_count) jump_link(src, dst, body);
}

// mechanism.wgsl:151-185
__global__ void __launch_bounds__(kMBlock) k_publish(StepBuffers b, MechBuffers m, MechParams p) {
    const uint32_t body = blockIdx.x * blockDim.x + threadIdx.x;
    if (body >= p.body_count) return;
    const Link L = ld_link(m.links_final, body);
    const uint32_t root = L.meta.x;
    if (body == root) return;
    const float4 rq = b.rot[root];
    b.pos[body] = f4(xyz(b.pos[root]) + quat_rotate(rq, xyz(L.pos)), 0.0f);
    b.rot[body] = normalize4(quat_multiply(rq, L.rot));
}

// articulated.wgsl:431-456 for the bodies of one depth level.
__global__ void __launch_bounds__(kMBlock) k_reconstruct_level(StepBuffers b, MechBuffers m, uint32_t begin,
                                                               uint32_t end) {
    const uint32_t t = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= end) return;
    const uint32_t body = m.level_bodies[t];
    const GpuMechanismBody mb = m.bodies[body];
    const uint32_t parent = mb.metadata[0];
    const GpuBearing& br = m.bearings[mb.metadata[1]];
    const float4 rp = b.rot[parent], rb = b.rot[body];
    f3 axis = normalize(quat_rotate(rp, r3(br.local_axis_a)));
    f3 pa = quat_rotate(rp, r3(br.local_anchor_a));
    f3 ca = quat_rotate(rb, r3(br.local_anchor_b));
    if (mb.metadata[2] != 0u) {
        axis = -normalize(quat_rotate(rp, r3(br.local_axis_b)));
        pa = quat_rotate(rp, r3(br.local_anchor_b));
        ca = quat_rotate(rb, r3(br.local_anchor_a));
    }
    const float speed = m.coords[br.metadata[2]].angular_velocity;
    const f3 wp = xyz(b.ang[parent]);
    const f3 angular = wp + axis * speed;
    const f3 av = xyz(b.lin[parent]) + cross(wp, pa);
    b.lin[body] = f4(av - cross(angular, ca), 0.0f);
    b.ang[body] = f4(angular, 0.0f);
}

// The same for deep, narrow trees.  A launch per level costs about 5 us whatever
// the level holds, so a tree of hundreds of levels is walked by one block
// instead: first a row per body (in level order) with the parts that do not
// depend on velocities, over the whole grid, then level by level with the
// velocities of the level before in shared memory and the rows of two levels
// loaded ahead; the results go to the rows' place, coalesced, and a last kernel
// puts them to their bodies (stored out of order by the walk: 315 us).  Bound:
// one block's issue and the barrier of each level.  100,000 bodies in 207
// levels (one B200, sum of kernel times): 207 launches 1,400 us, this 268 us.
// Rows, each an array over the level bodies: {axis * speed, parent's place in
// the level before} {parent's anchor arm} {child's anchor arm}.
__global__ void __launch_bounds__(kMBlock) k_reconstruct_rows(StepBuffers b, MechBuffers m, uint32_t count) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const uint32_t body = m.level_bodies[t];
    const GpuMechanismBody mb = m.bodies[body];
    const GpuBearing& br = m.bearings[mb.metadata[1]];
    const float4 rp = b.rot[mb.metadata[0]], rb = b.rot[body];
    const bool reversed = mb.metadata[2] != 0u;
    f3 axis = normalize(quat_rotate(rp, r3(reversed ? br.local_axis_b : br.local_axis_a)));
    if (reversed) axis = -axis;
    const f3 pa = quat_rotate(rp, r3(reversed ? br.local_anchor_b : br.local_anchor_a));
    const f3 ca = quat_rotate(rb, r3(reversed ? br.local_anchor_a : br.local_anchor_b));
    m.level_rows[t] = f4(axis * m.coords[br.metadata[2]].angular_velocity, __uint_as_float(m.level_parent[t]));
    m.level_rows[count + t] = f4(pa, 0.0f);
    m.level_rows[2ull * count + t] = f4(ca, 0.0f);
}

constexpr uint32_t kWalkThreads = 1024;
constexpr uint32_t kWalkSmem = 2 * 6 * kWalkWidth * sizeof(float);
__global__ void __launch_bounds__(kWalkThreads) k_reconstruct_walk(StepBuffers b, MechBuffers m, uint32_t levels,
                                                                   uint32_t count) {
    extern __shared__ float s_vel[];   // [level parity][component][place]
    struct Row {
        float4 r0, r1, r2;
    };
    float4* rows = m.level_rows;
    auto load = [&](uint32_t at, uint32_t end) -> Row {
        if (at >= end) return {};
        return {rows[at], rows[count + at], rows[2ull * count + at]};
    };
    // this thread's row of the level at hand and of the two after it (an L2 round trip is longer than a level)
    uint32_t begin = m.level_begin[1], end = m.level_begin[2];
    uint32_t end1 = 2 < levels ? m.level_begin[3] : end, end2 = 3 < levels ? m.level_begin[4] : end1;
    Row now = load(begin + threadIdx.x, end), next = load(end + threadIdx.x, end1);
    for (uint32_t l = 1; l < levels; ++l) {
        const Row after = load(end1 + threadIdx.x, end2);
        const uint32_t end3 = l + 3 < levels ? m.level_begin[l + 4] : end2;
        float* to = s_vel + (l & 1u) * 6u * kWalkWidth;
        const float* from = s_vel + ((l & 1u) ^ 1u) * 6u * kWalkWidth;
        for (uint32_t i = threadIdx.x; begin + i < end; i += kWalkThreads) {
            const Row r = i < kWalkThreads ? now : load(begin + i, end);
            const uint32_t up = __float_as_uint(r.r0.w);
            f3 lp, wp;
            if (l == 1) {   // `up` is the root's body
                lp = xyz(b.lin[up]);
                wp = xyz(b.ang[up]);
            } else {
                lp = mkf3(from[up], from[kWalkWidth + up], from[2 * kWalkWidth + up]);
                wp = mkf3(from[3 * kWalkWidth + up], from[4 * kWalkWidth + up], from[5 * kWalkWidth + up]);
            }
            const f3 angular = wp + xyz(r.r0);
            const f3 av = lp + cross(wp, xyz(r.r1));
            const f3 linear = av - cross(angular, xyz(r.r2));
            to[i] = linear.x; to[kWalkWidth + i] = linear.y; to[2 * kWalkWidth + i] = linear.z;
            to[3 * kWalkWidth + i] = angular.x; to[4 * kWalkWidth + i] = angular.y; to[5 * kWalkWidth + i] = angular.z;
            rows[begin + i] = f4(linear, 0.0f);
            rows[count + begin + i] = f4(angular, 0.0f);
        }
        begin = end;
        end = end1;
        end1 = end2;
        end2 = end3;
        now = next;
        next = after;
        __syncthreads();
    }
}
__global__ void __launch_bounds__(kMBlock) k_reconstruct_store(StepBuffers b, MechBuffers m, uint32_t count) {
    const uint32_t t = m.level_begin[1] + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const uint32_t body = m.level_bodies[t];
    b.lin[body] = m.level_rows[t];
    b.ang[body] = m.level_rows[count + t];
}

// articulated.wgsl:458-484
__global__ void __launch_bounds__(kMBlock) k_validate_state(StepBuffers b, MechBuffers m, MechParams p) {
    const uint32_t body = blockIdx.x * blockDim.x + threadIdx.x;
    if (body >= p.body_count) return;
    const float4 q = b.rot[body];
    const float rl = dot4(q, q);
    bool valid = finite4(b.pos[body]) && finite4(q) && finite4(b.lin[body]) && finite4(b.ang[body]) && rl > 0.5f &&
                 rl < 1.5f;
    const GpuMechanismBody mb = m.bodies[body];
    if (mb.metadata[3] == 0u) {
        const GpuMechanismCoordinate st = m.coords[m.bearings[mb.metadata[1]].metadata[2]];
        valid = valid && st.angle == st.angle && fabsf(st.angle) < kFloatMax && st.angular_velocity == st.angular_velocity &&
                fabsf(st.angular_velocity) < kFloatMax;
    }
    if (!valid) atomicOr(&b.diag->error_flags, MK_INVALID_NUMERIC_FLAG);
}

// bearings.wgsl:48-66
__device__ __forceinline__ void record_residual(GpuDiagnostics* d, f3 anchor_a, f3 anchor_b, f3 axis_a, f3 axis_b,
                                                bool closure) {
    const uint32_t um = round_u32(length(anchor_a - anchor_b) * 1000000.0f);
    const float deg = atan2_cr(length(cross(axis_a, axis_b)), clampf(dot(axis_a, axis_b), -1.0f, 1.0f)) * 57.295779513f;
    const uint32_t udeg = round_u32(deg * 1000000.0f);
    atomicMax(&d->max_anchor_micrometers, um);
    atomicMax(&d->max_axis_microdegrees, udeg);
    if (closure && (um > 10u || udeg > 1000u)) atomicOr(&d->error_flags, MK_CONSTRAINT_NON_CONVERGENCE_FLAG);
}

// bearings.wgsl:68-102 (world poses, or the final mechanism links).
__global__ void k_validate_bearings(const GpuBearing* __restrict__ bearings, uint32_t J, const float4* pos,
                                    const float4* rot, const GpuLinkState* links, GpuDiagnostics* diag) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= J) return;
    const GpuBearing br = bearings[i];
    const uint32_t a = br.metadata[0], c = br.metadata[1];
    float4 pa, qa, pc, qc;
    if (links) {
        const Link la = ld_link(links, a), lc = ld_link(links, c);
        pa = la.pos; qa = la.rot; pc = lc.pos; qc = lc.rot;
    } else {
        pa = pos[a]; qa = rot[a]; pc = pos[c]; qc = rot[c];
    }
    const f3 anchor_a = xyz(pa) + quat_rotate(qa, r3(br.local_anchor_a));
    const f3 anchor_b = xyz(pc) + quat_rotate(qc, r3(br.local_anchor_b));
    const f3 axis_a = normalize(quat_rotate(qa, r3(br.local_axis_a)));
    const f3 axis_b = normalize(quat_rotate(qc, r3(br.local_axis_b)));
    record_residual(diag, anchor_a, anchor_b, axis_a, axis_b, br.metadata[3] != 0u);
}

// ------------------------------------------------------------- closure loop
__device__ __forceinline__ float block_sum(float v, float* scratch) {
    // fixed tree order: warp shuffles, then warp 0 over the warp partials
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    __syncthreads();
    if (lane == 0) scratch[w] = v;
    __syncthreads();
    float r = 0.0f;
    if (w == 0) {
        r = lane < (blockDim.x >> 5) ? scratch[lane] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
        if (lane == 0) scratch[32] = r;
    }
    __syncthreads();
    return scratch[32];
}

// Dot products over the closure coordinates.  Up to kSerialDot coordinates
// one thread sums them in ascending coordinate order (the serial order of
// closure.wgsl:339-414, so small systems reproduce it bit for bit).  Larger
// systems sum per chunk of 1,024 coordinates: thread t of the chunk's block
// holds coordinate 1024 c + t, the block tree sums the chunk, and the chunk
// sums are added in chunk order -- the same result whether one block or the
// whole grid walks the chunks.
constexpr uint32_t kSerialDot = 512;
constexpr uint32_t kDotChunk = kClosureThreads;

// Sync of the closure loop: the block, or the whole cooperative grid.
template <bool kGrid>
__device__ __forceinline__ void loop_sync(uint32_t* barrier, uint32_t* error_flags) {
    if (kGrid) grid_barrier(barrier, error_flags, gridDim.x);
    else __syncthreads();
}

// Sums of the slot values of the closure coordinates whose runs are longer than
// kLongList slots (near the root of a large loop lattice a coordinate lies on a
// branch of nearly every closure: up to 176k slots).  Such a run is summed in two
// levels, so that no thread adds it alone: each chunk of kLongList consecutive
// slots serially, in parallel over the chunks, then the chunk sums serially in
// chunk order.  Runs of up to kLongList slots keep the one serial sum.  The
// accumulation order of the reference (CAS float atomics, closure.wgsl:128-192) is
// a race, so any fixed order is as faithful; the oracle restates this one.
// kEval: evaluation sums (a NaN gradient marks a slot without contribution, the
// diagonal summed beside it) into out_g / out_d; else plain sums into out_g.
template <bool kGrid, bool kEval>
__device__ void gather_long_runs(const MechBuffers& m, const MechParams& p, float* out_g, float* out_d,
                                 uint32_t* flags) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    for (uint32_t c = tid; c < p.long_chunks; c += nt) {
        const uint32_t w = m.chunk_long[c];
        const uint32_t q = m.long_q[w];
        const uint32_t begin = m.cq_off[q] + kLongList * (c - m.long_chunk_off[w]);
        const uint32_t end = min(begin + kLongList, m.cq_off[q + 1]);
        float g = 0.0f, d = 0.0f;
#pragma unroll 8
        for (uint32_t i = begin; i < end; ++i) {
            const float sg = __ldcg(m.slot_g + i);
            if (kEval) {
                if (sg == sg) { g += sg; d += __ldcg(m.slot_d + i); }
            } else {
                g += sg;
            }
        }
        m.chunk_g[c] = g;
        if (kEval) m.chunk_d[c] = d;
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
    for (uint32_t w = tid; w < p.long_coords; w += nt) {
        float g = 0.0f, d = 0.0f;
        for (uint32_t c = m.long_chunk_off[w]; c < m.long_chunk_off[w + 1]; ++c) {
            g += __ldcg(m.chunk_g + c);
            if (kEval) d += __ldcg(m.chunk_d + c);
        }
        const uint32_t cc = m.cq_coords[m.long_q[w]];
        out_g[cc] = g;
        if (kEval) out_d[cc] = d;
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
}

// The chunked dot: `part` is this thread's term for the coordinate of chunk
// `c` it holds (0 when none); the block tree sum of the chunk goes to
// chunk_part[c].  Call for every chunk the block walks, all threads together.
__device__ __forceinline__ void chunk_dot(float part, float* chunk_part, uint32_t c, float* scratch) {
    const float s = block_sum(part, scratch);
    if (threadIdx.x == 0) chunk_part[c] = s;
}

// The total after a loop_sync: serial over the coordinates (small systems) or
// the chunk sums in chunk order, computed by thread 0 of every block and
// shared through scratch[32].
__device__ __forceinline__ float dot_total(uint32_t nq, const MechBuffers& m, const float* a, const float* bvec,
                                           const float* chunk_part, float* scratch) {
    if (threadIdx.x == 0) {
        float acc = 0.0f;
        if (nq <= kSerialDot) {
            for (uint32_t q = 0; q < nq; ++q) {
                const uint32_t c = m.cq_coords[q];
                acc += a[c] * bvec[c];
            }
        } else {
            const uint32_t chunks = (nq + kDotChunk - 1) / kDotChunk;
            for (uint32_t c = 0; c < chunks; ++c) acc += chunk_part[c];
        }
        scratch[32] = acc;
    }
    __syncthreads();
    const float r = scratch[32];
    __syncthreads();
    return r;
}

// slot_g[sl] = the slot's share of J^T J x: per closure the branch products
// (sums over its slots in slot order, branch a then b) and their transposes,
// from the stored Jacobian columns; closures strided over the block or grid.
__device__ __forceinline__ bool long_run(const MechBuffers& m, uint32_t q) { return m.cq_off[q + 1] - m.cq_off[q] > kLongList; }

__device__ __forceinline__ void closure_products(const MechBuffers& m, const MechParams& p, const float* x) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    for (uint32_t k = tid; k < p.closures; k += nt) {
        const uint32_t s0 = m.cl_slot_off[k], s1 = m.cl_slot_off[k + 1], split = m.cl_split[k];
        // branch a's and branch b's sums in registers (no indexed array), unrolled so
        // the columns' loads issue together; each sum keeps slot order
        f3 pp_a = mkf3(0, 0, 0), pa_a = mkf3(0, 0, 0), pp_b = mkf3(0, 0, 0), pa_b = mkf3(0, 0, 0);
#pragma unroll 4
        for (uint32_t sl = s0; sl < s1; ++sl) {
            const f3 pd = xyz(m.slot_v[2 * sl]), ad = xyz(m.slot_v[2 * sl + 1]);
            const float dv = x[__float_as_uint(m.slot_v[2 * sl].w)];
            const f3 tp = pd * dv, ta = ad * dv;
            if (sl < split) {
                pp_a = pp_a + tp;
                pa_a = pa_a + ta;
            } else {
                pp_b = pp_b + tp;
                pa_b = pa_b + ta;
            }
        }
        const f3 pp = pp_a + pp_b, pa = pa_a + pa_b;
#pragma unroll 4
        for (uint32_t sl = s0; sl < s1; ++sl)
            m.slot_g[m.slot_pos[sl]] = dot(xyz(m.slot_v[2 * sl]), pp) + 1.0f * dot(xyz(m.slot_v[2 * sl + 1]), pa);
    }
}

// Joint frame of `body` in its root's frame (closure.wgsl:168-181).
__device__ __forceinline__ void joint_frame(const MechBuffers& m, uint32_t body, f3& axis, f3& anchor, uint32_t& coord) {
    const GpuMechanismBody mb = m.bodies[body];
    const GpuBearing& tb = m.bearings[mb.metadata[1]];
    const Link pp = ld_link(m.links_final, mb.metadata[0]);
    if (mb.metadata[2] == 0u) {
        axis = normalize(quat_rotate(pp.rot, r3(tb.local_axis_a)));
        anchor = xyz(pp.pos) + quat_rotate(pp.rot, r3(tb.local_anchor_a));
    } else {
        axis = -normalize(quat_rotate(pp.rot, r3(tb.local_axis_b)));
        anchor = xyz(pp.pos) + quat_rotate(pp.rot, r3(tb.local_anchor_b));
    }
    coord = tb.metadata[2];
}

__device__ __forceinline__ void closure_frames(const MechBuffers& m, const GpuBearing& br, f3& anc_a, f3& anc_b,
                                               f3& ax_a, f3& ax_b) {
    const Link pa = ld_link(m.links_final, br.metadata[0]), pb = ld_link(m.links_final, br.metadata[1]);
    anc_a = xyz(pa.pos) + quat_rotate(pa.rot, r3(br.local_anchor_a));
    anc_b = xyz(pb.pos) + quat_rotate(pb.rot, r3(br.local_anchor_b));
    ax_a = normalize(quat_rotate(pa.rot, r3(br.local_axis_a)));
    ax_b = normalize(quat_rotate(pb.rot, r3(br.local_axis_b)));
}

__device__ __forceinline__ bool finite3(f3 v) {
    return v.x == v.x && v.y == v.y && v.z == v.z && fabsf(v.x) < kFloatMax && fabsf(v.y) < kFloatMax &&
           fabsf(v.z) < kFloatMax;
}

// The closure loop of device.rs:973-1020: 12 Newton steps of
// closure.wgsl:268-427 (evaluate, finalize, 8-round diagonal PCG, step the
// coordinates), each followed by forward kinematics of the closure
// components.  Accumulations go through per-joint slots summed per
// coordinate in the serial order; dot products as above.  kGrid = false runs
// it in one block (few closures: block syncs are nearly free); kGrid = true
// spreads closures, coordinate chunks and bodies over a cooperative grid with
// grid barriers in place of the block syncs (thousands of closures).  Both
// compute the same values.
// evaluate_closures (closure.wgsl:268-319) for closure k: its residual against the
// tolerance (lane 0 of the walkers records the step's maxima), then the slots
// first + i * step of its branches: the joint's Jacobian column and the slot's
// gradient and diagonal contributions (NaN: none).  With step 32 a warp walks
// one closure; every slot's arithmetic is the same whoever computes it.
struct ClosureFrame {
    f3 aa, ab, xa, xb, rp, ra;   // anchors and axes of both bodies, their differences
    bool active;                 // the residual is above the tolerance
};
// The frame of closure k; `record` adds its residual to the step's maxima.
__device__ __forceinline__ ClosureFrame closure_frame(const MechBuffers& m, uint32_t k, uint32_t* st, uint32_t* flags,
                                                      bool record) {
    ClosureFrame f;
    closure_frames(m, m.bearings[m.cl_bearings[k]], f.aa, f.ab, f.xa, f.xb);
    f.rp = f.aa - f.ab;
    f.ra = f.xa - f.xb;
    f.active = true;
    if (!finite3(f.rp) || !finite3(f.ra)) {
        if (record) {
            atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
            atomicMax(&st[0], 0xffffffffu);
            atomicMax(&st[1], 0xffffffffu);
        }
        f.active = false;
    } else {
        const uint32_t um = round_u32(length(f.rp) * 1000000.0f);
        // axis error as atan2(|a x b|, a . b): FP32 acos (closure.wgsl:295) reads 0
        // below ~3.5e-4 rad, blind to the 1000 micro-degree tolerance
        const float deg =
            atan2_cr(length(cross(f.xa, f.xb)), clampf(dot(f.xa, f.xb), -1.0f, 1.0f)) * 57.295779513f;
        const uint32_t ud = round_u32(deg * 1000000.0f);
        if (record) {
            atomicMax(&st[0], um);
            atomicMax(&st[1], ud);
        }
        f.active = !(um <= 10u && ud <= 1000u);
    }
    return f;
}

// The slot's Jacobian column, stored; returns its coordinate.  The links do not
// move during the step's PCG rounds, so closure.wgsl:194-266's recomputation in
// every round gives these same floats (sign * v == v * sign).
__device__ __forceinline__ uint32_t slot_column(const MechBuffers& m, const ClosureFrame& f, uint32_t sl, bool side_a,
                                                uint32_t Q, f3& pd, f3& ad) {
    const f3 ea = side_a ? f.aa : f.ab, ex = side_a ? f.xa : f.xb;
    const float sign = side_a ? 1.0f : -1.0f;
    f3 axis, anchor;
    uint32_t coord;
    joint_frame(m, m.slot_body[sl], axis, anchor, coord);
    pd = cross(axis, ea - anchor) * sign;
    ad = cross(axis, ex) * sign;
    m.slot_v[2 * sl] = f4(pd, __uint_as_float(coord < Q ? coord : 0u));
    m.slot_v[2 * sl + 1] = f4(ad, 0.0f);
    return coord;
}

__device__ __forceinline__ void evaluate_closure(const MechBuffers& m, uint32_t k, uint32_t* st, uint32_t* flags,
                                                 uint32_t Q, uint32_t first, uint32_t step, bool record) {
    const ClosureFrame f = closure_frame(m, k, st, flags, record && first == 0);
    const f3 rp = f.rp, ra = f.ra;
    const bool active = f.active;
    const uint32_t s0 = m.cl_slot_off[k], s1 = m.cl_slot_off[k + 1], split = m.cl_split[k];
    for (uint32_t sl = s0 + first; sl < s1; sl += step) {
        float g = 0.0f, d = 0.0f;
        uint32_t valid = 0;
        f3 pd, ad;
        const uint32_t coord = slot_column(m, f, sl, sl < split, Q, pd, ad);
        if (active) {
            if (coord >= Q) {
                atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
            } else {
                g = dot(rp, pd) + 1.0f * dot(ra, ad);
                d = dot(pd, pd) + 1.0f * dot(ad, ad);
                if (g == g && d == d) valid = 1;
                else atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
            }
        }
        // NaN marks "no contribution" so the gather skips it
        m.slot_g[m.slot_pos[sl]] = valid ? g : __int_as_float(0x7fffffff);
        m.slot_d[m.slot_pos[sl]] = valid ? d : 0.0f;
    }
}

template <bool kGrid>
__global__ void __launch_bounds__(kClosureThreads) k_closure_loop(StepBuffers b, MechBuffers m, MechParams p) {
    __shared__ float s_red[33];
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, gnt = gridDim.x * blockDim.x;
    const uint32_t NC = p.closures, NQ = p.closure_coords, NB = p.closure_bodies, Q = p.coordinate_count;
    const uint32_t chunks = (NQ + kDotChunk - 1) / kDotChunk;
    float* sol = m.pcg;
    float* res = m.pcg + Q;
    float* pre = m.pcg + 2ull * Q;
    float* dir = m.pcg + 3ull * Q;
    float* op = m.pcg + 4ull * Q;
    uint32_t* flags = &b.diag->error_flags;
    // per-step residual maxima (zeroed at the start of the tick) and chunk sums
    uint32_t* state = m.loop_state;
    float* part_a = m.chunk_part;
    float* part_b = m.chunk_part + chunks;
    uint32_t steps = 0, rounds = 0;
    for (uint32_t step = 0; step < kClosureSteps; ++step) {
        uint32_t* st = state + 2 * step;
        // evaluate_closures (closure.wgsl:268-319): slot contributions
        if (p.wide_closures) {
            // closures of dozens of slots: the residuals alone first (a thread per closure).  A
            // converged step needs no slot: on the 100 x 100 x 10 loop lattice at rest (20M slots)
            // that takes the loop from 1,160 to 15 us.  Then a warp per closure, its slots
            // spread over the lanes.
            for (uint32_t k = gtid; k < NC; k += gnt) closure_frame(m, k, st, flags, true);
        } else {
            for (uint32_t k = gtid; k < NC; k += gnt) evaluate_closure(m, k, st, flags, Q, 0u, 1u, true);
        }
        loop_sync<kGrid>(m.grid_barrier, flags);
        const bool unconverged = ld_relaxed_u32(&st[0]) > 10u || ld_relaxed_u32(&st[1]) > 1000u;
        if (p.wide_closures && gtid == 0) *m.columns_stale = unconverged ? 0u : 1u;
        if (!unconverged) break;   // the steps after a converged one move nothing
        if (p.wide_closures) {
            for (uint32_t k = gtid >> 5; k < NC; k += gnt >> 5)
                evaluate_closure(m, k, st, flags, Q, threadIdx.x & 31u, 32u, false);
            loop_sync<kGrid>(m.grid_barrier, flags);
        }
        ++steps;
        if (p.long_coords) gather_long_runs<kGrid, true>(m, p, m.grad, m.diag, flags);   // long runs first
        // gather per coordinate in the serial accumulation order, then the PCG's
        // initial vectors (solve_closure_pcg, closure.wgsl:333-427), chunk by chunk
        for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
            const uint32_t q = c * kDotChunk + threadIdx.x;
            float part = 0.0f;
            if (q < NQ) {
                float g = 0.0f, d = 0.0f;
                if (long_run(m, q)) {
                    g = m.grad[m.cq_coords[q]];
                    d = m.diag[m.cq_coords[q]];
                } else {
                    for (uint32_t i = m.cq_off[q]; i < m.cq_off[q + 1]; ++i) {
                        const float sg = m.slot_g[i];
                        if (sg == sg) { g += sg; d += m.slot_d[i]; }
                    }
                }
                const uint32_t cc = m.cq_coords[q];
                m.grad[cc] = g;
                m.diag[cc] = d;
                float r = 0.0f, z = 0.0f;
                if (d > 1.0e-12f) { r = -g; z = r / d; }
                sol[cc] = 0.0f; res[cc] = r; pre[cc] = z; dir[cc] = z; op[cc] = 0.0f;
                part = r * z;
            }
            if (NQ > kSerialDot) chunk_dot(part, part_a, c, s_red);
        }
        {
            loop_sync<kGrid>(m.grid_barrier, flags);
            float rz = dot_total(NQ, m, res, pre, part_a, s_red);
            for (uint32_t round = 0; round < kClosureRounds; ++round) {
                // J^T J dir per closure: branch products then transposes
                // (closure.wgsl:194-266), from the step's stored columns
                closure_products(m, p, dir);
                loop_sync<kGrid>(m.grid_barrier, flags);
                if (p.long_coords) gather_long_runs<kGrid, false>(m, p, op, nullptr, flags);
                for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
                    const uint32_t q = c * kDotChunk + threadIdx.x;
                    float dpart = 0.0f;
                    if (q < NQ) {
                        float o = 0.0f;
                        if (long_run(m, q)) o = op[m.cq_coords[q]];
                        else
                            for (uint32_t i = m.cq_off[q]; i < m.cq_off[q + 1]; ++i) o += m.slot_g[i];
                        const uint32_t cc = m.cq_coords[q];
                        op[cc] = o;
                        dpart = dir[cc] * o;
                    }
                    if (NQ > kSerialDot) chunk_dot(dpart, part_b, c, s_red);
                }
                loop_sync<kGrid>(m.grid_barrier, flags);
                const float dop = dot_total(NQ, m, dir, op, part_b, s_red);
                const float alpha = fabsf(dop) > 1.0e-20f ? rz / dop : 0.0f;
                for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
                    const uint32_t q = c * kDotChunk + threadIdx.x;
                    float npart = 0.0f;
                    if (q < NQ) {
                        const uint32_t cc = m.cq_coords[q];
                        sol[cc] += alpha * dir[cc];
                        res[cc] -= alpha * op[cc];
                        const float d = m.diag[cc];
                        pre[cc] = 0.0f;
                        if (d > 1.0e-12f) pre[cc] = res[cc] / d;
                        npart = res[cc] * pre[cc];
                    }
                    if (NQ > kSerialDot) chunk_dot(npart, part_a, c, s_red);
                }
                loop_sync<kGrid>(m.grid_barrier, flags);
                const float nrz = dot_total(NQ, m, res, pre, part_a, s_red);
                const float beta = fabsf(rz) > 1.0e-20f ? nrz / rz : 0.0f;
                for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
                    const uint32_t q = c * kDotChunk + threadIdx.x;
                    if (q < NQ) {
                        const uint32_t cc = m.cq_coords[q];
                        dir[cc] = pre[cc] + beta * dir[cc];
                    }
                }
                rz = nrz;
                ++rounds;
                loop_sync<kGrid>(m.grid_barrier, flags);
            }
            // step every coordinate (coordinates off the closure branches add 0)
            for (uint32_t c = gtid; c < Q; c += gnt) {
                const float stp = clampf(0.35f * sol[c], -0.2f, 0.2f);
                if (stp == stp) m.coords[c].angle += stp;
                else atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
            }
            loop_sync<kGrid>(m.grid_barrier, flags);
            // forward kinematics of the closure components (mechanism.wgsl:72-149)
            for (uint32_t i = gtid; i < NB; i += gnt) prepare_link(m, m.cb_bodies[i]);
            loop_sync<kGrid>(m.grid_barrier, flags);
            bool a_src = true;
            for (uint32_t r = 0; r < p.jump_rounds; ++r) {
                for (uint32_t i = gtid; i < NB; i += gnt)
                    jump_link(a_src ? m.links_a : m.links_b, a_src ? m.links_b : m.links_a, m.cb_bodies[i]);
                loop_sync<kGrid>(m.grid_barrier, flags);
                a_src = !a_src;
            }
        }
    }
    if (gtid == 0) {
        atomicAdd(&b.diag->reserved_b, steps);
        atomicAdd(&b.diag->reserved_c, rounds);
    }
}

// The columns that a converged step of a wide system did not need, for a read of
// them (MK_BUF_CLOSURE_SLOTS): a warp per closure, from the links of that step.
__global__ void __launch_bounds__(kMBlock) k_closure_columns(MechBuffers m, MechParams p) {
    if (*m.columns_stale == 0u) return;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < p.closures; k += warps) {
        const ClosureFrame f = closure_frame(m, k, nullptr, nullptr, false);
        const uint32_t split = m.cl_split[k];
        f3 pd, ad;
        for (uint32_t sl = m.cl_slot_off[k] + (threadIdx.x & 31u); sl < m.cl_slot_off[k + 1]; sl += 32u)
            slot_column(m, f, sl, sl < split, p.coordinate_count, pd, ad);
    }
}

// ------------------------------------------------- closure PCG to a residual
// MK_CLOSURE_PCG_RESIDUAL: each Newton step of the closure loop solves
// (J^T J) dtheta = -g by preconditioned conjugate gradients until
// ||r|| <= closure_tol * ||r0|| (or closure_max_it iterations), with
// FP64 dot products and residual check (f32 vectors), instead of the
// reference's 8 diagonal-PCG rounds.  The preconditioner is block Jacobi
// over 2 x 2 blocks of consecutive closure coordinates (a whole loop's block
// would be the exact inverse of its independent component, leaving nothing
// to precondition); with the learned preconditioner the network's corrected
// block inverse replaces a block when it is positive definite.
//
// Each Newton step is two launches (evaluate, solve) with the network in
// between; a converged step sets `done` and the later launches return.

// Fixed-order FP64 block sum (1024 threads): per-thread partials, warp
// shuffle-down trees, then the same shuffle-down tree over the 32 warp sums,
// which every warp evaluates for itself (identical operands and order, so
// identical bits) instead of warp 0 publishing it through shared memory: two
// barriers per sum instead of four.
__device__ __forceinline__ double block_sum_d(double v, double* scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    __syncthreads();   // the previous sum's readers are done with scratch
    if (lane == 0) scratch[w] = v;
    __syncthreads();
    double r = lane < (blockDim.x >> 5) ? scratch[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    return __shfl_sync(0xffffffffu, r, 0);
}

// The FP64 dot product after a loop_sync: the chunk sums in chunk order (thread
// 0 of every block), shared through scratch[32].  Chunks of 1,024 coordinates
// with one coordinate per thread: up to 1,024 coordinates this is the block
// tree of the per-thread terms, and one block or the whole grid give the same.
__device__ __forceinline__ double chunk_total_d(const double* part, uint32_t chunks, double* scratch) {
    if (threadIdx.x == 0) {
        double acc = 0.0;
        for (uint32_t c = 0; c < chunks; ++c) acc += part[c];
        scratch[32] = acc;
    }
    __syncthreads();
    const double r = scratch[32];
    __syncthreads();
    return r;
}

// out[c] = (J^T J x)[c] for the closure coordinates, from the stored columns
// (the block, or with kGrid the whole cooperative grid).
template <bool kGrid>
__device__ void closure_apply(const MechBuffers& m, const MechParams& p, const float* x, float* out,
                              uint32_t* flags) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    closure_products(m, p, x);
    loop_sync<kGrid>(m.grid_barrier, flags);
    if (p.long_coords) gather_long_runs<kGrid, false>(m, p, out, nullptr, flags);
    for (uint32_t q = tid; q < p.closure_coords; q += nt) {
        if (long_run(m, q)) continue;
        float o = 0.0f;
        for (uint32_t i = m.cq_off[q]; i < m.cq_off[q + 1]; ++i) o += m.slot_g[i];
        out[m.cq_coords[q]] = o;
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
}

// (J^T J)[i][j] for two closure coordinates (positions qi, qj in the list).
__device__ __forceinline__ float closure_coupling(const MechBuffers& m, uint32_t qi, uint32_t qj) {
    float r = 0.0f;
    for (uint32_t a = m.cq_off[qi]; a < m.cq_off[qi + 1]; ++a) {
        const uint32_t sa = m.cq_slots[a];
        for (uint32_t bq = m.cq_off[qj]; bq < m.cq_off[qj + 1]; ++bq) {
            const uint32_t sb = m.cq_slots[bq];
            if (m.slot_closure[sa] != m.slot_closure[sb]) continue;
            r += dot(xyz(m.slot_v[2 * sa]), xyz(m.slot_v[2 * sb])) +
                 1.0f * dot(xyz(m.slot_v[2 * sa + 1]), xyz(m.slot_v[2 * sb + 1]));
        }
    }
    return r;
}

template <bool kGrid>
__global__ void __launch_bounds__(kClosureThreads) k_closure_eval(StepBuffers b, MechBuffers m, MechParams p,
                                                                  uint32_t step) {
    ClosureState* cs = m.cstate;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const uint32_t NC = p.closures, NQ = p.closure_coords, Q = p.coordinate_count;
    uint32_t* flags = &b.diag->error_flags;
    if (step == 0) {
        if (tid == 0) *cs = ClosureState{0u, 0u, 0u, 0u, 0u, 0u, 0.0};
    } else if (ld_acquire_u32(&cs->done)) {
        return;
    }
    uint32_t* s_state = m.loop_state + 2 * step;   // largest residuals of this step (zeroed per tick)
    // slot columns and their gradient / diagonal contributions (closure.wgsl:268-319)
    for (uint32_t k = tid; k < NC; k += nt) {
        const GpuBearing br = m.bearings[m.cl_bearings[k]];
        f3 aa, ab, xa, xb;
        closure_frames(m, br, aa, ab, xa, xb);
        const f3 rp = aa - ab, ra = xa - xb;
        const uint32_t s0 = m.cl_slot_off[k], s1 = m.cl_slot_off[k + 1], split = m.cl_split[k];
        bool active = true;
        if (!finite3(rp) || !finite3(ra)) {
            atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
            atomicMax(&s_state[0], 0xffffffffu);
            atomicMax(&s_state[1], 0xffffffffu);
            active = false;
        } else {
            const uint32_t um = round_u32(length(rp) * 1000000.0f);
            const float deg = atan2_cr(length(cross(xa, xb)), clampf(dot(xa, xb), -1.0f, 1.0f)) * 57.295779513f;
            const uint32_t ud = round_u32(deg * 1000000.0f);
            atomicMax(&s_state[0], um);
            atomicMax(&s_state[1], ud);
            active = !(um <= 10u && ud <= 1000u);
        }
        for (uint32_t sl = s0; sl < s1; ++sl) {
            const bool side_a = sl < split;
            const f3 ea = side_a ? aa : ab, ex = side_a ? xa : xb;
            const float sign = side_a ? 1.0f : -1.0f;
            f3 axis, anchor;
            uint32_t coord;
            joint_frame(m, m.slot_body[sl], axis, anchor, coord);
            f3 pd = mkf3(0, 0, 0), ad = mkf3(0, 0, 0);
            float g = 0.0f, d = 0.0f;
            uint32_t valid = 0;
            if (coord >= Q) {
                atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
                coord = 0;
            } else {
                pd = cross(axis, ea - anchor) * sign;
                ad = cross(axis, ex) * sign;
                if (active) {
                    g = dot(rp, pd) + 1.0f * dot(ra, ad);
                    d = dot(pd, pd) + 1.0f * dot(ad, ad);
                    if (g == g && d == d) valid = 1;
                    else atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
                }
            }
            m.slot_v[2 * sl] = f4(pd, __uint_as_float(coord));
            m.slot_v[2 * sl + 1] = f4(ad, __uint_as_float(m.slot_closure[sl]));
            m.slot_g[m.slot_pos[sl]] = valid ? g : __int_as_float(0x7fffffff);
            m.slot_d[m.slot_pos[sl]] = valid ? d : 0.0f;
        }
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
    if (p.long_coords) gather_long_runs<kGrid, true>(m, p, m.grad, m.diag, flags);
    for (uint32_t q = tid; q < NQ; q += nt) {
        const uint32_t c = m.cq_coords[q];
        if (!long_run(m, q)) {
            float g = 0.0f, d = 0.0f;
            for (uint32_t i = m.cq_off[q]; i < m.cq_off[q + 1]; ++i) {
                const float sg = m.slot_g[i];
                if (sg == sg) { g += sg; d += m.slot_d[i]; }
            }
            m.grad[c] = g;
            m.diag[c] = d;
        }
        // probe vectors: ones and alternating signs over the coordinate list
        m.pcg[c] = 1.0f;
        m.pcg[Q + c] = (q & 1u) ? -1.0f : 1.0f;
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
    const bool unconverged = ld_relaxed_u32(&s_state[0]) > 10u || ld_relaxed_u32(&s_state[1]) > 1000u;
    // the 2 x 2 blocks and the network's inputs, for the preconditioners that use them
    const bool pair_blocks = p.precond == MK_PRECOND_LEARNED || p.precond == MK_PRECOND_PAIR_BLOCKS;
    // A * ones and A * alternating signs (block inputs of the network)
    if (pair_blocks) closure_apply<kGrid>(m, p, m.pcg, m.probe, flags);
    if (pair_blocks) closure_apply<kGrid>(m, p, m.pcg + Q, m.probe + Q, flags);
    // block entries (a, b, d) and the plain 2 x 2 inverse
    float* blk_b = m.pcg + 2ull * Q;   // coupling of each block (free until the solve)
    for (uint32_t blk = tid; pair_blocks && blk < p.blocks; blk += nt) {
        const uint32_t qi = 2 * blk, qj = qi + 1;
        const bool pair = qj < NQ;
        const float a = m.diag[m.cq_coords[qi]], d = pair ? m.diag[m.cq_coords[qj]] : 0.0f;
        const float bij = pair ? closure_coupling(m, qi, qj) : 0.0f;
        float4 inv = make_float4(a > 1.0e-12f ? 1.0f / a : 0.0f, 0.0f, d > 1.0e-12f ? 1.0f / d : 0.0f, 0.0f);
        if (pair && a > 1.0e-12f && d > 1.0e-12f) {
            const float det = a * d - bij * bij;
            if (det > 1.0e-6f * (a * d)) inv = make_float4(d / det, -bij / det, a / det, 0.0f);
        }
        m.blk_m[blk] = inv;
        blk_b[blk] = bij;
    }
    if (pair_blocks) loop_sync<kGrid>(m.grid_barrier, flags);
    // network inputs: the diagonal-normalised entries of J^T J around the block,
    // with the partner block (blk ^ 1) and the couplings to it recovered from
    // the two probes (exact when the loop's coordinates are these two blocks)
    for (uint32_t blk = tid; pair_blocks && blk < p.blocks; blk += nt) {
        float4 f[4] = {make_float4(0, 0, 0, 0), make_float4(0, 0, 0, 0), make_float4(0, 0, 0, 0),
                       make_float4(0, 0, 0, 1.0f)};
        const uint32_t qi = 2 * blk, qj = qi + 1;
        const uint32_t ci = m.cq_coords[qi];
        const bool pair = qj < NQ;
        const uint32_t cj = pair ? m.cq_coords[qj] : ci;
        const float a = m.diag[ci], d = pair ? m.diag[cj] : 0.0f, bij = blk_b[blk];
        const uint32_t pb = blk ^ 1u;
        const bool partner = pb < p.blocks && 2 * pb + 1 < NQ;
        if (pair && partner && a > 1.0e-12f && d > 1.0e-12f) {
            const float pa = m.diag[m.cq_coords[2 * pb]], pd = m.diag[m.cq_coords[2 * pb + 1]];
            if (pa > 1.0e-12f && pd > 1.0e-12f) {
                const float s1i = m.probe[ci] - a - bij, ssi = m.probe[Q + ci] - a + bij;
                const float s1j = m.probe[cj] - bij - d, ssj = m.probe[Q + cj] - bij + d;
                const float sa = sqrtf(a), sd = sqrtf(d), spa = sqrtf(pa), spd = sqrtf(pd);
                f[0] = make_float4(bij / (sa * sd), blk_b[pb] / (spa * spd), 0.5f * (s1i + ssi) / (sa * spa),
                                   0.5f * (s1i - ssi) / (sa * spd));
                f[1] = make_float4(0.5f * (s1j + ssj) / (sd * spa), 0.5f * (s1j - ssj) / (sd * spd), logf(a / d),
                                   1.0f);
            }
        }
        float4* fo = m.blk_feat + 4ull * blk;
        fo[0] = f[0]; fo[1] = f[1]; fo[2] = f[2]; fo[3] = f[3];
    }
    // per-loop blocks: Cholesky of J^T J on the loop's coordinates plus a ridge of
    // 1e-6 x the mean diagonal; a failed pivot leaves the block diagonal (Jacobi).
    // Across the grid the off-diagonal couplings (chains of dependent loads) are
    // computed first, one entry per thread, into the block's packed storage, and
    // one thread per loop then factors it; in one block the loop's thread
    // computes them itself (the extra sync and round trip cost more there).
    if (p.precond == MK_PRECOND_BLOCK_JACOBI) {
        if (kGrid) {
            constexpr uint32_t kOff = kMaxLoop * (kMaxLoop - 1) / 2;   // strict lower entries of a block
            for (uint32_t e = tid; e < p.loops * kOff; e += nt) {
                const uint32_t lp = e / kOff;
                uint32_t r = e % kOff, i = 1;
                while (r >= i) { r -= i; ++i; }   // (i, r): row i > column r
                const uint32_t o = m.loop_off[lp], n = m.loop_off[lp + 1] - o;
                if (i < n)
                    m.loop_l[36ull * lp + i * (i + 1) / 2 + r] = closure_coupling(m, m.loop_q[o + i], m.loop_q[o + r]);
            }
            loop_sync<kGrid>(m.grid_barrier, flags);
        }
        for (uint32_t lp = tid; lp < p.loops; lp += nt) {
            const uint32_t o = m.loop_off[lp], n = m.loop_off[lp + 1] - o;
            float a[kMaxLoop * (kMaxLoop + 1) / 2];
            float mean = 0.0f;
            for (uint32_t i = 0; i < n; ++i) mean += m.diag[m.cq_coords[m.loop_q[o + i]]];
            mean = n ? mean / (float)n : 0.0f;
            for (uint32_t i = 0; i < n; ++i)
                for (uint32_t j = 0; j <= i; ++j)
                    a[i * (i + 1) / 2 + j] = i == j  ? m.diag[m.cq_coords[m.loop_q[o + i]]] + 1.0e-6f * mean
                                             : kGrid ? m.loop_l[36ull * lp + i * (i + 1) / 2 + j]
                                                     : closure_coupling(m, m.loop_q[o + i], m.loop_q[o + j]);
            bool ok = mean > 1.0e-12f;
            for (uint32_t j = 0; j < n && ok; ++j) {
                float dj = a[j * (j + 1) / 2 + j];
                for (uint32_t k = 0; k < j; ++k) dj -= a[j * (j + 1) / 2 + k] * a[j * (j + 1) / 2 + k];
                if (!(dj > 0.0f)) { ok = false; break; }
                const float ljj = sqrtf(dj);
                a[j * (j + 1) / 2 + j] = ljj;
                for (uint32_t i = j + 1; i < n; ++i) {
                    float v = a[i * (i + 1) / 2 + j];
                    for (uint32_t k = 0; k < j; ++k) v -= a[i * (i + 1) / 2 + k] * a[j * (j + 1) / 2 + k];
                    a[i * (i + 1) / 2 + j] = v / ljj;
                }
            }
            float* l = m.loop_l + 36ull * lp;
            for (uint32_t i = 0; i < n; ++i)
                for (uint32_t j = 0; j <= i; ++j) {
                    float v = a[i * (i + 1) / 2 + j];
                    if (!ok) {   // Jacobi: L = diag(sqrt(a_ii))
                        const float dii = m.diag[m.cq_coords[m.loop_q[o + i]]];
                        v = (i == j) ? (dii > 1.0e-12f ? sqrtf(dii) : 0.0f) : 0.0f;
                    }
                    l[i * (i + 1) / 2 + j] = v;
                }
        }
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
    if (tid == 0) {
        if (unconverged) {
            cs->live_blocks = p.blocks;
            ++cs->newton_steps;
        } else {
            cs->live_blocks = 0;
            st_release_u32(&cs->done, 1u);
        }
    }
}

template <bool kGrid>
__device__ __forceinline__ void precond_apply(const MechBuffers& m, const MechParams& p, const float* r, float* z,
                                              uint32_t* flags) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    if (p.precond == MK_PRECOND_DIAGONAL) {   // closure.wgsl:343-346, :396-400
        for (uint32_t q = tid; q < p.closure_coords; q += nt) {
            const uint32_t c = m.cq_coords[q];
            const float d = m.diag[c];
            z[c] = d > 1.0e-12f ? r[c] / d : 0.0f;
        }
        loop_sync<kGrid>(m.grid_barrier, flags);
        return;
    }
    if (p.precond == MK_PRECOND_BLOCK_JACOBI) {
        for (uint32_t lp = tid; lp < p.loops; lp += nt) {
            const uint32_t o = m.loop_off[lp], n = m.loop_off[lp + 1] - o;
            const float* l = m.loop_l + 36ull * lp;
            float y[kMaxLoop];
            for (uint32_t i = 0; i < n; ++i) {   // L y = r
                float v = r[m.cq_coords[m.loop_q[o + i]]];
                for (uint32_t k = 0; k < i; ++k) v -= l[i * (i + 1) / 2 + k] * y[k];
                const float lii = l[i * (i + 1) / 2 + i];
                y[i] = lii > 0.0f ? v / lii : 0.0f;
            }
            for (uint32_t ii = n; ii-- > 0;) {   // L^T z = y
                float v = y[ii];
                for (uint32_t k = ii + 1; k < n; ++k) v -= l[k * (k + 1) / 2 + ii] * y[k];
                const float lii = l[ii * (ii + 1) / 2 + ii];
                y[ii] = lii > 0.0f ? v / lii : 0.0f;
            }
            for (uint32_t i = 0; i < n; ++i) z[m.cq_coords[m.loop_q[o + i]]] = y[i];
        }
        loop_sync<kGrid>(m.grid_barrier, flags);
        return;
    }
    for (uint32_t blk = tid; blk < p.blocks; blk += nt) {
        const float4 mi = m.blk_m[blk];
        const uint32_t qi = 2 * blk, qj = qi + 1;
        const uint32_t ci = m.cq_coords[qi];
        if (qj < p.closure_coords) {
            const uint32_t cj = m.cq_coords[qj];
            const float ri = r[ci], rj = r[cj];
            z[ci] = mi.x * ri + mi.y * rj;
            z[cj] = mi.y * ri + mi.z * rj;
        } else {
            z[ci] = mi.x * r[ci];
        }
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
}

template <bool kGrid>
__global__ void __launch_bounds__(kClosureThreads) k_closure_pcg(StepBuffers b, MechBuffers m, MechParams p,
                                                                 uint32_t step) {
    __shared__ double s_red[33];
    ClosureState* cs = m.cstate;
    if (ld_acquire_u32(&cs->done)) return;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const uint32_t NQ = p.closure_coords, NB = p.closure_bodies, Q = p.coordinate_count;
    const uint32_t chunks = (NQ + kDotChunk - 1) / kDotChunk;
    uint32_t* flags = &b.diag->error_flags;
    double* part_a = m.chunk_part_d;            // chunk sums of the FP64 dot products
    double* part_b = m.chunk_part_d + chunks;
    // one block over one chunk: a dot product's block sum is its total (the chunk-order
    // total is 0.0 + the chunk sums), and the sum's barriers order the loop's writes, so
    // neither the chunk sums in memory nor the sync that publishes them are needed
    const bool one = !kGrid && chunks == 1;
    double one_a = 0.0, one_b = 0.0;
    float* sol = m.pcg;
    float* res = m.pcg + Q;
    float* pre = m.pcg + 2ull * Q;
    float* dir = m.pcg + 3ull * Q;
    float* op = m.pcg + 4ull * Q;
    // learned blocks: T' = S M^-1 S with S = diag(sqrt(a), sqrt(d)), from the network's
    // (y0, y1, y2) as t11 = e^y0, t22 = e^y1, t12 = 0.999 tanh(y2) sqrt(t11 t22): positive
    // definite by construction (the check below only catches overflow and NaN)
    if (p.learned_precond) {
        uint32_t used = 0, rejected = 0;
        for (uint32_t blk = tid; blk < p.blocks; blk += nt) {
            const float y0 = fminf(fmaxf(m.blk_out[3 * blk], -30.0f), 30.0f);
            const float y1 = fminf(fmaxf(m.blk_out[3 * blk + 1], -30.0f), 30.0f);
            const float t11 = expf(y0), t22 = expf(y1);
            const float t12 = 0.999f * tanhf(m.blk_out[3 * blk + 2]) * sqrtf(t11 * t22);
            float* h = m.blk_hist + 3ull * ((uint64_t)step * p.blocks + blk);
            h[0] = t11; h[1] = t12; h[2] = t22;
            const uint32_t qi = 2 * blk, qj = qi + 1;
            const uint32_t ci = m.cq_coords[qi];
            const bool pair = qj < NQ;
            const float a = m.diag[ci], d = pair ? m.diag[m.cq_coords[qj]] : 0.0f;
            if (pair) {
                if (a > 1.0e-12f && d > 1.0e-12f && t11 > 0.0f && t22 > 0.0f &&
                    t11 * t22 - t12 * t12 > 1.0e-6f * (t11 * t22)) {
                    const float sa = sqrtf(a), sd = sqrtf(d);
                    m.blk_m[blk] = make_float4(t11 / a, t12 / (sa * sd), t22 / d, 0.0f);
                    ++used;
                } else {
                    ++rejected;
                }
            } else if (a > 1.0e-12f && t11 > 0.0f) {
                m.blk_m[blk] = make_float4(t11 / a, 0.0f, 0.0f, 0.0f);
                ++used;
            } else {
                ++rejected;
            }
        }
        if (used) atomicAdd(&cs->learned_blocks, used);
        if (rejected) atomicAdd(&cs->rejected_blocks, rejected);
        loop_sync<kGrid>(m.grid_barrier, flags);
    }
    // r = -g, x = 0, z = M^-1 r, p = z
    for (uint32_t q = tid; q < NQ; q += nt) {
        const uint32_t c = m.cq_coords[q];
        sol[c] = 0.0f;
        res[c] = -m.grad[c];
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
    precond_apply<kGrid>(m, p, res, pre, flags);
    // coordinate loops that feed a dot product walk chunks of 1,024 coordinates
    // (thread t of the chunk's block holds coordinate 1024 c + t)
    for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const uint32_t q = c * kDotChunk + threadIdx.x;
        double prz = 0.0, prr = 0.0;
        if (q < NQ) {
            const uint32_t cc = m.cq_coords[q];
            dir[cc] = pre[cc];
            prz = (double)res[cc] * (double)pre[cc];
            prr = (double)res[cc] * (double)res[cc];
        }
        const double sz = block_sum_d(prz, s_red), sr = block_sum_d(prr, s_red);
        if (one) { one_a = sz; one_b = sr; }
        else if (threadIdx.x == 0) { part_a[c] = sz; part_b[c] = sr; }
    }
    if (!one) loop_sync<kGrid>(m.grid_barrier, flags);
    double rz = one ? 0.0 + one_a : chunk_total_d(part_a, chunks, s_red);
    const double rr0 = one ? 0.0 + one_b : chunk_total_d(part_b, chunks, s_red);
    double rr = rr0;
    const double tol2 = (double)p.closure_tol * (double)p.closure_tol;
    uint32_t it = 0;
    while (it < p.closure_max_it && rr > tol2 * rr0) {
        closure_apply<kGrid>(m, p, dir, op, flags);
        for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
            const uint32_t q = c * kDotChunk + threadIdx.x;
            double ppq = 0.0;
            if (q < NQ) {
                const uint32_t cc = m.cq_coords[q];
                ppq = (double)dir[cc] * (double)op[cc];
            }
            const double sq = block_sum_d(ppq, s_red);
            if (one) one_a = sq;
            else if (threadIdx.x == 0) part_a[c] = sq;
        }
        if (!one) loop_sync<kGrid>(m.grid_barrier, flags);
        const double pq = one ? 0.0 + one_a : chunk_total_d(part_a, chunks, s_red);
        const float alpha = fabs(pq) > 1.0e-30 ? (float)(rz / pq) : 0.0f;
        for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
            const uint32_t q = c * kDotChunk + threadIdx.x;
            double pr = 0.0;
            if (q < NQ) {
                const uint32_t cc = m.cq_coords[q];
                sol[cc] += alpha * dir[cc];
                res[cc] -= alpha * op[cc];
                pr = (double)res[cc] * (double)res[cc];
            }
            const double sr = block_sum_d(pr, s_red);
            if (one) one_b = sr;
            else if (threadIdx.x == 0) part_b[c] = sr;
        }
        if (!one) loop_sync<kGrid>(m.grid_barrier, flags);
        rr = one ? 0.0 + one_b : chunk_total_d(part_b, chunks, s_red);
        ++it;
        if (rr <= tol2 * rr0) break;
        precond_apply<kGrid>(m, p, res, pre, flags);
        for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
            const uint32_t q = c * kDotChunk + threadIdx.x;
            double pz = 0.0;
            if (q < NQ) {
                const uint32_t cc = m.cq_coords[q];
                pz = (double)res[cc] * (double)pre[cc];
            }
            const double sz = block_sum_d(pz, s_red);
            if (one) one_a = sz;
            else if (threadIdx.x == 0) part_a[c] = sz;
        }
        if (!one) loop_sync<kGrid>(m.grid_barrier, flags);
        const double nrz = one ? 0.0 + one_a : chunk_total_d(part_a, chunks, s_red);
        const float beta = fabs(rz) > 1.0e-300 ? (float)(nrz / rz) : 0.0f;
        for (uint32_t q = tid; q < NQ; q += nt) {
            const uint32_t cc = m.cq_coords[q];
            dir[cc] = pre[cc] + beta * dir[cc];
        }
        rz = nrz;
        loop_sync<kGrid>(m.grid_barrier, flags);
    }
    if (tid == 0) {
        cs->pcg_iterations += it;
        const double rel = rr0 > 0.0 ? sqrt(rr / rr0) : 0.0;
        if (rel > cs->max_relative_residual) cs->max_relative_residual = rel;
    }
    // step the closure coordinates (closure.wgsl:416-427)
    for (uint32_t q = tid; q < NQ; q += nt) {
        const uint32_t c = m.cq_coords[q];
        const float stp = clampf(0.35f * sol[c], -0.2f, 0.2f);
        if (stp == stp) m.coords[c].angle += stp;
        else atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
    }
    loop_sync<kGrid>(m.grid_barrier, flags);
    // forward kinematics of the closure components (mechanism.wgsl:72-149)
    for (uint32_t i = tid; i < NB; i += nt) prepare_link(m, m.cb_bodies[i]);
    loop_sync<kGrid>(m.grid_barrier, flags);
    bool a_src = true;
    for (uint32_t r = 0; r < p.jump_rounds; ++r) {
        for (uint32_t i = tid; i < NB; i += nt)
            jump_link(a_src ? m.links_a : m.links_b, a_src ? m.links_b : m.links_a, m.cb_bodies[i]);
        loop_sync<kGrid>(m.grid_barrier, flags);
        a_src = !a_src;
    }
}

// ------------------------------------------------ closure solve in one block
// A closure system that fits one block's shared memory is solved there: its
// Jacobian columns, slot values, search direction and (PCG) preconditioner stay
// in shared memory, the PCG vectors in the registers of their coordinate's
// thread, and all Newton steps run in one launch.  The kernels above keep all
// of that in global memory, where every phase of a round is a chain of L2 round
// trips.  The evaluation (a thread per slot) and the forward kinematics (a
// thread per body) are spread over a cluster of blocks when the system is
// large; the columns go straight to block 0's shared memory.  Each sum keeps
// the order of those kernels (slots of a closure, slots of a coordinate, the
// dot products' trees and chunks), so the results are theirs bit for bit.
// Bound: the dependent chain of each phase and its barrier.  One B200, a tick's
// closure solve: 380 loops of five bodies in the reference's loop 1,550 us in
// the kernels above, 500 us here; 49 such loops by PCG to 1e-5 500 us (24
// launches), 196 us.  The line (closure_block_shape) is what the registers and
// the shared memory hold; systems with runs over kLongList slots keep the
// kernels above.
//
// Slots are laid out by their place j in their closure, closures sorted by
// falling slot count: slot j of closure k is column_off[j] + k, so the threads
// of neighbouring closures read neighbouring words.
constexpr uint32_t kClosureCluster = 8;                    // blocks of a spread system (portable cluster size)
constexpr uint32_t kClosureFew = 256;                      // up to this many threads: compiled for 255 registers
// Slots or bodies above which a system is spread over the cluster.  Reference
// loop and PCG, one block / eight: 80 five-body loops (320 slots) 471 / 475 and
// 193 / 207 us, 130 loops (520 slots) 333 / 323 and 217 / 222 us, 380 loops
// 590 / 499 us; beyond, a block walks its slots and bodies in several rounds.
constexpr uint32_t kClosureSpread = 512;
constexpr uint32_t kPieceEntries = kLoopPiece * (kLoopPiece + 1) / 2;

// Word offsets of the dynamic shared memory.
struct ClosureLayout {
    uint32_t all_max, clos, frame, slot, fk, angle, link_pos, link_rot, col_off;   // every block
    uint32_t terms, len, sums, col, g, d, qi, pos, off, dir;                       // block 0
    uint32_t diag, res, z, cqs, loop_off, loop_q, l, words;                        // block 0, PCG to a residual
};
__host__ __device__ inline ClosureLayout closure_layout(const MechParams& p, uint32_t blocks, bool pcg) {
    ClosureLayout L{};
    const uint32_t NC = p.closures, S = p.slots, NQ = p.closure_coords;
    const uint32_t per = (NC + blocks - 1) / blocks, bodies = (p.closure_bodies + blocks - 1) / blocks;
    uint32_t w = 0;
    auto take = [&](uint32_t n) { const uint32_t at = w; w += (n + 3u) & ~3u; return at; };
    L.all_max = take(2 * kClosureCluster);
    L.clos = take(15 * per);   // positions of its bodies, local anchors and axes of the closure bearing, its row
    L.frame = take(13 * per);  // its world anchors and axes of the step, and whether it is active
    L.slot = take(8 * per * p.closure_depth);   // parent's position (with side and direction), local axis and anchor
                                                // of the joint, place of its value in the runs
    L.fk = take(14 * bodies);  // axis, anchors and bind rotation of the body's joint, and its direction
    L.angle = take(bodies);    // the joint's angle
    L.link_pos = take(2 * 4 * bodies);   // the links of the forward kinematics, two buffers:
    L.link_rot = take(2 * 4 * bodies);   // {position, parent's position in the list | done}, rotation
    L.col_off = take(p.closure_depth + 1);
    L.terms = take(kBlockChunks * 32 * 33 * 2);   // terms of a dot product, 32-term groups 33 words apart
    L.len = take(NC);          // slots of the closure, and of its branch a
    L.sums = take(6 * NC);     // branch products of the closure
    L.col = take(6 * S);       // the joint's Jacobian column
    L.g = take(S);             // slot values, at their position in the coordinates' runs
    L.d = take(S);
    L.qi = take(S);            // coordinate (position in the list) and closure of the slot
    L.pos = take(S);
    L.off = take(NQ + 1);      // first slot value of each coordinate's run
    L.dir = take(NQ);
    if (pcg) {
        L.diag = take(NQ);
        L.res = take(NQ);
        L.z = take(NQ);
        L.cqs = take(S);
        L.loop_off = take(p.loops + 1);
        L.loop_q = take(NQ);
        L.l = take(kPieceEntries * p.loops);
    }
    L.words = w;
    return L;
}

constexpr uint32_t kSlotSideA = 1u << 30, kSlotReversed = 1u << 31, kSlotParent = kSlotSideA - 1u;
constexpr uint32_t kLinkDone = 1u << 31;   // the link is relative to its root

// The dot products of the one-block solve, in the order of chunk_dot and
// dot_total (FP32) and of block_sum_d and chunk_total_d (FP64): the tree of a
// shuffle-down over 32 consecutive terms, the same tree over a chunk's 32 group
// sums, the chunks in order.  The terms go through shared memory: a thread sums
// a group (its words 33 apart, so no two threads of the warp share a bank) and
// one warp a chunk, which costs a third of the shuffles by every warp.  Terms
// past `nq` stay zero.
template <class T>
__device__ __forceinline__ T block_dot(const T (&part)[kBlockChunks], uint32_t nq, T* terms, T* totals) {
    const uint32_t tid = threadIdx.x, w = warp_id(), lane = lane_id();
#pragma unroll
    for (uint32_t c = 0; c < kBlockChunks; ++c)
        if (c * kDotChunk + tid < nq) terms[c * 32 * 33 + tid + tid / 32] = part[c];
    __syncthreads();
    if (w < kBlockChunks && w * kDotChunk < nq) {
        const T* r = terms + w * 32 * 33 + lane * 33;
        T h[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) h[k] = (r[k] + r[k + 16]) + (r[k + 8] + r[k + 24]);
        T v = ((h[0] + h[4]) + (h[2] + h[6])) + ((h[1] + h[5]) + (h[3] + h[7]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) totals[w] = v;
    }
    __syncthreads();
    T acc = (T)0;
#pragma unroll
    for (uint32_t c = 0; c < kBlockChunks; ++c)
        if (c * kDotChunk < nq) acc += totals[c];
    return acc;
}

// Barrier over the cluster's blocks (release / acquire, global memory included).
__device__ __forceinline__ void cluster_sync(uint32_t blocks) {
    if (blocks == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}
// The address in block `rank`'s shared memory that corresponds to `v` in this block's.
template <class T>
__device__ __forceinline__ T* cluster_map(T* v, uint32_t rank) {
    T* out;
    asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(v), "r"(rank));
    return out;
}

template <bool kPcg, uint32_t kThreads>
__global__ void __launch_bounds__(kThreads) k_closure_block(StepBuffers b, MechBuffers m, MechParams p) {
    extern __shared__ __align__(16) float s_dyn[];
    __shared__ uint32_t s_max[2];
    __shared__ double s_tot[kBlockChunks];
    const uint32_t blocks = gridDim.x, rank = blockIdx.x;   // the grid is one cluster of 2^shift blocks
    const uint32_t shift = 31u - __clz(blocks), rank_mask = blocks - 1u;
    const ClosureLayout L = closure_layout(p, blocks, kPcg);
    const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = lane_id();
    const uint32_t NC = p.closures, S = p.slots, NQ = p.closure_coords, Q = p.coordinate_count;
    const uint32_t per = (NC + blocks - 1) / blocks;                   // closures of a block, [k0, k0 + per)
    const uint32_t k0 = rank * per, mine = k0 < NC ? min(per, NC - k0) : 0u;
    const uint32_t rows = (p.closure_bodies + blocks - 1) / blocks;    // bodies of a block: one per thread
    const uint32_t place = tid * blocks + rank;                        // this thread's body in the list
    const bool has_body = tid < rows && place < p.closure_bodies;
    uint32_t* flags = &b.diag->error_flags;
    uint32_t* all_max = reinterpret_cast<uint32_t*>(s_dyn + L.all_max);
    float* clos = s_dyn + L.clos;
    float* frame = s_dyn + L.frame;
    float* slot = s_dyn + L.slot;
    float* fk = s_dyn + L.fk;
    float* angle_s = s_dyn + L.angle;
    float4* link_pos = reinterpret_cast<float4*>(s_dyn + L.link_pos);
    float4* link_rot = reinterpret_cast<float4*>(s_dyn + L.link_rot);
    uint32_t* col_off = reinterpret_cast<uint32_t*>(s_dyn + L.col_off);
    uint32_t* len = reinterpret_cast<uint32_t*>(s_dyn + L.len);
    float* sums = s_dyn + L.sums;
    float* col = s_dyn + L.col;
    float* sg = s_dyn + L.g;
    float* sd = s_dyn + L.d;
    uint32_t* qi = reinterpret_cast<uint32_t*>(s_dyn + L.qi);
    uint32_t* pos = reinterpret_cast<uint32_t*>(s_dyn + L.pos);
    uint32_t* off = reinterpret_cast<uint32_t*>(s_dyn + L.off);
    float* dir_s = s_dyn + L.dir;
    auto at3 = [](const float* base, uint32_t i, uint32_t stride, uint32_t k) {
        return mkf3(base[i * stride + k], base[(i + 1) * stride + k], base[(i + 2) * stride + k]);
    };
    auto put3 = [](float* base, uint32_t i, uint32_t stride, uint32_t k, f3 v) {
        base[i * stride + k] = v.x;
        base[(i + 1) * stride + k] = v.y;
        base[(i + 2) * stride + k] = v.z;
    };
    // the link of the body at `at` in the list (in the memory of the block that owns it)
    auto load_link = [&](uint32_t buffer, uint32_t at, float4& lp, float4& lr) {
        const uint32_t i = buffer * rows + (at >> shift), owner = at & rank_mask;
        lp = *cluster_map(link_pos + i, owner);
        lr = *cluster_map(link_rot + i, owner);
    };
    const uint32_t final_buffer = p.final_is_a ? 0u : 1u;
    // ---- the system's constant rows: this block's closures, joints and bodies
    const uint32_t tasks = p.closure_depth * per;   // (place j, closure) of this block's slots
    for (uint32_t j = tid; j <= p.closure_depth; j += nt) col_off[j] = m.cl_columns[j];
    for (uint32_t i = tid; i < mine; i += nt) {
        const uint32_t k = m.cl_order[k0 + i];
        const GpuBearing br = m.bearings[m.cl_bearings[k]];
        clos[i] = __uint_as_float(m.cl_places[2 * k]);
        clos[per + i] = __uint_as_float(m.cl_places[2 * k + 1]);
        put3(clos, 2, per, i, r3(br.local_anchor_a));
        put3(clos, 5, per, i, r3(br.local_anchor_b));
        put3(clos, 8, per, i, r3(br.local_axis_a));
        put3(clos, 11, per, i, r3(br.local_axis_b));
    }
    for (uint32_t t = tid; t < tasks; t += nt) {
        const uint32_t j = t / per, i = t - j * per;
        if (i >= mine || k0 + i >= m.cl_columns[j + 1] - m.cl_columns[j]) continue;
        const uint32_t k = m.cl_order[k0 + i], sl = m.cl_slot_off[k] + j;
        const GpuMechanismBody* mb = m.bodies + m.slot_body[sl];
        const GpuBearing& tb = m.bearings[mb->metadata[1]];
        const bool reversed = mb->metadata[2] != 0u;
        slot[t] = __uint_as_float(m.slot_parent[sl] | (sl < m.cl_split[k] ? kSlotSideA : 0u) |
                                  (reversed ? kSlotReversed : 0u));
        put3(slot, 1, tasks, t, reversed ? r3(tb.local_axis_b) : r3(tb.local_axis_a));
        put3(slot, 4, tasks, t, reversed ? r3(tb.local_anchor_b) : r3(tb.local_anchor_a));
        slot[7 * tasks + t] = __uint_as_float(m.slot_pos[sl]);
    }
    bool root = false;
    uint32_t body = 0, parent = 0;
    if (has_body) {   // prepare_link's constant part, and the links as they stand
        body = m.cb_bodies[place];
        parent = m.cb_parents[place];
        const GpuMechanismBody mb = m.bodies[body];
        root = mb.metadata[3] != 0u;
        if (!root) {
            const GpuBearing& br = m.bearings[mb.metadata[1]];
            const bool reversed = mb.metadata[2] != 0u;
            put3(fk, 0, rows, tid, normalize(reversed ? r3(br.local_axis_b) : r3(br.local_axis_a)));
            put3(fk, 3, rows, tid, reversed ? r3(br.local_anchor_b) : r3(br.local_anchor_a));
            put3(fk, 6, rows, tid, reversed ? r3(br.local_anchor_a) : r3(br.local_anchor_b));
            const float4 bind = r4(mb.bind_relative_rotation);
            put3(fk, 9, rows, tid, xyz(bind));
            fk[12 * rows + tid] = bind.w;
            fk[13 * rows + tid] = reversed ? -1.0f : 1.0f;
            // the reference's loop adds 0 to the coordinates off the closure branches
            const float angle = m.coords[br.metadata[2]].angle;
            angle_s[tid] = kPcg ? angle : angle + 0.0f;
        }
        const Link l = ld_link(m.links_final, body);
        link_pos[final_buffer * rows + tid] = l.pos;
        link_rot[final_buffer * rows + tid] = l.rot;
    }
    uint32_t coord[kBlockChunks], child[kBlockChunks];   // this thread's coordinates and their joints' bodies
    float angle[kBlockChunks];
#pragma unroll
    for (uint32_t c = 0; c < kBlockChunks; ++c) {
        coord[c] = child[c] = 0u;
        angle[c] = 0.0f;
    }
    if (rank == 0) {
        for (uint32_t q = tid; q <= NQ; q += nt) off[q] = m.cq_off[q];
        for (uint32_t i = tid; i < kBlockChunks * 32 * 33 * 2; i += nt) s_dyn[L.terms + i] = 0.0f;
        for (uint32_t k = tid; k < NC; k += nt) {
            const uint32_t c = m.cl_order[k], s0 = m.cl_slot_off[c], n = m.cl_slot_off[c + 1] - s0;
            len[k] = n | ((m.cl_split[c] - s0) << 16);
        }
        if (kPcg) {
            for (uint32_t i = tid; i <= p.loops; i += nt)
                reinterpret_cast<uint32_t*>(s_dyn + L.loop_off)[i] = m.loop_off[i];
            for (uint32_t i = tid; i < NQ; i += nt) reinterpret_cast<uint32_t*>(s_dyn + L.loop_q)[i] = m.loop_q[i];
        }
#pragma unroll
        for (uint32_t c = 0; c < kBlockChunks; ++c) {
            const uint32_t q = c * kDotChunk + tid;
            if (q >= NQ) continue;
            coord[c] = m.cq_coords[q];
            child[c] = m.cq_child[q];
            angle[c] = m.coords[coord[c]].angle;
        }
        for (uint32_t at = tid; at < S; at += nt) {
            qi[at] = m.col_coord[at];
            pos[at] = m.col_pos[at];
            if (kPcg) reinterpret_cast<uint32_t*>(s_dyn + L.cqs)[pos[at]] = at;
        }
    }
    if (tid == 0) s_max[0] = s_max[1] = 0u;
    cluster_sync(blocks);   // every block's shared memory is up before another reads or writes it
    float* col0 = cluster_map(col, 0u);
    float* sg0 = cluster_map(sg, 0u);
    float* sd0 = cluster_map(sd, 0u);

    // sg[slot position] = the slot's share of J^T J dir (closure_products): the branch
    // products, a closure's position or axis rows per thread, then a slot per thread
    auto products = [&]() {
        for (uint32_t t = tid; t < 2u * NC; t += nt) {
            const uint32_t half = t >= NC ? 3u : 0u, k = t >= NC ? t - NC : t;
            const uint32_t n = len[k] & 0xffffu, split = len[k] >> 16;
            f3 sum_a = mkf3(0, 0, 0), sum_b = mkf3(0, 0, 0);
#pragma unroll 4
            for (uint32_t j = 0; j < n; ++j) {
                const uint32_t at = col_off[j] + k;
                const f3 term = at3(col, half, S, at) * dir_s[qi[at] & 0xffffu];
                if (j < split) sum_a = sum_a + term;
                else sum_b = sum_b + term;
            }
            put3(sums, half, NC, k, sum_a + sum_b);
        }
        __syncthreads();
        for (uint32_t at = tid; at < S; at += nt) {
            const uint32_t k = qi[at] >> 16;
            sg[pos[at]] = dot(at3(col, 0, S, at), at3(sums, 0, NC, k)) + 1.0f * dot(at3(col, 3, S, at), at3(sums, 3, NC, k));
        }
    };
    auto run_sum = [&](uint32_t q) {
        float o = 0.0f;
        for (uint32_t i = off[q]; i < off[q + 1]; ++i) o += sg[i];
        return o;
    };
    // a dot product of the reference's loop: serial up to kSerialDot coordinates
    auto dot_f = [&](const float (&x)[kBlockChunks], const float (&y)[kBlockChunks]) -> float {
        if (NQ <= kSerialDot) {
            float* prod = s_dyn + L.terms;
            if (tid < NQ) prod[tid] = x[0] * y[0];
            __syncthreads();
            if (tid == 0) {
                float acc = 0.0f;
                const uint32_t whole = NQ & ~3u;
#pragma unroll 8
                for (uint32_t q = 0; q < whole; q += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(prod + q);
                    acc = (((acc + v.x) + v.y) + v.z) + v.w;
                }
                for (uint32_t q = whole; q < NQ; ++q) acc += prod[q];
                reinterpret_cast<float*>(s_tot)[0] = acc;
            }
            __syncthreads();
            return reinterpret_cast<float*>(s_tot)[0];
        }
        float part[kBlockChunks];
#pragma unroll
        for (uint32_t c = 0; c < kBlockChunks; ++c) part[c] = c * kDotChunk + tid < NQ ? x[c] * y[c] : 0.0f;
        return block_dot<float>(part, NQ, s_dyn + L.terms, reinterpret_cast<float*>(s_tot));
    };
    auto dot_d = [&](const float (&x)[kBlockChunks], const float (&y)[kBlockChunks]) -> double {
        double part[kBlockChunks];
#pragma unroll
        for (uint32_t c = 0; c < kBlockChunks; ++c)
            part[c] = c * kDotChunk + tid < NQ ? (double)x[c] * (double)y[c] : 0.0;
        return block_dot<double>(part, NQ, reinterpret_cast<double*>(s_dyn + L.terms), s_tot);
    };
    uint32_t steps = 0, rounds = 0, done = 0, newton = 0, iterations = 0;
    double worst = 0.0;
    for (uint32_t step = 0; step < kClosureSteps; ++step) {
        // ---- evaluate_closures (closure.wgsl:268-319): frames and residuals
        uint32_t um = 0u, ud = 0u;
        for (uint32_t i = tid; i < mine; i += nt) {
            float4 pa, ra4, pb, rb4;
            load_link(final_buffer, __float_as_uint(clos[i]), pa, ra4);
            load_link(final_buffer, __float_as_uint(clos[per + i]), pb, rb4);
            const f3 aa = xyz(pa) + quat_rotate(ra4, at3(clos, 2, per, i));
            const f3 ab = xyz(pb) + quat_rotate(rb4, at3(clos, 5, per, i));
            const f3 xa = normalize(quat_rotate(ra4, at3(clos, 8, per, i)));
            const f3 xb = normalize(quat_rotate(rb4, at3(clos, 11, per, i)));
            const f3 rp = aa - ab, ra = xa - xb;
            bool active = false;
            if (!finite3(rp) || !finite3(ra)) {
                atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
                um = ud = 0xffffffffu;
            } else {
                const uint32_t u = round_u32(length(rp) * 1000000.0f);
                const float deg = atan2_cr(length(cross(xa, xb)), clampf(dot(xa, xb), -1.0f, 1.0f)) * 57.295779513f;
                const uint32_t v = round_u32(deg * 1000000.0f);
                active = !(u <= 10u && v <= 1000u);
                um = max(um, u);
                ud = max(ud, v);
            }
            put3(frame, 0, per, i, aa);
            put3(frame, 3, per, i, ab);
            put3(frame, 6, per, i, xa);
            put3(frame, 9, per, i, xb);
            frame[12 * per + i] = active ? 1.0f : 0.0f;
        }
        um = __reduce_max_sync(0xffffffffu, um);
        ud = __reduce_max_sync(0xffffffffu, ud);
        if (lane == 0 && um) atomicMax(&s_max[0], um);
        if (lane == 0 && ud) atomicMax(&s_max[1], ud);
        __syncthreads();
        if (tid < blocks) {   // this block's maxima to every block
            uint32_t* to = cluster_map(all_max, tid);
            to[2 * rank] = s_max[0];
            to[2 * rank + 1] = s_max[1];
        }
        // ---- the joints' columns and their gradient and diagonal contributions
        for (uint32_t t = tid; t < tasks; t += nt) {
            const uint32_t j = t / per, i = t - j * per;
            const uint32_t at = col_off[j] + k0 + i;
            if (i >= mine || at >= col_off[j + 1]) continue;
            const uint32_t word = __float_as_uint(slot[t]);
            const bool side_a = word & kSlotSideA;
            float4 lpos, lrot;
            load_link(final_buffer, word & kSlotParent, lpos, lrot);
            const uint32_t where = __float_as_uint(slot[7 * tasks + t]);
            f3 axis = normalize(quat_rotate(lrot, at3(slot, 1, tasks, t)));
            if (word & kSlotReversed) axis = -axis;
            const f3 anchor = xyz(lpos) + quat_rotate(lrot, at3(slot, 4, tasks, t));
            const f3 aa = at3(frame, 0, per, i), ab = at3(frame, 3, per, i);
            const f3 xa = at3(frame, 6, per, i), xb = at3(frame, 9, per, i);
            const f3 rp = aa - ab, ra = xa - xb;
            const f3 ea = side_a ? aa : ab, ex = side_a ? xa : xb;
            const float sign = side_a ? 1.0f : -1.0f;
            const f3 pd = cross(axis, ea - anchor) * sign;
            const f3 ad = cross(axis, ex) * sign;
            put3(col0, 0, S, at, pd);
            put3(col0, 3, S, at, ad);
            float g = __int_as_float(0x7fffffff), d = 0.0f;   // NaN: no contribution
            if (frame[12 * per + i] != 0.0f) {
                const float gg = dot(rp, pd) + 1.0f * dot(ra, ad), dd = dot(pd, pd) + 1.0f * dot(ad, ad);
                if (gg == gg && dd == dd) {
                    g = gg;
                    d = dd;
                } else {
                    atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
                }
            }
            sg0[where] = g;
            sd0[where] = d;
        }
        cluster_sync(blocks);
        um = ud = 0u;
        for (uint32_t r = 0; r < blocks; ++r) {
            um = max(um, all_max[2 * r]);
            ud = max(ud, all_max[2 * r + 1]);
        }
        if (tid == 0) s_max[0] = s_max[1] = 0u;
        if (!(um > 10u || ud > 1000u)) {   // every block takes the same branch
            done = 1;
            break;
        }
        ++steps;
        if (rank == 0) {
        // ---- per coordinate: gradient and diagonal in the serial accumulation order
        float grad[kBlockChunks], diag[kBlockChunks];
#pragma unroll
        for (uint32_t c = 0; c < kBlockChunks; ++c) {
            const uint32_t q = c * kDotChunk + tid;
            float g = 0.0f, d = 0.0f;
            if (q < NQ)
                for (uint32_t i = off[q]; i < off[q + 1]; ++i) {
                    const float v = sg[i];
                    if (v == v) { g += v; d += sd[i]; }
                }
            grad[c] = g;
            diag[c] = d;
        }
        float sol[kBlockChunks], res[kBlockChunks], dir[kBlockChunks], pre[kBlockChunks], op[kBlockChunks];
        if constexpr (!kPcg) {   // solve_closure_pcg (closure.wgsl:333-427)
#pragma unroll
            for (uint32_t c = 0; c < kBlockChunks; ++c) {
                const uint32_t q = c * kDotChunk + tid;
                sol[c] = 0.0f;
                res[c] = pre[c] = 0.0f;
                if (diag[c] > 1.0e-12f) {
                    res[c] = -grad[c];
                    pre[c] = res[c] / diag[c];
                }
                dir[c] = pre[c];
                if (q < NQ) dir_s[q] = dir[c];
            }
            float rz = dot_f(res, pre);
            if (NQ == 0) __syncthreads();
            for (uint32_t round = 0; round < kClosureRounds; ++round) {
                products();   // dir_s was published by the barrier of the dot product or the round before
                __syncthreads();
#pragma unroll
                for (uint32_t c = 0; c < kBlockChunks; ++c) {
                    const uint32_t q = c * kDotChunk + tid;
                    op[c] = q < NQ ? run_sum(q) : 0.0f;
                }
                const float dop = dot_f(dir, op);
                const float alpha = fabsf(dop) > 1.0e-20f ? rz / dop : 0.0f;
#pragma unroll
                for (uint32_t c = 0; c < kBlockChunks; ++c) {
                    sol[c] += alpha * dir[c];
                    res[c] -= alpha * op[c];
                    pre[c] = 0.0f;
                    if (diag[c] > 1.0e-12f) pre[c] = res[c] / diag[c];
                }
                const float nrz = dot_f(res, pre);
                const float beta = fabsf(rz) > 1.0e-20f ? nrz / rz : 0.0f;
#pragma unroll
                for (uint32_t c = 0; c < kBlockChunks; ++c) {
                    const uint32_t q = c * kDotChunk + tid;
                    dir[c] = pre[c] + beta * dir[c];
                    if (q < NQ) dir_s[q] = dir[c];
                }
                rz = nrz;
                ++rounds;
                __syncthreads();
            }
        } else {   // PCG to a residual
            float* diag_s = s_dyn + L.diag;
            float* res_s = s_dyn + L.res;
            float* z_s = s_dyn + L.z;
            const uint32_t* cqs = reinterpret_cast<const uint32_t*>(s_dyn + L.cqs);
            const uint32_t* loop_off = reinterpret_cast<const uint32_t*>(s_dyn + L.loop_off);
            const uint32_t* loop_q = reinterpret_cast<const uint32_t*>(s_dyn + L.loop_q);
            float* lf = s_dyn + L.l;   // packed lower triangles, entry-major
            const uint32_t loops = p.loops;
            const bool loop_blocks = p.precond == MK_PRECOND_BLOCK_JACOBI;
#pragma unroll
            for (uint32_t c = 0; c < kBlockChunks; ++c) {
                const uint32_t q = c * kDotChunk + tid;
                sol[c] = 0.0f;
                res[c] = -grad[c];
                if (q < NQ) {
                    diag_s[q] = diag[c];
                    res_s[q] = res[c];
                }
            }
            if (loop_blocks) {   // couplings of each loop's coordinates (closure_coupling), one entry per thread
                constexpr uint32_t kOff = kLoopPiece * (kLoopPiece - 1) / 2;
                for (uint32_t e = tid; e < loops * kOff; e += nt) {
                    const uint32_t lp = e / kOff;
                    uint32_t j = e % kOff, i = 1;
                    while (j >= i) { j -= i; ++i; }   // (i, j): row i > column j
                    const uint32_t o = loop_off[lp], n = loop_off[lp + 1] - o;
                    if (i >= n) continue;
                    const uint32_t a = loop_q[o + i], c = loop_q[o + j];
                    float r = 0.0f;
                    for (uint32_t x = off[a]; x < off[a + 1]; ++x) {
                        const uint32_t sa = cqs[x];
                        const uint32_t ka = qi[sa] >> 16;
                        for (uint32_t y = off[c]; y < off[c + 1]; ++y) {
                            const uint32_t sb = cqs[y];
                            if (ka != qi[sb] >> 16) continue;
                            r += dot(at3(col, 0, S, sa), at3(col, 0, S, sb)) +
                                 1.0f * dot(at3(col, 3, S, sa), at3(col, 3, S, sb));
                        }
                    }
                    lf[(i * (i + 1) / 2 + j) * loops + lp] = r;
                }
            }
            __syncthreads();
            if (loop_blocks && tid < loops) {   // Cholesky with a ridge; a failed pivot leaves the block diagonal
                const uint32_t o = loop_off[tid], n = loop_off[tid + 1] - o;
                float a[kPieceEntries], dg[kLoopPiece];
                float mean = 0.0f;
#pragma unroll
                for (uint32_t i = 0; i < kLoopPiece; ++i) {
                    dg[i] = i < n ? diag_s[loop_q[o + i]] : 0.0f;
                    if (i < n) mean += dg[i];
                }
                mean = n ? mean / (float)n : 0.0f;
#pragma unroll
                for (uint32_t i = 0; i < kLoopPiece; ++i)
#pragma unroll
                    for (uint32_t j = 0; j <= i; ++j) {
                        const uint32_t e = i * (i + 1) / 2 + j;
                        a[e] = i >= n ? 0.0f : i == j ? dg[i] + 1.0e-6f * mean : lf[e * loops + tid];
                    }
                bool ok = mean > 1.0e-12f;
#pragma unroll
                for (uint32_t j = 0; j < kLoopPiece; ++j) {
                    if (j < n && ok) {
                        float dj = a[j * (j + 1) / 2 + j];
#pragma unroll
                        for (uint32_t k = 0; k < j; ++k) dj -= a[j * (j + 1) / 2 + k] * a[j * (j + 1) / 2 + k];
                        if (!(dj > 0.0f)) {
                            ok = false;
                        } else {
                            const float ljj = sqrtf(dj);
                            a[j * (j + 1) / 2 + j] = ljj;
#pragma unroll
                            for (uint32_t i = j + 1; i < kLoopPiece; ++i) {
                                if (i < n) {
                                    float v = a[i * (i + 1) / 2 + j];
#pragma unroll
                                    for (uint32_t k = 0; k < j; ++k)
                                        v -= a[i * (i + 1) / 2 + k] * a[j * (j + 1) / 2 + k];
                                    a[i * (i + 1) / 2 + j] = v / ljj;
                                }
                            }
                        }
                    }
                }
#pragma unroll
                for (uint32_t i = 0; i < kLoopPiece; ++i)
#pragma unroll
                    for (uint32_t j = 0; j <= i; ++j) {
                        const uint32_t e = i * (i + 1) / 2 + j;
                        float v = a[e];
                        if (!ok) v = i == j ? (dg[i] > 1.0e-12f ? sqrtf(dg[i]) : 0.0f) : 0.0f;
                        if (i < n) lf[e * loops + tid] = v;   // read by this thread only
                    }
            }
            // pre = M^-1 res (precond_apply); res_s is published, z_s free
            auto precondition = [&]() {
                if (!loop_blocks) {
#pragma unroll
                    for (uint32_t c = 0; c < kBlockChunks; ++c) pre[c] = diag[c] > 1.0e-12f ? res[c] / diag[c] : 0.0f;
                    return;
                }
                if (tid < loops) {
                    const uint32_t o = loop_off[tid], n = loop_off[tid + 1] - o;
                    float y[kLoopPiece];
#pragma unroll
                    for (uint32_t i = 0; i < kLoopPiece; ++i) {
                        y[i] = 0.0f;
                        if (i < n) {
                            float v = res_s[loop_q[o + i]];
#pragma unroll
                            for (uint32_t k = 0; k < i; ++k) v -= lf[(i * (i + 1) / 2 + k) * loops + tid] * y[k];
                            const float lii = lf[(i * (i + 1) / 2 + i) * loops + tid];
                            y[i] = lii > 0.0f ? v / lii : 0.0f;
                        }
                    }
#pragma unroll
                    for (uint32_t x = kLoopPiece; x > 0; --x) {
                        const uint32_t i = x - 1;
                        if (i < n) {
                            float v = y[i];
#pragma unroll
                            for (uint32_t k = i + 1; k < kLoopPiece; ++k)
                                if (k < n) v -= lf[(k * (k + 1) / 2 + i) * loops + tid] * y[k];
                            const float lii = lf[(i * (i + 1) / 2 + i) * loops + tid];
                            y[i] = lii > 0.0f ? v / lii : 0.0f;
                        }
                    }
#pragma unroll
                    for (uint32_t i = 0; i < kLoopPiece; ++i)
                        if (i < n) z_s[loop_q[o + i]] = y[i];
                }
                __syncthreads();
#pragma unroll
                for (uint32_t c = 0; c < kBlockChunks; ++c) {
                    const uint32_t q = c * kDotChunk + tid;
                    pre[c] = q < NQ ? z_s[q] : 0.0f;
                }
            };
            precondition();
#pragma unroll
            for (uint32_t c = 0; c < kBlockChunks; ++c) {
                const uint32_t q = c * kDotChunk + tid;
                dir[c] = pre[c];
                if (q < NQ) dir_s[q] = dir[c];
            }
            double rz = dot_d(res, pre);
            const double rr0 = dot_d(res, res);
            double rr = rr0;
            const double tol2 = (double)p.closure_tol * (double)p.closure_tol;
            uint32_t it = 0;
            while (it < p.closure_max_it && rr > tol2 * rr0) {
                products();
                __syncthreads();
#pragma unroll
                for (uint32_t c = 0; c < kBlockChunks; ++c) {
                    const uint32_t q = c * kDotChunk + tid;
                    op[c] = q < NQ ? run_sum(q) : 0.0f;
                }
                const double pq = dot_d(dir, op);
                const float alpha = fabs(pq) > 1.0e-30 ? (float)(rz / pq) : 0.0f;
#pragma unroll
                for (uint32_t c = 0; c < kBlockChunks; ++c) {
                    const uint32_t q = c * kDotChunk + tid;
                    sol[c] += alpha * dir[c];
                    res[c] -= alpha * op[c];
                    if (q < NQ) res_s[q] = res[c];
                }
                rr = dot_d(res, res);
                ++it;
                if (rr <= tol2 * rr0) break;
                precondition();
                const double nrz = dot_d(res, pre);
                const float beta = fabs(rz) > 1.0e-300 ? (float)(nrz / rz) : 0.0f;
#pragma unroll
                for (uint32_t c = 0; c < kBlockChunks; ++c) {
                    const uint32_t q = c * kDotChunk + tid;
                    dir[c] = pre[c] + beta * dir[c];
                    if (q < NQ) dir_s[q] = dir[c];
                }
                rz = nrz;
                __syncthreads();
            }
            ++newton;
            iterations += it;
            const double rel = rr0 > 0.0 ? sqrt(rr / rr0) : 0.0;
            if (rel > worst) worst = rel;
        }
        // ---- step the coordinates (closure.wgsl:416-427), to their joints' bodies
#pragma unroll
        for (uint32_t c = 0; c < kBlockChunks; ++c) {
            if (c * kDotChunk + tid >= NQ) continue;
            const float stp = clampf(0.35f * sol[c], -0.2f, 0.2f);
            if (stp == stp) angle[c] += stp;
            else atomicOr(flags, MK_INVALID_NUMERIC_FLAG);
            *cluster_map(angle_s + (child[c] >> shift), child[c] & rank_mask) = angle[c];
        }
        }
        cluster_sync(blocks);
        // ---- forward kinematics of the closure components (prepare_link, jump_link), a body per thread
        float4 lp = make_float4(0, 0, 0, 0), lr = make_float4(0, 0, 0, 1);
        uint32_t up = parent | (root ? kLinkDone : 0u);
        if (has_body) {
            if (!root) {
                const float h = (fk[13 * rows + tid] * angle_s[tid]) * 0.5f;
                const f3 v = at3(fk, 0, rows, tid) * sin_cr(h);
                const float4 bind = f4(at3(fk, 9, rows, tid), fk[12 * rows + tid]);
                lr = quat_multiply(make_float4(v.x, v.y, v.z, cos_cr(h)), bind);
                lp = f4(at3(fk, 3, rows, tid) - quat_rotate(lr, at3(fk, 6, rows, tid)), 0.0f);
            }
            link_pos[tid] = f4(xyz(lp), __uint_as_float(up));
            link_rot[tid] = lr;
        }
        cluster_sync(blocks);
        uint32_t src = 0;
        for (uint32_t r = 0; r < p.jump_rounds; ++r) {
            if (has_body) {
                if (!(up & kLinkDone)) {
                    float4 up_pos, up_rot;
                    load_link(src, up, up_pos, up_rot);
                    lp = f4(xyz(up_pos) + quat_rotate(up_rot, xyz(lp)), 0.0f);
                    lr = normalize4(quat_multiply(up_rot, lr));
                    up = __float_as_uint(up_pos.w);
                }
                link_pos[(src ^ 1u) * rows + tid] = f4(xyz(lp), __uint_as_float(up));
                link_rot[(src ^ 1u) * rows + tid] = lr;
            }
            cluster_sync(blocks);
            src ^= 1u;
        }
    }
    // ---- results: the links, the coordinates and the columns of the last evaluated step
    if (steps && has_body) {
        const float4 lp = link_pos[final_buffer * rows + tid], lr = link_rot[final_buffer * rows + tid];
        const uint32_t up = __float_as_uint(lp.w);
        st_link(m.links_final, body,
                {f4(xyz(lp), 0.0f), lr, make_uint4(m.cb_bodies[up & ~kLinkDone], up >> 31, 0u, 0u)});
    }
    if (rank == 0) {
        if (!kPcg && steps) {
            for (uint32_t c = tid; c < Q; c += nt) m.coords[c].angle += 0.0f;   // those off the closure branches
            __syncthreads();
        }
#pragma unroll
        for (uint32_t c = 0; c < kBlockChunks; ++c)
            if (steps && c * kDotChunk + tid < NQ) m.coords[coord[c]].angle = angle[c];
        for (uint32_t at = tid; at < S; at += nt) {
            const uint32_t k = qi[at] >> 16, row = m.cl_order[k];
            const uint32_t sl = m.cq_slots[pos[at]];
            m.slot_v[2 * sl] = f4(at3(col, 0, S, at), __uint_as_float(m.cq_coords[qi[at] & 0xffffu]));
            m.slot_v[2 * sl + 1] = f4(at3(col, 3, S, at), kPcg ? __uint_as_float(row) : 0.0f);
        }
    }
    cluster_sync(blocks);   // no block leaves while another may still read its links
    if (rank == 0 && tid == 0) {
        if constexpr (kPcg) {
            *m.cstate = ClosureState{done, done ? 0u : p.blocks, newton, iterations, 0u, 0u, worst};
        } else {
            atomicAdd(&b.diag->reserved_b, steps);
            atomicAdd(&b.diag->reserved_c, rounds);
        }
    }
}

// --------------------------------------------------------------- launches
static inline uint32_t nblocks(uint32_t n) { return (n + kMBlock - 1) / kMBlock; }

// The pose-only parts of the bearing rows, before a set of projection passes.
static cudaError_t bearing_cache(MechBuffers& m, const StepBuffers& b, const MechParams& p, cudaStream_t s) {
    if (p.bearing_count) k_bearing_cache<<<nblocks(p.bearing_count), kMBlock, 0, s>>>(b, m, p);
    return cudaGetLastError();
}

// The two velocity buffer pairs that the passes alternate between: the live
// velocities and the first iteration pair of the cooperative solve (not used
// while bearings are projected).
static void velocity_buffers(const StepBuffers& b, const MechParams& p, float4* lin[2], float4* ang[2]) {
    lin[0] = b.lin;
    ang[0] = b.ang;
    lin[1] = b.vel_iter;
    ang[1] = b.vel_iter + p.body_count;
}
static uint32_t side_blocks(const MechParams& p) { return p.padded_sides / kPassBlock; }
static uint32_t rest_blocks(const MechParams& p) {
    return (p.body_count - p.bearing_bodies + kPassBlock - 1) / kPassBlock;
}

// `iterations` projection passes over the live velocities (bodies without
// bearings get their apply of zeros with the first one; it changes nothing after that).
static cudaError_t bearing_projections(MechBuffers& m, const StepBuffers& b, const MechParams& p, cudaStream_t s) {
    float4 *lin[2], *ang[2];
    velocity_buffers(b, p, lin, ang);
    const uint32_t sides = side_blocks(p), hubs = p.hub_chunks, passes = std::max(1u, p.iterations);
    for (uint32_t it = 0; it < passes; ++it) {
        const uint32_t from = it & 1u, to = from ^ 1u;
        const uint32_t rest = it == 0 ? rest_blocks(p) : 0u;
        if (sides + hubs + rest == 0) continue;
        const VelocityPass f{lin[from], ang[from], lin[to], ang[to], lin[from], ang[from], nullptr, nullptr};
        auto* kernel = hubs ? k_bearing_pass<false, true> : k_bearing_pass<false, false>;
        kernel<<<sides + hubs + rest, kPassBlock, 0, s>>>(b, m, p, f, sides, hubs);
    }
    if ((passes & 1u) && p.bearing_bodies)
        k_pass_back<<<nblocks(p.bearing_bodies), kMBlock, 0, s>>>(m, p.bearing_bodies,
                                                                  VelocityPass{lin[1], ang[1], lin[0], ang[0]});
    return cudaGetLastError();
}

static cudaError_t forward_kinematics(MechBuffers& m, const MechParams& p, cudaStream_t s) {
    k_prepare_links<<<nblocks(p.body_count), kMBlock, 0, s>>>(m, p);
    bool a_src = true;
    for (uint32_t r = 0; r < p.jump_rounds; ++r) {
        k_jump<<<nblocks(p.body_count), kMBlock, 0, s>>>(a_src ? m.links_a : m.links_b, a_src ? m.links_b : m.links_a,
                                                         p);
        a_src = !a_src;
    }
    return cudaGetLastError();
}

static cudaError_t reconstruct(MechBuffers& m, const StepBuffers& b, const MechParams& p, cudaStream_t s) {
    if (p.walk_levels) {
        const uint32_t count = m.level_offsets[m.level_count];
        k_reconstruct_rows<<<nblocks(count), kMBlock, 0, s>>>(b, m, count);
        k_reconstruct_walk<<<1, kWalkThreads, kWalkSmem, s>>>(b, m, m.level_count, count);
        k_reconstruct_store<<<nblocks(count), kMBlock, 0, s>>>(b, m, count);
        return cudaGetLastError();
    }
    for (uint32_t l = 1; l < m.level_count; ++l) {
        const uint32_t begin = m.level_offsets[l], end = m.level_offsets[l + 1];
        if (end > begin) k_reconstruct_level<<<nblocks(end - begin), kMBlock, 0, s>>>(b, m, begin, end);
    }
    return cudaGetLastError();
}

// Closure solves (the reference's loop and the PCG to a residual), all with the
// same values: a system that fits takes k_closure_block (closure_block_shape);
// of the others, those below kGridClosures closures take one block of the
// kernels that keep their vectors in global memory, the rest the whole grid.
// The tuning forces one block (1) or the grid (2) of the latter.  Mechanism
// stage on one B200, reference loop and PCG, k_closure_block / one block / grid:
// 300 loops of five bodies 540 / 1,155 / 1,756 and 332 / 818 / 1,019 us; loops
// of three bodies, 512 476 / 754 / 1,532 and 307 / 555 / 844, 700 559 / 1,102 /
// 1,463 and 354 / 723 / 852, 1,000 629 / 1,262 / 1,622 (PCG does not fit); one
// loop of 200 bodies 983 / 3,040 / 6,952.
constexpr uint32_t kGridClosures = 512;
static uint32_t g_closure_grid = 0;
void set_closure_grid(uint32_t mode) { g_closure_grid = mode <= 2u ? mode : 0u; }
uint32_t closure_grid_mode() { return g_closure_grid; }

// Launch shape of the one-block closure solve (blocks of its cluster, threads,
// dynamic shared memory); false where the system does not fit it.  A thread per
// coordinate (two above 1,024), per closure body of a block and per closure of
// a block; the run positions and closures of the slots are 16-bit.  A cluster
// where a block would walk its slots or bodies in several rounds.
struct ClosureShape {
    uint32_t blocks, threads, bytes;
};
static bool closure_block_shape(const MechParams& p, ClosureShape& sh) {
    const bool pcg = pcg_residual_mode(p);
    if (!p.block_solve) return false;
    if ((uint64_t)p.closure_depth * p.closures > 64u * kClosureSmem) return false;   // 32-bit word offsets
    if (pcg && p.precond != MK_PRECOND_BLOCK_JACOBI && p.precond != MK_PRECOND_DIAGONAL) return false;
    sh.blocks = std::max(p.slots, p.closure_bodies) > kClosureSpread ? kClosureCluster : 1u;
    const uint32_t rows = (p.closure_bodies + sh.blocks - 1) / sh.blocks;
    if (rows > kClosureThreads) return false;
    const uint32_t want = std::max({rows, std::min(p.closure_coords, kClosureThreads), 128u});
    sh.threads = p.closure_coords > kDotChunk ? kClosureThreads : std::min(kClosureThreads, (want + 31u) & ~31u);
    sh.bytes = 4u * closure_layout(p, sh.blocks, pcg).words;
    return sh.bytes <= kClosureSmem;
}

// Dynamic shared memory of the one-block closure solves, set once per device
// (outside stream capture: at handle creation).
cudaError_t mechanism_prepare() {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load() & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(k_reconstruct_walk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWalkSmem);
    for (const void* k : {(const void*)k_closure_block<false, kClosureFew>, (const void*)k_closure_block<true, kClosureFew>,
                          (const void*)k_closure_block<false, kClosureThreads>,
                          (const void*)k_closure_block<true, kClosureThreads>})
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClosureSmem);
    if (e == cudaSuccess) done.fetch_or(bit);
    return e;
}

static cudaError_t launch_closure_block(const MechBuffers& m, const StepBuffers& b, const MechParams& p,
                                        const ClosureShape& sh, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sh.blocks);
    cfg.blockDim = dim3(sh.threads);
    cfg.dynamicSmemBytes = sh.bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = sh.blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (sh.threads <= kClosureFew)
        return pcg_residual_mode(p) ? cudaLaunchKernelEx(&cfg, k_closure_block<true, kClosureFew>, b, m, p)
                                    : cudaLaunchKernelEx(&cfg, k_closure_block<false, kClosureFew>, b, m, p);
    return pcg_residual_mode(p) ? cudaLaunchKernelEx(&cfg, k_closure_block<true, kClosureThreads>, b, m, p)
                                : cudaLaunchKernelEx(&cfg, k_closure_block<false, kClosureThreads>, b, m, p);
}

// One co-resident 1,024-thread block per SM for the grid-wide closure kernels
// (cooperative launch: they sync with grid barriers).  `step` is passed when
// the kernel takes one (kNoStep: it does not).
constexpr uint32_t kNoStep = 0xffffffffu;
static cudaError_t launch_grid(const void* kernel, const StepBuffers& b, const MechBuffers& m, const MechParams& p,
                               uint32_t step, cudaStream_t s) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kClosureThreads, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    StepBuffers bb = b;
    MechBuffers mm = m;
    MechParams pp = p;
    uint32_t st = step;
    void* args3[] = {&bb, &mm, &pp};
    void* args4[] = {&bb, &mm, &pp, &st};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((uint32_t)sms);
    cfg.blockDim = dim3(kClosureThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, kernel, step == kNoStep ? args3 : args4);
}

cudaError_t refresh_closure_columns(const MechBuffers& m, const MechParams& p, cudaStream_t s) {
    if (p.closures == 0 || !p.wide_closures || pcg_residual_mode(p)) return cudaSuccess;
    k_closure_columns<<<std::min(4096u, (p.closures + 7u) / 8u), kMBlock, 0, s>>>(m, p);
    return cudaGetLastError();
}

void mechanism_tick_clears(const MechBuffers& m, const MechParams& p, void** ptr, uint64_t* bytes, uint32_t* count) {
    *count = 0;
    if (p.closures == 0) return;
    ptr[0] = m.grid_barrier;
    bytes[0] = 64 * sizeof(uint32_t);
    ptr[1] = m.loop_state;
    bytes[1] = 2ull * kClosureSteps * sizeof(uint32_t);
    *count = 2;
}

// device.rs:963-1048
cudaError_t enqueue_mechanism(MechBuffers& m, const StepBuffers& b, const MechParams& p, cudaStream_t s) {
    cudaError_t e;
    if ((e = bearing_cache(m, b, p, s)) != cudaSuccess) return e;
    if ((e = bearing_projections(m, b, p, s)) != cudaSuccess) return e;
    k_advance_coordinates<<<nblocks(p.body_count), kMBlock, 0, s>>>(b, m, p);
    if ((e = forward_kinematics(m, p, s)) != cudaSuccess) return e;
    const uint32_t mode = g_closure_grid;
    const bool grid = p.closures > 0 && (mode == 2u || (mode == 0u && p.closures >= kGridClosures));
    ClosureShape shape;
    if (mode == 0u && closure_block_shape(p, shape)) {
        if ((e = launch_closure_block(m, b, p, shape, s)) != cudaSuccess) return e;
    } else if (pcg_residual_mode(p)) {
        for (uint32_t step = 0; step < kClosureSteps; ++step) {
            if (grid) {
                if ((e = launch_grid((const void*)k_closure_eval<true>, b, m, p, step, s)) != cudaSuccess) return e;
            } else {
                k_closure_eval<false><<<1, kClosureThreads, 0, s>>>(b, m, p, step);
            }
            if (p.learned_precond) {
                e = mlp::forward(m.precond_params, reinterpret_cast<const float*>(m.blk_feat), 0,
                                 &m.cstate->live_blocks, p.blocks, m.blk_out, 3, &b.diag->error_flags, s);
                if (e != cudaSuccess) return e;
            }
            if (grid) {
                if ((e = launch_grid((const void*)k_closure_pcg<true>, b, m, p, step, s)) != cudaSuccess) return e;
            } else {
                k_closure_pcg<false><<<1, kClosureThreads, 0, s>>>(b, m, p, step);
            }
        }
    } else if (p.closures > 0) {
        if (grid) {
            if ((e = launch_grid((const void*)k_closure_loop<true>, b, m, p, kNoStep, s)) != cudaSuccess) return e;
        } else {
            k_closure_loop<false><<<1, kClosureThreads, 0, s>>>(b, m, p);
        }
    }
    k_publish<<<nblocks(p.body_count), kMBlock, 0, s>>>(b, m, p);
    if ((e = reconstruct(m, b, p, s)) != cudaSuccess) return e;
    // the published poses hold for the rest of the tick: the projection passes
    // during and after the contact solve share one cache
    return bearing_cache(m, b, p, s);
}

// device.rs:1343-1416 with a dynamic mechanism root
cudaError_t enqueue_contact_solver_with_bearings(MechBuffers& m, const StepBuffers& b, const StepParams& sp,
                                                 const MechParams& p, const StepLaunch& l, int parity,
                                                 cudaStream_t s) {
    if (p.serial_contacts)
        return launch_contact_solver_serial(b, sp, l, parity, [&]() {
            k_project_bearings_serial<<<1, 32, 0, s>>>(b, m, p);
            return cudaGetLastError();
        }, s);
    float4 *lin[2], *ang[2];
    velocity_buffers(b, p, lin, ang);
    const uint32_t sides = side_blocks(p), hubs = p.hub_chunks, iterations = std::max(1u, l.iterations);
    cudaError_t e = launch_contact_solver_passes(b, sp, l, parity, lin, ang, [&](uint32_t it, int32_t* deltas, int32_t* clear) {
        const uint32_t from = it & 1u, to = from ^ 1u;
        auto* kernel = hubs ? k_bearing_pass<true, true> : k_bearing_pass<true, false>;
        kernel<<<sides + hubs + rest_blocks(p), kPassBlock, 0, s>>>(
            b, m, p, VelocityPass{lin[from], ang[from], lin[to], ang[to], lin[to], ang[to], deltas, clear}, sides, hubs);
        return cudaGetLastError();
    }, s);
    if (e == cudaSuccess && (iterations & 1u)) {
        k_pass_back<<<nblocks(p.body_count), kMBlock, 0, s>>>(m, p.body_count,
                                                              VelocityPass{lin[1], ang[1], lin[0], ang[0]});
        e = cudaGetLastError();
    }
    return e;
}

// device.rs:1128-1155
cudaError_t enqueue_post_contact(MechBuffers& m, const StepBuffers& b, const MechParams& p, cudaStream_t s) {
    cudaError_t e;
    if (!p.has_dynamic_root && (e = bearing_projections(m, b, p, s)) != cudaSuccess) return e;
    k_capture_coordinates<<<nblocks(p.body_count), kMBlock, 0, s>>>(b, m, p);
    if (!p.has_dynamic_root) return reconstruct(m, b, p, s);
    return cudaGetLastError();
}

void enqueue_validate_state(MechBuffers& m, const StepBuffers& b, const MechParams& p, cudaStream_t s) {
    k_validate_state<<<nblocks(p.body_count), kMBlock, 0, s>>>(b, m, p);
}

void enqueue_validate_bearings(MechBuffers& m, const StepBuffers& b, const MechParams& p, bool mechanism_active,
                               cudaStream_t s) {
    if (p.bearing_count == 0) return;
    k_validate_bearings<<<nblocks(p.bearing_count), kMBlock, 0, s>>>(m.bearings, p.bearing_count, b.pos, b.rot,
                                                                      mechanism_active ? m.links_final : nullptr,
                                                                      b.diag);
}

void read_mechanism_readback(const MechBuffers& m, const MechParams& p, const GpuDiagnostics& d,
                             const ClosureState* cs, MkTickReadback* out) {
    (void)m;
    if (pcg_residual_mode(p) && cs) {
        out->closure_iterations = cs->pcg_iterations;
        out->closure_relative_residual = cs->max_relative_residual;
    } else {
        out->closure_iterations = d.reserved_c;
        out->closure_relative_residual = 0.0;
    }
}

}  // namespace mk
