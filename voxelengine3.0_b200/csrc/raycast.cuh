// raycast.cuh — the octree DDA on the device.
//
// Result-identical to the reference's restart-from-root Raycast /
// RaycastCounted (internal.glsl:297-400): the same slab arithmetic, the same
// step counting (entry intersection counts one check, loop test
// `q++ <= controlchecks`), the same out-of-range-reads-zero rule.  What
// differs is how the descent finds the terminal cell of a DDA step:
//
//   The node read at descent level k depends only on the bits D..D-k of the
//   integer position.  Consecutive DDA positions share their high bits, so a
//   descent restarts at the first level whose bits changed, reusing the
//   child-block offsets `base[k]` the previous descent recorded.  When the
//   new position lies in the previous terminal (empty) cell the previous
//   result is reused outright.  The node words read per ray are then the
//   distinct nodes along its walk instead of (depth+1) per step.
//
//   A descent that restarts above level T0 reads one word of the scene's
//   top table instead of levels 0..T0-1: per cell of the level-(T0-1)
//   grid, the child-block offset reached at level T0, or the size of the
//   terminal cell when the walk ends higher up (built from the node words by
//   k_build_top, bit-identical to walking them).  The grid has one layer of
//   cells beyond 2^D on every axis, for the positions with a coordinate equal
//   to 2^D that the bounds test admits.  Fetch-counting runs (COUNT) walk
//   every level.
//
//   Where the table reaches the leaves (T0 = D, every scene of depth 3..10),
//   a restart below level D is one table word and then the leaf word: FlatRay
//   and flat_step below, the walk of every frame kernel.
#pragma once
#include "ve_device.cuh"

namespace ve {
namespace dev {

struct RayCount {
    uint32_t fetch = 0;
    uint32_t steps = 0;
};

__device__ __forceinline__ uint32_t fetch_node(const uint32_t* __restrict__ nodes, uint64_t n, uint32_t off) {
    return off < n ? __ldg(nodes + off) : 0u;
}


// The bound of a node array as the trace kernel keeps it: offsets are 32-bit,
// so a bound clamped to 2^32 - 1 rejects exactly the same offsets.
__device__ __forceinline__ uint32_t word_bound(uint64_t n) { return n < 0xFFFFFFFFull ? uint32_t(n) : 0xFFFFFFFFu; }
// The DDA as a resumable state machine: dda_init performs the origin advance
// and the entry intersection, dda_step one iteration of the reference loop
// `while (inBounds(r_pos) && q++ <= controlchecks)`.  Both return true when
// the ray is finished, with the result in `h`.
struct Dda {
    f3 o, d, inv;
    float t;  // the position is d * t + o (recomputed each step: the same operations as storing it)
    float t_end;  // CLIP: past this distance the ray can hit nothing (set by the caller)
    uint32_t q, cc;
    uint32_t lux, luy, luz, e_last;
    uint32_t base[17];
};

__device__ __forceinline__ bool dda_init(Dda& s, f3 o, f3 d, uint32_t controlchecks, uint32_t D, Hit& h) {
    const float Lf = float(1u << D);
    h.status = kEscaped;
    h.id = 0;
    h.material = 0;
    h.x = h.y = h.z = 0;
    h.size = 0;
    s.inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    s.d = d;
    s.o = add(o, muls(d, 4.0f));
    s.q = 0;
    s.cc = controlchecks;
    s.base[0] = 0u;
    // no position yet: every bit differs from the first step's, which
    // therefore restarts at level 0
    s.lux = s.luy = s.luz = 0xFFFFFFFFu;
    s.e_last = 0;
    if (in_bounds(s.o, Lf)) {
        s.t = 0.0f;
    } else {
        const f3 t1 = mul(mk((0.0f - s.o.x) + 0.001f, (0.0f - s.o.y) + 0.001f, (0.0f - s.o.z) + 0.001f), s.inv);
        const f3 t2 = mul(mk((Lf - s.o.x) - 0.001f, (Lf - s.o.y) - 0.001f, (Lf - s.o.z) - 0.001f), s.inv);
        const float t_enter = gmax(gmax(gmin(t1.x, t2.x), gmin(t1.y, t2.y)), gmin(t1.z, t2.z));
        const float t_exit = gmin(gmin(gmax(t1.x, t2.x), gmax(t1.y, t2.y)), gmax(t1.z, t2.z));
        s.q++;
        if (t_exit < t_enter || t_exit < 0.0f) {
            h.checks = s.q;
            return true;
        }
        s.t = t_enter;
    }
    return false;
}

// Layout of the top table: 2^(T0-1) cells and the layer beyond 2^D along each
// axis, y slowest, then x, then z in rows of a multiple of 16 bytes.  Worlds
// extend along x and z and have most of their content in a band of y, so the
// part of the table that rays read is one contiguous range: a depth-10
// terrain's is a sixth of its 556 MB, and with x slowest that sixth lay on every
// page of it (trace of a 1080p frame 0.694 against 0.631 ms).
__host__ __device__ constexpr uint32_t top_side(uint32_t T0) { return (1u << (T0 - 1u)) + 1u; }
__host__ __device__ constexpr uint32_t top_row(uint32_t T0) { return (1u << (T0 - 1u)) + 16u; }
// Top-table entry of the cell containing (x, y, z): (offset << 1) | 1 when
// levels 0..T0-1 are internal (offset = child block of the level-T0 node),
// else (size of the terminal cell - 1) << 1.
__device__ __forceinline__ uint32_t top_index(uint32_t x, uint32_t y, uint32_t z, uint32_t D, uint32_t T0) {
    const uint32_t sh = D - T0 + 1u;
    return ((y >> sh) * top_side(T0) + (x >> sh)) * top_row(T0) + (z >> sh);
}

// WORD: a hit reports the leaf's node word in h.id instead of its slot (the
// bounce trace keeps the word for shading; the slot is the GBuffer's field).
// CLIP: the ray also ends, as escaped, once its distance passes s.t_end —
// for callers to whom an escape and a timeout are the same result.
template <bool COUNT, bool WORD = false, bool CLIP = false>
__device__ __forceinline__ bool dda_step(Dda& s, const uint32_t* __restrict__ nodes, uint64_t n_words, uint32_t D,
                                         const uint32_t* __restrict__ top, uint32_t T0, Hit& h, RayCount& rc) {
    const uint32_t L = 1u << D;
    const float Lf = float(L);
    const f3 r = add(muls(s.d, s.t), s.o);
    if (!in_bounds(r, Lf) || (CLIP && s.t > s.t_end)) {
        h.status = kEscaped;
        h.checks = s.q;
        return true;
    }
    if (!(s.q++ <= s.cc)) {
        h.status = kTimeout;
        h.checks = s.q;
        return true;
    }
    if (COUNT) rc.steps++;
    const uint32_t ux = uint32_t(r.x), uy = uint32_t(r.y), uz = uint32_t(r.z);
    bool reuse = false;
    uint32_t start = 0;
    {
        const uint32_t xd = (ux ^ s.lux) | (uy ^ s.luy) | (uz ^ s.luz);
        if (xd == 0u) {
            reuse = true;
        } else {
            const uint32_t hb = 31u - uint32_t(__clz(xd));
            start = hb >= D ? 0u : D - hb;
            reuse = start > s.e_last;
        }
    }
    uint32_t k = s.e_last;
    if (!reuse) {
        s.lux = ux; s.luy = uy; s.luz = uz;
        bool found = false;
        uint32_t off = 0;
        k = start;
        // child index at level k: bit D-k of x, y, z as bits 2, 1, 0
        const uint32_t sx = ux << 2, sy = uy << 1;
        if (!COUNT && start < T0) {
            const uint32_t ent = __ldg(top + top_index(ux, uy, uz, D, T0));
            if (ent & 1u) {
                s.base[T0] = ent >> 1;
                k = T0;
            } else {
                k = D - uint32_t(__popc(ent >> 1));  // cell size 2^(D-k)
                found = true;
            }
        }
        for (; !found && k < D; k++) {
            const uint32_t b = D - k;  // the position bit level k tests
            off = s.base[k] + (((sx >> b) & 4u) | ((sy >> b) & 2u) | ((uz >> b) & 1u));
            const uint32_t raw = fetch_node(nodes, n_words, off);
            if (COUNT) rc.fetch++;
            if (!(raw & 1u)) {
                found = true;
                break;
            }
            s.base[k + 1] = raw >> 4;
        }
        s.e_last = k;
        if (!found) {
            off = s.base[D] + ((sx & 4u) | (sy & 2u) | (uz & 1u));
            const uint32_t raw = fetch_node(nodes, n_words, off);
            if (COUNT) rc.fetch++;
            const uint32_t mat = (raw & 254u) >> 1;
            if (mat != 0u) {
                h.status = kHit;
                h.id = WORD ? raw : off;
                h.material = mat;
                h.x = ux; h.y = uy; h.z = uz;
                h.size = 1u;
                h.checks = s.q;
                return true;
            }
        }
    }
    const uint32_t size = L >> k;
    const uint32_t px = ux & ~(size - 1u), py = uy & ~(size - 1u), pz = uz & ~(size - 1u);
    // exit of the cell: the reference takes, per axis, the larger of the two
    // slab distances ((min - o) - 0.001) / d and ((max - o) + 0.001) / d.
    // Rounding is monotone and the first numerator is below the second, so
    // that larger one is always the second where 1/d > 0 (+inf included) and
    // the first elsewhere: only that plane is computed, with the same
    // operations, giving the same bits (3-4 % less trace time than both).
    const bool ax = s.inv.x > 0.0f, ay = s.inv.y > 0.0f, az = s.inv.z > 0.0f;
    const float tx = ((float(px + (ax ? size : 0u)) - s.o.x) + (ax ? 0.001f : -0.001f)) * s.inv.x;
    const float ty = ((float(py + (ay ? size : 0u)) - s.o.y) + (ay ? 0.001f : -0.001f)) * s.inv.y;
    const float tz = ((float(pz + (az ? size : 0u)) - s.o.z) + (az ? 0.001f : -0.001f)) * s.inv.z;
    const float t_exit = gmin(gmin(tx, ty), tz);
    s.t = t_exit;
    return false;
}

// ---------------------------------------------------------------------------
// The walk of scenes whose top table reaches the leaves (T0 = D).
//
// Bound by issue: a step is arithmetic between two dependent loads, so it is
// written for few instructions.  With the result stores moved to the refill
// (k_trace) it took the trace of a 1080p depth-10 frame (4 spp x 3 bounces)
// from 0.963 to 0.694 ms (155.9 M -> 88.2 M warp instructions in the first
// pass of its 960x540 form) and the primary pass from 0.382 to 0.346 ms.
//   * Positions are kept as the bits of r + 1.5 * 2^23 rounded toward zero
//     (r in [0, 2^16]: the low 22 bits are trunc(r) exactly), one full-rate
//     add in place of a quarter-rate conversion, and the far plane of a cell
//     goes back to a float by subtracting that constant (exact).  The plane
//     itself is one logic operation: with c = the bits of -1.5 * 2^23 + 1 for
//     a rising axis (low 22 bits all ones) and of -1.5 * 2^23 for a falling one
//     (all zeros), ((b ^ c) & ~m) ^ c is the cell's last coordinate or its
//     first one (m = cell size - 1), and adding c as a float gives the plane.
//   * The cell is its table entry: no level, no leading-zero count.
//   * min/max of three operands are one instruction each.  They return what
//     the glm selects of dda_step return: inside the volume no exit distance
//     is NaN (an axis with 1/d = +-inf has a non-zero numerator of its sign),
//     and the bounds test propagates NaN to "outside" as the comparisons do.
//   * The table's index arithmetic runs on the biased bits; the table pointer
//     takes the bias out (flat_scene).
// Table entries below 2^31 and blocks at most n_words (k_build_top clamps; the
// node array ends with 8 zero words) make both loads unconditional.
// ---------------------------------------------------------------------------
constexpr float kPosBias = 12582912.0f;         // 1.5 * 2^23
constexpr uint32_t kPosBits = 0x4B400000u;      // its bits
constexpr uint32_t kPlaneRise = 0xCB3FFFFFu;    // bits of 1 - 1.5 * 2^23
enum : uint32_t { kWalking = 3u };              // flat_step: the ray goes on

struct FlatRay {
    f3 o, d, inv;
    float t, t_end;
    uint32_t left;        // steps before the timeout
    uint32_t bx, by, bz;  // biased position bits
    uint32_t ent;         // table entry of its cell; after a hit: the leaf's word (WORD) or slot
};

// Table pointer such that the index of the biased bits, modulo 2^32, lands on
// the cell: index + K, K = (kPosBits >> 1) * ((S + 1) * row + 1) mod 2^32,
// must not wrap for any table.
__host__ __device__ constexpr uint32_t flat_bias(uint32_t D) {
    return (kPosBits >> 1) * ((top_side(D) + 1u) * top_row(D) + 1u);
}
constexpr bool flat_bias_fits(uint32_t D) {
    return uint64_t(flat_bias(D)) + uint64_t(top_side(D)) * top_side(D) * top_row(D) < (1ull << 32);
}
static_assert(flat_bias_fits(3) && flat_bias_fits(4) && flat_bias_fits(5) && flat_bias_fits(6) && flat_bias_fits(7) &&
                  flat_bias_fits(8) && flat_bias_fits(9) && flat_bias_fits(10),
              "a biased table index wraps");
struct FlatScene {
    const uint32_t* nodes;
    const uint32_t* topb;  // the table, biased
    uint32_t side, row;
    float Lf;
};
__host__ __device__ __forceinline__ FlatScene flat_scene(const uint32_t* nodes, const uint32_t* top, uint32_t D) {
    return FlatScene{nodes, reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(top) - 4ull * flat_bias(D)),
                     top_side(D), top_row(D), float(1u << D)};
}
__device__ __forceinline__ float min3_nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Distance to the far plane of the cell along one axis.
__device__ __forceinline__ float flat_exit(uint32_t b, uint32_t m, float o, float inv) {
    const uint32_t neg = __float_as_uint(inv) >> 31;
    const uint32_t c = kPlaneRise + neg;
    const float plane = __uint_as_float(((b ^ c) & ~m) ^ c) + __uint_as_float(c);
    const float e = __uint_as_float((__float_as_uint(inv) & 0x80000000u) | __float_as_uint(0.001f));
    return ((plane - o) + e) * inv;
}

// The position at distance t: false when it lies outside (or, CLIP, t beyond
// t_end).
template <bool CLIP>
__device__ __forceinline__ bool flat_at(const FlatRay& s, const FlatScene& w, uint32_t& bx, uint32_t& by, uint32_t& bz) {
    const f3 r = add(muls(s.d, s.t), s.o);
    const float lo = min3_nan(r.x, r.y, r.z), hi = max3_nan(r.x, r.y, r.z);
    bx = __float_as_uint(__fadd_rz(r.x, kPosBias));
    by = __float_as_uint(__fadd_rz(r.y, kPosBias));
    bz = __float_as_uint(__fadd_rz(r.z, kPosBias));
    return 0.0f <= lo && hi <= w.Lf && !(CLIP && s.t > s.t_end);
}
__device__ __forceinline__ uint32_t flat_entry(const FlatScene& w, uint32_t bx, uint32_t by, uint32_t bz) {
    return __ldg(w.topb + (((by >> 1) * w.side + (bx >> 1)) * w.row + (bz >> 1)));
}

// The ray's set-up up to its first position's distance: false when it misses
// the volume (escaped; `left` is then one less than the checks allow).
__device__ __forceinline__ bool flat_init(FlatRay& s, f3 o, f3 d, uint32_t controlchecks, float Lf) {
    s.inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    s.d = d;
    s.o = add(o, muls(d, 4.0f));
    s.left = controlchecks + 1u;
    s.t = 0.0f;
    if (!in_bounds(s.o, Lf)) {
        const f3 t1 = mul(mk((0.0f - s.o.x) + 0.001f, (0.0f - s.o.y) + 0.001f, (0.0f - s.o.z) + 0.001f), s.inv);
        const f3 t2 = mul(mk((Lf - s.o.x) - 0.001f, (Lf - s.o.y) - 0.001f, (Lf - s.o.z) - 0.001f), s.inv);
        const float t_enter = gmax(gmax(gmin(t1.x, t2.x), gmin(t1.y, t2.y)), gmin(t1.z, t2.z));
        const float t_exit = gmin(gmin(gmax(t1.x, t2.x), gmax(t1.y, t2.y)), gmax(t1.z, t2.z));
        s.left--;
        if (t_exit < t_enter || t_exit < 0.0f) return false;
        s.t = t_enter;
    }
    return true;
}
// The first position's checks and table entry: kWalking, or how the ray ended.
template <bool CLIP>
__device__ __forceinline__ uint32_t flat_first(FlatRay& s, const FlatScene& w) {
    if (!flat_at<CLIP>(s, w, s.bx, s.by, s.bz)) return kEscaped;
    if (s.left == 0u) return kTimeout;
    s.left--;
    s.ent = flat_entry(w, s.bx, s.by, s.bz);
    return kWalking;
}

// One iteration of the reference loop, from the lookup of the current
// position's cell to the checks of the next one: kWalking, or how the ray
// ended (kHit / kEscaped / kTimeout).  The cell's exit depends on its table
// entry but not on its leaf word, so the next position's table entry is loaded
// while the leaf word is on its way: a step waits for one load, not two (1080p
// depth-10 frame: trace 0.594 -> 0.545 ms, primary 0.351 -> 0.324; 256x256
// depth 7: 0.047 -> 0.042 and 0.0345 -> 0.0273).  A ray that hits has loaded
// one entry in vain.  The entry is loaded at every step, also inside the leaf
// block or cell it was loaded for: the test that spared those (cached) loads
// cost more (2160p 8 spp frame: trace 2.93 -> 2.77 ms without it, 1080p 0.520 ->
// 0.508).
// WORD: a hit leaves the leaf's word in ent, else its slot.  CLIP as in
// dda_step.
template <bool WORD, bool CLIP>
__device__ __forceinline__ uint32_t flat_step(FlatRay& s, const FlatScene& w) {
    const uint32_t blk = s.ent >> 1;
    const bool leaf = (s.ent & 1u) != 0u;
    const uint32_t m = leaf ? 0u : blk;  // size - 1 of the cell
    const uint32_t off = blk + (((s.bx << 2) & 4u) | ((s.by << 1) & 2u) | (s.bz & 1u));
    uint32_t raw = 0u;
    if (leaf) raw = __ldg(w.nodes + off);
    s.t = fminf(fminf(flat_exit(s.bx, m, s.o.x, s.inv.x), flat_exit(s.by, m, s.o.y, s.inv.y)),
                flat_exit(s.bz, m, s.o.z, s.inv.z));
    uint32_t bx, by, bz;
    const bool in = flat_at<CLIP>(s, w, bx, by, bz);
    uint32_t ent = 0u;
    if (in) ent = flat_entry(w, bx, by, bz);
    if ((raw & 254u) != 0u || !in || s.left == 0u) {
        const bool hit = (raw & 254u) != 0u;
        if (hit) s.ent = WORD ? raw : off;
        return hit ? kHit : in ? kTimeout : kEscaped;
    }
    s.left--;
    s.bx = bx; s.by = by; s.bz = bz;
    s.ent = ent;
    return kWalking;
}

template <bool COUNT>
__device__ __forceinline__ Hit raycast(const uint32_t* __restrict__ nodes, uint64_t n_words, uint32_t D,
                                       const uint32_t* __restrict__ top, uint32_t T0, f3 o, f3 d,
                                       uint32_t controlchecks, RayCount& rc) {
    Hit h;
    if (!COUNT && T0 == D) {
        const FlatScene w = flat_scene(nodes, top, D);
        FlatRay s;
        h.status = kEscaped;
        h.id = h.material = h.x = h.y = h.z = h.size = 0;
        if (flat_init(s, o, d, controlchecks, w.Lf)) {
            h.status = flat_first<false>(s, w);
            while (h.status == kWalking) h.status = flat_step<false, false>(s, w);
        }
        // the reference's count includes the check that found no steps left
        h.checks = controlchecks + 1u - s.left + (h.status == kTimeout ? 1u : 0u);
        if (h.status == kHit) {
            h.id = s.ent;
            h.material = (__ldg(nodes + s.ent) & 254u) >> 1;
            h.x = s.bx - kPosBits; h.y = s.by - kPosBits; h.z = s.bz - kPosBits;
            h.size = 1u;
        }
        return h;
    }
    Dda s;
    if (dda_init(s, o, d, controlchecks, D, h)) return h;
    while (!dda_step<COUNT>(s, nodes, n_words, D, top, T0, h, rc)) {
    }
    return h;
}

}  // namespace dev
}  // namespace ve
