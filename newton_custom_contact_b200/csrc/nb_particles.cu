// XPBD particle path: soft contacts between particles and shapes, and the
// particle substep (integration, particle-shape and particle-particle
// contacts, springs, position corrections).
//
// Layout: particles are SoA float3 rows ([P,3]).  Each particle GATHERS its corrections (its own soft contacts,
// its neighbours, its springs) in a fixed order and writes its delta once, in
// place of the reference's per-constraint atomic scatter: no atomics on the
// data path and the same bits on every run.
//
// Particle-particle neighbours come from a hashed cell grid, rebuilt every
// iteration from the positions it reads (struct Grid below): the apply kernel
// of iteration i counts every particle into its bucket as it writes its new
// position, and two small kernels put the particles' entries in bucket order.
#include <cuda_runtime.h>

#include <cstdint>

#include "nb_kernels.cuh"
#include "nb_math.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kScanThreads = 1024;
constexpr int kCollideParticles = 1 << 2;  // ShapeFlags.COLLIDE_PARTICLES

NB_D bool active(const NbParticleDesc& pd, int p) { return (pd.particle_flags[p] & NB_PARTICLE_ACTIVE) != 0; }
NB_D V3 ld3(const float* a, int i) { return V3{a[3 * i], a[3 * i + 1], a[3 * i + 2]}; }
NB_D void st3(float* a, int i, V3 v) {
    a[3 * i] = v.x;
    a[3 * i + 1] = v.y;
    a[3 * i + 2] = v.z;
}
// wp.sign: -1 for negative arguments, +1 otherwise
NB_D float warp_sign(float x) { return x < 0.0f ? -1.0f : 1.0f; }

// atan2 from the library's asin (nb_math.cuh), so the CPU oracle reproduces it bit for bit: the angle
// is asin of the smaller of |x|, |y| over the radius (argument at most 1/sqrt 2, where asin is well
// conditioned), shifted into its quadrant.  atan2(0, 0) = 0.
NB_D float nb_atan2(float y, float x) {
    const float r = sqrtf(x * x + y * y);
    if (r == 0.0f) return 0.0f;
    if (fabsf(y) <= fabsf(x)) {
        const float a = nb_asin(y / r);
        if (x > 0.0f) return a;
        return y < 0.0f ? -3.1415927410125732f - a : 3.1415927410125732f - a;
    }
    const float a = 1.5707963705062866f - nb_asin(x / r);
    return y < 0.0f ? -a : a;
}

// Signed distance and outward gradient in the shape frame (newton/_src/geometry/
// kernels.py:165-330 sdf_sphere/_grad, sdf_box/_grad, sdf_capsule/_grad with the
// Z up axis, 568-590 sdf_plane).
NB_D void shape_sdf(int type, V3 p, V3 s, float& d, V3& n) {
    d = 1.0e6f;
    n = V3{0.0f, 0.0f, 0.0f};
    if (type == NB_GEO_SPHERE) {
        d = length(p) - s.x;
        const float l = length(p);
        n = l > 1.0e-8f ? divs(p, l) : V3{0.0f, 0.0f, 1.0f};
    } else if (type == NB_GEO_BOX) {
        const float qx = fabsf(p.x) - s.x, qy = fabsf(p.y) - s.y, qz = fabsf(p.z) - s.z;
        const V3 e = V3{fmaxw(qx, 0.0f), fmaxw(qy, 0.0f), fmaxw(qz, 0.0f)};
        d = length(e) + fminw(fmaxw(qx, fmaxw(qy, qz)), 0.0f);
        if (qx > 0.0f || qy > 0.0f || qz > 0.0f) {
            const V3 c = V3{clampw(p.x, -s.x, s.x), clampw(p.y, -s.y, s.y), clampw(p.z, -s.z, s.z)};
            n = normalize(sub(p, c));
        } else if ((qx > qy && qx > qz) || (qy == 0.0f && qz == 0.0f)) {
            n = V3{warp_sign(p.x), 0.0f, 0.0f};
        } else if ((qy > qx && qy > qz) || (qx == 0.0f && qz == 0.0f)) {
            n = V3{0.0f, warp_sign(p.y), 0.0f};
        } else {
            n = V3{0.0f, 0.0f, warp_sign(p.z)};
        }
    } else if (type == NB_GEO_CAPSULE) {
        const float r = s.x, hh = s.y;
        V3 v;
        V3 fallback;
        if (p.z > hh) {
            v = V3{p.x, p.y, p.z - hh};
            fallback = V3{0.0f, 0.0f, 1.0f};
        } else if (p.z < -hh) {
            v = V3{p.x, p.y, p.z + hh};
            fallback = V3{0.0f, 0.0f, -1.0f};
        } else {
            v = V3{p.x, p.y, 0.0f};
            fallback = V3{0.0f, 0.0f, 1.0f};
        }
        d = length(v) - r;
        const float l = length(v);
        n = l > 1.0e-8f ? divs(v, l) : fallback;
    } else if (type == NB_GEO_PLANE) {
        const float w = s.x * 0.5f, l = s.y * 0.5f;
        if (w > 0.0f && l > 0.0f) {
            const float dd = fmaxw(fabsf(p.x) - w, fabsf(p.y) - l);
            d = fmaxw(dd, fabsf(p.z));
        } else {
            d = p.z;
        }
        n = V3{0.0f, 0.0f, 1.0f};
    }
}

// One (particle, shape) test of create_soft_contacts (newton/_src/geometry/kernels.py:1029-1140).
// Returns true for a contact and fills its body-frame point, velocity and world normal.
NB_D bool soft_contact(const NbParticleDesc& pd, const float* body_q, int p, int s, V3 px, float radius,
                       float margin, V3& body_pos, V3& body_vel, V3& world_normal) {
    if ((pd.shape_flags[s] & kCollideParticles) == 0) return false;
    const int pw = pd.particle_world[p], sw = pd.shape_world[s];
    if (pw != -1 && sw != -1 && pw != sw) return false;
    const int rigid = pd.shape_body[s];
    const TF X_wb = rigid >= 0 ? load_tf(body_q + 7 * rigid) : tf_identity();
    const TF X_bs = load_tf(pd.shape_transform + 7 * s);
    const TF X_ws = tf_mul(X_wb, X_bs);
    const TF X_sw = tf_inverse(X_ws);
    const V3 x_local = tf_point(X_sw, px);
    float d;
    V3 n;
    shape_sdf(pd.shape_type[s], x_local, load_v3(pd.shape_scale + 3 * s), d, n);
    if (!(d < margin + radius)) return false;
    body_pos = tf_point(X_bs, sub(x_local, mul(n, d)));
    body_vel = tf_vector(X_bs, V3{0.0f, 0.0f, 0.0f});
    world_normal = tf_vector(X_ws, n);
    return true;
}

NB_D int particle_soft_count(const NbParticleDesc& pd, const float* body_q, int p, const float* q, float margin) {
    if (!active(pd, p)) return 0;
    const V3 px = ld3(q, p);
    const float radius = pd.particle_radius[p];
    int c = 0;
    for (int s = 0; s < pd.shape_count; ++s) {
        V3 a, b, n;
        c += soft_contact(pd, body_q, p, s, px, radius, margin, a, b, n) ? 1 : 0;
    }
    return c;
}

// Exclusive scan of one value per thread over a block of kScanThreads threads.
__device__ int block_exclusive_scan(int v, int& total) {
    __shared__ int warp_sums[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < kScanThreads / 32 ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kScanThreads / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    total = warp_sums[kScanThreads / 32 - 1];
    const int before = warp > 0 ? warp_sums[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

// Pass 1: every particle's contact count (kept in particle_start[p]) and each block's sum.
__global__ void __launch_bounds__(kScanThreads) soft_count_kernel(NbParticleDesc pd, const float* q,
                                                                  const float* body_q, NbSoftContacts sc) {
    const int p = blockIdx.x * kScanThreads + threadIdx.x;
    const int P = pd.particle_count;
    const int c = p < P ? particle_soft_count(pd, body_q, p, q, sc.margin) : 0;
    if (p < P) sc.particle_start[p] = c;
    int total;
    block_exclusive_scan(c, total);
    if (threadIdx.x == 0) sc.particle_start[P + 1 + blockIdx.x] = total;
}

// Pass 2 (one block): exclusive scan of the block sums; the grand total is the contact count.
__global__ void __launch_bounds__(kScanThreads) soft_scan_blocks_kernel(NbParticleDesc pd, NbSoftContacts sc,
                                                                        int blocks) {
    const int P = pd.particle_count;
    int* sums = sc.particle_start + P + 1;
    int carry = 0;
    for (int base = 0; base < blocks; base += kScanThreads) {
        const int b = base + threadIdx.x;
        const int v = b < blocks ? sums[b] : 0;
        int total;
        const int ex = block_exclusive_scan(v, total);
        if (b < blocks) sums[b] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) {
        sc.particle_start[P] = carry;
        sc.count[0] = carry;
    }
}

// Pass 3: each particle's first contact, then its contacts in shape order (the first max are stored).
__global__ void __launch_bounds__(kScanThreads) soft_write_kernel(NbParticleDesc pd, const float* q,
                                                                  const float* body_q, NbSoftContacts sc) {
    const int p = blockIdx.x * kScanThreads + threadIdx.x;
    const int P = pd.particle_count;
    const int c = p < P ? sc.particle_start[p] : 0;
    int total;
    const int ex = block_exclusive_scan(c, total);
    if (p >= P) return;
    int at = sc.particle_start[P + 1 + blockIdx.x] + ex;
    sc.particle_start[p] = at;
    if (c == 0) return;
    const V3 px = ld3(q, p);
    const float radius = pd.particle_radius[p];
    for (int s = 0; s < pd.shape_count && at < sc.max; ++s) {
        V3 bp, bv, n;
        if (!soft_contact(pd, body_q, p, s, px, radius, sc.margin, bp, bv, n)) continue;
        sc.particle[at] = p;
        sc.shape[at] = s;
        st3(sc.body_pos, at, bp);
        st3(sc.body_vel, at, bv);
        st3(sc.normal, at, n);
        ++at;
    }
}

// ---------------------------------------------------------------- substep
// Neighbour search.  Cells have the size of the largest contact distance; a cell's bucket is
// (cx + cy K1 + cz K2) mod M, so cells that follow each other in x are buckets that follow each other,
// and the up to 3 cells of one (cy, cz) row around a particle are one run of the particles in bucket
// order: 9 runs in place of 27 chains.  Two forms:
//   sorted: per iteration the particles are counted into the buckets (integrate / apply), the buckets
//           get their ranges (particle_ranges_kernel) and the particles' entries are written there
//           (particle_scatter_kernel).  An entry is 8 bytes: the position within 4 cells, 10 bits per
//           axis, and the particle -- enough to reject most candidates with one load.  Up to 2 P buckets:
//           most candidates of a scattered particle are strangers that share a bucket with its cells, and
//           half as many buckets have twice as many of them (us per substep of 4 iterations, up to P / up to
//           2 P buckets: 100,000 scattered particles 245 / 210, piled ones 276 / 260).
//   lists:  linked lists per bucket (head / next), for scratch too small for the sorted form.
struct Grid {
    int32_t* head;   // lists: [2][M] first particle of a bucket, -1 empty
    int32_t* next;   // lists: [P] next particle of the same bucket
    int2* entry;     // sorted: [P] (packed position, particle) in bucket order
    int32_t* first;  // sorted: first entries of the buckets and the blocks' ends (bucket_at)
    int32_t* count;  // sorted: [M] particles of a bucket; all zero outside counting .. scatter
    int32_t* cursor; // sorted: [1] entries handed out so far; the active particles once all are
    uint32_t mask;   // M - 1
    float inv_h;
    bool on, sorted;
    bool small;      // sorted, rebuilt by one block (particle_regrid_kernel)
};

constexpr int kRangeBuckets = 1024;  // buckets whose ranges one block lays out contiguously
constexpr int kSmallParticles = 3072;  // most particles one block rebuilds the grid of
constexpr int kSmallBuckets = 4096;     // their buckets: fewer than twice as many, a power of two
constexpr int kMinSorted = 8;        // fewest buckets of the sorted form: a row of 5 cells never wraps onto itself

// place of bucket b's first entry; the place behind it holds its end, which is the next bucket's first entry or
// the end of the block
__host__ __device__ __forceinline__ uint32_t bucket_at(uint32_t b) { return b + b / kRangeBuckets; }
NB_D int cell_of(float x, float inv_h) { return (int)floorf(x * inv_h); }
// the last of the cells searched from `first` on: at most 5, which keeps the loops bounded whatever the
// scale, and none past the largest int, where far positions end up
NB_D int last_cell(float x, float inv_h, int first) {
    return min(cell_of(x, inv_h), first < INT32_MAX - 4 ? first + 4 : INT32_MAX);
}
NB_D uint32_t cell_hash(int cx, int cy, int cz, uint32_t mask) {
    return ((uint32_t)cx + (uint32_t)cy * 0x9E3779B1u + (uint32_t)cz * 0x85EBCA77u) & mask;
}
// position within 4 cells in 1/256 cells
NB_D uint32_t pack_axis(float x, float inv_h) {
    const float t = x * inv_h, c = floorf(t);
    const int f = (int)((t - c) * 256.0f);
    return (((uint32_t)(int)c & 3u) << 8) | (uint32_t)min(max(f, 0), 255);
}
NB_D uint32_t pack_pos(V3 x, float inv_h) {
    return pack_axis(x.x, inv_h) | (pack_axis(x.y, inv_h) << 10) | (pack_axis(x.z, inv_h) << 20);
}
// An entry's first word: the packed position, with kLargeEntry set for a particle beyond the model's
// particle_max_radius (a program may change radii later): it may touch particles whose reach, which counts on
// that radius, ends before it.
constexpr uint32_t kLargeEntry = 1u << 30;
NB_D uint32_t entry_word(const NbParticleDesc& pd, int p, V3 x, float inv_h) {
    return pack_pos(x, inv_h) | (pd.particle_radius[p] > pd.particle_max_radius ? kLargeEntry : 0u);
}
NB_D void grid_insert(const Grid& g, int table, int p, V3 x) {
    const uint32_t b = cell_hash(cell_of(x.x, g.inv_h), cell_of(x.y, g.inv_h), cell_of(x.z, g.inv_h), g.mask);
    if (g.sorted) atomicAdd(&g.count[b], 1);
    else g.next[p] = atomicExch(&g.head[(size_t)table * (g.mask + 1u) + b], p);
}

// Ranges of kRangeBuckets buckets per block: an exclusive scan of their counts from a base taken off the
// cursor.  Which block comes first decides only where its entries lie; within the block they are in
// bucket order.
__global__ void __launch_bounds__(kThreads) particle_ranges_kernel(Grid g) {
    __shared__ int s_warp[kThreads / 32];
    __shared__ int s_base;
    constexpr int kPer = kRangeBuckets / kThreads;
    const uint32_t b0 = blockIdx.x * kRangeBuckets + threadIdx.x * kPer;
    int c[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        c[k] = b0 + k <= g.mask ? g.count[b0 + k] : 0;
        sum += c[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int w = 0; w < kThreads / 32; ++w) {
            const int v = s_warp[w];
            s_warp[w] = run;
            run += v;
        }
        s_base = run > 0 ? atomicAdd(g.cursor, run) : 0;
    }
    __syncthreads();
    int at = s_base + s_warp[warp] + x - sum;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const uint32_t b = b0 + k;
        if (b <= g.mask) g.first[bucket_at(b)] = at;
        at += c[k];
        if (b == g.mask || (b < g.mask && b % kRangeBuckets == kRangeBuckets - 1)) g.first[bucket_at(b) + 1] = at;
    }
}

// The particles' entries into their buckets' ranges; leaves every count at zero.
__global__ void __launch_bounds__(kThreads) particle_scatter_kernel(NbParticleDesc pd, const float* xq, Grid g) {
    const int p = blockIdx.x * kThreads + threadIdx.x;
    if (p >= pd.particle_count || !active(pd, p)) return;
    const V3 x = ld3(xq, p);
    const uint32_t b = cell_hash(cell_of(x.x, g.inv_h), cell_of(x.y, g.inv_h), cell_of(x.z, g.inv_h), g.mask);
    const int at = g.first[bucket_at(b)] + atomicSub(&g.count[b], 1) - 1;
    g.entry[at] = make_int2((int)entry_word(pd, p, x, g.inv_h), p);
}

// integrate_particles (newton/_src/solvers/solver.py:11-47): semi-implicit Euler, gravity on
// particles with positive inverse mass, velocity clamp.  An inactive particle keeps its state.
__global__ void __launch_bounds__(kThreads) particle_integrate_kernel(NbParticleDesc pd, NbParticleIO io,
                                                                      float dt, Grid g) {
    const int p = blockIdx.x * kThreads + threadIdx.x;
    if (p >= pd.particle_count) return;
    if (p == 0 && g.sorted) g.cursor[0] = 0;
    const V3 x0 = ld3(io.particle_q, p);
    const V3 v0 = ld3(io.particle_qd, p);
    if (!active(pd, p)) {
        st3(io.particle_q_out, p, x0);
        st3(io.particle_qd_out, p, v0);
        return;
    }
    const V3 f0 = io.particle_f ? ld3(io.particle_f, p) : V3{0.0f, 0.0f, 0.0f};
    const float inv_mass = pd.particle_inv_mass[p];
    const int w = pd.particle_world[p];
    const V3 grav = ld3(pd.gravity, w > 0 ? w : 0);
    const float gate = -inv_mass < 0.0f ? 1.0f : 0.0f;  // wp.step(-inv_mass)
    V3 v1 = add(v0, mul(add(mul(f0, inv_mass), mul(grav, gate)), dt));
    const float v1_mag = length(v1);
    if (v1_mag > pd.particle_max_velocity) v1 = mul(v1, pd.particle_max_velocity / v1_mag);
    const V3 x1 = add(x0, mul(v1, dt));
    st3(io.particle_q_out, p, x1);
    st3(io.particle_qd_out, p, v1);
    if (g.on && !g.small) grid_insert(g, 0, p, x1);
}

// The corrections of one particle in one iteration: soft contacts (kernels.py:114-222, static
// shapes), particle neighbours (kernels.py:225-289) and springs (kernels.py:292-356), summed in
// that order.  kGroup lanes serve one particle: they filter the candidates of its cell rows by the packed
// positions, kept ones go to a list in shared memory, each lane tests its share of the list exactly and
// then computes the contributions of its share of the contacting ones (and of the springs); every lane
// sums them in ascending neighbour (spring) index.  Which lane computes a contribution does not change its
// bits, so the result equals a sequential sum in that order.
// Bound by the latency of the dependent loads and, at size, by instructions, so the steps are few and
// wide: one row lookup per lane, candidates in runs of 32, all arrays of a kept candidate at once; the
// sorted form takes the particles in bucket order, so that a block's particles share their candidates in
// L1.  Measured at 110,002 particles (4 contacts each on average; 8 iterations, per substep) with 4 / 8 / 16 /
// 32 lanes and up to P buckets: 1369 / 990 / 967 / 1440 us; at 3,010 particles (4 iterations): 286 / 205 / 150 /
// 147 us; now, with 16 lanes and up to 2 P buckets, 953 and 136 us.  Linked lists of the cells, whose candidates
// are one dependent load after another, with one lane sorting and summing for its group of 8, took 2215 and
// 240 us; they stay faster by 1.15 to 1.3 times where hardly any particles meet (20,000 scattered ones 120
// against 156 us per substep of 8 iterations, 100,000 368 against 426), for they need two kernels less.
constexpr int kGroup = 16;                 // lanes per particle
constexpr int kSlots = kThreads / kGroup;  // particles per block
constexpr int kAhead = 2;                  // candidate loads a lane has in flight
constexpr int kMaybe = 2 * kAhead * kGroup;

// A group's scratch: the candidates' runs and list, then (in the same place) the contributions.
struct GroupScratch {
    // runs of entries (a row may be cut in two): entry minus running index, running index past the run,
    // low cell bits of the row where the packed position has them, row
    union {
        struct {
            int4 seg[2 * kGroup];
            int maybe[kMaybe];                         // candidates to be tested exactly
        };
        float c[NB_PARTICLE_MAX_NEIGHBORS][3];     // the accepted neighbours' contributions, in ascending index
    };
    int j[NB_PARTICLE_MAX_NEIGHBORS];              // accepted neighbours
    int n;                                         // neighbours accepted
};

template <bool kSorted>
__global__ void __launch_bounds__(kThreads, 4)
particle_constraints_kernel(NbParticleDesc pd, NbParticleIO io, NbSoftContacts sc, int has_sc, float dt,
                            float relaxation, Grid g, int table) {
    __shared__ GroupScratch s_group[kSlots];
    const int tid = blockIdx.x * kThreads + threadIdx.x;
    if (!kSorted && g.on) {
        // clears the lists the following apply fills
        int32_t* other = g.head + (size_t)(table ^ 1) * (g.mask + 1u);
        for (uint32_t t = tid; t <= g.mask; t += gridDim.x * kThreads) other[t] = -1;
    }
    const int lane = threadIdx.x & (kGroup - 1);
    const unsigned gmask = ((1u << kGroup) - 1u) << (threadIdx.x & 31 & ~(kGroup - 1));
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;  // the lanes before this one
    GroupScratch& G = s_group[threadIdx.x / kGroup];
    int i = blockIdx.x * kSlots + threadIdx.x / kGroup;
    if constexpr (kSorted) {
        if (i >= g.cursor[0]) return;  // the whole group; inactive particles have no entry and need no delta
        i = g.entry[i].y;
    } else {
        if (i >= pd.particle_count || !active(pd, i)) return;
    }
    const float* xq = io.particle_q_out;
    const float* vq = io.particle_qd_out;
    const V3 x = ld3(xq, i), v = ld3(vq, i);
    const float w1 = pd.particle_inv_mass[i], radius = pd.particle_radius[i];
    const int spring_lo = pd.spring_count > 0 ? pd.particle_spring_start[i] : 0;
    const int spring_hi = pd.spring_count > 0 ? pd.particle_spring_start[i + 1] : 0;
    const int soft_lo = has_sc ? sc.particle_start[i] : 0;
    const int soft_hi = has_sc ? min(sc.particle_start[i + 1], min(sc.max, sc.count[0])) : 0;
    if (lane == 0) G.n = 0;
    __syncwarp(gmask);

    if (g.on) {
        const float reach = (radius + pd.particle_max_radius + pd.particle_cohesion) * 1.001f + 1.0e-6f;
        // the reach is at most ~1 cell (cell size 2 * max radius + cohesion), so a span of 3 cells per axis
        const int x0 = cell_of(x.x - reach, g.inv_h), x1 = last_cell(x.x + reach, g.inv_h, x0);
        const int y0 = cell_of(x.y - reach, g.inv_h), y1 = last_cell(x.y + reach, g.inv_h, y0);
        const int z0 = cell_of(x.z - reach, g.inv_h), z1 = last_cell(x.z + reach, g.inv_h, z0);
        // tests candidate j exactly
        auto consider = [&](int j) {
            const V3 xj = ld3(xq, j);
            const float rj = pd.particle_radius[j], wj = pd.particle_inv_mass[j];
            const int cx = cell_of(xj.x, g.inv_h), cy = cell_of(xj.y, g.inv_h), cz = cell_of(xj.z, g.inv_h);
            const V3 n = sub(x, xj);
            const float d = length(n);
            const float err = d - radius - rj;
            const float denom = w1 + wj;
            if (cx >= x0 && cx <= x1 && cy >= y0 && cy <= y1 && cz >= z0 && cz <= z1 && err <= pd.particle_cohesion &&
                denom > 0.0f) {
                const int at = atomicAdd(&G.n, 1);
                if (at < NB_PARTICLE_MAX_NEIGHBORS) G.j[at] = j;
            }
        };
        const int ny = y1 - y0 + 1, rows = ny * (z1 - z0 + 1);
        if constexpr (kSorted) {
            // squared reach in the packed positions' units: a packed difference is off by less than 1 per
            // axis, and by the rounding of x * inv_h far from the origin; past half the packed period
            // nothing is rejected, nor is a particle larger than the reach counts on
            const float far = fmaxf(fabsf(x.x), fmaxf(fabsf(x.y), fabsf(x.z))) + reach;
            const float ru = (reach * 256.0f + far * 1.0e-4f) * g.inv_h + 2.0f;
            const int r2 = ru < 500.0f ? (int)(ru * ru) + 1 : 0x7fffffff;
            const uint32_t mine = pack_pos(x, g.inv_h);
            const uint32_t bm = min((uint32_t)kRangeBuckets - 1u, g.mask);
            // a candidate belongs to the row it is met in (rows may share buckets): by its cells' low two
            // bits, which tell up to 4 rows apart, or by its cells where there are 5
            const bool wide = ny > 4 || rows > 4 * ny;
            for (int r0 = 0; r0 < rows; r0 += kGroup) {
                // each lane looks one row up: one run of entries, or two where the row leaves its block
                const int r = r0 + lane;
                int beg = 0, len = 0, beg2 = 0, tot = 0;
                uint32_t key = 0u;
                if (r < rows) {
                    const int rz = (int)__fdividef((float)r + 0.5f, (float)ny);  // r / ny: both below 32
                    const int cy = y0 + r - rz * ny, cz = z0 + rz;
                    key = (((uint32_t)cy & 3u) << 18) | (((uint32_t)cz & 3u) << 28);
                    const uint32_t b = cell_hash(x0, cy, cz, g.mask);
                    const uint32_t e = b + (uint32_t)(x1 - x0), cut = b | bm;
                    beg = g.first[bucket_at(b)];
                    len = g.first[bucket_at(min(e, cut)) + 1] - beg;
                    tot = len;
                    if (e > cut) {
                        beg2 = g.first[bucket_at((cut + 1u) & g.mask)];
                        tot += g.first[bucket_at(e & g.mask) + 1] - beg2;
                    }
                }
                int run = tot;
#pragma unroll
                for (int o = 1; o < kGroup; o <<= 1) {
                    const int y = __shfl_up_sync(gmask, run, o, kGroup);
                    if (lane >= o) run += y;
                }
                const int total = __shfl_sync(gmask, run, kGroup - 1, kGroup);
                if (total <= 0) continue;
                run -= tot;
                G.seg[2 * lane] = make_int4(beg - run, run + len, (int)key, r);
                G.seg[2 * lane + 1] = make_int4(beg2 - run - len, run + tot, (int)key, r);
                __syncwarp(gmask);
                int q = 0, nm = 0;  // nm: candidates listed, the same number in every lane
                int4 seg = G.seg[0];
                for (int base = 0; base < total; base += kAhead * kGroup) {
                    int2 en[kAhead];
                    uint32_t row_key[kAhead];
#pragma unroll
                    for (int u = 0; u < kAhead; ++u) {
                        const int a = base + u * kGroup + lane;
                        en[u].y = i;  // none
                        if (a < total) {
                            while (a >= seg.y) seg = G.seg[++q];
                            en[u] = g.entry[seg.x + a];
                            row_key[u] = (uint32_t)seg.z;
                            if (wide) {
                                const V3 xj = ld3(xq, en[u].y);
                                const int rz = seg.w / ny;
                                if (cell_of(xj.y, g.inv_h) != y0 + seg.w - rz * ny ||
                                    cell_of(xj.z, g.inv_h) != z0 + rz)
                                    en[u].y = i;
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kAhead; ++u) {
                        const uint32_t w = (uint32_t)en[u].x;
                        const int dx = (int)((w - mine) << 22) >> 22;
                        const int dy = (int)(((w >> 10) - (mine >> 10)) << 22) >> 22;
                        const int dz = (int)(((w >> 20) - (mine >> 20)) << 22) >> 22;
                        const bool keep = en[u].y != i && ((w ^ row_key[u]) & 0x300C0000u) == 0u &&
                                          (dx * dx + dy * dy + dz * dz <= r2 || (w & kLargeEntry) != 0u);
                        const unsigned kept = __ballot_sync(gmask, keep) & gmask;
                        if (keep) G.maybe[nm + __popc(kept & below)] = en[u].y;
                        nm += __popc(kept);
                    }
                    // the list is tested when another round might not fit, and at the end; every lane counts
                    // it from the ballots, so that the whole group comes here or goes on to the next round
                    if (nm > kMaybe - kAhead * kGroup || base + kAhead * kGroup >= total) {
                        __syncwarp(gmask);  // the list is visible
                        for (int a = lane; a < nm; a += kGroup) consider(G.maybe[a]);
                        __syncwarp(gmask);  // ... and read
                        nm = 0;
                    }
                }
            }
        } else {
            const int nx = x1 - x0 + 1, ncell = nx * rows;
            const int32_t* head = g.head + (size_t)table * (g.mask + 1u);
            for (int c = lane; c < ncell; c += kGroup) {
                const int cx = x0 + c % nx, cy = y0 + (c / nx) % ny, cz = z0 + c / (nx * ny);
                for (int j = head[cell_hash(cx, cy, cz, g.mask)]; j >= 0; j = g.next[j]) {
                    if (j == i) continue;
                    const V3 xj = ld3(xq, j);
                    // each particle sits in one cell: skip other cells hashed to this bucket
                    if (cell_of(xj.x, g.inv_h) == cx && cell_of(xj.y, g.inv_h) == cy && cell_of(xj.z, g.inv_h) == cz)
                        consider(j);
                }
            }
            __syncwarp(gmask);
        }
        if (lane == 0 && G.n > NB_PARTICLE_MAX_NEIGHBORS) atomicOr(io.status, NB_STATUS_NEIGHBOR_OVERFLOW);
        const int count = min(G.n, NB_PARTICLE_MAX_NEIGHBORS);
        for (int a = lane; a < count; a += kGroup) {
            const int j = G.j[a];
            const V3 vj = ld3(vq, j);
            V3 n = sub(x, ld3(xq, j));
            const float d = length(n);
            const float err = d - radius - pd.particle_radius[j];
            const float denom = w1 + pd.particle_inv_mass[j];
            int rank = 0;
            for (int b = 0; b < count; ++b) rank += G.j[b] < j ? 1 : 0;
            n = divs(n, d);
            const V3 vrel = sub(v, vj);
            const float lambda_n = err;
            const V3 delta_n = mul(n, lambda_n);
            const float vn = dot(n, vrel);
            const V3 vt = sub(vrel, mul(n, vn));
            const float lambda_f = fmaxw(pd.particle_mu * lambda_n, -length(vt) * dt);
            const V3 delta_f = mul(normalize(vt), lambda_f);
            const V3 contrib = divs(sub(delta_f, delta_n), denom);
            G.c[rank][0] = contrib.x;
            G.c[rank][1] = contrib.y;
            G.c[rank][2] = contrib.z;
        }
        __syncwarp(gmask);
    }

    V3 delta = V3{0.0f, 0.0f, 0.0f};
    for (int k = soft_lo; k < soft_hi; ++k) {
        const int s = sc.shape[k];
        // static shape: identity body transform, zero body velocity
        const TF X_wb = tf_identity();
        const V3 bx = tf_point(X_wb, ld3(sc.body_pos, k));
        const V3 r = sub(bx, tf_point(X_wb, V3{0.0f, 0.0f, 0.0f}));
        const V3 n = ld3(sc.normal, k);
        const V3 body_vel = ld3(sc.body_vel, k);
        const float mu = 0.5f * (pd.soft_contact_mu + pd.shape_mu[s]);
        if (pd.shape_body[s] >= 0) {
            if (lane == 0) atomicOr(io.status, NB_STATUS_PARTICLE_BODY_CONTACT);
            continue;
        }
        const float c = dot(n, sub(x, bx)) - radius;
        if (c > pd.particle_adhesion) continue;
        const V3 body_w = V3{0.0f, 0.0f, 0.0f}, body_v = V3{0.0f, 0.0f, 0.0f};
        const V3 bv = add(add(body_v, cross(body_w, r)), tf_vector(X_wb, body_vel));
        const V3 vr = sub(v, bv);
        const float lambda_n = c;
        const V3 delta_n = mul(n, lambda_n);
        const float vn = dot(n, vr);
        const V3 vt = sub(vr, mul(n, vn));
        const float denom = w1 + 0.0f;
        if (denom == 0.0f) continue;
        const float lambda_f = fmaxw(mu * lambda_n, -length(vt) * dt);
        const V3 delta_f = mul(normalize(vt), lambda_f);
        const V3 delta_total = mul(divs(sub(delta_f, delta_n), denom), relaxation);
        delta = add(delta, smul(w1, delta_total));
    }

    if (g.on) {
        const int count = min(G.n, NB_PARTICLE_MAX_NEIGHBORS);
        V3 dpp = V3{0.0f, 0.0f, 0.0f};
        for (int k = 0; k < count; ++k) {
            const float* c = G.c[k];
            dpp = add(dpp, V3{c[0], c[1], c[2]});
        }
        delta = add(delta, mul(mul(dpp, w1), relaxation));
    }

    {
        const int s_hi = spring_hi;
        for (int k0 = spring_lo; k0 < s_hi; k0 += kGroup) {
            // each lane one spring: its direction (toward increasing delta of particle i) and magnitude
            V3 dir = V3{0.0f, 0.0f, 0.0f};
            float mag = 0.0f;
            bool on = false;
            if (k0 + lane < s_hi) {
                const int s = pd.particle_spring_list[k0 + lane];
                const int a = pd.spring_indices[2 * s], b = pd.spring_indices[2 * s + 1];
                const float ke = pd.spring_stiffness[s], kd = pd.spring_damping[s], rest = pd.spring_rest_length[s];
                const V3 xij = sub(ld3(xq, a), ld3(xq, b));
                const V3 vij = sub(ld3(vq, a), ld3(vq, b));
                const float l = length(xij);
                const V3 n = divs(xij, l);
                const float c = l - rest;
                const float wi = pd.particle_inv_mass[a], wj = pd.particle_inv_mass[b];
                const float denom = wi + wj;
                on = l != 0.0f && !(denom <= 0.0f || ke <= 0.0f || kd < 0.0f);
                const float alpha = 1.0f / (ke * dt * dt);
                const float gamma = kd / (ke * dt);
                const float grad_c_dot_v = dt * dot(n, vij);
                const float lambda_prev = 0.0f;  // the solver zeroes the spring multipliers every iteration
                const float dlambda =
                    -1.0f * (c + alpha * lambda_prev + gamma * grad_c_dot_v) / ((1.0f + gamma) * denom + alpha);
                // a spring's ends are two particles (l != 0)
                dir = i == a ? n : smul(-1.0f, n);
                mag = i == a ? wi * dlambda : wj * dlambda;
            }
            const int nk = min(s_hi - k0, kGroup);
            for (int k = 0; k < nk; ++k) {
                const V3 kd3 = V3{__shfl_sync(gmask, dir.x, k, kGroup), __shfl_sync(gmask, dir.y, k, kGroup),
                                  __shfl_sync(gmask, dir.z, k, kGroup)};
                const float km = __shfl_sync(gmask, mag, k, kGroup);
                if (__shfl_sync(gmask, on ? 1 : 0, k, kGroup)) delta = add(delta, mul(kd3, km));
            }
        }
    }
    if (lane == 0) st3(io.delta, i, delta);
}

NB_D float det3(const M33& m) {
    return m.m[0][0] * (m.m[1][1] * m.m[2][2] - m.m[1][2] * m.m[2][1]) -
           m.m[0][1] * (m.m[1][0] * m.m[2][2] - m.m[1][2] * m.m[2][0]) +
           m.m[0][2] * (m.m[1][0] * m.m[2][1] - m.m[1][1] * m.m[2][0]);
}
NB_D M33 matmul3(const M33& a, const M33& b) {
    M33 r;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) r.m[i][j] = a.m[i][0] * b.m[0][j] + a.m[i][1] * b.m[1][j] + a.m[i][2] * b.m[2][j];
    return r;
}
NB_D M33 from_cols(V3 a, V3 b, V3 c) {
    M33 r;
    r.m[0][0] = a.x; r.m[1][0] = a.y; r.m[2][0] = a.z;
    r.m[0][1] = b.x; r.m[1][1] = b.y; r.m[2][1] = b.z;
    r.m[0][2] = c.x; r.m[1][2] = c.y; r.m[2][2] = c.z;
    return r;
}
NB_D V3 col(const M33& m, int c) { return V3{m.m[0][c], m.m[1][c], m.m[2][c]}; }

// One lane's terms: up to 4 vertices' corrections grad * mag (bit r of `on` when vertex r is the
// particle and the term is live).
struct ElemTerms {
    V3 grad[4];
    float mag[4];
    unsigned on;
};

// The terms of the group's first `lanes` lanes added to every lane's delta, lane after lane, vertex after
// vertex.
template <int kLanes>
NB_D V3 add_terms(const ElemTerms& t, unsigned gmask, int lanes, V3 delta) {
    if constexpr (kLanes == 1) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if ((t.on >> r) & 1u) delta = add(delta, mul(t.grad[r], t.mag[r]));
    } else {
        for (int k = 0; k < lanes; ++k) {
            const unsigned on = __shfl_sync(gmask, t.on, k, kLanes);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (!((on >> r) & 1u)) continue;
                const V3 gr = V3{__shfl_sync(gmask, t.grad[r].x, k, kLanes),
                                 __shfl_sync(gmask, t.grad[r].y, k, kLanes),
                                 __shfl_sync(gmask, t.grad[r].z, k, kLanes)};
                delta = add(delta, mul(gr, __shfl_sync(gmask, t.mag[r], k, kLanes)));
            }
        }
    }
    return delta;
}

// One bending edge (bending_constraint, kernels.py:358-457) as seen by particle i.
NB_D void edge_terms(const NbParticleDesc& pd, const float* xq, const float* vq, int i, int e, float dt,
                     ElemTerms& t) {
    t.on = 0u;
    const int* ix = pd.edge_indices + 4 * e;
    const float ke = pd.edge_bending_properties[2 * e], kd = pd.edge_bending_properties[2 * e + 1];
    const V3 x1 = ld3(xq, ix[0]), x2 = ld3(xq, ix[1]), x3 = ld3(xq, ix[2]), x4 = ld3(xq, ix[3]);
    const float w[4] = {pd.particle_inv_mass[ix[0]], pd.particle_inv_mass[ix[1]], pd.particle_inv_mass[ix[2]],
                        pd.particle_inv_mass[ix[3]]};
    const V3 n1 = cross(sub(x3, x1), sub(x4, x1));
    const V3 n2 = cross(sub(x4, x2), sub(x3, x2));
    const V3 ev = sub(x4, x3);
    const float n1_length = length(n1), n2_length = length(n2), e_length = length(ev);
    if (n1_length < 1.0e-6f || n2_length < 1.0e-6f || e_length < 1.0e-6f) return;
    const V3 n1_hat = divs(n1, n1_length), n2_hat = divs(n2, n2_length), e_hat = divs(ev, e_length);
    const float cos_theta = dot(n1_hat, n2_hat);
    const float sin_theta = dot(cross(n1_hat, n2_hat), e_hat);
    const float c = nb_atan2(sin_theta, cos_theta) - pd.edge_rest_angle[e];
    V3* grad = t.grad;
    grad[0] = mul(neg(n1_hat), e_length);
    grad[1] = mul(neg(n2_hat), e_length);
    grad[2] = sub(mul(neg(n1_hat), dot(sub(x1, x4), e_hat)), mul(n2_hat, dot(sub(x2, x4), e_hat)));
    grad[3] = sub(mul(neg(n1_hat), dot(sub(x3, x1), e_hat)), mul(n2_hat, dot(sub(x3, x2), e_hat)));
    const float denominator = w[0] * length_sq(grad[0]) + w[1] * length_sq(grad[1]) + w[2] * length_sq(grad[2]) +
                              w[3] * length_sq(grad[3]);
    if (denominator <= 0.0f || ke <= 0.0f || kd < 0.0f) return;
    const float alpha = 1.0f / (ke * dt * dt);
    const float gamma = kd / (ke * dt);
    const float grad_dot_v = dt * (dot(grad[0], ld3(vq, ix[0])) + dot(grad[1], ld3(vq, ix[1])) +
                                   dot(grad[2], ld3(vq, ix[2])) + dot(grad[3], ld3(vq, ix[3])));
    const float lambda_prev = 0.0f;
    const float dlambda =
        -1.0f * (c + alpha * lambda_prev + gamma * grad_dot_v) / ((1.0f + gamma) * denominator + alpha);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        t.mag[r] = w[r] * dlambda;
        if (ix[r] == i) t.on |= 1u << r;
    }
}

// The two terms of a tetrahedron (solve_tetrahedra, kernels.py:459-628) as seen by particle i, added to its
// delta: the stretch (trace(F^T F) - 3), then the volume (det F - 1), each a compliant constraint with
// compliance `relaxation` (the solver's soft_body_relaxation) scaled by the inverse rest volume.
NB_D V3 tet_terms(const NbParticleDesc& pd, const float* xq, int i, int e, float dt, V3 delta) {
    const int* ix = pd.tet_indices + 4 * e;
    const V3 x0 = ld3(xq, ix[0]), x1 = ld3(xq, ix[1]), x2 = ld3(xq, ix[2]), x3 = ld3(xq, ix[3]);
    const float w[4] = {pd.particle_inv_mass[ix[0]], pd.particle_inv_mass[ix[1]], pd.particle_inv_mass[ix[2]],
                        pd.particle_inv_mass[ix[3]]};
    const M33 Ds = from_cols(sub(x1, x0), sub(x2, x0), sub(x3, x0));
    M33 Dm, inv_QT;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) Dm.m[r][c] = pd.tet_poses[9 * e + 3 * r + c];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) inv_QT.m[r][c] = Dm.m[c][r];
    const float inv_rest_volume = det3(Dm) * 6.0f;
    const M33 Fm = matmul3(Ds, Dm);
    const V3 f1 = col(Fm, 0), f2 = col(Fm, 1), f3 = col(Fm, 2);
    const float tr = dot(f1, f1) + dot(f2, f2) + dot(f3, f3);
    for (int term = 0; term < 2; ++term) {
        float C;
        M33 dC;
        if (term == 0) {
            C = tr - 3.0f;
            for (int r = 0; r < 3; ++r)
                for (int c = 0; c < 3; ++c) dC.m[r][c] = Fm.m[r][c] * 2.0f;
        } else {
            C = det3(Fm) - 1.0f;
            dC = from_cols(cross(f2, f3), cross(f3, f1), cross(f1, f2));
        }
        if (C == 0.0f) continue;
        const M33 dP = matmul3(dC, inv_QT);
        V3 grad[4];
        grad[1] = col(dP, 0);
        grad[2] = col(dP, 1);
        grad[3] = col(dP, 2);
        grad[0] = sub(sub(neg(grad[1]), grad[2]), grad[3]);
        const float wsum = dot(grad[0], grad[0]) * w[0] + dot(grad[1], grad[1]) * w[1] +
                           dot(grad[2], grad[2]) * w[2] + dot(grad[3], grad[3]) * w[3];
        if (!(wsum > 0.0f)) continue;
        float alpha = pd.soft_body_relaxation / dt / dt;
        if (inv_rest_volume > 0.0f) alpha *= inv_rest_volume;
        const float dlambda = -C / (wsum + alpha);
        for (int r = 0; r < 4; ++r)
            if (ix[r] == i) delta = add(delta, mul(grad[r], w[r] * dlambda));
    }
    return delta;
}

// Bending edges, then tetrahedra, of one particle, added to its delta after the constraint kernel's terms
// (the same order as one sequential sum).  A kernel of its own so that the constraint kernel keeps its
// register budget.  The solver zeroes the multipliers every iteration.  kLanes lanes serve one particle: an
// inner cloth particle has 4 bending edges, so with 4 each lane computes one, and the lanes then add all of
// them in ascending index; tetrahedra, whose two terms share most of their work, take one lane.  Which form
// runs: elements_by_lanes below.
template <int kLanes>
__global__ void __launch_bounds__(kThreads) particle_bending_kernel(NbParticleDesc pd, NbParticleIO io, float dt) {
    const int lane = threadIdx.x & (kLanes - 1);
    const unsigned gmask = ((1u << kLanes) - 1u) << (threadIdx.x & 31 & ~(kLanes - 1));
    const int i = blockIdx.x * (kThreads / kLanes) + threadIdx.x / kLanes;
    if (i >= pd.particle_count) return;
    const int e_lo = pd.edge_count > 0 ? pd.particle_edge_start[i] : 0;
    const int e_hi = pd.edge_count > 0 ? pd.particle_edge_start[i + 1] : 0;
    int t_lo = 0, t_hi = 0;
    if (kLanes == 1 && pd.tet_count > 0) {
        t_lo = pd.particle_tet_start[i];
        t_hi = pd.particle_tet_start[i + 1];
    }
    if (e_lo == e_hi && t_lo == t_hi) return;
    const float* xq = io.particle_q_out;
    const float* vq = io.particle_qd_out;
    V3 delta = ld3(io.delta, i);
    ElemTerms t;
    for (int k = e_lo; k < e_hi; k += kLanes) {
        t.on = 0u;
        if (k + lane < e_hi) edge_terms(pd, xq, vq, i, pd.particle_edge_list[k + lane], dt, t);
        delta = add_terms<kLanes>(t, gmask, min(e_hi - k, kLanes), delta);
    }
    if constexpr (kLanes == 1)
        for (int k = t_lo; k < t_hi; ++k) delta = tet_terms(pd, xq, i, pd.particle_tet_list[k], dt, delta);
    if (lane == 0) st3(io.delta, i, delta);
}

// apply_particle_deltas (kernels.py:776-807) for one active particle, in place; returns its new position.
NB_D V3 apply_delta(const NbParticleDesc& pd, const NbParticleIO& io, float dt, int p) {
    const V3 x0 = ld3(io.particle_q, p);
    const V3 xp = ld3(io.particle_q_out, p);
    const V3 x_new = add(xp, ld3(io.delta, p));
    V3 v_new = divs(sub(x_new, x0), dt);
    const float v_mag = length(v_new);
    if (v_mag > pd.particle_max_velocity) v_new = mul(v_new, pd.particle_max_velocity / v_mag);
    st3(io.particle_q_out, p, x_new);
    st3(io.particle_qd_out, p, v_new);
    return x_new;
}

// The deltas applied; then each particle is counted into its bucket of the next iteration's grid.
__global__ void __launch_bounds__(kThreads) particle_apply_kernel(NbParticleDesc pd, NbParticleIO io, float dt,
                                                                  Grid g, int next_table, int insert) {
    const int p = blockIdx.x * kThreads + threadIdx.x;
    if (p == 0 && g.sorted) g.cursor[0] = 0;  // for the next iteration's ranges
    if (p >= pd.particle_count || !active(pd, p)) return;
    const V3 x_new = apply_delta(pd, io, dt, p);
    if (insert) grid_insert(g, next_table, p, x_new);
}

// One block applies the deltas (`apply`; the first grid of a substep has none yet) and rebuilds the whole
// grid: counts in shared memory, their scan, ranges and entries.  It saves two launches of the three kernels it
// replaces (apply, ranges, scatter), and its one SM's work grows with the particles where theirs is latency.
// us per substep of 4 iterations, one block / three kernels, launched one by one: 1,902 particles 114 / 130,
// 2,560 122 / 132, 3,072 123 / 132, 3,584 132 / 133, 4,096 131 / 131; replayed from a captured graph, where
// launches cost less: 88 / 92, 96 / 91, 101 / 94, 106 / 94, 108 / 88.  The line is between the two crossings.
__global__ void __launch_bounds__(1024) particle_regrid_kernel(NbParticleDesc pd, NbParticleIO io, float dt, Grid g,
                                                               int apply) {
    constexpr int kT = 1024, kPer = kSmallParticles / kT, kBuckets = kSmallBuckets / kT;  // per thread
    __shared__ int s_count[kSmallBuckets];
    __shared__ int s_warp[kT / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int M = (int)g.mask + 1;
    for (int b = t; b < M; b += kT) s_count[b] = 0;
    __syncthreads();
    int bucket[kPer], rank[kPer];
    uint32_t word[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int p = t + k * kT;
        bucket[k] = -1;
        if (p >= pd.particle_count || !active(pd, p)) continue;
        const V3 x = apply ? apply_delta(pd, io, dt, p) : ld3(io.particle_q_out, p);
        bucket[k] = (int)cell_hash(cell_of(x.x, g.inv_h), cell_of(x.y, g.inv_h), cell_of(x.z, g.inv_h), g.mask);
        word[k] = entry_word(pd, p, x, g.inv_h);
        rank[k] = atomicAdd(&s_count[bucket[k]], 1);
    }
    __syncthreads();
    int c[kBuckets], sum = 0;
#pragma unroll
    for (int k = 0; k < kBuckets; ++k) {
        const int b = t * kBuckets + k;
        c[k] = b < M ? s_count[b] : 0;
        sum += c[k];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        s_warp[lane] = w;
        if (lane == 31) g.cursor[0] = w;
    }
    __syncthreads();
    int at = x - sum + (warp > 0 ? s_warp[warp - 1] : 0);
#pragma unroll
    for (int k = 0; k < kBuckets; ++k) {
        const int b = t * kBuckets + k;
        if (b < M) {
            g.first[bucket_at(b)] = at;
            s_count[b] = at;  // this thread alone reads and writes bucket b here
            if (b == M - 1 || b % kRangeBuckets == kRangeBuckets - 1) g.first[bucket_at(b) + 1] = at + c[k];
        }
        at += c[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (bucket[k] >= 0) g.entry[s_count[bucket[k]] + rank[k]] = make_int2((int)word[k], t + k * kT);
}

// apply_particle_shape_restitution (kernels.py:34-112) for static shapes: contacts tested at the
// substep's start position; each particle adds the velocity change of its contacts, in list order, to
// its velocity after the iterations (every change computed from that velocity).
__global__ void __launch_bounds__(kThreads) particle_restitution_kernel(NbParticleDesc pd, NbParticleIO io,
                                                                        NbSoftContacts sc) {
    const int p = blockIdx.x * kThreads + threadIdx.x;
    if (p >= pd.particle_count || !active(pd, p)) return;
    const int lim = min(sc.max, sc.count[0]);
    const int lo = sc.particle_start[p], hi = min(sc.particle_start[p + 1], lim);
    if (lo >= hi) return;
    const V3 v_new = ld3(io.particle_qd_out, p);
    const V3 px = ld3(io.particle_q, p);
    const V3 v_old = ld3(io.particle_qd, p);
    V3 v_out = v_new;
    for (int k = lo; k < hi; ++k) {
        if (pd.shape_body[sc.shape[k]] >= 0) continue;  // body-attached shapes: not coupled
        const TF X_wb = tf_identity(), X_wb_prev = tf_identity();
        const V3 bx = tf_point(X_wb, ld3(sc.body_pos, k));
        const V3 n = ld3(sc.normal, k);
        const float c = dot(n, sub(px, bx)) - pd.particle_radius[p];
        if (c > pd.particle_adhesion) continue;
        const V3 bv_contact = tf_vector(X_wb_prev, ld3(sc.body_vel, k));
        const float rel_vel_old = dot(n, sub(v_old, bv_contact));
        const float rel_vel_new = dot(n, sub(v_new, bv_contact));
        if (rel_vel_old < 0.0f) {
            const V3 dv = mul(n, -rel_vel_new + fmaxw(-pd.soft_contact_restitution * rel_vel_old, 0.0f));
            v_out = add(v_out, dv);
        }
    }
    st3(io.particle_qd_out, p, v_out);
}

bool check_pd(const NbParticleDesc* pd) {
    if (!pd || pd->particle_count < 0 || pd->spring_count < 0 || pd->shape_count < 0 || pd->world_count < 1)
        return false;
    if (pd->particle_count == 0) return true;
    if (!pd->particle_inv_mass || !pd->particle_radius || !pd->particle_flags || !pd->particle_world ||
        !pd->gravity)
        return false;
    if (pd->spring_count > 0 && (!pd->spring_indices || !pd->spring_rest_length || !pd->spring_stiffness ||
                                 !pd->spring_damping || !pd->particle_spring_start || !pd->particle_spring_list))
        return false;
    if (pd->tet_count < 0 || (pd->tet_count > 0 && (!pd->tet_indices || !pd->tet_poses || !pd->particle_tet_start ||
                                                     !pd->particle_tet_list)))
        return false;
    if (pd->edge_count < 0 || (pd->edge_count > 0 && (!pd->edge_indices || !pd->edge_rest_angle ||
                                                       !pd->edge_bending_properties || !pd->particle_edge_start ||
                                                       !pd->particle_edge_list)))
        return false;
    if (pd->shape_count > 0 && (!pd->shape_body || !pd->shape_type || !pd->shape_transform || !pd->shape_scale ||
                                !pd->shape_world || !pd->shape_flags || !pd->shape_mu))
        return false;
    return true;
}

// Lays the neighbour search out in the caller's scratch: grid_head [2 n] and grid_next [P].  The sorted form
// keeps its entries, buckets and cursor in grid_head, and the counts of its M buckets in grid_next where they fit
// (M <= P), else in grid_head too.  M is the largest power of two below 2 P that fits: with about one particle
// per bucket few strangers are met.  Below P / 4 buckets, or kMinSorted, the lists, which use all n buckets, are
// taken.  n >= 2 P holds the sorted form for P > 8.
cudaError_t grid_layout(Grid& g, const NbParticleIO* io, int P, cudaStream_t st) {
    const long long room = 2LL * io->grid_size - 1;  // ints, after up to one to align
    auto ints = [&](long long M) {
        return 2LL * P + M + (M + kRangeBuckets - 1) / kRangeBuckets + 1 + (M > P ? M : 0);
    };
    long long M = 1;
    while (M < P) M *= 2;
    while (M > 1 && ints(M) > room) M /= 2;
    g.sorted = M >= kMinSorted && 4 * M >= P && ints(M) <= room;
    if (!g.sorted) {
        g.head = io->grid_head;
        g.next = io->grid_next;
        g.mask = (uint32_t)io->grid_size - 1u;
        return cudaMemsetAsync(g.head, 0xff, sizeof(int32_t) * (size_t)io->grid_size, st);
    }
    int32_t* base = io->grid_head + (((uintptr_t)io->grid_head & 7u) ? 1 : 0);
    g.entry = reinterpret_cast<int2*>(base);
    g.first = base + 2LL * P;
    g.cursor = g.first + bucket_at((uint32_t)M - 1u) + 2;
    g.count = M > P ? g.cursor + 1 : io->grid_next;
    g.mask = (uint32_t)(M - 1);
    g.small = P <= kSmallParticles;
    if (g.small) return cudaSuccess;
    return cudaMemsetAsync(g.count, 0, sizeof(int32_t) * (size_t)M, st);
}

// Whether a particle's bending edges get 4 lanes.  They shorten its chain, but repeat its loads and sums: worth
// it while the blocks with edges (about one particle per edge, 64 to a block) run all at once, 2 per SM, and the
// blocks without do not count.  us per substep of 4 iterations (148 SMs), 4 lanes / 1: sheets of 3,604 / 10,004 /
// 16,904 / 19,604 / 40,004 particles 45 / 58, 57 / 70, 64 / 76, 80 / 78, 125 / 110; a sheet of 10,000 beside
// 100,000 / 200,000 / 300,000 loose particles 408 / 422, 715 / 718, 965 / 964.  Tetrahedra share most of their
// two terms' work in one lane: blocks of 125 / 4,096 / 29,791 particles, the terms on lanes of their own 147 /
// 180 / 349, in one 107 / 181 / 237.
bool elements_by_lanes(const NbParticleDesc& pd) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long wave = 2LL * sms * (kThreads / 4);
    return pd.tet_count == 0 && pd.edge_count <= wave && pd.particle_count <= 12 * wave;
}

void launch_bending(const NbParticleDesc& pd, const NbParticleIO& io, float dt, cudaStream_t st) {
    const int P = pd.particle_count;
    if (elements_by_lanes(pd))
        particle_bending_kernel<4><<<(P + kThreads / 4 - 1) / (kThreads / 4), kThreads, 0, st>>>(pd, io, dt);
    else
        particle_bending_kernel<1><<<(P + kThreads - 1) / kThreads, kThreads, 0, st>>>(pd, io, dt);
}

}  // namespace

extern "C" {

int nb_soft_collide(const NbParticleDesc* pd, const float* particle_q, const float* body_q,
                    const NbSoftContacts* sc, void* stream) {
    if (!check_pd(pd) || !sc || !sc->count || sc->max < 0) return NB_ERR_INVALID;
    const cudaStream_t st = (cudaStream_t)stream;
    const int P = pd->particle_count;
    if (P == 0 || pd->shape_count == 0)
        return nb_cuda_rc(cudaMemsetAsync(sc->count, 0, sizeof(int32_t), st));
    if (!particle_q || !sc->particle_start) return NB_ERR_INVALID;
    if (sc->max > 0 && (!sc->particle || !sc->shape || !sc->body_pos || !sc->body_vel || !sc->normal))
        return NB_ERR_INVALID;
    const int blocks = (P + kScanThreads - 1) / kScanThreads;
    soft_count_kernel<<<blocks, kScanThreads, 0, st>>>(*pd, particle_q, body_q, *sc);
    soft_scan_blocks_kernel<<<1, kScanThreads, 0, st>>>(*pd, *sc, blocks);
    soft_write_kernel<<<blocks, kScanThreads, 0, st>>>(*pd, particle_q, body_q, *sc);
    return nb_cuda_rc(cudaGetLastError());
}

int nb_particle_step(const NbParticleDesc* pd, const NbParticleIO* io, const NbSoftContacts* sc, float dt,
                     int32_t iterations, float relaxation, void* stream) {
    if (!check_pd(pd) || !io || iterations < 0 || !(dt > 0.0f)) return NB_ERR_INVALID;
    const int P = pd->particle_count;
    if (P == 0) return NB_OK;
    if (!io->particle_q || !io->particle_qd || !io->particle_q_out || !io->particle_qd_out || !io->delta ||
        !io->status)
        return NB_ERR_INVALID;
    if (sc && (!sc->count || !sc->particle_start || sc->max < 0 ||
               (sc->max > 0 && (!sc->shape || !sc->body_pos || !sc->body_vel || !sc->normal))))
        return NB_ERR_INVALID;
    const cudaStream_t st = (cudaStream_t)stream;
    Grid g{};
    g.on = pd->particle_max_radius > 0.0f && P > 1;
    if (g.on) {
        const float h = 2.0f * pd->particle_max_radius + pd->particle_cohesion;
        const int32_t n = io->grid_size;
        if (!io->grid_head || !io->grid_next || n <= 0 || (n & (n - 1)) != 0 || !(h > 0.0f)) return NB_ERR_INVALID;
        g.inv_h = 1.0f / h;
        const cudaError_t e = grid_layout(g, io, P, st);
        if (e != cudaSuccess) return nb_cuda_rc(e);
    }
    NbSoftContacts none{};
    const int has_sc = sc != nullptr && pd->shape_count > 0;
    const NbSoftContacts scv = sc ? *sc : none;
    const int blocks = (P + kThreads - 1) / kThreads;
    particle_integrate_kernel<<<blocks, kThreads, 0, st>>>(*pd, *io, dt, g);
    const int con_blocks = (P + kSlots - 1) / kSlots;
    for (int it = 0; it < iterations; ++it) {
        const int table = it & 1;
        if (g.on && g.sorted) {
            if (!g.small) {
                particle_ranges_kernel<<<(g.mask + kRangeBuckets) / kRangeBuckets, kThreads, 0, st>>>(g);
                particle_scatter_kernel<<<blocks, kThreads, 0, st>>>(*pd, io->particle_q_out, g);
            } else if (it == 0) {
                particle_regrid_kernel<<<1, 1024, 0, st>>>(*pd, *io, dt, g, 0);
            }
            particle_constraints_kernel<true><<<con_blocks, kThreads, 0, st>>>(*pd, *io, scv, has_sc, dt, relaxation,
                                                                               g, table);
        } else {
            particle_constraints_kernel<false><<<con_blocks, kThreads, 0, st>>>(*pd, *io, scv, has_sc, dt, relaxation,
                                                                                g, table);
        }
        if (pd->edge_count > 0 || pd->tet_count > 0)
            launch_bending(*pd, *io, dt, st);
        if (g.small && it + 1 < iterations)
            particle_regrid_kernel<<<1, 1024, 0, st>>>(*pd, *io, dt, g, 1);
        else
            particle_apply_kernel<<<blocks, kThreads, 0, st>>>(*pd, *io, dt, g, table ^ 1,
                                                               g.on && it + 1 < iterations ? 1 : 0);
    }
    if (io->enable_restitution && has_sc)
        particle_restitution_kernel<<<blocks, kThreads, 0, st>>>(*pd, *io, scv);
    return nb_cuda_rc(cudaGetLastError());
}

}  // extern "C"
