// Device rasteriser (material classes per E-component Yee point) and the
// combo/bounding-box passes that turn class maps into the stepper's
// one-byte-per-voxel material index.
//
// The CSG evaluation restates composite_object::in and the primitives'
// in() (src/cgs.cpp:34-120, 403-449) with the reference's operation order:
// matrix rows are summed left to right starting from 0 (src/geometry.hpp:88-99),
// dot products left to right (src/geometry.hpp:199-201), and no fused
// multiply-add, so that points lying exactly on a face get the same answer.
#include <cmath>

#include "sj_internal.h"

namespace sj {

__device__ __forceinline__ void mat_vec(const double* __restrict__ m, double x, double y, double z,
                                        double& ox, double& oy, double& oz) {
    ox = __dadd_rn(__dadd_rn(__dadd_rn(0.0, __dmul_rn(m[0], x)), __dmul_rn(m[1], y)), __dmul_rn(m[2], z));
    oy = __dadd_rn(__dadd_rn(__dadd_rn(0.0, __dmul_rn(m[3], x)), __dmul_rn(m[4], y)), __dmul_rn(m[5], z));
    oz = __dadd_rn(__dadd_rn(__dadd_rn(0.0, __dmul_rn(m[6], x)), __dmul_rn(m[7], y)), __dmul_rn(m[8], z));
}

// Which of a node's transforms are the identity: bit 0 the ancestors' (m),
// bit 1 the primitive's own (t).  At a finite point the product with an
// identity gives the point back, up to the sign of a zero, which no primitive
// can tell (t's point, r - c, is finite where neither number is near overflow);
// the flags are formed once per block.
constexpr int RASTER_MAX_NODES = SJ_MAX_CSG_NODES * SJ_MAX_REGIONS;
__device__ __forceinline__ bool is_identity(const double* m) {
    bool id = true;
    for (int q = 0; q < 9; ++q) {
        const unsigned long long w = (unsigned long long)__double_as_longlong(m[q]);
        id = id && (q % 4 == 0 ? w == 0x3ff0000000000000ull : (w << 1) == 0ull);
    }
    return id;
}
constexpr double MODERATE = 1e100, FAR = 1e307;
__device__ void identity_flags(const sj_csg_node* __restrict__ nodes, int n, bool finite, uint8_t* flags) {
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        const sj_csg_node& nd = nodes[q];
        const bool centre = fabs(nd.c[0]) < FAR && fabs(nd.c[1]) < FAR && fabs(nd.c[2]) < FAR;
        flags[q] = finite ? (uint8_t)((is_identity(nd.m) ? 1 : 0) | (centre && is_identity(nd.t) ? 2 : 0)) : 0;
    }
    __syncthreads();
}

// Do a row's ends decide every primitive of the scene (leaf_code)?  No
// transforms, and every number so far from overflow that no infinity or NaN can
// come up on the way.
bool raster_rows(const sj_scene_desc* sc, const double* offs, size_t n_offs) {
    for (size_t q = 0; q < n_offs; ++q)
        if (!(std::fabs(offs[q]) < MODERATE)) return false;
    auto identity = [](const double* m) {
        for (int q = 0; q < 9; ++q)
            if (m[q] != (q % 4 == 0 ? 1.0 : 0.0)) return false;
        return true;
    };
    for (int r = 0; r < sc->n_regions; ++r)
        for (int q = 0; q < sc->regions[r].n_nodes; ++q) {
            const sj_csg_node& nd = sc->regions[r].nodes[q];
            if (nd.op > SJ_CSG_PLANE) continue;
            if (!identity(nd.m) || !identity(nd.t)) return false;
            for (int a = 0; a < 4; ++a)
                if (!(std::fabs(nd.p[a]) < MODERATE)) return false;
            for (int a = 0; a < 3; ++a)
                if (!(std::fabs(nd.c[a]) < MODERATE)) return false;
        }
    return true;
}

// The operand stack after one operator
__device__ __forceinline__ unsigned long long combine(const sj_csg_node& nd, unsigned long long stk) {
    const int op = nd.op;
    if (op == SJ_CSG_UNION || op == SJ_CSG_INTERSECT) {
        const int b = (int)(stk & 1ull);
        stk >>= 1;
        const int a = (int)(stk & 1ull);
        stk >>= 1;
        return (stk << 1) | (unsigned long long)(nd.invert ^ (op == SJ_CSG_UNION ? (a | b) : (a & b)));
    }
    if (op == SJ_CSG_PASS) return (stk & ~1ull) | (unsigned long long)(nd.invert ^ (int)(stk & 1ull));
    if (op == SJ_CSG_CONST) return (stk << 1) | (unsigned long long)(nd.invert & 1);
    return stk << 1;  // NOOP
}

// Evaluate one region's postfix program at r; returns in_root(r) in {0,1}.
// The operand stack is a 64-bit word: push = shift left, pop = shift right.
// Bound by the FP64 pipe (19 cycles per warp operation and SM): a box under
// two identities costs three subtractions and three comparisons, z first (a
// thin film's z decides most points of a row at once), instead of 36
// operations.  256 x 256 x 192 bowtie scene, every point: 16.3 ms before, 2.9 ms.
__device__ int eval_program(const sj_csg_node* __restrict__ nodes, const uint8_t* flags, int n, double x, double y,
                            double z) {
    unsigned long long stk = 0;
    for (int q = 0; q < n; ++q) {
        const sj_csg_node& nd = nodes[q];
        const int op = nd.op;
        int v = 0;
        if (op <= SJ_CSG_PLANE) {
            const int id = flags[q];
            double rx = x, ry = y, rz = z;
            if (!(id & 1)) mat_vec(nd.m, x, y, z, rx, ry, rz);
            if (op == SJ_CSG_PLANE) {
                const double d = __dadd_rn(__dadd_rn(__dmul_rn(rx, nd.p[0]), __dmul_rn(ry, nd.p[1])),
                                           __dmul_rn(rz, nd.p[2]));
                v = d > nd.p[3] ? 0 : 1;
            } else {
                bool out;
                if (op == SJ_CSG_BOX && (id & 2)) {
                    out = fabs(__dsub_rn(rz, nd.c[2])) > nd.p[2] || fabs(__dsub_rn(ry, nd.c[1])) > nd.p[1] ||
                          fabs(__dsub_rn(rx, nd.c[0])) > nd.p[0];
                } else {
                    double qx = __dsub_rn(rx, nd.c[0]), qy = __dsub_rn(ry, nd.c[1]), qz = __dsub_rn(rz, nd.c[2]);
                    if (!(id & 2)) mat_vec(nd.t, qx, qy, qz, qx, qy, qz);
                    if (op == SJ_CSG_BOX) {
                        out = fabs(qx) > nd.p[0] || fabs(qy) > nd.p[1] || fabs(qz) > nd.p[2];
                    } else if (op == SJ_CSG_SPHERE) {
                        const double s2 = __dadd_rn(__dadd_rn(__dadd_rn(0.0, __dmul_rn(qx, qx)), __dmul_rn(qy, qy)),
                                                    __dmul_rn(qz, qz));
                        out = __dsqrt_rn(s2) > nd.p[0];
                    } else {  // cylinder: p = height, r1^2, r2^2
                        const double h = nd.p[0], r1 = nd.p[1], r2 = nd.p[2];
                        if (qz < 0 || qz > h) {
                            out = true;
                        } else {
                            const double cr = __dadd_rn(__dmul_rn(qx, qx), __dmul_rn(qy, qy));
                            out = __dmul_rn(cr, h) > __dadd_rn(__dmul_rn(__dsub_rn(r2, r1), qz), __dmul_rn(r1, h));
                        }
                    }
                }
                v = out ? nd.invert : 1 - nd.invert;
            }
            stk = (stk << 1) | (unsigned long long)v;
        } else {
            stk = combine(nd, stk);
        }
    }
    return (int)(stk & 1ull);
}

// Where x stands to a primitive without transforms, at a fixed y and z: 0 in,
// else out, by y or z alone (2) or on x's lower (-1) or upper (1) side; a plane
// 0 or 1.  Rounded sums and products are monotone in each operand, so along
// a row a plane's dot product and a box's distance are monotone and a sphere's
// or cylinder's radius is on either side of its centre: two points with one
// code have it all the way between them.
__device__ __forceinline__ int leaf_code(const sj_csg_node& nd, double x, double y, double z) {
    if (nd.op == SJ_CSG_PLANE) {
        const double d = __dadd_rn(__dadd_rn(__dmul_rn(x, nd.p[0]), __dmul_rn(y, nd.p[1])), __dmul_rn(z, nd.p[2]));
        return d > nd.p[3] ? 1 : 0;
    }
    const double qx = __dsub_rn(x, nd.c[0]), qy = __dsub_rn(y, nd.c[1]), qz = __dsub_rn(z, nd.c[2]);
    const int side = qx < 0 ? -1 : 1;
    if (nd.op == SJ_CSG_BOX) {
        if (fabs(qz) > nd.p[2] || fabs(qy) > nd.p[1]) return 2;
        return fabs(qx) > nd.p[0] ? side : 0;
    }
    if (nd.op == SJ_CSG_SPHERE) {
        const double s2 = __dadd_rn(__dadd_rn(__dadd_rn(0.0, __dmul_rn(qx, qx)), __dmul_rn(qy, qy)), __dmul_rn(qz, qz));
        return __dsqrt_rn(s2) > nd.p[0] ? side : 0;
    }
    const double h = nd.p[0], r1 = nd.p[1], r2 = nd.p[2];
    if (qz < 0 || qz > h) return 2;
    const double cr = __dadd_rn(__dmul_rn(qx, qx), __dmul_rn(qy, qy));
    return __dmul_rn(cr, h) > __dadd_rn(__dmul_rn(__dsub_rn(r2, r1), qz), __dmul_rn(r1, h)) ? side : 0;
}

// eval_program on the row of points from (xa, y, z) to (xb, y, z): in_root
// where it is one answer by every primitive's code at the ends, else -1.
__device__ int eval_row(const sj_csg_node* __restrict__ nodes, int n, double xa, double xb, double y, double z) {
    unsigned long long stk = 0;
    for (int q = 0; q < n; ++q) {
        const sj_csg_node& nd = nodes[q];
        const int op = nd.op;
        if (op <= SJ_CSG_PLANE) {
            const int code = leaf_code(nd, xa, y, z);
            if (code != 2 && leaf_code(nd, xb, y, z) != code) return -1;
            const int out = code != 0;
            stk = (stk << 1) | (unsigned long long)(op == SJ_CSG_PLANE ? 1 - out : out ? nd.invert : 1 - nd.invert);
        } else {
            stk = combine(nd, stk);
        }
    }
    return (int)(stk & 1ull);
}

// every point of the grid has coordinates below FAR (1), of moderate size (3)
static int finite_grid(int nx, int ny, int nz, double dx, const double* o) {
    const int n[3] = {nx, ny, nz};
    int f = 3;
    for (int a = 0; a < 3; ++a) {
        const double end = o[a] + (n[a] + 1.0) * dx;
        if (!(std::fabs(o[a]) < FAR && std::fabs(end) < FAR)) return 0;
        if (std::fabs(o[a]) >= MODERATE || std::fabs(end) >= MODERATE) f = 1;
    }
    return f;
}

// Region start table carried by value in the kernel's parameters.
struct RegionStarts {
    int s[SJ_MAX_REGIONS + 1];
    __device__ int operator[](int g) const { return s[g]; }
};

// voxel t of the grid, by 32-bit division where the grid allows
__device__ __forceinline__ void voxel_of(long long t, long long total, int nx, int ny, int& i, int& j, int& k) {
    if (total < (1ll << 32)) {
        const unsigned u = (unsigned)t, r = u / (unsigned)nx;
        i = (int)(u - r * (unsigned)nx);
        k = (int)(r / (unsigned)ny);
        j = (int)(r - (unsigned)k * (unsigned)ny);
    } else {
        i = (int)(t % nx);
        const long long r = t / nx;
        j = (int)(r % ny);
        k = (int)(r / ny);
    }
}

// The mask of component c's point (i, j, k): bit g = in region g.
template <typename Starts>
__device__ __forceinline__ unsigned point_mask(const sj_csg_node* __restrict__ nodes, const Starts& rstart,
                                               const uint8_t* flags, int n_regions, int c, int i, int j, int k,
                                               double dx, double ox, double oy, double oz) {
    const double x = __dadd_rn(ox, __dmul_rn((double)i + (c == 0 ? 0.5 : 0.0), dx));
    const double y = __dadd_rn(oy, __dmul_rn((double)j + (c == 1 ? 0.5 : 0.0), dx));
    const double z = __dadd_rn(oz, __dmul_rn((double)k + (c == 2 ? 0.5 : 0.0), dx));
    unsigned m = 0;
    for (int g = 0; g < n_regions; ++g) {
        const int s = rstart[g], e = rstart[g + 1];
        if (eval_program(nodes + s, flags + s, e - s, x, y, z)) m |= 1u << g;
    }
    return m;
}

// Masks for the Ex, Ey and Ez points.  A thread takes a segment of SEG points
// of a row: where every primitive's code is the same at its ends the segment
// has one mask (eval_row), the others are listed and the block then goes over
// their points one by one.  SEG = 1 (also for scenes with a transform): a
// point.  Starts is a device pointer to the region start table or a
// RegionStarts value.  Ends decide 3 of 4 segments of the 256 x 256 x 192 bowtie:
// 2.91 ms with every point evaluated, 0.62 with segments of 16 (8: 0.88); 192^3
// on quartz 0.74 and 0.10.  A segment's two ends and then its block's list are
// a serial chain, so grids of fewer than RASTER_FEW points take one per thread
// (spheres and cylinders, 48^3: 43 us, 169 in segments; 80^3 171 and 172;
// 96^3 283 and 171).
constexpr int RASTER_SEG = 16, RASTER_THREADS = 128;
constexpr long long RASTER_FEW = 1 << 19;
template <typename Starts, int SEG>
__global__ void __launch_bounds__(RASTER_THREADS, 10)
k_rasterize(const sj_csg_node* __restrict__ nodes, const Starts rstart, int n_regions, int nx, int ny, int nz, double dx,
            double ox, double oy, double oz, int finite, uint8_t* __restrict__ masks, long long cpitch, int px) {
    __shared__ uint8_t flags[RASTER_MAX_NODES];
    __shared__ int3 seg[RASTER_THREADS];                 // first point of each thread's segment
    __shared__ unsigned short list[3 * RASTER_THREADS];  // component * RASTER_THREADS + segment
    __shared__ int n_list;
    if (threadIdx.x == 0) n_list = 0;
    identity_flags(nodes, rstart[n_regions], finite != 0, flags);
    const int nseg = (nx + SEG - 1) / SEG;
    const long long t = blockIdx.x * (long long)RASTER_THREADS + threadIdx.x;
    const long long total = (long long)nseg * ny * nz;
    int i = nx, j = 0, k = 0;
    if (t < total) {
        voxel_of(t, total, nseg, ny, i, j, k);
        i *= SEG;
    }
    const int len = min(SEG, nx - i);
    for (int c = 0; c < 3 && len > 0; ++c) {
        uint8_t* const out = masks + c * cpitch + ((long long)k * ny + j) * px + i;
        if (SEG == 1) {
            *out = (uint8_t)point_mask(nodes, rstart, flags, n_regions, c, i, j, k, dx, ox, oy, oz);
            continue;
        }
        const double xa = __dadd_rn(ox, __dmul_rn((double)i + (c == 0 ? 0.5 : 0.0), dx));
        const double xb = __dadd_rn(ox, __dmul_rn((double)(i + len - 1) + (c == 0 ? 0.5 : 0.0), dx));
        const double y = __dadd_rn(oy, __dmul_rn((double)j + (c == 1 ? 0.5 : 0.0), dx));
        const double z = __dadd_rn(oz, __dmul_rn((double)k + (c == 2 ? 0.5 : 0.0), dx));
        unsigned m = 0;
        bool one = true;
        for (int g = 0; g < n_regions && one; ++g) {
            const int v = eval_row(nodes + rstart[g], rstart[g + 1] - rstart[g], xa, xb, y, z);
            one = v >= 0;
            if (v > 0) m |= 1u << g;
        }
        if (!one) {
            list[atomicAdd(&n_list, 1)] = (unsigned short)(c * RASTER_THREADS + threadIdx.x);
        } else if (len == 16 && (reinterpret_cast<size_t>(out) & 15) == 0) {
            const unsigned w = m * 0x01010101u;
            *reinterpret_cast<uint4*>(out) = make_uint4(w, w, w, w);
        } else {
            for (int q = 0; q < len; ++q) out[q] = (uint8_t)m;
        }
    }
    if (SEG == 1) return;
    seg[threadIdx.x] = make_int3(i, j, k);
    __syncthreads();
    for (int u = threadIdx.x; u < n_list * SEG; u += RASTER_THREADS) {
        const int e = list[u / SEG], c = e / RASTER_THREADS;
        const int3 f = seg[e % RASTER_THREADS];
        const int p = f.x + u % SEG;
        if (p < nx)
            masks[c * cpitch + ((long long)f.z * ny + f.y) * px + p] =
                (uint8_t)point_mask(nodes, rstart, flags, n_regions, c, p, f.y, f.z, dx, ox, oy, oz);
    }
}

// A kernel's segment length by the grid, and its blocks
static bool raster_segments(int nx, int ny, int nz, bool rows, int finite, unsigned& blocks) {
    const bool seg = rows && finite == 3 && (long long)nx * ny * nz >= RASTER_FEW;
    const long long threads = (long long)(seg ? (nx + RASTER_SEG - 1) / RASTER_SEG : nx) * ny * nz;
    blocks = (unsigned)((threads + RASTER_THREADS - 1) / RASTER_THREADS);
    return seg;
}
template <typename Starts>
static cudaError_t rasterize_with(const sj_csg_node* d_nodes, const Starts& starts, int n_regions, bool rows, int nx, int ny,
                                  int nz, double dx, const double* o, uint8_t* d_masks, long long cpitch, int px,
                                  cudaStream_t s) {
    const int finite = finite_grid(nx, ny, nz, dx, o);
    unsigned blocks;
    if (raster_segments(nx, ny, nz, rows, finite, blocks))
        k_rasterize<Starts, RASTER_SEG><<<blocks, RASTER_THREADS, 0, s>>>(d_nodes, starts, n_regions, nx, ny, nz, dx, o[0],
                                                                          o[1], o[2], finite, d_masks, cpitch, px);
    else
        k_rasterize<Starts, 1><<<blocks, RASTER_THREADS, 0, s>>>(d_nodes, starts, n_regions, nx, ny, nz, dx, o[0], o[1], o[2],
                                                                 finite, d_masks, cpitch, px);
    return cudaGetLastError();
}

cudaError_t launch_rasterize(const sj_csg_node* d_nodes, const int* d_region_start, int n_regions, bool rows,
                             int nx, int ny, int nz, double dx, const double* origin,
                             uint8_t* d_masks, long long mask_pitch_elems, int px, cudaStream_t s) {
    return rasterize_with(d_nodes, d_region_start, n_regions, rows, nx, ny, nz, dx, origin, d_masks, mask_pitch_elems, px, s);
}

// ------------------------------------------------------------ smoothing
// Stochastic smoothing (cgs_material_function::in_bound, src/disp.cpp:264-283):
// at each E-component Yee point, region g's count is in(r) plus in(r + d_j)
// over the n_offs offsets, r + d_j formed by one rounded add per axis as there.
// A point's key packs the counts 8 bits per region (at most 8 * 31 + 1 = 249,
// so the all-ones word never occurs and marks an empty slot of the key set).
constexpr unsigned long long SMOOTH_EMPTY = ~0ull;

__device__ __forceinline__ unsigned smooth_slot(unsigned long long key, unsigned cap) {
    key ^= key >> 29;
    key *= 0xbf58476d1ce4e5b9ull;
    key ^= key >> 32;
    return (unsigned)key & (cap - 1);
}

// Insert key into the open-addressing set (cap a power of two); at most cap
// probes, after which *overflow is raised.
__device__ void smooth_insert(unsigned long long* set, unsigned cap, unsigned long long key, int* overflow) {
    unsigned h = smooth_slot(key, cap);
    for (unsigned probe = 0; probe < cap; ++probe) {
        const unsigned long long cur = ((volatile unsigned long long*)set)[h];
        if (cur == key) return;
        if (cur == SMOOTH_EMPTY) {
            const unsigned long long prev = atomicCAS(set + h, SMOOTH_EMPTY, key);
            if (prev == SMOOTH_EMPTY || prev == key) return;
        }
        h = (h + 1) & (cap - 1);
    }
    atomicExch(overflow, 1);
}

// The key of the row of points from (xa, y, z) to (xb, y, z) where every sample
// of every region is decided by its ends, else SMOOTH_EMPTY.
__device__ __forceinline__ unsigned long long row_key(const sj_csg_node* __restrict__ nodes, const int* __restrict__ rstart,
                                                      int n_regions, const double* __restrict__ offs, int n_offs, double xa,
                                                      double xb, double y, double z) {
    unsigned long long key = 0;
    for (int g = 0; g < n_regions; ++g) {
        const sj_csg_node* p = nodes + rstart[g];
        const int n = rstart[g + 1] - rstart[g];
        const int in = eval_row(p, n, xa, xb, y, z);
        if (in < 0) return SMOOTH_EMPTY;
        unsigned cnt = (unsigned)in;
        for (int q = 0; q < n_offs; ++q) {
            const double dx = offs[3 * q];
            const int v = eval_row(p, n, __dadd_rn(xa, dx), __dadd_rn(xb, dx), __dadd_rn(y, offs[3 * q + 1]),
                                   __dadd_rn(z, offs[3 * q + 2]));
            if (v < 0) return SMOOTH_EMPTY;
            cnt += (unsigned)v;
        }
        key |= (unsigned long long)cnt << (8 * g);
    }
    return key;
}

// Keys of the Ex, Ey and Ez points; with a set, every distinct key also goes
// into it (one insert per distinct key of a warp's points).  Segments of SEG
// points of a row as in k_rasterize: one key where their ends decide every
// sample (rounded offsets keep the order of x), else point by point.
// smooth_n = 1, every point and in segments: 256 x 256 x 192 bowtie 23.8 and
// 5.3 ms, 192^3 junction 2.9 and 0.5 (FP64 operations of what stays undecided).
template <int SEG>
__global__ void __launch_bounds__(RASTER_THREADS, 8)
k_rasterize_counts(const sj_csg_node* __restrict__ nodes, const int* __restrict__ rstart, int n_regions, int nx, int ny,
                   int nz, double dx, double ox, double oy, double oz, int finite, const double* __restrict__ offs,
                   int n_offs, unsigned long long* __restrict__ keys, long long kpitch, int px,
                   unsigned long long* __restrict__ set, unsigned cap, int* __restrict__ overflow) {
    __shared__ uint8_t flags[RASTER_MAX_NODES];
    __shared__ int3 seg[RASTER_THREADS];                 // first point of each thread's segment
    __shared__ unsigned short list[3 * RASTER_THREADS];  // component * RASTER_THREADS + segment
    __shared__ unsigned long long row[3][RASTER_THREADS];  // its key
    __shared__ int n_list;
    if (threadIdx.x == 0) n_list = 0;
    bool all = finite != 0;
    for (int q = threadIdx.x; q < 3 * n_offs; q += RASTER_THREADS) all = all && fabs(offs[q]) < FAR;
    identity_flags(nodes, rstart[n_regions], __syncthreads_and(all) != 0, flags);
    const int nseg = (nx + SEG - 1) / SEG;
    const long long t = blockIdx.x * (long long)RASTER_THREADS + threadIdx.x;
    const long long total = (long long)nseg * ny * nz;
    int i = nx, j = 0, k = 0;
    if (t < total) {
        voxel_of(t, total, nseg, ny, i, j, k);
        i *= SEG;
    }
    auto insert = [&](unsigned long long key) {
        if (!set) return;
        const unsigned peers = __match_any_sync(__activemask(), key);
        if ((threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) smooth_insert(set, cap, key, overflow);
    };
    // component c's key at point (p, q, r)
    auto point = [&](int c, int p, int q, int r) {
        const double x = __dadd_rn(ox, __dmul_rn((double)p + (c == 0 ? 0.5 : 0.0), dx));
        const double y = __dadd_rn(oy, __dmul_rn((double)q + (c == 1 ? 0.5 : 0.0), dx));
        const double z = __dadd_rn(oz, __dmul_rn((double)r + (c == 2 ? 0.5 : 0.0), dx));
        unsigned long long key = 0;
        for (int g = 0; g < n_regions; ++g) {
            const int s = rstart[g], e = rstart[g + 1];
            unsigned cnt = (unsigned)eval_program(nodes + s, flags + s, e - s, x, y, z);
            for (int m = 0; m < n_offs; ++m)
                cnt += (unsigned)eval_program(nodes + s, flags + s, e - s, __dadd_rn(x, offs[3 * m]),
                                              __dadd_rn(y, offs[3 * m + 1]), __dadd_rn(z, offs[3 * m + 2]));
            key |= (unsigned long long)cnt << (8 * g);
        }
        keys[c * kpitch + ((long long)r * ny + q) * px + p] = key;
        insert(key);
    };
    const int len = min(SEG, nx - i);
    for (int c = 0; c < 3 && len > 0; ++c) {
        if (SEG == 1) {
            point(c, i, j, k);
            continue;
        }
        const double xa = __dadd_rn(ox, __dmul_rn((double)i + (c == 0 ? 0.5 : 0.0), dx));
        const double xb = __dadd_rn(ox, __dmul_rn((double)(i + len - 1) + (c == 0 ? 0.5 : 0.0), dx));
        const double y = __dadd_rn(oy, __dmul_rn((double)j + (c == 1 ? 0.5 : 0.0), dx));
        const double z = __dadd_rn(oz, __dmul_rn((double)k + (c == 2 ? 0.5 : 0.0), dx));
        const unsigned long long key = row_key(nodes, rstart, n_regions, offs, n_offs, xa, xb, y, z);
        row[c][threadIdx.x] = key;
        if (key == SMOOTH_EMPTY)
            list[atomicAdd(&n_list, 1)] = (unsigned short)(c * RASTER_THREADS + threadIdx.x);
        else
            insert(key);
    }
    if (SEG == 1) return;
    seg[threadIdx.x] = make_int3(i, j, k);
    __syncthreads();
    for (int u = threadIdx.x; u < RASTER_THREADS * SEG; u += RASTER_THREADS) {
        const int3 f = seg[u / SEG];
        const int p = f.x + u % SEG;
        if (p >= nx) continue;
        for (int c = 0; c < 3; ++c) {
            if (row[c][u / SEG] != SMOOTH_EMPTY)
                keys[c * kpitch + ((long long)f.z * ny + f.y) * px + p] = row[c][u / SEG];
        }
    }
    for (int u = threadIdx.x; u < n_list * SEG; u += RASTER_THREADS) {
        const int e = list[u / SEG];
        const int3 f = seg[e % RASTER_THREADS];
        const int p = f.x + u % SEG;
        if (p < nx) point(e / RASTER_THREADS, p, f.y, f.z);
    }
}

cudaError_t launch_rasterize_counts(const sj_csg_node* d_nodes, const int* d_region_start, int n_regions, bool rows,
                                    int nx, int ny, int nz, double dx, const double* origin,
                                    const double* d_offs, int n_offs, unsigned long long* d_keys,
                                    long long key_pitch_elems, int px, unsigned long long* d_set,
                                    unsigned cap, int* d_overflow, cudaStream_t s) {
    const int finite = finite_grid(nx, ny, nz, dx, origin);
    unsigned blocks;
    const bool seg = raster_segments(nx, ny, nz, rows, finite, blocks);
    (seg ? k_rasterize_counts<RASTER_SEG> : k_rasterize_counts<1>)<<<blocks, RASTER_THREADS, 0, s>>>(
        d_nodes, d_region_start, n_regions, nx, ny, nz, dx, origin[0], origin[1], origin[2], finite, d_offs, n_offs, d_keys,
        key_pitch_elems, px, d_set, cap, d_overflow);
    return cudaGetLastError();
}

// Replace each point's key by its index in the sorted list of distinct keys
// (n_keys <= 256): the point's material class.
__global__ void k_class_assign(const unsigned long long* __restrict__ keys, long long pitch, int nx, int ny,
                               int nz, int px, const unsigned long long* __restrict__ sorted, int n_keys,
                               uint8_t* __restrict__ cls) {
    __shared__ unsigned long long sk[256];
    for (int q = threadIdx.x; q < n_keys; q += blockDim.x) sk[q] = sorted[q];
    __syncthreads();
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = (long long)nx * ny * nz;
    if (t >= total) return;
    const int i = (int)(t % nx);
    const long long r = t / nx;
    const int j = (int)(r % ny);
    const int k = (int)(r / ny);
    const long long o = ((long long)k * ny + j) * px + i;
    for (int c = 0; c < 3; ++c) {
        const unsigned long long key = keys[c * pitch + o];
        int lo = 0, hi = n_keys - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sk[mid] < key)
                lo = mid + 1;
            else
                hi = mid;
        }
        cls[c * pitch + o] = (uint8_t)lo;
    }
}

cudaError_t launch_class_assign(const unsigned long long* d_keys, long long pitch, int nx, int ny, int nz,
                                int px, const unsigned long long* d_sorted, int n_keys, uint8_t* d_cls,
                                cudaStream_t s) {
    const long long total = (long long)nx * ny * nz;
    k_class_assign<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_keys, pitch, nx, ny, nz, px, d_sorted,
                                                                   n_keys, d_cls);
    return cudaGetLastError();
}

// Mark every (class_x, class_y, class_z) triple present in a 2^24-bit set.
__global__ void k_combo_mark(const uint8_t* __restrict__ cls, long long cpitch, int nx, int ny,
                             int nz, int px, uint32_t* __restrict__ bitmap) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = (long long)nx * ny * nz;
    if (t >= total) return;
    const int i = (int)(t % nx);
    const long long r = t / nx;
    const int j = (int)(r % ny);
    const int k = (int)(r / ny);
    const long long o = ((long long)k * ny + j) * px + i;
    const uint32_t key = (uint32_t)cls[o] | ((uint32_t)cls[cpitch + o] << 8) |
                         ((uint32_t)cls[2 * cpitch + o] << 16);
    const uint32_t bit = 1u << (key & 31u);
    uint32_t* w = bitmap + (key >> 5);
    if ((*((volatile uint32_t*)w) & bit) == 0) atomicOr(w, bit);
}

cudaError_t launch_combo_mark(const uint8_t* d_cls, long long cpitch, int nx, int ny, int nz,
                              int px, uint32_t* d_bitmap, cudaStream_t s) {
    const long long total = (long long)nx * ny * nz;
    k_combo_mark<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_cls, cpitch, nx, ny, nz, px, d_bitmap);
    return cudaGetLastError();
}

// The set bits of the triple bitmap as a key list (unordered; the host sorts
// the at most cap it reads back).  *count gets the number of set bits.
__global__ void k_combo_compact(const uint32_t* __restrict__ bitmap, int n_words, uint32_t* __restrict__ keys,
                                int cap, int* __restrict__ count) {
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += gridDim.x * blockDim.x) {
        uint32_t bits = bitmap[w];
        while (bits) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1;
            const int slot = atomicAdd(count, 1);
            if (slot < cap) keys[slot] = (uint32_t)w * 32u + (uint32_t)b;
        }
    }
}

cudaError_t launch_combo_compact(const uint32_t* d_bitmap, int n_words, uint32_t* d_keys, int cap, int* d_count,
                                 cudaStream_t s) {
    k_combo_compact<<<608, 256, 0, s>>>(d_bitmap, n_words, d_keys, cap, d_count);
    return cudaGetLastError();
}

// Replace each voxel's triple by its index in the sorted key list.
__global__ void k_combo_assign(const uint8_t* __restrict__ cls, long long cpitch, int nx, int ny,
                               int nz, int px, const uint32_t* __restrict__ keys, int n_keys,
                               uint8_t* __restrict__ combo) {
    __shared__ uint32_t sk[256];
    for (int q = threadIdx.x; q < n_keys; q += blockDim.x) sk[q] = keys[q];
    __syncthreads();
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = (long long)nx * ny * nz;
    if (t >= total) return;
    const int i = (int)(t % nx);
    const long long r = t / nx;
    const int j = (int)(r % ny);
    const int k = (int)(r / ny);
    const long long o = ((long long)k * ny + j) * px + i;
    const uint32_t key = (uint32_t)cls[o] | ((uint32_t)cls[cpitch + o] << 8) |
                         ((uint32_t)cls[2 * cpitch + o] << 16);
    int lo = 0, hi = n_keys - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sk[mid] < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    combo[o] = (uint8_t)lo;
}

cudaError_t launch_combo_assign(const uint8_t* d_cls, long long cpitch, int nx, int ny, int nz,
                                int px, const uint32_t* d_keys, int n_keys, uint8_t* d_combo,
                                cudaStream_t s) {
    const long long total = (long long)nx * ny * nz;
    k_combo_assign<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_cls, cpitch, nx, ny, nz, px,
                                                                   d_keys, n_keys, d_combo);
    return cudaGetLastError();
}

// Bounding box of voxels whose combo carries a polarisation: box = {min i,j,k, max i,j,k}.
__global__ void k_disp_bbox(const uint8_t* __restrict__ combo, const uint8_t* __restrict__ cflag,
                            int nx, int ny, int nz, int px, int* box) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = (long long)nx * ny * nz;
    if (t >= total) return;
    const int i = (int)(t % nx);
    const long long r = t / nx;
    const int j = (int)(r % ny);
    const int k = (int)(r / ny);
    const long long o = ((long long)k * ny + j) * px + i;
    if (cflag[combo[o]] & 1) {
        atomicMin(box + 0, i);
        atomicMin(box + 1, j);
        atomicMin(box + 2, k);
        atomicMax(box + 3, i);
        atomicMax(box + 4, j);
        atomicMax(box + 5, k);
    }
}

cudaError_t launch_disp_bbox(const uint8_t* d_combo, const uint8_t* d_cflag, int nx, int ny,
                             int nz, int px, int* d_box, cudaStream_t s) {
    const long long total = (long long)nx * ny * nz;
    k_disp_bbox<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_combo, d_cflag, nx, ny, nz, px, d_box);
    return cudaGetLastError();
}

}  // namespace sj

namespace sj {
// 256-bin histogram of the combo map (voxel counts per material combo).
__global__ void k_combo_hist(const uint8_t* __restrict__ combo, int nx, int ny, int nz, int px,
                             unsigned long long* __restrict__ hist) {
    __shared__ unsigned int h[256];
    for (int q = threadIdx.x; q < 256; q += blockDim.x) h[q] = 0;
    __syncthreads();
    const long long total = (long long)nx * ny * nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % nx);
        const long long r = t / nx;
        const int j = (int)(r % ny);
        const int k = (int)(r / ny);
        atomicAdd(&h[combo[((long long)k * ny + j) * px + i]], 1u);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 256; q += blockDim.x)
        if (h[q]) atomicAdd(hist + q, (unsigned long long)h[q]);
}

cudaError_t launch_combo_hist(const uint8_t* d_combo, int nx, int ny, int nz, int px,
                              unsigned long long* d_hist, cudaStream_t s) {
    k_combo_hist<<<608, 256, 0, s>>>(d_combo, nx, ny, nz, px, d_hist);
    return cudaGetLastError();
}
}  // namespace sj

// ---------------------------------------------------------------------------
// Allocation-free rasteriser (sj_rasterize_static).
//
// The concatenated CSG programs live in one file-scope device array instead
// of cudaMalloc'd buffers; the region start table travels by value in the
// kernel's parameters.  Host code never names the array directly: its device
// address comes from cudaGetSymbolAddress, looked up with the device current
// and cached per device together with the context it was taken in, so a
// context torn down and created again (cudaDeviceReset) gets a fresh lookup.
#include <cuda.h>
#include <mutex>

namespace sj {

constexpr size_t RASTER_SCRATCH_BYTES = (size_t)SJ_RASTER_STATIC_NODES * sizeof(sj_csg_node);

static __device__ __align__(256) unsigned char g_raster_scratch[RASTER_SCRATCH_BYTES];

namespace {
constexpr int MAX_DEVICES = 64;
std::mutex g_scratch_mu;
unsigned char* g_scratch_ptr[MAX_DEVICES] = {};
CUcontext g_scratch_ctx[MAX_DEVICES] = {};

typedef CUresult (*CtxGetCurrentFn)(CUcontext*);

// The driver's current context, through the runtime's entry-point table (the
// library links only the CUDA runtime).
cudaError_t current_context(CUcontext* out) {
    static CtxGetCurrentFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 4000, cudaEnableDefault, &q);
        if (e != cudaSuccess) return e;
        if (q != cudaDriverEntryPointSuccess || !p) return cudaErrorNotSupported;
        fn = reinterpret_cast<CtxGetCurrentFn>(p);
    }
    return fn(out) == CUDA_SUCCESS ? cudaSuccess : cudaErrorContextIsDestroyed;
}

// Device address of g_raster_scratch on the current device.
cudaError_t raster_scratch(unsigned char** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    CUcontext ctx = nullptr;
    e = current_context(&ctx);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!ctx || !g_scratch_ptr[dev] || g_scratch_ctx[dev] != ctx) {
        // no context yet (first CUDA call of this thread) or a new one: the
        // lookup makes the device's primary context current if none is
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_raster_scratch);
        if (e != cudaSuccess) return e;
        e = current_context(&ctx);
        if (e != cudaSuccess) return e;
        g_scratch_ptr[dev] = static_cast<unsigned char*>(p);
        g_scratch_ctx[dev] = ctx;
    }
    *out = g_scratch_ptr[dev];
    return cudaSuccess;
}
}  // namespace

// Returns 0 or an SJ_E_* code; *msg gets a static description on failure.
int rasterize_static(const sj_grid_desc* g, const sj_scene_desc* sc, uint8_t* d_out, cudaStream_t s,
                     const char** msg) {
    if (!g || !sc || !d_out) {
        *msg = "NULL argument";
        return SJ_E_INVALID;
    }
    if (g->nx < 1 || g->ny < 1 || g->nz < 1 || !(g->dx > 0)) {
        *msg = "bad grid";
        return SJ_E_INVALID;
    }
    if (sc->n_regions < 0 || sc->n_regions > SJ_MAX_REGIONS || (sc->n_regions > 0 && !sc->regions)) {
        *msg = "scene n_regions must be in [0, 8]";
        return SJ_E_INVALID;
    }
    if (sc->smooth_n != 0) {
        *msg = "a smoothed scene has fill counts, not region masks (sj_rasterize_counts)";
        return SJ_E_INVALID;
    }
    RegionStarts start = {};
    for (int r = 0; r < sc->n_regions; ++r) {
        const sj_region_desc& rg = sc->regions[r];
        if (rg.n_nodes < 1 || !rg.nodes) {
            *msg = "region without CSG nodes";
            return SJ_E_INVALID;
        }
        int depth = 0;
        for (int q = 0; q < rg.n_nodes; ++q) {
            const int op = rg.nodes[q].op;
            if (op < 0 || op > SJ_CSG_NOOP) {
                *msg = "unknown CSG op";
                return SJ_E_INVALID;
            }
            if (op <= SJ_CSG_PLANE || op == SJ_CSG_CONST || op == SJ_CSG_NOOP)
                ++depth;
            else if (op == SJ_CSG_UNION || op == SJ_CSG_INTERSECT)
                depth = depth >= 2 ? depth - 1 : -1000;
            else if (depth < 1)
                depth = -1000;
            if (depth < 0 || depth > 64) {
                *msg = "malformed CSG program";
                return SJ_E_INVALID;
            }
        }
        if (depth != 1) {
            *msg = "CSG program must leave exactly one value";
            return SJ_E_INVALID;
        }
        if (start.s[r] + rg.n_nodes > SJ_RASTER_STATIC_NODES) {
            *msg = "scene has more CSG nodes than SJ_RASTER_STATIC_NODES (512)";
            return SJ_E_RANGE;
        }
        start.s[r + 1] = start.s[r] + rg.n_nodes;
    }
    unsigned char* base = nullptr;
    cudaError_t e = raster_scratch(&base);
    if (e != cudaSuccess) {
        *msg = "cudaGetSymbolAddress of the rasteriser scratch array failed";
        return SJ_E_CUDA;
    }
    // the program is overwritten in full by every call; nothing needs clearing
    sj_csg_node* d_nodes = reinterpret_cast<sj_csg_node*>(base);
    for (int r = 0; r < sc->n_regions && e == cudaSuccess; ++r)
        e = cudaMemcpyAsync(d_nodes + start.s[r], sc->regions[r].nodes,
                            (size_t)sc->regions[r].n_nodes * sizeof(sj_csg_node), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        const long long nv = (long long)g->nx * g->ny * g->nz;
        e = rasterize_with(d_nodes, start, sc->n_regions, raster_rows(sc), g->nx, g->ny, g->nz, g->dx, g->origin, d_out, nv,
                           g->nx, s);
    }
    if (e != cudaSuccess) {
        *msg = "CUDA call failed in sj_rasterize_static";
        return SJ_E_CUDA;
    }
    return SJ_OK;
}

}  // namespace sj
