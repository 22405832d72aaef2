// Column density through the octree: pytreegrav's ray-traced and angle-binned walks
// (treewalk.py:904-1030, frontend.py:1321-1458) over the tree's FP64 arrays, in the reference's order
// of operations with every operation rounded once (explicit _rn intrinsics, no FMA contraction).
//
// The ray-traced walk has no truncation: a node opens whenever its bounding sphere, inflated by its
// largest particle radius, can meet the ray, and only particles contribute, each as a uniform sphere
// of its mass and radius (the softening). One thread walks one (target, ray) pair; lanes of a warp
// take consecutive targets (Morton order) for the same ray, so their walks stay together.
#include "tg_tree.cuh"

namespace tg {
namespace {

constexpr double FAC_DENSITY = 3.0 / (4.0 * 3.141592653589793);  // 3 / (4 pi), as numpy evaluates it
constexpr double FOUR_PI = 4.0 * 3.141592653589793;
constexpr double BIN_SOLID_ANGLE = (4.0 * 3.141592653589793) / 6.0;  // angular_bin_size

struct ColumnTree {
    const double *coord, *mass, *soft, *size, *delta;
    const int64_t *first, *next;
    int64_t npart, nelem;
    int64_t max_visits;  // visits one walk may make (one per element always suffices)
    // FP32 copy for the screen, three words per element: coordinates split hi + lo, with the radius
    // (hi.w) and, for nodes, size * sqrt(3)/2 + delta (lo.w); then the links (next, first; LINK_NONE:
    // none) and whether the radius is positive in FP64
    const float4 *rec;
    // output row of target i: rows[i] (the targets are the tree's own particles, results go back to
    // the caller's order), or i when null
    const int64_t *rows = nullptr;
    __device__ int64_t row(int64_t i) const { return rows ? rows[i] : i; }
};

__device__ __forceinline__ void split_f(double v, float &hi, float &lo) { d2f_split(v, hi, lo); }

constexpr uint32_t LINK_NONE = 0xffffffffu;  // elements number below 2^32 - 1 (N < 2^31 and fewer nodes)
__device__ __forceinline__ uint32_t pack_link(int64_t e) { return e < 0 ? LINK_NONE : (uint32_t)e; }

__global__ void k_column_prep(ColumnTree t, float4 *rec) {
    chain_next();
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= t.nelem) return;
    float4 a, b;
    split_f(t.coord[3 * e], a.x, b.x);
    split_f(t.coord[3 * e + 1], a.y, b.y);
    split_f(t.coord[3 * e + 2], a.z, b.z);
    const double h = t.soft[e];
    a.w = d2f(h);
    b.w = e < t.npart ? 0.f : (float)(t.size[e] * 0.8660254037844386 + t.delta[e]);
    rec[3 * e] = a;
    rec[3 * e + 1] = b;
    rec[3 * e + 2] = make_float4(__uint_as_float(pack_link(t.next[e])), __uint_as_float(pack_link(t.first[e])),
                                 __uint_as_float(h > 0.0 ? 1u : 0u), 0.f);
}

__device__ __forceinline__ float sqrt_approx(float x) {  // relative error below 2^-22; subnormals as 0
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Offset, distance and along-ray coordinate of element no from a ray's origin in FP64, and r^2 - z^2:
// the reference's expressions.
struct RayOffset {
    double r, z, b2;
};
__device__ __forceinline__ RayOffset ray_offset(const ColumnTree &t, int64_t no, const double *p, const double *ray) {
    const double dx = dsub(t.coord[3 * no], p[0]), dy = dsub(t.coord[3 * no + 1], p[1]);
    const double dz = dsub(t.coord[3 * no + 2], p[2]);
    const double r2 = dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
    RayOffset o;
    o.r = __dsqrt_rn(r2);
    o.z = dadd(dadd(dmul(ray[0], dx), dmul(ray[1], dy)), dmul(ray[2], dz));
    o.b2 = dsub(r2, dmul(o.z, o.z));
    return o;
}

// A particle's share of the column (treewalk.py:940-962), added to it.
__device__ __forceinline__ double column_particle(const ColumnTree &t, int64_t no, const double *p, const double *ray,
                                                  double column) {
    const RayOffset o = ray_offset(t, no, p, ray);
    const double h_no = t.soft[no];
    if (o.b2 < 0.0 || !(h_no > 0.0)) return column;
    const double h_inv = ddiv(1.0, h_no);
    const double fac = dmul(dmul(dmul(FAC_DENSITY, t.mass[no]), h_inv), h_inv);
    const double r_proj = __dsqrt_rn(o.b2);
    const double q = dmul(r_proj, h_inv);
    if (r_proj < h_no) {
        if (o.r > h_no) {
            if (o.z > 0.0) column = dadd(column, dmul(dmul(fac, 2.0), __dsqrt_rn(dsub(1.0, dmul(q, q)))));
        } else {
            const double dzh = dmul(o.z, h_inv);
            column = dadd(column, dmul(fac, dadd(dzh, __dsqrt_rn(dsub(1.0, dmul(q, q))))));
        }
    }
    return column;
}

// ColumnDensityWalk_singleray (treewalk.py:904-973) of one (target, ray) pair per lane, a warp's lanes
// visiting one element each per step. Each visited element is first screened in FP32: distance r,
// along-ray coordinate z and impact parameter b (from |d x n|, which does not cancel). Their FP32
// errors are a few 1e-7 of r, so with a margin of 4e-6 r the screen's "certainly" answers are the FP64
// decisions. A node whose decision is within the margin is decided in FP64, in the reference's order,
// including its skip of elements whose r^2 - z^2 rounds below zero.
// A particle that may contribute does not steer the walk, so it is only put in its lane's queue in shared
// memory; once a lane's queue is full, the whole warp evaluates its queues, each lane its own entries in
// the order of its walk (the same sum, bit for bit). A step's FP64 evaluation would run with one
// lane or two of 32, and GB300 takes ~76 cycles for an FP64 warp instruction with any number of them.
// A step reads one 48-byte record, links included, so that its loads are one round trip, and decides
// without branches; the screen's roots are approximate (their error is inside the margin).
// 60000 Plummer particles, six rays each: 4211 us with the particles' FP64 in the step (FP64 pipe 59 % busy)
// and the links read after the decision; 2877 us with the queues and records (FP64 pipe 8 %), 2527 us
// branch-free. What bounds it now: issue (2.1 of 4 per cycle) and the records' latency, in walks whose lanes
// are 74 % together.
// *runaway is set if a walk does not end within one visit per element (a malformed tree).
constexpr int COL_THREADS = 128;
constexpr int COL_BLOCKS_PER_SM = 8;  // 64 registers (2527 us against 2565 at 66, 7 blocks)
constexpr int COL_QUEUE = 8;  // entries per lane (4 to 24: within 3 %)

__device__ double column_walk(const ColumnTree &t, bool active, const double *p, const double *ray, int *runaway,
                              uint32_t (*queue)[COL_THREADS]) {
    const uint32_t N = (uint32_t)t.npart, ne = (uint32_t)t.nelem;
    const float n0 = (float)ray[0], n1 = (float)ray[1], n2 = (float)ray[2];
    float phx, phy, phz, plx, ply, plz;
    split_f(p[0], phx, plx);
    split_f(p[1], phy, ply);
    split_f(p[2], phz, plz);
    // absolute part of the margin: the lo parts' own rounding, and distances whose squares underflow
    const float m_abs = 1e-13f * (fabsf(phx) + fabsf(phy) + fabsf(phz)) + 1.2e-19f;
    double column = 0.0;
    uint32_t no = active ? N : LINK_NONE;
    const uint32_t stop = pack_link(t.next[N]);
    const uint32_t max_visits = (uint32_t)t.max_visits;  // at most the number of elements
    uint32_t visits = 0;
    int queued = 0;
    auto flush = [&]() {
        for (int k = 0; __any_sync(FULL, k < queued); k++)
            if (k < queued) column = column_particle(t, queue[k][threadIdx.x], p, ray, column);
        queued = 0;
    };
    for (;;) {
        if (no != LINK_NONE && no != stop) {
            if (visits++ > max_visits || no >= ne) {
                atomicOr(runaway, 1);
                no = LINK_NONE;
            }
        } else {
            no = LINK_NONE;
        }
        if (!__any_sync(FULL, no != LINK_NONE)) break;
        if (no != LINK_NONE) {
            const float4 ah = t.rec[3 * (int64_t)no], al = t.rec[3 * (int64_t)no + 1], lk = t.rec[3 * (int64_t)no + 2];
            const uint32_t next = __float_as_uint(lk.x), first = __float_as_uint(lk.y);
            const float fx = (ah.x - phx) + (al.x - plx), fy = (ah.y - phy) + (al.y - ply);
            const float fz = (ah.z - phz) + (al.z - plz), hf = ah.w;
            const float rf = sqrt_approx(fx * fx + fy * fy + fz * fz);
            const float zf = n0 * fx + n1 * fy + n2 * fz;
            const float cx = n1 * fz - n2 * fy, cy = n2 * fx - n0 * fz, cz = n0 * fy - n1 * fx;
            const float bf = sqrt_approx(cx * cx + cy * cy + cz * cz);
            const float m = 4e-6f * rf + m_abs;  // error margin of r, z and b
            const float reach = hf + al.w;  // Softenings[no] + R_eff (a particle's R_eff is 0)
            const bool out = rf - m > reach * 1.000001f, miss = bf - m > reach * 1.000001f;  // certainly
            const bool part = no < N;
            // A particle makes no contribution when it is point-like, when the ray certainly misses it
            // (which also makes r^2 - z^2 certainly positive), or when it lies certainly behind the target
            // and does not hold it. A node, with r^2 - z^2 certainly positive (b > m), is skipped when it is
            // certainly outside and behind or missed, and opened when it certainly holds the target's
            // neighbourhood, or is ahead and hit.
            const bool skip = out && (zf < -m || miss);
            const bool none = skip || miss || __float_as_uint(lk.z) == 0u;
            const bool hit = rf + m < reach * 0.999999f || (out && zf > m && bf + m < reach * 0.999999f);
            const bool clear = bf > m;
            bool open = !part && clear && hit;
            if (part && !none) queue[queued++][threadIdx.x] = no;
            if (!part && !(clear && (hit || skip))) {  // FP64, the reference's expression
                const RayOffset o = ray_offset(t, no, p, ray);
                if (!(o.b2 < 0.0)) {
                    const double h_no = t.soft[no];
                    const double R_eff = dadd(dmul(t.size[no], 0.8660254037844386), t.delta[no]);
                    if (o.r < dadd(h_no, R_eff)) {
                        open = true;
                    } else if (o.z > 0.0) {
                        const double reach64 = dadd(h_no, R_eff);
                        open = o.b2 < dmul(reach64, reach64);
                    }
                }
            }
            no = open ? first : next;
        }
        if (__any_sync(FULL, queued == COL_QUEUE)) flush();
    }
    flush();
    return column;
}

// rays shared by all targets (ray_stride 0) or per target (ray_stride 3 * nrays): pair p is
// target p % n on ray p / n
__global__ void __launch_bounds__(COL_THREADS, COL_BLOCKS_PER_SM) k_column_rays(ColumnTree t, const double *pos, int64_t n,
                                                             const double *rays, int64_t nrays, int64_t ray_stride,
                                                             double *out, int *runaway) {
    chain_wait();
    chain_next();
    __shared__ uint32_t queue[COL_QUEUE][COL_THREADS];
    const int64_t pair = (int64_t)blockIdx.x * COL_THREADS + threadIdx.x;
    const bool active = pair < n * nrays;
    const int64_t i = active ? pair % n : 0, j = active ? pair / n : 0;
    const double *src = rays + i * ray_stride + 3 * j;
    const double p[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]}, ray[3] = {src[0], src[1], src[2]};
    const double column = column_walk(t, active, p, ray, runaway, queue);
    if (active) out[t.row(i) * nrays + j] = column;
}

// angular_bin (treewalk.py:49-70)
__device__ __forceinline__ int angular_bin(double dx, double dy, double dz) {
    if (fabs(dx) > fabs(dy) && fabs(dx) > fabs(dz)) return dx > 0.0 ? 0 : 1;
    if (fabs(dy) > fabs(dz)) return dy > 0.0 ? 2 : 3;
    return dz > 0.0 ? 4 : 5;
}

// ColumnDensityWalk_binned (treewalk.py:976-1030): one thread per target, six sky bins.
__global__ void k_column_binned(ColumnTree t, const double *pos, int64_t n, double theta, double *out,
                                int *runaway) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double px = pos[3 * i], py = pos[3 * i + 1], pz = pos[3 * i + 2];
    double col[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const int64_t N = t.npart;
    int64_t no = N;
    const int64_t stop = t.next[N];
    for (int64_t guard = 0; no > -1 && no != stop; guard++) {
        if (guard > t.max_visits || no >= t.nelem) {
            atomicOr(runaway, 1);
            break;
        }
        const double dx = dsub(t.coord[3 * no], px), dy = dsub(t.coord[3 * no + 1], py);
        const double dz = dsub(t.coord[3 * no + 2], pz);
        const double r2 = dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
        const double h = t.soft[no];
        if (no < N) {
            const int bin = angular_bin(dx, dy, dz);
            if (r2 > dmul(h, h)) {
                const double c = ddiv(ddiv(t.mass[no], r2), BIN_SOLID_ANGLE);
#pragma unroll
                for (int k = 0; k < 6; k++)
                    if (k == bin) col[k] = dadd(col[k], c);
            } else if (h > 0.0) {
                const double col0 = dmul(t.mass[no], ddiv(3.0, dmul(dmul(FOUR_PI, h), h)));
                const double fac = ddiv(__dsqrt_rn(r2), h);
                const double iso = dmul(dsub(1.0, fac), col0);
                const double peak = dmul(dmul(col0, fac), 2.0);
#pragma unroll
                for (int k = 0; k < 6; k++) {
                    col[k] = dadd(col[k], iso);
                    if (k == bin) col[k] = dadd(col[k], peak);
                }
            }
            no = t.next[no];
        } else {
            const double size = t.size[no], delta = t.delta[no];
            const double crit = pymax(dadd(ddiv(size, theta), delta), dadd(dadd(h, dmul(size, 0.6)), delta));
            if (__dsqrt_rn(r2) > crit) {
                const double c = ddiv(ddiv(t.mass[no], r2), BIN_SOLID_ANGLE);
                const int bin = angular_bin(dx, dy, dz);
#pragma unroll
                for (int k = 0; k < 6; k++)
                    if (k == bin) col[k] = dadd(col[k], c);
                no = t.next[no];
            } else {
                no = t.first[no];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 6; k++) out[6 * t.row(i) + k] = col[k];
}

// ColumnDensityBinned_grouped (treewalk.py:1197-1294): one warp per group of gsz (<= 32)
// consecutive targets, lane k holding target k. The group's bounding box decides every node for all
// its targets, so the warp walks one path; each lane adds its own target's share of every accepted
// node and particle, in the walk's order.
__global__ void k_column_binned_grouped(ColumnTree t, const double *pos, int64_t n, double theta, int gsz,
                                        double *out, int *runaway) {
    const int64_t a = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * gsz;
    const int lane = threadIdx.x & 31;
    if (a >= n) return;  // whole warps leave together
    const int cnt = (int)(n - a < (int64_t)gsz ? n - a : (int64_t)gsz);
    const bool mine = lane < cnt;
    const int64_t ti = a + (mine ? lane : 0);
    const double px = pos[3 * ti], py = pos[3 * ti + 1], pz = pos[3 * ti + 2];
    double bmin[3] = {px, py, pz}, bmax[3] = {px, py, pz};
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            bmin[k] = fmin(bmin[k], __shfl_xor_sync(FULL, bmin[k], o));
            bmax[k] = fmax(bmax[k], __shfl_xor_sync(FULL, bmax[k], o));
        }
    double col[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const int64_t N = t.npart;
    int64_t no = N;
    const int64_t stop = t.next[N];
    for (int64_t guard = 0; no > -1 && no != stop; guard++) {
        if (guard > t.max_visits || no >= t.nelem) {
            if (lane == 0) atomicOr(runaway, 1);
            break;
        }
        const double cx = t.coord[3 * no], cy = t.coord[3 * no + 1], cz = t.coord[3 * no + 2];
        const double h_no = t.soft[no], M = t.mass[no];
        if (no < N) {
            const double hh = dmul(h_no, h_no);
            const double d0 = dsub(cx, px), d1 = dsub(cy, py), d2 = dsub(cz, pz);
            const double r2 = dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
            const int bin = angular_bin(d0, d1, d2);
            if (r2 > hh) {
                const double c = ddiv(ddiv(M, r2), BIN_SOLID_ANGLE);
#pragma unroll
                for (int k = 0; k < 6; k++)
                    if (k == bin) col[k] = dadd(col[k], c);
            } else if (h_no > 0.0) {
                const double col0 = dmul(M, ddiv(3.0, dmul(FOUR_PI, hh)));
                const double fac = ddiv(__dsqrt_rn(r2), h_no);
                const double iso = dmul(dsub(1.0, fac), col0);
                const double peak = dmul(dmul(col0, fac), 2.0);
#pragma unroll
                for (int k = 0; k < 6; k++) {
                    col[k] = dadd(col[k], iso);
                    if (k == bin) col[k] = dadd(col[k], peak);
                }
            }
            no = t.next[no];
        } else {
            const double c3[3] = {cx, cy, cz};
            double dm[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                dm[k] = 0.0;
                if (c3[k] < bmin[k]) dm[k] = dsub(bmin[k], c3[k]);
                else if (c3[k] > bmax[k]) dm[k] = dsub(c3[k], bmax[k]);
            }
            const double r_min = __dsqrt_rn(dadd(dadd(dmul(dm[0], dm[0]), dmul(dm[1], dm[1])), dmul(dm[2], dm[2])));
            const double size = t.size[no], delta = t.delta[no];
            const double crit = pymax(dadd(ddiv(size, theta), delta), dadd(dadd(h_no, dmul(size, 0.6)), delta));
            if (r_min > crit) {  // the same answer on every lane
                const double d0 = dsub(cx, px), d1 = dsub(cy, py), d2 = dsub(cz, pz);
                const double r2 = dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
                const double c = ddiv(ddiv(M, r2), BIN_SOLID_ANGLE);
                const int bin = angular_bin(d0, d1, d2);
#pragma unroll
                for (int k = 0; k < 6; k++)
                    if (k == bin) col[k] = dadd(col[k], c);
                no = t.next[no];
            } else {
                no = t.first[no];
            }
        }
    }
    if (mine)
#pragma unroll
        for (int k = 0; k < 6; k++) out[6 * t.row(ti) + k] = col[k];
}

}  // namespace
}  // namespace tg

using namespace tg;

extern "C" {

tg_status tg_tree_column_density(tg_tree t, const double *pos, int64_t n, const double *rays, int64_t nrays,
                                 int64_t ray_stride, int binned, double theta, int group_size, int mem, double *out,
                                 void *stream) {
    if (!t || !out || n < 0) return TG_ERR_BAD_ARG;
    const bool own = !pos;  // the tree's own particles, results in the caller's order
    if (own && n != t->ntot) return TG_ERR_BAD_ARG;
    if (binned && (group_size < 0 || group_size > 32)) return TG_ERR_BAD_ARG;
    if (mem != TG_MEM_HOST && mem != TG_MEM_DEVICE) return TG_ERR_BAD_ARG;
    if (binned) {
        if (!(theta > 0)) return TG_ERR_BAD_ARG;
        nrays = 6;
        ray_stride = 0;
    } else if (!rays || nrays < 1 || (ray_stride != 0 && ray_stride != 3 * nrays)) {
        return TG_ERR_BAD_ARG;
    }
    if (t->nsys != 1) {
        set_last_error_msg("column density needs a tree of one particle system");
        return TG_ERR_BAD_ARG;
    }
    if (n == 0) return TG_OK;
    cudaStream_t st = (cudaStream_t)stream;
    tree_wait_built(t, st);
    ColumnTree ct;
    ct.coord = t->coord; ct.mass = t->mass; ct.soft = t->soft; ct.size = t->size; ct.delta = t->delta;
    ct.first = t->first; ct.next = t->next;
    ct.npart = t->ntot;
    ct.nelem = t->ntot + t->mtot;
    ct.max_visits = loop_limits().column_visits > 0 ? std::min<int64_t>(loop_limits().column_visits, ct.nelem) : ct.nelem;
    ct.rows = own ? t->walk_idx : nullptr;
    const int64_t nray_vals = binned ? 0 : (ray_stride ? n * ray_stride : 3 * nrays);
    const double *dpos = pos, *drays = rays;
    double *dout = out, *owned = nullptr;
    int *flag = nullptr;
    // one allocation: flag, positions, rays and output when they come from or go to the host
    size_t bytes = 16;
    if (mem == TG_MEM_HOST) bytes += sizeof(double) * ((own ? 0 : 3 * n) + nray_vals + n * nrays);
    TG_CUDA(dev_malloc((void **)&owned, bytes, st));
    flag = (int *)owned;
    TG_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), st));
    if (own) dpos = t->coord;  // rows [0, N) of the arena: the particles in walk order
    if (mem == TG_MEM_HOST) {
        double *p = owned + 2;
        if (!own) {
            TG_CUDA(cudaMemcpyAsync(p, pos, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, st));
            dpos = p;
            p += 3 * n;
        }
        if (nray_vals) {
            TG_CUDA(cudaMemcpyAsync(p, rays, sizeof(double) * nray_vals, cudaMemcpyHostToDevice, st));
            drays = p;
            p += nray_vals;
        }
        dout = p;
    }
    float4 *fcopy = nullptr;
    ct.rec = nullptr;
    if (binned && group_size >= 1) {
        const int64_t ngroups = (n + group_size - 1) / group_size;
        k_column_binned_grouped<<<div_up(ngroups * 32, 128), 128, 0, st>>>(ct, dpos, n, theta, group_size, dout, flag);
        note_launch();
    } else if (binned) {
        k_column_binned<<<div_up(n, 128), 128, 0, st>>>(ct, dpos, n, theta, dout, flag);
        note_launch();
    } else {
        TG_CUDA(dev_malloc((void **)&fcopy, sizeof(float4) * 3 * ct.nelem, st));
        ct.rec = fcopy;
        k_column_prep<<<div_up(ct.nelem, 256), 256, 0, st>>>(ct, fcopy);
        note_launch();
        TG_CHAIN(k_column_rays, div_up(n * nrays, COL_THREADS), COL_THREADS, 0, st, ct, dpos, n, drays, nrays,
                 ray_stride, dout, flag);
    }
    TG_CUDA(cudaGetLastError());
    int hflag = 0;
    if (mem == TG_MEM_HOST)
        TG_CUDA(cudaMemcpyAsync(out, dout, sizeof(double) * n * nrays, cudaMemcpyDeviceToHost, st));
    TG_CUDA(cudaMemcpyAsync(&hflag, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    TG_CUDA(cudaFreeAsync(owned, st));
    if (fcopy) TG_CUDA(cudaFreeAsync(fcopy, st));
    TG_CUDA(cudaStreamSynchronize(st));
    if (hflag) {
        set_last_error_msg("column density walk did not end within one visit per element");
        return TG_ERR_ITER_LIMIT;
    }
    return TG_OK;
}

}  // extern "C"
