// mps_group.cuh -- neighbour walks with a group of lanes per particle.
//
// One thread per particle leaves a scene of some ten thousand particles with two or three warps
// per scheduler, each running a serial chain of several hundred dependent loads; time is then
// latency alone. Here G lanes share a particle and a warp's 32 / G particles share one candidate
// list:
//   1. the rows that the warp's particles reach are found lane by lane (one row per lane) and
//      their table indices written to shared memory, in visiting order;
//   2. the group tests G candidates at a time, and a ballot gives each accepted one its place in
//      the particle's neighbour list (shared memory), again in visiting order;
//   3. the group computes G neighbours' terms at a time;
//   4. the terms are added in visiting order, one lane per component, so every sum is the sum
//      of the walk per particle.
// The candidate list is the union of the particles' own candidates (they are consecutive slots,
// mostly of one or two adjacent fine cells), and each particle tests all of it exactly.
#pragma once
#include <climits>
#include <type_traits>

#include "mps_device.cuh"
#include "mps_exact.cuh"

namespace mps {

constexpr int kGroupRows = 81;     // 9 x 9 fine rows
constexpr int kGroupSpan = 2;      // buckets along x of particles walked together
constexpr int kGroupChunk = 32;    // neighbours whose terms are kept at a time
constexpr int kGroupPitch = kGroupChunk + 4;
constexpr unsigned kFull = 0xffffffffu;

// one warp's scratch
template <class T, int P, int NT> struct GroupMem {
    static constexpr int kWindow = 384;  // candidates listed at a time
    alignas(16) T term[NT][P][kGroupPitch];
    alignas(16) int kidx[kWindow];   // table index of each listed candidate, then zeros
    unsigned short hit[P][kWindow];  // accepted candidates' places in kidx
    int base[kGroupRows + 1], lo[kGroupRows];  // per row: first candidate's number, table index
};

template <int G> struct Group {
    static constexpr int P = 32 / G;
    int lane, l, g;  // lane of the warp, lane of the group, group of the warp
    __device__ __forceinline__ Group() {
        lane = threadIdx.x & 31;
        l = lane & (G - 1);
        g = lane / G;
    }
    // this group's bits of a warp ballot
    __device__ __forceinline__ unsigned mine(unsigned ballot) const {
        return G == 32 ? ballot : (ballot >> (g * G)) & ((1u << (G & 31)) - 1u);
    }
    __device__ __forceinline__ unsigned below() const { return (1u << l) - 1u; }
    // value of the group's lane i
    template <class T> __device__ __forceinline__ T from(T v, int i) const {
        return __shfl_sync(kFull, v, g * G + i);
    }
};

// order-preserving integer of a float, for integer minima and maxima
__device__ __forceinline__ unsigned ord_bits(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord_float(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
// distance from [v0, v1] to fine cell f along one axis (fine_gap of the nearer end)
__device__ __forceinline__ float fine_gap_box(float v0, float v1, int f, float hf) {
    const float lo = float(f - 3) * hf;
    return fmaxf(fmaxf(lo - v1, v0 - (lo + hf)), 0.0f);
}

// The particles of one warp that are walked together (a run of its lanes in one bucket row,
// kGroupSpan + 1 buckets at most): their bucket range and the box around them, relative to the
// grid minimum. All fields are uniform over the warp.
struct GroupSet {
    unsigned lanes;
    int ixl, ixh, iy, iz;
    float x0, x1, y0, y1, z0, z1;
};

// the next set out of the lanes `pend`; row: this lane's bucket row (its first bucket's number)
template <class R>
__device__ __forceinline__ GroupSet group_next(unsigned pend, int row, const RowCtx<R>& c) {
    const int lane = threadIdx.x & 31, lead = __ffs(pend) - 1;
    GroupSet t;
    const int row0 = __shfl_sync(kFull, row, lead);
    t.ixl = __shfl_sync(kFull, c.ix, lead);
    t.iy = __shfl_sync(kFull, c.iy, lead);
    t.iz = __shfl_sync(kFull, c.iz, lead);
    const bool in = ((pend >> lane) & 1u) && row == row0 && c.ix >= t.ixl && c.ix <= t.ixl + kGroupSpan;
    t.lanes = __ballot_sync(kFull, in);
    t.ixh = __reduce_max_sync(kFull, in ? c.ix : INT_MIN);
    t.x0 = ord_float(__reduce_min_sync(kFull, in ? ord_bits(c.rx) : 0xffffffffu));
    t.x1 = ord_float(__reduce_max_sync(kFull, in ? ord_bits(c.rx) : 0u));
    t.y0 = ord_float(__reduce_min_sync(kFull, in ? ord_bits(c.ry) : 0xffffffffu));
    t.y1 = ord_float(__reduce_max_sync(kFull, in ? ord_bits(c.ry) : 0u));
    t.z0 = ord_float(__reduce_min_sync(kFull, in ? ord_bits(c.rz) : 0xffffffffu));
    t.z1 = ord_float(__reduce_max_sync(kFull, in ? ord_bits(c.rz) : 0u));
    return t;
}

// Appends the rows of one round (this lane's [lo, hi)) to the row list, empty ones left out.
template <class M>
__device__ __forceinline__ void group_push(M& m, int lo, int hi, int& nrow, int& total) {
    const int lane = threadIdx.x & 31, n = max(hi - lo, 0);
    const unsigned some = __ballot_sync(kFull, n > 0);
    int incl = n;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
    }
    if (n > 0) {
        const int r = nrow + __popc(some & ((1u << lane) - 1u));
        m.base[r] = total + incl - n;
        m.lo[r] = lo;
    }
    nrow += __popc(some);
    total += __shfl_sync(kFull, incl, 31);
    if (lane == 0) m.base[nrow] = total;
}

// The fluid rows that the set's box reaches within sqrt(B): ranges of the row-ordered copy
// (start table csr). Every step is monotone in the coordinates, so the box's range of a row
// covers the range of each particle in it.
template <class M, class R, class RN>
__device__ __forceinline__ void group_fluid_rows(M& m, const SceneDev<R, RN>& sc,
                                                 const int* __restrict__ csr, const GroupSet& t, R B,
                                                 int& nrow, int& total) {
    const int lane = threadIdx.x & 31;
    const float b = float(B), s = sqrtf(b), hf = sc.hf, ih = sc.ihf;
    const int fx0 = 3 * t.ixl - 3, fx1 = 3 * t.ixh - 3, fy0 = 3 * t.iy - 3, fz0 = 3 * t.iz - 3;
    const int zl = fine_at(t.z0 - s, ih, fz0), zh = fine_at(t.z1 + s, ih, fz0);
    const int yl = fine_at(t.y0 - s, ih, fy0), yh = fine_at(t.y1 + s, ih, fy0);
    const int ny = yh - yl + 1, n = (zh - zl + 1) * ny;
    const float iny = 1.0f / float(ny);
    const int nfx = 3 * sc.nbx, nfxy = 9 * sc.nbxy;
    nrow = total = 0;
    for (int r0 = 0; r0 < n; r0 += 32) {
        const int r = r0 + lane;
        int lo = 0, hi = 0;
        if (r < n) {
            const int dz = int((float(r) + 0.5f) * iny);
            const int fz = zl + dz, fy = yl + r - dz * ny;
            const float gz = fine_gap_box(t.z0, t.z1, fz, hf), gy = fine_gap_box(t.y0, t.y1, fy, hf);
            const float g = b - gz * gz - gy * gy;
            if (!(g < 0.0f)) {
                const float sx = sqrtf(g);
                const int xl = int(fminf(fmaxf(fmaf(t.x0 - sx, ih, 3.0f), float(fx0)), float(fx0 + 8)));
                const int xh = int(fminf(fmaxf(fmaf(t.x1 + sx, ih, 3.0f), float(fx1)), float(fx1 + 8)));
                const int row = sc.fbase + fz * nfxy + fy * nfx;
                lo = __ldg(csr + row + xl);
                hi = __ldg(csr + row + xh + 1);
            }
        }
        group_push(m, lo, hi, nrow, total);
    }
    __syncwarp();
}

// The bucket rows around the set within sqrt(B) of its box, for a table in bucket order
// (mirrors, walls)
template <class M, class R, class RN>
__device__ __forceinline__ void group_bucket_rows(M& m, const SceneDev<R, RN>& sc,
                                                  const int* __restrict__ cs, const GroupSet& t, R B,
                                                  int& nrow, int& total) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = 0;
    if (lane < 9) {
        const int dz = lane / 3 - 1, dy = lane % 3 - 1;
        const float db = float(sc.db), b = float(B);
        const float gz = dz < 0 ? t.z0 - float(t.iz - 1) * db : (dz > 0 ? float(t.iz) * db - t.z1 : 0.0f);
        const float gy = dy < 0 ? t.y0 - float(t.iy - 1) * db : (dy > 0 ? float(t.iy) * db - t.y1 : 0.0f);
        const float gz0 = fmaxf(gz, 0.0f), gy0 = fmaxf(gy, 0.0f);
        const float left = b - gz0 * gz0 - gy0 * gy0;
        if (!(left < 0.0f)) {
            const float gl = fmaxf(t.x0 - float(t.ixl - 1) * db, 0.0f),
                        gh = fmaxf(float(t.ixh) * db - t.x1, 0.0f);
            const int row = sc.cbase + (t.iz + dz) * sc.nbxy + (t.iy + dy) * sc.nbx;
            lo = __ldg(cs + row + (gl * gl > left ? t.ixl : t.ixl - 1));
            hi = __ldg(cs + row + (gh * gh > left ? t.ixh : t.ixh + 1) + 1);
        }
    }
    nrow = total = 0;
    group_push(m, lo, hi, nrow, total);
    __syncwarp();
}

// Lists the candidates [w0, w0 + n) of the rows, n <= M::kWindow, padded with index 0 to a
// multiple of 4 G; n is returned
template <int G, class M> __device__ __forceinline__ int group_list(M& m, int nrow, int total, int w0) {
    const int lane = threadIdx.x & 31, n = min(M::kWindow, total - w0);
    __syncwarp();
    for (int r = lane; r < nrow; r += 32) {
        const int b = m.base[r] - w0, k0 = m.lo[r];
        const int i1 = min(m.base[r + 1] - w0, n) - b;
        for (int i = max(0, -b); i < i1; ++i) m.kidx[b + i] = k0 + i;
    }
    for (int i = n + lane; i < (n + 4 * G - 1) / (4 * G) * (4 * G); i += 32) m.kidx[i] = 0;
    __syncwarp();
    return n;
}

// Tests the n listed candidates of `table`, one per lane, against each of the warp's particles in
// turn: near(i, k, q) says whether particle i (of group i) accepts candidate k at q. A ballot per
// particle gives each accepted candidate its place in m.hit[i], in order. Returns the number that
// this lane's particle accepted.
template <int G, class M, class R, class N>
__device__ __forceinline__ int group_test(M& m, const Group<G>& gr, const V4<R>* __restrict__ table,
                                          int n, N&& near) {
    constexpr int P = 32 / G;
    int cnt[P];
#pragma unroll
    for (int i = 0; i < P; ++i) cnt[i] = 0;
    const unsigned below = (1u << gr.lane) - 1u;
#pragma unroll 2
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int o = c0 + gr.lane;
        const V4<R> q = ldg4(table + m.kidx[min(o, n - 1)]);
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const bool ok = near(i, q) && o < n;
            const unsigned b = __ballot_sync(kFull, ok);
            if (ok) m.hit[i][cnt[i] + __popc(b & below)] = (unsigned short)o;
            cnt[i] += __popc(b);
        }
    }
    __syncwarp();
    int mine = cnt[0];
#pragma unroll
    for (int i = 1; i < P; ++i)
        if (gr.g == i) mine = cnt[i];
    return mine;
}

// Particle i's values for every lane of the warp: its position, slot and whether it takes part
template <class R, int P> struct GroupPts {
    R x[P], y[P], z[P];
    int s[P];
    unsigned in;
    template <int G>
    __device__ __forceinline__ GroupPts(const Group<G>&, const V4<R>& p, int slot, unsigned lanes) {
        in = 0u;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            x[i] = __shfl_sync(kFull, p.x, i * G);
            y[i] = __shfl_sync(kFull, p.y, i * G);
            z[i] = __shfl_sync(kFull, p.z, i * G);
            s[i] = __shfl_sync(kFull, slot, i * G);
            in |= ((lanes >> (i * G)) & 1u) << i;
        }
    }
    __device__ __forceinline__ R d2(int i, const V4<R>& q) const {
        const R dx = q.x - x[i], dy = q.y - y[i], dz = q.z - z[i];
        return dot3(dx, dy, dz, dx, dy, dz);
    }
    __device__ __forceinline__ bool on(int i) const { return (in >> i) & 1u; }
};

// s = fma(term[c][i], term[w][i], s) over entries [0, n) in order, for this lane's component c;
// entries are padded with zeros to a multiple of four
__device__ __forceinline__ float chain4(const float* a, const float* w, float s) {
    const float4 x = *reinterpret_cast<const float4*>(a), y = *reinterpret_cast<const float4*>(w);
    s = __fmaf_rn(x.x, y.x, s);
    s = __fmaf_rn(x.y, y.y, s);
    s = __fmaf_rn(x.z, y.z, s);
    return __fmaf_rn(x.w, y.w, s);
}
__device__ __forceinline__ double chain4(const double* a, const double* w, double s) {
    const double2 x = *reinterpret_cast<const double2*>(a), y = *reinterpret_cast<const double2*>(w),
                  p = *reinterpret_cast<const double2*>(a + 2), q = *reinterpret_cast<const double2*>(w + 2);
    s = __fma_rn(x.x, y.x, s);
    s = __fma_rn(x.y, y.y, s);
    s = __fma_rn(p.x, q.x, s);
    return __fma_rn(p.y, q.y, s);
}
__device__ __forceinline__ float add4(const float* a, float s) {
    const float4 x = *reinterpret_cast<const float4*>(a);
    return (((s + x.x) + x.y) + x.z) + x.w;
}
__device__ __forceinline__ double add4(const double* a, double s) {
    const double2 x = *reinterpret_cast<const double2*>(a), y = *reinterpret_cast<const double2*>(a + 2);
    return (((s + x.x) + x.y) + y.x) + y.y;
}

// Vector terms of the cnt accepted candidates, kGroupChunk at a time: f(h, on, k) gives the term
// of neighbour h (table index k) as (x, y, z, w), zeros where `on` is false; the sum of this
// lane's component (lanes 0-2 of a group: x, y, z) advances by fma(x, w, s) in order. t0: the
// first of four term arrays.
template <int G, class M, class R, class F>
__device__ __forceinline__ void group_sum(M& m, const Group<G>& gr, int cnt, R& s, F&& f) {
    const int most = G == 32 ? cnt : __reduce_max_sync(kFull, cnt);
    for (int h0 = 0; h0 < most; h0 += kGroupChunk) {
        const int n = min(kGroupChunk, most - h0);
#pragma unroll 2
        for (int u = 0; u < n; u += G) {
            const int h = h0 + u + gr.l;
            const bool on = h < cnt;
            const V4<R> t = f(h, on, m.kidx[on ? m.hit[gr.g][h] : 0]);
            m.term[0][gr.g][u + gr.l] = t.x;
            m.term[1][gr.g][u + gr.l] = t.y;
            m.term[2][gr.g][u + gr.l] = t.z;
            m.term[3][gr.g][u + gr.l] = t.w;
        }
        __syncwarp();
        if (gr.l < 3)
            for (int i = 0; i < n; i += 4)
                s = chain4(&m.term[gr.l][gr.g][i], &m.term[3][gr.g][i], s);
        __syncwarp();
    }
}

// Whether positions p and q lie in adjacent buckets. Asked of pairs whose distance is within
// rounding of the bucket width only, so out of line.
template <class R, class RN>
__device__ __noinline__ bool bucket_adjacent(const SceneDev<R, RN>& sc, R px, R py, R pz, R qx, R qy,
                                             R qz) {
    int ix, iy, iz, jx, jy, jz;
    cell_of(sc, px, py, pz, ix, iy, iz);
    cell_of(sc, qx, qy, qz, jx, jy, jz);
    return abs(jx - ix) <= 1 && abs(jy - iy) <= 1 && abs(jz - iz) <= 1;
}

}  // namespace mps
