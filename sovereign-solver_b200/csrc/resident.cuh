// resident.cuh -- an LP's iterations inside one thread-block cluster.
//
// The iteration of a small LP is latency: a pass of it is one load of the row's
// extent, one of its entries, one gather and one store, each a trip to L2,
// whatever the LP's size. Here a cluster keeps an LP in its shared memory and
// iterates there (the updates of src/l1/pdhg.cpp:295-331 as fast_common.cuh
// writes them). Each CTA owns a range of A^T's rows (columns) and one of A's,
// with their entries, bounds and iterates, and a copy of the two gathered
// vectors, x_bar and y. After each pass a CTA sends its slice of the vector it
// wrote to the others' copies, and a cluster barrier (a block barrier where the
// cluster is one CTA) stands where the kernel boundary stood.
//
// What a pass costs is shared-memory bandwidth and instructions, so the rows
// are ordered by length and stored lane-interleaved in slices of one warp: a
// slice's lanes run the same number of steps and its entries are read without
// bank conflicts; only the gathers conflict. Row by row (each lane reading its
// own row's entries) a pass over 500 rows of 12 entries took 3,900 cycles of
// one SM. A long row's sum has long_row_dot's order; a short one's is that of
// the kernels over all instances only where those give it as many lanes (here
// at most four, batch.cu lanes_log2), so the iterates differ by rounding.
//
// Measured on a B200, in cycles: block barrier 43, cluster barrier 470 at any
// size, a vector of 4 KB / 16 KB / 40 KB to all CTAs with the barrier 1,140 /
// 1,640 / 2,650 for eight CTAs in 16-byte stores (by each row's owner in
// 8-byte stores twice that). So an LP gets as few CTAs as hold it.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "engine.cuh"
#include "fast_common.cuh"

namespace pdhg {
namespace {

namespace cg = cooperative_groups;

// Dynamic shared memory a CTA may have, beside the kernels' static part (up to
// 10.6 KB): together the 227 KB of a block. Past that no cluster could be
// scheduled (res_largest_cluster), and every LP would take the slower kernels;
// so each kernel asserts its part.
constexpr uint32_t kResMaxSmem = 216 * 1024;
constexpr uint32_t kResStaticSmem = 227 * 1024 - kResMaxSmem;
constexpr int kResWeights = 64;    // Halpern weights tabulated at a time

__host__ __device__ constexpr uint32_t res_align(uint32_t b) { return (b + 15u) / 16u * 16u; }

// Shared memory is addressed by 32-bit offsets into the CTA's dynamic part, so
// that every access is a shared-memory instruction with a short address.
extern __shared__ __align__(16) unsigned char res_smem[];
template <class V>
__device__ __forceinline__ V& res_at(uint32_t off) {
    return *reinterpret_cast<V*>(res_smem + off);
}

template <class T>
struct ResVec;
template <>
struct ResVec<float> {
    using Two = float2;
};
template <>
struct ResVec<double> {
    using Two = double2;
};

// A part's entries: value and column's byte offset in the gathered vector
// (FP32: one 8-byte pair, so that an entry costs two loads and a
// multiply-add; FP64: the value, and the column apart in 16 bits).
// FAR: in global memory instead, for an LP whose entries no cluster's shared
// memory holds; its vectors and operands stay in shared memory, the entries
// stream from L2 every iteration, read by the CTA that wrote them.
template <class T, bool FAR>
struct ResEntries;
template <>
struct ResEntries<float, false> {
    uint32_t e = 0;
    __host__ __device__ static uint32_t bytes(uint32_t nnz) { return res_align(8 * nnz); }
    __device__ uint32_t place(uint32_t p, uint32_t nnz) {
        e = p;
        return p + bytes(nnz);
    }
    __device__ __forceinline__ void set(uint32_t k, uint32_t col, float v) const {
        res_at<uint2>(e + 8u * k) = make_uint2(__float_as_uint(v), 4u * col);
    }
    __device__ __forceinline__ void get(uint32_t k, uint32_t& off, float& v) const {
        const uint2 q = res_at<uint2>(e + 8u * k);
        v = __uint_as_float(q.x);
        off = q.y;
    }
};
template <>
struct ResEntries<double, false> {
    uint32_t v = 0, c = 0;
    __host__ __device__ static uint32_t bytes(uint32_t nnz) { return res_align(8 * nnz) + res_align(2 * nnz); }
    __device__ uint32_t place(uint32_t p, uint32_t nnz) {
        v = p;
        c = p + res_align(8 * nnz);
        return p + bytes(nnz);
    }
    __device__ __forceinline__ void set(uint32_t k, uint32_t col, double x) const {
        res_at<uint16_t>(c + 2u * k) = static_cast<uint16_t>(col);
        res_at<double>(v + 8u * k) = x;
    }
    __device__ __forceinline__ void get(uint32_t k, uint32_t& off, double& x) const {
        off = 8u * res_at<uint16_t>(c + 2u * k);
        x = res_at<double>(v + 8u * k);
    }
};
template <>
struct ResEntries<float, true> {
    uint2* e = nullptr;
    __host__ __device__ static uint32_t bytes(uint32_t) { return 0; }
    __device__ uint32_t place(uint32_t p, uint32_t) { return p; }
    __device__ void place_far(unsigned char* at, uint32_t) { e = reinterpret_cast<uint2*>(at); }
    __device__ __forceinline__ void set(uint32_t k, uint32_t col, float v) const {
        e[k] = make_uint2(__float_as_uint(v), 4u * col);
    }
    __device__ __forceinline__ void get(uint32_t k, uint32_t& off, float& v) const {
        const uint2 q = e[k];
        v = __uint_as_float(q.x);
        off = q.y;
    }
};
template <>
struct ResEntries<double, true> {
    double* v = nullptr;
    uint16_t* c = nullptr;
    __host__ __device__ static uint32_t bytes(uint32_t) { return 0; }
    __device__ uint32_t place(uint32_t p, uint32_t) { return p; }
    __device__ void place_far(unsigned char* at, uint32_t nnz) {
        v = reinterpret_cast<double*>(at);
        c = reinterpret_cast<uint16_t*>(at + 8 * static_cast<size_t>(nnz));
    }
    __device__ __forceinline__ void set(uint32_t k, uint32_t col, double x) const {
        c[k] = static_cast<uint16_t>(col);
        v[k] = x;
    }
    __device__ __forceinline__ void get(uint32_t k, uint32_t& off, double& x) const {
        off = 8u * c[k];
        x = v[k];
    }
};
constexpr uint32_t kResFarEntry = 10;  // bytes of an entry in global memory, at most

// The cluster: this CTA's rank, and the CTAs.
struct ResCluster {
    int rank, size;
    __device__ ResCluster() {
        const cg::cluster_group c = cg::this_cluster();
        rank = static_cast<int>(c.block_rank());
        size = static_cast<int>(c.num_blocks());
    }
    __device__ __forceinline__ void sync() const {
        __syncwarp();
        if (size > 1) cg::this_cluster().sync();
        else __syncthreads();
    }
    // Entries [r0, r1) of the vector at `v` into the other CTAs' copies, then
    // the barrier. r0 is a multiple of four and so is r1 but for the vector's
    // end, which is padded: whole 16-byte stores, the warps dealt out to the
    // CTAs.
    template <int NT, class T>
    __device__ __forceinline__ void publish(uint32_t v, int r0, int r1) const {
        __syncthreads();
        if (size == 1) return;
        const int nv = static_cast<int>((static_cast<uint32_t>(r1 - r0) * sizeof(T) + 15u) / 16u);
        const int warp = static_cast<int>(threadIdx.x >> 5), others = size - 1;
        const int subs = (NT / 32) / others;  // warps per other CTA
        if (warp < subs * others) {
            const int d = 1 + warp % others;
            const int to = rank + d < size ? rank + d : rank + d - size;
            int4* src = &res_at<int4>(v + static_cast<uint32_t>(r0) * static_cast<uint32_t>(sizeof(T)));
            int4* dst = cg::this_cluster().map_shared_rank(src, to);
            for (int x = (warp / others) * 32 + static_cast<int>(threadIdx.x & 31); x < nv; x += 32 * subs)
                dst[x] = src[x];
        }
        sync();
    }
};

// The rows of one matrix that a CTA owns: rows [r0, r1), counted from the
// LP's first. `perm` lists them by slot: first the n_short rows of at most
// kLongRow entries, longest first, 32 >> lg to a slice, then the n_long
// others, each summed by a warp. Slice s's step k is the 32 entries at
// meta[s].x + 32 k, lane l on entry (l mod lanes) + k lanes of its row; a short
// row's missing entries are zeros at the vector's zero slot. Long row q's
// entries are [ext[q].x, ext[q].y), with its skew (res_long_dot) in the upper
// two bits of ext[q].y. A slot's operands are one record of four,
// {x, sum, c, anchor of x} for a column and {s, sum, lower, upper bound} for a
// row, and one pair: the column's bounds, or the row's anchors of s and y
// (Halpern).
template <class T, bool FAR>
struct ResSlab {
    int r0 = 0, r1 = 0;
    int lg = 0;  // log2 of the lanes per row
    int n_short = 0, n_slice = 0, n_long = 0;
    uint32_t meta = 0, perm = 0, ext = 0, rec = 0, pair = 0;
    ResEntries<T, FAR> e;

    // Entries of `rows` rows with `nnz` entries in slices, padding included:
    // each lane's rounding up, and the slices' steps, which only fall from the
    // longest short row's.
    __host__ __device__ static uint32_t entries(uint32_t rows, uint32_t nnz, uint32_t longest, int lg) {
        return nnz + (((1u << lg) - 1u) * rows) + 32u * ((longest >> lg) + 2u);
    }
    __host__ __device__ static uint32_t slices(uint32_t rows, int lg) { return ((rows << lg) + 31u) / 32u + 1u; }
    __host__ __device__ static uint32_t longs(uint32_t nnz) { return nnz / (kLongRow + 1u) + 1u; }
    __host__ __device__ static uint32_t bytes(uint32_t rows, uint32_t nnz, uint32_t longest, int lg, bool pairs) {
        constexpr uint32_t t = sizeof(T);
        return res_align(4 * t * rows) + (pairs ? res_align(2 * t * rows) : 0) +
               ResEntries<T, FAR>::bytes(entries(rows, nnz, longest, lg)) + res_align(8 * slices(rows, lg)) +
               res_align(4 * rows) + res_align(8 * longs(nnz));
    }
    __device__ uint32_t place(uint32_t p, uint32_t rows, uint32_t nnz, uint32_t longest, int lg_, bool pairs) {
        constexpr uint32_t t = sizeof(T);
        lg = lg_;
        rec = p;
        p += res_align(4 * t * rows);
        pair = p;
        if (pairs) p += res_align(2 * t * rows);
        p = e.place(p, entries(rows, nnz, longest, lg));
        meta = p;
        p += res_align(8 * slices(rows, lg));
        perm = p;
        p += res_align(4 * rows);
        ext = p;
        return p + res_align(8 * longs(nnz));
    }
    __device__ __forceinline__ int row_of(int slot) const {
        return res_at<int32_t>(perm + 4u * static_cast<uint32_t>(slot));
    }
    __device__ __forceinline__ T& operand(int slot, int q) const {
        return res_at<T>(rec + (4u * static_cast<uint32_t>(slot) + static_cast<uint32_t>(q)) * sizeof(T));
    }
    __device__ __forceinline__ T& paired(int slot, int q) const {
        return res_at<T>(pair + (2u * static_cast<uint32_t>(slot) + static_cast<uint32_t>(q)) * sizeof(T));
    }
};

// Scratch of res_load_rows.
struct ResBuild {
    int count[kLongRow + 2], at[kLongRow + 2];
};

// Rows [r0, r1) of M's rows from row0 on (columns from col0 on; `zero`: the
// gathered vector's zero slot) into S.
template <int NT, class T, bool FAR>
__device__ __forceinline__ void res_load_rows(ResSlab<T, FAR>& S, const DevCsr& M, int row0, int col0, int r0, int r1,
                                              uint32_t zero, ResBuild& B) {
    S.r0 = r0;
    S.r1 = r1;
    const int nr = r1 - r0, lg = S.lg, vw = 1 << lg;
    const int32_t* __restrict__ rp = M.rp + row0 + r0;
    const T* __restrict__ vals = mvals<T>(M);
    const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, warp = tid >> 5;
    constexpr int kLong = kLongRow + 1;
    auto width = [&](int i) {  // steps of a short row
        const int len = __ldg(rp + i + 1) - __ldg(rp + i);
        return len <= kLongRow ? (len + vw - 1) >> lg : kLong;
    };
    for (int q = tid; q <= kLong; q += NT) B.count[q] = 0;
    __syncthreads();
    for (int i = tid; i < nr; i += NT) atomicAdd(&B.count[width(i)], 1);
    __syncthreads();
    if (warp == 0) {  // slots of each width, the widest first
        int at = 0;
        for (int w0 = kLongRow; w0 >= 0; w0 -= 32) {
            const int w = w0 - lane;
            int sum = w >= 0 ? B.count[w] : 0;
            const int own = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += y;
            }
            if (w >= 0) B.at[w] = at + sum - own;
            at += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) B.at[kLong] = at;
    }
    __syncthreads();
    S.n_short = B.at[kLong];
    S.n_long = nr - S.n_short;
    __syncthreads();
    for (int i = tid; i < nr; i += NT)
        res_at<int32_t>(S.perm + 4u * static_cast<uint32_t>(atomicAdd(&B.at[width(i)], 1))) = i;
    __syncthreads();
    const int per = 32 >> lg;  // rows of a slice
    S.n_slice = (S.n_short + per - 1) / per;
    if (warp == 0) {  // the slices' extents, then the long rows'
        int at = 0;
        for (int s0 = 0; s0 < S.n_slice; s0 += 32) {
            const int s = s0 + lane;
            const int w = s < S.n_slice ? width(S.row_of(s * per)) : 0;
            int sum = w;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += y;
            }
            if (s < S.n_slice)
                res_at<int2>(S.meta + 8u * static_cast<uint32_t>(s)) = make_int2(at + 32 * (sum - w), w);
            at += 32 * __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0)
            for (int q = 0; q < S.n_long; ++q) {
                const int i = S.row_of(S.n_short + q), b = __ldg(rp + i), len = __ldg(rp + i + 1) - b;
                const uint32_t skew = static_cast<uint32_t>(b) % (16u / sizeof(T));
                res_at<int2>(S.ext + 8u * static_cast<uint32_t>(q)) =
                    make_int2(at, static_cast<int>(static_cast<uint32_t>(at + len) | skew << 30));
                at += len;
            }
    }
    __syncthreads();
    for (int s = warp; s < S.n_slice; s += NT / 32) {
        const int2 m = res_at<int2>(S.meta + 8u * static_cast<uint32_t>(s));
        const int slot = s * per + (lane >> lg);
        int b = 0, e = 0;
        if (slot < S.n_short) {
            const int i = S.row_of(slot);
            b = __ldg(rp + i) + (lane & (vw - 1));
            e = __ldg(rp + i + 1);
        }
        for (int k = 0; k < m.y; ++k) {
            const int src = b + (k << lg);
            const bool ok = src < e;
            S.e.set(static_cast<uint32_t>(m.x + 32 * k + lane),
                    ok ? static_cast<uint32_t>(__ldg(M.ci + src) - col0) : zero, ok ? __ldg(vals + src) : T(0));
        }
    }
    for (int q = warp; q < S.n_long; q += NT / 32) {
        const int2 x = res_at<int2>(S.ext + 8u * static_cast<uint32_t>(q));
        const int b = __ldg(rp + S.row_of(S.n_short + q)), len = (x.y & 0x3fffffff) - x.x;
        for (int k = lane; k < len; k += 32)
            S.e.set(static_cast<uint32_t>(x.x + k), static_cast<uint32_t>(__ldg(M.ci + b + k) - col0),
                    __ldg(vals + b + k));
    }
    __syncthreads();
}

// What a pass needs besides its slab.
template <class T>
struct ResStep {
    T tau, sigma, w;  // w: the Halpern weight
    int zero_sums;
};

// epi_load and epi_store (fast_common.cuh) of one slot, z's x part always
// stored; the new x_bar or y entry goes to `out` (y's old one is read there).
template <class T, bool PRIMAL, bool HALPERN, bool FAR>
__device__ __forceinline__ void res_update(const ResSlab<T, FAR>& S, int slot, T& out, T dot, const ResStep<T>& p) {
    using Two = typename ResVec<T>::Two;
    constexpr uint32_t t = sizeof(T);
    const uint32_t at = S.rec + 4u * t * static_cast<uint32_t>(slot);
    const uint32_t at2 = S.pair + 2u * t * static_cast<uint32_t>(slot);
    const Two r0 = res_at<Two>(at), r1 = res_at<Two>(at + 2u * t);
    const T ps = HALPERN || p.zero_sums ? T(0) : r0.y;
    Two st;
    if (PRIMAL) {
        const Two box = res_at<Two>(at2);
        const T xo = r0.x;
        const T xn = clampT<T>(xo - p.tau * (r1.x - dot), box.x, box.y);
        const T xb = T(2) * xn - xo;
        st.x = HALPERN ? halpern_mix<T>(p.w, xb, r1.y) : xn;
        st.y = HALPERN ? xn : ps + xn;
        out = xb;
    } else {
        const T yo = out, so = r0.x;
        const T sn = clampT<T>(so - p.tau * yo, r1.x, r1.y);
        const T sb = T(2) * sn - so;
        const T yn = yo + p.sigma * (sb - dot);
        if (HALPERN) {
            const Two a = res_at<Two>(at2);
            st.x = halpern_mix<T>(p.w, sb, a.x);
            st.y = yn;
            out = halpern_mix<T>(p.w, T(2) * yn - yo, a.y);
        } else {
            st.x = sn;
            st.y = ps + yn;
            out = yn;
        }
    }
    res_at<Two>(at) = st;
}

// `cnt` entries k, k + 32, ... added in this order, four of each stream in
// flight.
template <class T, bool FAR>
__device__ __forceinline__ T res_dot(const ResEntries<T, FAR>& E, uint32_t k, int cnt, uint32_t xg) {
    T acc = T(0);
    for (; cnt >= 4; cnt -= 4, k += 128u) {
        uint32_t c[4];
        T v[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) E.get(k + 32u * u, c[u], v[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) g[u] = res_at<T>(xg + c[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) acc += v[u] * g[u];
    }
    if (cnt & 2) {
        uint32_t c0, c1;
        T v0, v1;
        E.get(k, c0, v0);
        E.get(k + 32u, c1, v1);
        const T g0 = res_at<T>(xg + c0), g1 = res_at<T>(xg + c1);
        acc += v0 * g0;
        acc += v1 * g1;
        k += 64u;
    }
    if (cnt & 1) {
        uint32_t c0;
        T v0;
        E.get(k, c0, v0);
        acc += v0 * res_at<T>(xg + c0);
    }
    return acc;
}

// Long row [b, e) of the local entries by one warp in long_row_dot's order: the
// kBlock threads' sums (over whole 16-byte vectors of the row's values in
// global memory, whose entry 0 of the row is `skew` past a vector's start), the
// tree over each 32 of them, the tree over those.
template <class T, bool FAR>
__device__ __forceinline__ T res_long_dot(const ResEntries<T, FAR>& E, int b, int e, int skew, uint32_t xg) {
    constexpr int W = 16 / sizeof(T);
    const int lane = static_cast<int>(threadIdx.x & 31);
    int bA = b + (W - skew) % W;
    if (bA > e) bA = e;
    const int nvec = (e - bA) / W;
    T tot[kBlock / 32];
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) {
        const int t = 32 * w + lane;
        T acc = T(0);
        auto one = [&](int k) {
            uint32_t c;
            T v;
            E.get(static_cast<uint32_t>(k), c, v);
            acc += v * res_at<T>(xg + c);
        };
        for (int k = b + t; k < bA; k += kBlock) one(k);
        for (int q = t; q < nvec; q += kBlock) {
            uint32_t c[W];
            T v[W];
#pragma unroll
            for (int u = 0; u < W; ++u) E.get(static_cast<uint32_t>(bA + W * q + u), c[u], v[u]);
            if constexpr (W == 4) {
                acc += v[0] * res_at<T>(xg + c[0]) + v[1] * res_at<T>(xg + c[1]) + v[2] * res_at<T>(xg + c[2]) +
                       v[3] * res_at<T>(xg + c[3]);
            } else {
                acc += v[0] * res_at<T>(xg + c[0]) + v[1] * res_at<T>(xg + c[1]);
            }
        }
        for (int k = bA + nvec * W + t; k < e; k += kBlock) one(k);
        __syncwarp();
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        tot[w] = acc;
    }
    return ((tot[0] + tot[4]) + (tot[2] + tot[6])) + ((tot[1] + tot[5]) + (tot[3] + tot[7]));
}

// One pass (primal: rows of A^T gather y; dual: rows of A gather x_bar) over
// the CTA's rows; xg: the gathered vector, vec: the other one.
template <int NT, class T, bool PRIMAL, bool HALPERN, bool FAR>
__device__ __forceinline__ void res_pass(const ResSlab<T, FAR>& S, uint32_t xg, uint32_t vec, const ResStep<T>& p) {
    constexpr uint32_t t = sizeof(T);
    const uint32_t out = vec + t * static_cast<uint32_t>(S.r0);
    const int lane = static_cast<int>(threadIdx.x & 31), warp = static_cast<int>(threadIdx.x >> 5);
    const int lg = S.lg, vw = 1 << lg;
    for (int s = warp; s < S.n_slice; s += NT / 32) {
        const int2 m = res_at<int2>(S.meta + 8u * static_cast<uint32_t>(s));
        const int slot = s * (32 >> lg) + (lane >> lg);
        T acc = res_dot(S.e, static_cast<uint32_t>(m.x + lane), m.y, xg);
        for (int o = vw >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if ((lane & (vw - 1)) == 0 && slot < S.n_short)
            res_update<T, PRIMAL, HALPERN, FAR>(S, slot, res_at<T>(out + t * static_cast<uint32_t>(S.row_of(slot))), acc, p);
        __syncwarp();
    }
    for (int q = warp; q < S.n_long; q += NT / 32) {
        const int2 x = res_at<int2>(S.ext + 8u * static_cast<uint32_t>(q));
        const int slot = S.n_short + q;
        const T acc = res_long_dot(S.e, x.x, x.y & 0x3fffffff, static_cast<int>(static_cast<uint32_t>(x.y) >> 30), xg);
        if (lane == 0)
            res_update<T, PRIMAL, HALPERN, FAR>(S, slot, res_at<T>(out + t * static_cast<uint32_t>(S.row_of(slot))), acc, p);
        __syncwarp();
    }
}

// An LP on a cluster: its vectors (one entry more than the LP's, the zero
// slot) and its two slabs, P over A^T's rows and D over A's.
template <class T, bool FAR>
struct ResLp {
    int n = 0, m = 0;  // columns, rows
    uint32_t xb = 0, y = 0;
    ResSlab<T, FAR> P, D;
    __host__ __device__ static uint32_t vec_bytes(uint32_t n, uint32_t m) {
        constexpr uint32_t t = sizeof(T);
        return res_align(t * (n + 1)) + res_align(t * (m + 1));
    }
    __device__ uint32_t place(int n_, int m_) {
        constexpr uint32_t t = sizeof(T);
        n = n_;
        m = m_;
        xb = 0;
        y = res_align(t * (static_cast<uint32_t>(n) + 1u));
        return vec_bytes(static_cast<uint32_t>(n), static_cast<uint32_t>(m));
    }
};

template <class T>
__device__ __forceinline__ T* sums_x(const Iterates<T>& it) {
    if constexpr (std::is_same<T, float>::value) return it.psx;
    else return it.xsum;
}
template <class T>
__device__ __forceinline__ T* sums_y(const Iterates<T>& it) {
    if constexpr (std::is_same<T, float>::value) return it.psy;
    else return it.ysum;
}

// The operands of an LP whose columns start at c0 and rows at r0 of the
// arrays: what stays, and the iterates before and after a run.
template <int NT, class T, bool FAR>
__device__ __forceinline__ void res_load_fixed(const ResLp<T, FAR>& L, const PV<T>& pv, int c0, int r0) {
    constexpr uint32_t t = sizeof(T);
    const int nc = L.P.r1 - L.P.r0, nr = L.D.r1 - L.D.r0;
    for (int i = threadIdx.x; i < nc; i += NT) {
        const int g = c0 + L.P.r0 + L.P.row_of(i);
        L.P.operand(i, 2) = pv.c[g];
        L.P.paired(i, 0) = pv.lo[g];
        L.P.paired(i, 1) = pv.hi[g];
    }
    for (int i = threadIdx.x; i < nr; i += NT) {
        const int g = r0 + L.D.r0 + L.D.row_of(i);
        L.D.operand(i, 2) = pv.rlo[g];
        L.D.operand(i, 3) = pv.rhi[g];
    }
    // the vectors' zero slots and padding
    for (uint32_t i = threadIdx.x + static_cast<uint32_t>(L.n); t * i < L.y - L.xb; i += NT) res_at<T>(L.xb + t * i) = T(0);
    const uint32_t ym = res_align(t * (static_cast<uint32_t>(L.m) + 1u));
    for (uint32_t i = threadIdx.x + static_cast<uint32_t>(L.m); t * i < ym; i += NT) res_at<T>(L.y + t * i) = T(0);
}
template <int NT, class T, bool FAR>
__device__ __forceinline__ void res_load_iterates(const ResLp<T, FAR>& L, const Iterates<T>& it, int c0, int r0) {
    constexpr uint32_t t = sizeof(T);
    const int nc = L.P.r1 - L.P.r0, nr = L.D.r1 - L.D.r0;
    const T *px = sums_x(it), *py = sums_y(it);
    for (int i = threadIdx.x; i < nc; i += NT) {
        const int g = c0 + L.P.r0 + L.P.row_of(i);
        L.P.operand(i, 0) = it.x[g];
        if (it.halpern) L.P.operand(i, 3) = it.xa[g];
        else L.P.operand(i, 1) = px[g];
    }
    for (int i = threadIdx.x; i < nr; i += NT) {
        const int g = r0 + L.D.r0 + L.D.row_of(i);
        L.D.operand(i, 0) = it.s[g];
        if (it.halpern) {
            L.D.paired(i, 0) = it.sa[g];
            L.D.paired(i, 1) = it.ya[g];
        } else {
            L.D.operand(i, 1) = py[g];
        }
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < L.m; i += NT) res_at<T>(L.y + t * static_cast<uint32_t>(i)) = it.y[r0 + i];
}
template <int NT, class T, bool FAR>
__device__ __forceinline__ void res_store_iterates(const ResLp<T, FAR>& L, const Iterates<T>& it, int c0, int r0) {
    constexpr uint32_t t = sizeof(T);
    const int nc = L.P.r1 - L.P.r0, nr = L.D.r1 - L.D.r0;
    T *px = sums_x(it), *py = sums_y(it);
    for (int i = threadIdx.x; i < nc; i += NT) {
        const int g = c0 + L.P.r0 + L.P.row_of(i);
        it.x[g] = L.P.operand(i, 0);
        px[g] = L.P.operand(i, 1);
        it.xbar[c0 + L.P.r0 + i] = res_at<T>(L.xb + t * static_cast<uint32_t>(L.P.r0 + i));
    }
    for (int i = threadIdx.x; i < nr; i += NT) {
        const int g = r0 + L.D.r0 + L.D.row_of(i);
        it.s[g] = L.D.operand(i, 0);
        py[g] = L.D.operand(i, 1);
        it.y[r0 + L.D.r0 + i] = res_at<T>(L.y + t * static_cast<uint32_t>(L.D.r0 + i));
    }
}

// Iterations [0, count) of a check period. weights: kResWeights of shared
// memory.
template <int NT, class T, bool HALPERN, bool FAR>
__device__ __forceinline__ void res_iterate(const ResLp<T, FAR>& L, const ResCluster& cl, ResStep<T>& p,
                                            const Iterates<T>& it, long long since, long long count, bool fresh,
                                            T* weights) {
    for (long long t = 0; t < count; ++t) {
        if (HALPERN) {
            const int q = static_cast<int>(t % kResWeights);
            if (q == 0) {
                __syncthreads();
                if (threadIdx.x < kResWeights)
                    weights[threadIdx.x] = halpern_weight<T>(it, since + t, static_cast<int>(threadIdx.x)).w;
                __syncthreads();
            }
            p.w = weights[q];
        }
        // FP32 sums are the period's, FP64 ones go on until a restart
        p.zero_sums = t == 0 && (std::is_same<T, float>::value || fresh);
        res_pass<NT, T, true, HALPERN, FAR>(L.P, L.y, L.xb, p);
        cl.publish<NT, T>(L.xb, L.P.r0, L.P.r1);
        res_pass<NT, T, false, HALPERN, FAR>(L.D, L.xb, L.y, p);
        cl.publish<NT, T>(L.y, L.D.r0, L.D.r1);
    }
}

// ---- host side ----------------------------------------------------------------

// Shared memory of an LP (its matrices' parts) on `c` CTAs in precision T, more
// than kResMaxSmem where it cannot be addressed, and the most entries of a
// CTA's two slabs.
struct ResSize {
    uint32_t smem = 0;
    uint32_t entries[2] = {0, 0};
};
template <class T, bool FAR>
ResSize res_size(const ResParts& pt, const ResParts& pa, int c, int lgt, int lga, bool halpern) {
    ResSize z;
    z.smem = kResMaxSmem + 1;
    const int64_t n = pt.row[kResMaxCluster], m = pa.row[kResMaxCluster];
    if (n > 0xfffe || m > 0xfffe) return z;
    const int per = kResMaxCluster / c;
    int64_t rows[2] = {0, 0}, nnz[2] = {0, 0};
    for (int w = 0; w < 2; ++w) {
        const ResParts& p = w ? pa : pt;
        for (int q = 0; q + per <= kResMaxCluster; q += per) {
            if (p.row[q + per] - p.row[q] > rows[w]) rows[w] = p.row[q + per] - p.row[q];
            if (p.nz[q + per] - p.nz[q] > nnz[w]) nnz[w] = p.nz[q + per] - p.nz[q];
        }
    }
    if (nnz[0] > (1 << 24) || nnz[1] > (1 << 24)) return z;  // 32-bit sizes below
    const uint32_t r0 = static_cast<uint32_t>(rows[0]), r1 = static_cast<uint32_t>(rows[1]);
    const uint32_t z0 = static_cast<uint32_t>(nnz[0]), z1 = static_cast<uint32_t>(nnz[1]);
    const uint32_t l0 = static_cast<uint32_t>(pt.longest), l1 = static_cast<uint32_t>(pa.longest);
    z.entries[0] = ResSlab<T, FAR>::entries(r0, z0, l0, lgt);
    z.entries[1] = ResSlab<T, FAR>::entries(r1, z1, l1, lga);
    z.smem = ResLp<T, FAR>::vec_bytes(static_cast<uint32_t>(n), static_cast<uint32_t>(m)) +
             ResSlab<T, FAR>::bytes(r0, z0, l0, lgt, true) + ResSlab<T, FAR>::bytes(r1, z1, l1, lga, halpern);
    return z;
}

// Lets `kernel` use kResMaxSmem and clusters up to 16; the largest size (a
// power of two) the device schedules that way, 0 on an error. active: how many
// clusters of 1, 2, ... 16 CTAs with that much run at once (an SM each, and a
// cluster's SMs near each other: fewer than the SMs would give).
template <class K>
int res_largest_cluster(K kernel, int threads, int* active = nullptr) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kResMaxSmem)) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return 0;
    int largest = 1;
    for (int c = 1, q = 0; c <= kResMaxCluster; c *= 2, ++q) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(c));
        cfg.blockDim = dim3(static_cast<unsigned>(threads));
        cfg.dynamicSmemBytes = kResMaxSmem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = static_cast<unsigned>(c);
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) cudaGetLastError();
        if (active != nullptr) active[q] = n;
        if (n > 0) largest = c;
    }
    return largest;
}

template <class... P, class... Q>
cudaError_t res_launch(void (*kernel)(P...), int clusters, int size, int threads, uint32_t smem, cudaStream_t s,
                       const Q&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * size));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = static_cast<unsigned>(size);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = size > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace
}  // namespace pdhg
