// exact_resident.cu -- a check period's FP64-exact iterations of a small LP in
// one launch of one cluster (resident.cuh): what as many ex_primal and ex_dual
// passes do, every product and sum rounded in the reference's order
// (src/l1/pdhg.cpp:295-331).
//
// Bound: the latency of a pass (barrier, one row's chain of ordered sums, the
// publication to the cluster); a launched pass costs 2-3 us whatever the LP's
// size. One lane takes a row, so rows of more than kExactRow entries would be
// the pass: those LPs keep the passes.
//
// Measured, us an iteration with its share of the check, passes -> here: 60 x
// 150 4.9 -> 1.8 (0.9 without the check), 200 x 500 5.5 -> 2.8, 1,000 x 2,500
// 7.5 -> 4.9, 2,000 x 5,000 (eight CTAs) 7.4 -> 6.0, 2,500 x 6,000 (sixteen)
// 9.4 -> 7.2: faster wherever a cluster holds the LP.
#include <algorithm>
#include <atomic>

#include "resident.cuh"

namespace pdhg {

namespace {

constexpr int kExactRow = 128;

__device__ __forceinline__ double exact_clamp(double v, double lo, double hi) {
    if (v < lo) v = lo;
    if (v > hi) v = hi;
    return v;
}

// One pass over the CTA's rows, a slice per warp at a time. A short row's
// padding adds -0 (primal) or +0 to a sum that is never -0: no change.
template <int NT, bool PRIMAL>
__device__ __forceinline__ void exact_pass(const ResSlab<double, false>& S, uint32_t xg, uint32_t vec, double tau,
                                           double sigma, bool fresh) {
    const uint32_t out = vec + 8u * static_cast<uint32_t>(S.r0);
    const int lane = static_cast<int>(threadIdx.x & 31), warp = static_cast<int>(threadIdx.x >> 5);
    const auto term = [&](uint32_t k) {
        uint32_t c;
        double v;
        S.e.get(k, c, v);
        const double g = res_at<double>(xg + c);
        return __dmul_rn(v, PRIMAL ? -g : g);
    };
    for (int s = warp; s < S.n_slice; s += NT / 32) {
        const int2 m = res_at<int2>(S.meta + 8u * static_cast<uint32_t>(s));
        const int slot = 32 * s + lane;
        const bool mine = slot < S.n_short;
        double acc = PRIMAL && mine ? S.operand(slot, 2) : 0.0;
        uint32_t k = static_cast<uint32_t>(m.x + lane);
        int cnt = m.y;
        for (; cnt >= 4; cnt -= 4, k += 128u) {
            double t[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) t[u] = term(k + 32u * u);
#pragma unroll
            for (int u = 0; u < 4; ++u) acc = __dadd_rn(acc, t[u]);
        }
        for (; cnt > 0; --cnt, k += 32u) acc = __dadd_rn(acc, term(k));
        if (mine) {
            const uint32_t at = S.rec + 32u * static_cast<uint32_t>(slot);
            const double2 r0 = res_at<double2>(at), r1 = res_at<double2>(at + 16u);
            double& o = res_at<double>(out + 8u * static_cast<uint32_t>(S.row_of(slot)));
            double2 st;
            if (PRIMAL) {
                const double2 box = res_at<double2>(S.pair + 16u * static_cast<uint32_t>(slot));
                st.x = exact_clamp(__dadd_rn(r0.x, __dmul_rn(-tau, acc)), box.x, box.y);
                st.y = fresh ? st.x : __dadd_rn(r0.y, st.x);
                o = __dadd_rn(2.0 * st.x, -r0.x);
            } else {
                const double yo = o;
                st.x = exact_clamp(__dadd_rn(r0.x, __dmul_rn(-tau, yo)), r1.x, r1.y);
                const double kb = __dadd_rn(-acc, __dadd_rn(2.0 * st.x, -r0.x));
                const double yn = __dadd_rn(yo, __dmul_rn(sigma, kb));
                st.y = fresh ? yn : __dadd_rn(r0.y, yn);
                o = yn;
            }
            res_at<double2>(at) = st;
        }
        __syncwarp();
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) exact_resident(ExactIter a, ResParts pt, ResParts pa, long long iters) {
    __shared__ ResBuild build;
    static_assert(sizeof(build) <= kResStaticSmem, "beside kResMaxSmem of dynamic shared memory");
    DevState* st = a.st;
    if (st->done) return;  // written by the check kernels only: the same for every CTA
    const ResCluster cl;
    const int per = kResMaxCluster / cl.size, p0 = cl.rank * per, p1 = p0 + per;
    ResLp<double, false> L;
    uint32_t at = L.place(a.AT.rows, a.A.rows);
    at = L.P.place(at, pt.row[p1] - pt.row[p0], pt.nz[p1] - pt.nz[p0], pt.longest, 0, true);
    L.D.place(at, pa.row[p1] - pa.row[p0], pa.nz[p1] - pa.nz[p0], pa.longest, 0, false);
    res_load_rows<NT>(L.P, a.AT, 0, 0, pt.row[p0], pt.row[p1], static_cast<uint32_t>(a.A.rows), build);
    res_load_rows<NT>(L.D, a.A, 0, 0, pa.row[p0], pa.row[p1], static_cast<uint32_t>(a.AT.rows), build);
    res_load_fixed<NT>(L, pvec<double>(a.P), 0, 0);
    res_load_iterates<NT>(L, a.it, 0, 0);
    const double tau = st->tau, sigma = st->sigma;
    const bool fresh0 = st->fresh != 0;
    cl.sync();  // every CTA has its copies before a neighbour writes into them
    if (cl.rank == 0 && threadIdx.x == 0) st->restart = 0;  // consumed by ex_restart
    for (long long t = 0; t < iters; ++t) {
        const bool fresh = t == 0 && fresh0;
        exact_pass<NT, true>(L.P, L.y, L.xb, tau, sigma, fresh);
        cl.publish<NT, double>(L.xb, L.P.r0, L.P.r1);
        exact_pass<NT, false>(L.D, L.xb, L.y, tau, sigma, fresh);
        cl.publish<NT, double>(L.y, L.D.r0, L.D.r1);
    }
    res_store_iterates<NT>(L, a.it, 0, 0);
}

constexpr int kFewThreads = 256, kManyThreads = 1024;
std::atomic<int> g_exact_cluster{0};  // the largest cluster the device schedules

}  // namespace

void init_exact_resident() {
    const int few = res_largest_cluster(exact_resident<kFewThreads>, kFewThreads);
    const int many = res_largest_cluster(exact_resident<kManyThreads>, kManyThreads);
    g_exact_cluster = few > 0 ? many : 0;
}

// The fewest CTAs that hold the LP with at most kExactNnz entries each. Us an
// iteration, with its share of the check, at 1,000 / 2,000 / 4,000 / 8,192
// entries: 200 x 500 3.7 / 3.8 / 2.8 / 2.8, 500 x 1,200 4.0 / 4.1 / 4.5 / 4.5,
// 1,000 x 2,500 5.1 / 5.1 / 4.9 / 5.3.
constexpr int64_t kExactNnz = 4096;
ExactPlan plan_exact_resident(const ResParts& pt, const ResParts& pa, int longest) {
    ExactPlan p;
    const int64_t nnz = pa.nz[kResMaxCluster];
    if (pt.row[kResMaxCluster] < 1 || pa.row[kResMaxCluster] < 1 || longest > kExactRow)
        return p;
    const int most = g_exact_cluster;
    for (int c = 1; c <= most; c *= 2) {
        const ResSize z = res_size<double, false>(pt, pa, c, 0, 0, false);
        if (z.smem > kResMaxSmem || (nnz > kExactNnz * c && 2 * c <= most)) continue;
        p.size = c;
        p.smem = z.smem;
        p.threads = c == 1 && nnz <= 3000 ? kFewThreads : kManyThreads;
        return p;
    }
    return p;
}

void launch_exact_resident(const ExactIter& a, const ExactPlan& p, const ResParts& pt, const ResParts& pa,
                           long long iters, cudaStream_t s) {
    auto run = [&](auto kernel) { res_launch(kernel, 1, p.size, p.threads, p.smem, s, a, pt, pa, iters); };
    if (p.threads == kFewThreads) run(exact_resident<kFewThreads>);
    else run(exact_resident<kManyThreads>);
}

}  // namespace pdhg
