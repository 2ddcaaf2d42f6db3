// batch_resident.cuh -- a batch whose instances fit the shared memory of a
// cluster each: one cluster runs one instance's whole solve (resident.cuh),
// every check period of it with the check, the decision and the restart, and
// the next instance takes its place. No instance waits for another: an
// instance that converges early frees its SMs, where the kernels over all
// instances (batch_kernels.cu) launch two passes an iteration until the slowest
// is done. Those remain for batches with an instance that does not fit.
//
// Bound: an iteration's two dependent passes over shared memory (per entry 8-12
// bytes and a gather that conflicts) and two barriers; many instances: the SMs.
// Measured per iteration, instances of one size, FP32: 60 x 150 1.3 us, 500 x
// 1,200 3.4 us (one or 67 of them), 2,000 x 5,000 4.4 us, 5,000 x 15,000
// (entries in global memory) 10 us. 67 FP64 instances of 500 x 1,200: a check
// period of 40 iterations 519 -> 205 us; 256 FP32 instances of 50 to 5,000 rows
// 2,009 -> 1,173 us. 1,024 threads at 64 registers or 512 at
// 128 for the large classes: within 10% of each other either way.
//
// A translation unit per precision (batch_resident_f32.cu, _f64.cu): the first
// kernel used of one loads all of it onto the device, 5 ms each.
#pragma once

#include <algorithm>
#include <atomic>
#include <cmath>
#include <vector>

#include "batch_device.cuh"
#include "batch_kernels.cuh"
#include "resident.cuh"

namespace pdhg {

namespace {

constexpr int K = kBatchCheckVals;

// Block maxima (values 0..7) and sums (8..15), the warps' results combined in
// warp order: thread q < K gets value q.
template <int NT>
__device__ __forceinline__ double reduce_vals(const double (&v)[K], double (*red)[NT / 32]) {
    const int lane = static_cast<int>(threadIdx.x & 31), warp = static_cast<int>(threadIdx.x >> 5);
#pragma unroll
    for (int q = 0; q < K; ++q) {
        double x = v[q];
        for (int o = 16; o > 0; o >>= 1) {
            const double y = __shfl_xor_sync(0xffffffffu, x, o);
            x = q < 8 ? fmax(x, y) : x + y;
        }
        if (lane == 0) red[q][warp] = x;
    }
    __syncthreads();
    double x = 0.0;
    if (threadIdx.x < K)
        for (int w = 0; w < NT / 32; ++w)
            x = threadIdx.x < 8 ? fmax(x, red[threadIdx.x][w]) : x + red[threadIdx.x][w];
    __syncthreads();
    return x;
}

// The check's products and terms (inst_pass) over the CTA's rows or columns.
template <int NT, class T, bool COLS, bool HALPERN, bool FAR>
__device__ __forceinline__ void check_rows(const BatchView& b, const Iterates<T>& it, const BatchParams& p,
                                           const ResSlab<T, FAR>& S, int first, double inv, double sign, Terms& t) {
    const DevCsr& M = COLS ? b.AT : b.A;
    const int vw = 1 << S.lg;
    const int lane = static_cast<int>(threadIdx.x) & (vw - 1);
    const int r1 = first + S.r1;
    for (int r = first + S.r0 + (static_cast<int>(threadIdx.x) >> S.lg); r < r1; r += NT >> S.lg) {
        double ac = 0.0, aa = 0.0;
        const int e = M.rp[r + 1];
        for (int q = M.rp[r] + lane; q < e; q += vw) {
            const int c = M.ci[q];
            const double v = M.v64[q];
            if (!HALPERN) ac += v * static_cast<double>(COLS ? it.y[c] : it.x[c]);
            aa += v * (COLS ? avg_y<T, HALPERN>(it, c, inv) : avg_x<T, HALPERN>(it, c, inv));
        }
        if (!HALPERN) ac = group_sum(ac, vw);
        aa = group_sum(aa, vw);
        if (HALPERN) ac = aa;  // only T(z) is measured
        if (lane == 0) {
            if (COLS) inst_col_terms(b, it, p, sign, r, ac, aa, inv, t);
            else inst_row_terms(b, it, p, r, ac, aa, inv, t);
        }
    }
}

struct ResJob {
    const int32_t* list;    // instances, one per cluster
    const ResParts* parts;  // per instance: of A^T's rows, of A's
    int lgt, lga;           // log2 of the lanes per row
    // FAR: each cluster's entries in global memory, at `far` + base, P's then
    // D's `entries` per CTA
    const ResFar* where;
    unsigned char* far;
};

// The kernel's static shared memory.
template <class T, int NT>
struct BatchShared {
    union {
        ResBuild build;
        double sum[2][kBlock];
    } scratch;
    double red[K][NT / 32];
    double part[kResMaxCluster][K];  // rank 0: the CTAs' values
    T weights[kResWeights];
    int stop_all;
};

template <class T, int NT, bool FAR>
__global__ void __launch_bounds__(NT, NT == 256 ? 4 : NT == 512 ? 2 : 1)
    batch_resident(BatchView b, Iterates<T> it, BatchParams p, ResJob job, long long iter0, long long n_periods,
                   long long tail) {
    __shared__ BatchShared<T, NT> sh;
    static_assert(sizeof(sh) <= kResStaticSmem, "beside kResMaxSmem of dynamic shared memory");
    auto& scratch = sh.scratch;
    auto& part = sh.part;
    const ResCluster cl;
    const int k = job.list[blockIdx.x / static_cast<unsigned>(cl.size)];
    InstState& s = b.is[k];
    if (s.done) return;  // the same for the cluster's CTAs, which alone run this instance
    const bool lead = cl.rank == 0 && threadIdx.x == 0;
    // A stop request, to the whole cluster. (No CTA writes into another's shared
    // memory before a barrier has shown that it has started.)
    const auto stop_requested = [&]() -> int {
        cl.sync();
        if (lead) {
            const int stop = b.mail != nullptr ? b.mail->stop_request : 0;
            for (int c = 0; c < cl.size; ++c) *cg::this_cluster().map_shared_rank(&sh.stop_all, c) = stop;
        }
        cl.sync();
        return sh.stop_all;
    };
    // ends the instance where it is, `iters` iterations done
    const auto stop_here = [&](int stop, long long iters) {
        if (!lead) return;
        s.done = 1;
        s.status = stop;
        s.stop_iter = iters;
        atomicMax(&b.g->iter, iters);
        finish_instance(b, s);
    };
    // one that came while the instance waited for its cluster
    if (const int stop = stop_requested(); stop != 0) return stop_here(stop, iter0);
    const int c0 = b.col_off[k], r0 = b.row_off[k];
    const int n = b.col_off[k + 1] - c0, m = b.row_off[k + 1] - r0;
    const ResParts &pt = job.parts[2 * k], &pa = job.parts[2 * k + 1];
    const int per = kResMaxCluster / cl.size, p0 = cl.rank * per, p1 = p0 + per;
    ResLp<T, FAR> L;
    uint32_t at = L.place(n, m);
    at = L.P.place(at, pt.row[p1] - pt.row[p0], pt.nz[p1] - pt.nz[p0], pt.longest, job.lgt, true);
    L.D.place(at, pa.row[p1] - pa.row[p0], pa.nz[p1] - pa.nz[p0], pa.longest, job.lga, it.halpern != 0);
    if constexpr (FAR) {
        const ResFar w = job.where[blockIdx.x / static_cast<unsigned>(cl.size)];
        unsigned char* mine = job.far + w.base +
                              static_cast<int64_t>(kResFarEntry) * (w.entries[0] + w.entries[1]) * cl.rank;
        L.P.e.place_far(mine, w.entries[0]);
        L.D.e.place_far(mine + static_cast<int64_t>(kResFarEntry) * w.entries[0], w.entries[1]);
    }
    res_load_rows<NT>(L.P, b.AT, c0, r0, pt.row[p0], pt.row[p1], static_cast<uint32_t>(m), scratch.build);
    res_load_rows<NT>(L.D, b.A, r0, c0, pa.row[p0], pa.row[p1], static_cast<uint32_t>(n), scratch.build);
    const PV<T> pv = pvec<T>(b.P);
    res_load_fixed<NT>(L, pv, c0, r0);
    const double sign = s.obj_sign;
    bool done = false;
    long long periods = 0;
    // whole check periods, then the tail: one body, so that the slabs stay in
    // registers (as a function of its own it reads them from local memory:
    // FP64 500 x 1,200 instances 4.8 -> 8.5 us an iteration)
    for (bool checked = n_periods > 0; !done; checked = periods < n_periods) {
        const long long count = checked ? p.period : tail;
        if (!checked) {
            if (count == 0) break;
            if (periods > 0)
                if (const int stop = stop_requested(); stop != 0) return stop_here(stop, iter0 + periods * p.period);
        }
        res_load_iterates<NT>(L, it, c0, r0);
        ResStep<T> step;
        step.tau = static_cast<T>(s.tau);
        step.sigma = static_cast<T>(s.sigma);
        const long long since = s.since_restart;
        const bool fresh = s.fresh != 0;
        cl.sync();  // every CTA has its copies before a neighbour writes into them
        if (it.halpern) res_iterate<NT, T, true>(L, cl, step, it, since, count, fresh, sh.weights);
        else res_iterate<NT, T, false>(L, cl, step, it, since, count, fresh, sh.weights);
        res_store_iterates<NT>(L, it, c0, r0);
        cl.sync();  // the stored vectors, seen by the whole cluster
        if (!checked) break;
        const long long iter = iter0 + periods * p.period;
        ++periods;
        // ---- check
        // read ahead of its products, so that nobody waits for the host's memory
        const int stop = lead && b.mail != nullptr ? b.mail->stop_request : 0;
        const double inv = it.halpern ? 1.0 : 1.0 / static_cast<double>(s.since_restart + p.period);
        Terms t;
        if (it.halpern) {
            check_rows<NT, T, false, true, FAR>(b, it, p, L.D, r0, inv, sign, t);
            check_rows<NT, T, true, true, FAR>(b, it, p, L.P, c0, inv, sign, t);
        } else {
            check_rows<NT, T, false, false, FAR>(b, it, p, L.D, r0, inv, sign, t);
            check_rows<NT, T, true, false, FAR>(b, it, p, L.P, c0, inv, sign, t);
        }
        __syncwarp();
        const double v[K] = {t.cp,     t.cd,     t.ap,     t.ad,     t.ocp, t.ocd, t.oap, t.oad,
                             t.pobj_c, t.dobj_c, t.pobj_a, t.dobj_a, t.ppc, t.ddc, t.ppa, t.dda};
        const double mine = reduce_vals<NT>(v, sh.red);
        if (threadIdx.x < K) *cg::this_cluster().map_shared_rank(&part[cl.rank][threadIdx.x], 0) = mine;
        cl.sync();
        if (lead) {  // merged in rank order
            double w[K];
            for (int q = 0; q < K; ++q) {
                w[q] = part[0][q];
                for (int c = 1; c < cl.size; ++c) w[q] = q < 8 ? smax(w[q], part[c][q]) : w[q] + part[c][q];
            }
            batch_decide(b, p, s, w, it.halpern != 0, std::is_same<T, float>::value, iter, stop);
        }
        cl.sync();
        // ---- restart
        const int restart = s.restart, fold = s.fold;
        done = s.done != 0;
        if (restart || fold) {
            const bool to_avg = s.restart_to_avg != 0;
            const double ri = s.inv;
            if (restart && p.primal_weight_update) {
                // the weight's sums in batch_restart's order, whatever the
                // cluster, so the step sizes do not depend on its size
                if (cl.rank == 0) {
                    double dx2 = 0.0, dy2 = 0.0;
                    if (NT == kBlock || threadIdx.x < kBlock)
                        for (int j = c0 + static_cast<int>(threadIdx.x); j < c0 + n; j += kBlock) {
                            const double d = restart_move_col<T>(it, p, pv, j, to_avg, ri);
                            dx2 += d * d;
                        }
                    if (NT == kBlock || (threadIdx.x >= kBlock && threadIdx.x < 2 * kBlock))
                        for (int i = r0 + static_cast<int>(threadIdx.x % kBlock); i < r0 + m; i += kBlock) {
                            const double d = restart_move_row<T>(it, p, i, to_avg, ri);
                            dy2 += d * d;
                        }
                    // block_sum_det's tree, x's and y's sums side by side
                    double(*sum)[kBlock] = scratch.sum;
                    const int t = static_cast<int>(threadIdx.x);
                    if (NT == kBlock) {
                        sum[0][t] = dx2;
                        sum[1][t] = dy2;
                    } else if (t < 2 * kBlock) {
                        sum[t / kBlock][t % kBlock] = t < kBlock ? dx2 : dy2;
                    }
                    __syncthreads();
                    for (int o = kBlock / 2; o > 0; o >>= 1) {
                        if (t < 2 * o) sum[t / o][t % o] += sum[t / o][t % o + o];
                        __syncthreads();
                    }
                    if (lead) restart_weight(s, sum[0][0], sum[1][0]);
                }
                cl.sync();  // read before it changes
            }
            for (int j = c0 + L.P.r0 + static_cast<int>(threadIdx.x); j < c0 + L.P.r1; j += NT)
                restart_col<T>(it, p, pv, j, restart, to_avg, ri);
            for (int i = r0 + L.D.r0 + static_cast<int>(threadIdx.x); i < r0 + L.D.r1; i += NT)
                restart_row<T>(it, p, pv, i, restart, to_avg, ri);
        }
        cl.sync();  // every CTA has read the flags
        if (lead) {
            s.restart = 0;
            s.fold = 0;
        }
        cl.sync();
    }
    if (lead) {
        // as the period count of the kernels over all instances: the period in
        // which the last instance ends is not counted
        s.spent = done ? 0 : 1;
        atomicMax(&b.g->iter, iter0 + (done ? (periods - 1) * p.period : periods * p.period + tail));
        atomicMax(&b.g->checks, periods);
    }
}

template <class T>
cudaError_t launch_class(const ResClass& c, const BatchView& b, const Iterates<T>& it, const BatchParams& p,
                         const ResJob& job, long long iter0, long long n_periods, long long tail, cudaStream_t s) {
    auto run = [&](auto kernel) {
        return res_launch(kernel, c.count, c.size, c.threads, c.smem, s, b, it, p, job, iter0, n_periods, tail);
    };
    if (c.far) return run(batch_resident<T, 1024, true>);
    if (c.threads == 256) return run(batch_resident<T, 256, false>);
    if (c.threads == 512) return run(batch_resident<T, 512, false>);
    return run(batch_resident<T, 1024, false>);
}

// The largest cluster the device schedules at the largest shared memory, and how
// many of 1, 2, ... 16 CTAs at once (on a B200 148, 74, 33, 15, 7).
std::atomic<int> g_res_cluster{0};
std::atomic<int> g_res_active[5];
// Instances of class c at once.
int res_at_once(int c, int size) {
    int q = 0;
    while ((1 << q) < size) ++q;
    return g_res_active[q] * (c == 0 ? 4 : c == 1 ? 2 : 1);
}

}  // namespace

template <class T>
void init_resident_kernels() {
    int active[2][5] = {};
    const int c[4] = {res_largest_cluster(batch_resident<T, 1024, false>, 1024, active[0]),
                      res_largest_cluster(batch_resident<T, 1024, true>, 1024, active[1]),
                      res_largest_cluster(batch_resident<T, 512, false>, 512),
                      res_largest_cluster(batch_resident<T, 256, false>, 256)};
    for (int q = 0; q < 5; ++q) g_res_active[q] = std::min(active[0][q], active[1][q]);
    g_res_cluster = *std::min_element(c, c + 4) == 0 ? 0 : std::min(c[0], c[1]);
}
// Classes of like CTAs, tried in the order of their CTAs; the largest instances
// first (a class's launch ends with its last instance).
constexpr ResClass kClasses[kResClasses] = {
    {1, 256}, {1, 512}, {1, 1024}, {1, 1024, 0, 0, 0, true}, {2, 1024}, {2, 1024, 0, 0, 0, true},
    {4, 1024}, {4, 1024, 0, 0, 0, true}, {8, 1024}, {8, 1024, 0, 0, 0, true}, {16, 1024, 0, 0, 0, true}};
// ... of an instance. per = 0: its own time counts, the CTAs that hold its
// entries, at most eight (60 KB to all CTAs of a cluster: 3,500 cycles for
// eight, 4,600 for sixteen). Else SM time does: the fewest CTAs that hold it at
// up to `per` entries each, its entries in global memory where they do not fit.
template <class T>
int res_class(const ResParts& pt, const ResParts& pa, int lgt, int lga, bool halpern, int64_t per, ResSize* z) {
    const int32_t nnz = pa.nz[kResMaxCluster];
    int last = -1;
    for (int c = 2; c < kResClasses; ++c) {
        const ResClass& k = kClasses[c];
        if (k.size > g_res_cluster) continue;
        const ResSize y = k.far ? res_size<T, true>(pt, pa, k.size, lgt, lga, halpern)
                                : res_size<T, false>(pt, pa, k.size, lgt, lga, halpern);
        if (y.smem > kResMaxSmem) continue;
        if (per == 0 && k.far && k.size < 8) continue;
        last = c;
        *z = y;
        if (per == 0 || k.size >= 8 || nnz <= per * k.size) break;
    }
    if (last == 2 && nnz <= 3000 && z->smem <= kResMaxSmem / 4) return 0;   // four to an SM
    if (last == 2 && nnz <= 12000 && z->smem <= kResMaxSmem / 2) return 1;  // two
    return last;
}

// Each instance at its own time if all of them run at once that way; else at
// the fewest entries a CTA with which they do; else, with more instances than
// that, at 32,768. FP32, a check period of 40 iterations of 256 instances of 50
// x 100 to 5,000 x 15,000: 1,483 us at their own time's clusters; at 8,192 /
// 16,384 / 32,768 / 65,536 entries a CTA 1,483 / 1,244 / 1,184 / 1,218 us. Where
// they just do not run at once at their own time's clusters, an iteration there
// / here: 20 FP32 instances of 3,000 x 9,000 19.5 / 11.6 us, 16 FP64 ones of
// 1,000 x 4,000 with 20 entries a column 18.2 / 13.5, of 300 x 10,000 20.0 /
// 12.2.
constexpr int64_t kResPer[] = {0, 4096, 8192, 16384, 32768};

// The kernels over all instances, us an iteration: 9 and what their entries and
// rows take, and a CTA along the longest row: within 15% of what batches of 1 to
// 64 instances of 300 x 10,000 to 10,000 x 23,000 measured, and badly scaled ones.
template <class T>
double over_all_us(const std::vector<ResParts>& parts) {
    constexpr bool f32 = std::is_same<T, float>::value;
    double nnz = 0.0, rows = 0.0, longest = 0.0;
    for (const ResParts& p : parts) {
        nnz += 0.5 * p.nz[kResMaxCluster];
        rows += p.row[kResMaxCluster];
        longest = std::max(longest, static_cast<double>(p.longest_row));
    }
    return 9.0 + (f32 ? 9.5e-6 : 13.5e-6) * nnz + (f32 ? 12e-6 : 13e-6) * rows + 6e-3 * longest;
}

template <class T>
bool plan_resident(const std::vector<ResParts>& parts, int lgt, int lga, bool halpern, ResPlan& plan) {
    plan = ResPlan{};
    const size_t count = parts.size() / 2;
    if (g_res_cluster == 0) return false;
    struct Item {
        int32_t k, nnz, cls;
        ResFar far;
    };
    std::vector<Item> items(count);
    ResClass all[kResClasses];
    // the longest row of more than kResLongRow entries in global memory, and what
    // of the GPU the instances with such rows take at once
    constexpr int kResLongRow = 2048;
    int far_row = 0;
    double far_fill = 0.0;
    for (const int64_t per : kResPer) {
        std::copy(kClasses, kClasses + kResClasses, all);
        plan.far_bytes = 0;
        far_row = 0;
        far_fill = 0.0;
        double fill = 0.0;  // of the GPU, by all instances at once
        for (size_t k = 0; k < count; ++k) {
            const ResParts &pt = parts[2 * k], &pa = parts[2 * k + 1];
            ResSize z;
            const int cls = res_class<T>(pt, pa, lgt, lga, halpern, per, &z);
            if (cls < 0) return false;
            items[k] = {static_cast<int32_t>(k), pa.nz[kResMaxCluster], cls, ResFar{}};
            if (all[cls].far) {
                const int row = std::max(pt.longest_row, pa.longest_row);
                if (row > kResLongRow) far_fill += 1.0 / res_at_once(cls, all[cls].size);
                if (row > kResLongRow) far_row = std::max(far_row, row);
                // whole 16-byte vectors per CTA
                for (int w = 0; w < 2; ++w) items[k].far.entries[w] = (z.entries[w] + 7u) / 8u * 8u;
                items[k].far.base = plan.far_bytes;
                plan.far_bytes += static_cast<int64_t>(kResFarEntry) *
                                  (items[k].far.entries[0] + items[k].far.entries[1]) * all[cls].size;
                plan.far_bytes = (plan.far_bytes + 255) / 256 * 256;
            }
            all[cls].count += 1;
            all[cls].smem = std::max(all[cls].smem, z.smem);
            fill += 1.0 / res_at_once(cls, all[cls].size);
        }
        if (fill <= 1.0) break;
    }
    // Not where the clusters alone would take longer than the kernels over all
    // instances: several waves of sixteen CTAs (11 us an iteration each: 64 FP32
    // instances of 10,000 x 23,000 102 us on clusters, 72 not), or a warp along a
    // long row from global memory (FP64, badly scaled: 4,000 x 9,000 with a row of
    // 6,000 entries 55 / 47 us, 40 of 2,000 x 5,000 with one of 3,500 56 / 47, 150
    // of them in two waves 145 / 126; shorter rows are not what takes the time: 300
    // of 500 x 1,200 with one of 870 49 / 72; in FP32 the clusters are as fast or
    // faster).
    const ResClass& wide = all[kResClasses - 1];
    const int waves = wide.count > 0 ? (wide.count - 1) / res_at_once(kResClasses - 1, wide.size) + 1 : 0;
    double least = waves > 1 ? 11.0 * waves : 0.0;
    if (!std::is_same<T, float>::value && far_row > 0)
        least = std::max(least, std::ceil(far_fill) * (3.0 + 15e-3 * far_row));
    if (least > over_all_us<T>(parts)) return false;
    std::sort(items.begin(), items.end(), [](const Item& a, const Item& b) {
        return a.cls != b.cls ? a.cls > b.cls : a.nnz != b.nnz ? a.nnz > b.nnz : a.k < b.k;
    });
    for (const Item& i : items) {
        plan.list.push_back(i.k);
        plan.where.push_back(i.far);
    }
    int32_t first = 0;
    for (int c = kResClasses - 1; c >= 0; --c) {
        if (all[c].count == 0) continue;
        all[c].first = first;
        first += all[c].count;
        plan.classes.push_back(all[c]);
    }
    return true;
}

template <class T>
cudaError_t launch_batch_resident(const std::vector<ResClass>& classes, const ResBuffers& buf, int lgt, int lga,
                                  const BatchView& b, const Iterates<T>& it, const BatchParams& p, long long iter0,
                                  long long n_periods, long long tail, cudaStream_t s, const ResStreams& side) {
    cudaError_t e = cudaEventRecord(side.fork, s);
    for (size_t c = 0; c < classes.size() && e == cudaSuccess; ++c) {
        const cudaStream_t to = c == 0 ? s : side.stream[c - 1];
        if (c > 0) e = cudaStreamWaitEvent(to, side.fork, 0);
        if (e == cudaSuccess)
            e = launch_class<T>(classes[c], b, it, p, ResJob{buf.list + classes[c].first, buf.parts, lgt, lga,
                                       buf.where + classes[c].first, buf.far}, iter0, n_periods, tail,
                                to);
        if (c > 0 && e == cudaSuccess) e = cudaEventRecord(side.join[c - 1], to);
        if (c > 0 && e == cudaSuccess) e = cudaStreamWaitEvent(s, side.join[c - 1], 0);
    }
    return e;
}

}  // namespace pdhg
