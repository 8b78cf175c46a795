// mhist.cu -- FP64 multihistogram density of states on the GPU.
//
// The fixed point of src/cae_estimator.cc:172-253 (Ferrenberg-Swendsen /
// Newman-Barkema multihistogram): for energy bins e_i = emin + i*estep,
//   ln g(e_i) = ln sum_j N_j(e_i) - ln sum_j exp(ln n - ln Z_j - beta_j e_i)
//   ln Z_j    = ln sum_i exp(ln g(e_i) - beta_j e_i)
// iterated from ln Z = 0 until sum_j ((lnZ_j - lnZ'_j)/lnZ'_j)^2 <= tol.
// The reference accumulates every sum with a pairwise log-add in index order;
// here the sums are those of the exponentials themselves, the numerator is
// the exact integer count sum, and sums are reduced in parallel -- the same
// quantities to FP64 rounding.  FP64 is kept throughout: the exponents span
// thousands of nats.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <vector>

#include "mhist_job.h"

namespace pticm {

namespace cg = cooperative_groups;

// Whole fixed point on the device, one cluster of CTAs per instance (many
// instances per launch), each CTA holding a slice of the bins.
//
// What bounds it is the FP64 pipe (about two multiply-adds a clock and SM):
// with an exponential for every (bin, temperature) in each of the two sums,
// 33 temperatures and 1742 bins took 0.38 ms an iteration on one SM, 517 ms
// for 1338 iterations.  exp(-beta_j e_i) does not change over the iterations,
// so they are products with a fixed matrix.  With a reference a0_j (the
// a_j = ln n - ln Z_j of some iteration) and x_j = exp(a_j - a0_j),
//   K_ij = exp(a0_j - beta_j e_i - m_i),  m_i = max_j (...)
//   S_i  = sum_j K_ij x_j,   T_j = sum_i K_ij c_i / S_i,
//   ln Z'_j = ln T_j - a0_j,  x'_j = n / T_j,
// two matrix-vector products and no exponential: 10.4 ms instead of 504 ms, 7.8
// us an iteration over 16 SMs (the two products about 3 us of FP64 pipe, the
// rest the divisions, the sums' short chains and the cluster's barrier).
// Against extended precision ln g is off by 2e-16 of its scale, the
// exponentials of every iteration's a_j were off by up to 8e-14.  The reference moves to the
// current a_j when an x_j leaves [e^-20, e^20] (27 times in those 1338
// iterations).  K_ij below e^-120 is zero: with every |ln x_j| at most 35 the
// dropped terms of S_i are below e^-50 of it, and of T_j below e^-65.
//
// An iteration that moves some ln Z_j by kFarNats or more (the first one or
// two), or gives a T_j that is not a positive number, is made in the log
// domain instead, with the exponentials shifted by each sum's own largest
// term, by the cluster's first CTA.
namespace {
constexpr float kDropNats = 60.f;     // log-domain iteration: terms this far below the shift are dropped
constexpr double kZeroNats = 120.0;   // K_ij this far below its row's largest is zero
constexpr float kRefNats = 20.f;      // |ln x_j| beyond which the reference moves
constexpr float kFarNats = 15.f;      // change of a ln Z_j that needs the log domain
constexpr int kMhThreads = 512;
constexpr size_t kMhSmem = 200 * 1024;   // per CTA: the fixed arrays and, when it fits, the slice's matrix

// Row stride of K (odd: a column's rows fall into different banks).
__host__ __device__ constexpr int mh_pitch(int nt) { return nt | 1; }
// A CTA's slice: K, then c, g, m and the range of kept temperatures per row.
__host__ __device__ constexpr size_t mh_slice_bytes(long long rows, int nt) {
    return (size_t)rows * ((size_t)mh_pitch(nt) * 8 + 3 * 8 + 8);
}
__host__ __device__ constexpr size_t mh_fixed_bytes(int nt, int cs) {
    return ((size_t)nt * 8 * 7 + (size_t)(nt > kMhThreads ? nt : kMhThreads) * 8 + (size_t)2 * cs * nt * 8 +
            (size_t)nt * 4 * 2 + 127) & ~size_t(127);
}
}  // namespace

// The log-domain iteration over all bins of a job, by one CTA: reads sZ,
// writes sNew.  The shifts and the test that drops a term come from FP32
// shadows of the same quantities; every kept term and every sum is FP64.  A
// term more than 60 nats below the shift is dropped: 60 nats is 1e-26
// relative, so even 10^7 such terms stay below half an ulp of a sum >= 1.
__device__ void mh_log_iteration(const MhJob& J, const double* sZ, double* sA, const double* sB, float* sAf,
                                 const float* sBf, const double* lc, double* ld, float* lf, double* sNew) {
    const int nt = J.nt, tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    const long long nb = J.nbins;
    for (int j = tid; j < nt; j += T) {
        sA[j] = J.logn - sZ[j];
        sAf[j] = (float)sA[j];
    }
    __syncthreads();
    for (long long i = tid; i < nb; i += T) {
        const double lci = lc[i];
        if (lci == -DBL_MAX) {
            ld[i] = -DBL_MAX;
            lf[i] = -FLT_MAX;
            continue;
        }
        const double e = J.min_emin + (double)i * J.estep;
        const float ef = (float)e;
        float mf = -FLT_MAX;
        for (int j = 0; j < nt; j++) mf = fmaxf(mf, sAf[j] - sBf[j] * ef);
        const double m = (double)mf;
        double s = 0.0;
        for (int j = 0; j < nt; j++) {
            if (sAf[j] - sBf[j] * ef - mf < -kDropNats) continue;
            s += exp(sA[j] - sB[j] * e - m);
        }
        const double v = lci - (m + log(s));
        ld[i] = v;
        lf[i] = (float)v;
    }
    __syncthreads();
    // one warp per ln Z_j
    for (int j = warp; j < nt; j += nw) {
        const float bf = sBf[j];
        const double bj = sB[j];
        float mf = -FLT_MAX;
        for (long long i = lane; i < nb; i += 32) {
            const float v = lf[i];
            if (v == -FLT_MAX) continue;
            mf = fmaxf(mf, v - bf * (float)(J.min_emin + (double)i * J.estep));
        }
        for (int o = 16; o > 0; o >>= 1) mf = fmaxf(mf, __shfl_xor_sync(0xffffffffu, mf, o));
        const double m = (double)mf;
        double s = 0.0;
        for (long long i = lane; i < nb; i += 32) {
            const float v = lf[i];
            if (v == -FLT_MAX) continue;
            const double e = J.min_emin + (double)i * J.estep;
            if (v - bf * (float)e - mf < -kDropNats) continue;
            s += exp(ld[i] - bj * e - m);
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) sNew[j] = m + log(s);
    }
    __syncthreads();
}

// The convergence sum in histogram order, as src/cae_estimator.cc:245-251.
__device__ bool mh_converged(const double* zold, const double* znew, int nt) {
    double metric = 0.0;
    for (int j = 0; j < nt; j++) {
        const double q = fabs(zold[j] - znew[j]) / fabs(znew[j]);
        metric += q * q;
    }
    return !(metric > 1e-7);
}

// MANY: the clusters take the jobs in turn (else one job each).
template <bool MANY>
__global__ void __launch_bounds__(kMhThreads, 1)
mh_solve_kernel(int njobs, const MhJob* jobs, const uint32_t* hist, const uint64_t* hoff, const uint64_t* hlen,
                const double* emin, const double* beta, double* logdos, double* logc, float* ldf, double* logZ,
                unsigned long long* iters, long long max_iters, uint8_t* work, size_t slot, int* taken, size_t smem_bytes) {
    cg::cluster_group cluster = cg::this_cluster();
    const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int mine = (int)blockIdx.x / cs, clusters = (int)gridDim.x / cs;
    __shared__ int s_job;
    // the cluster's first job, then those that no cluster has taken
    for (int job = mine; !MANY || job < njobs;) {
    const MhJob J = jobs[job];
    const int nt = J.nt, tid = threadIdx.x, T = blockDim.x, p = mh_pitch(nt);
    const long long per = (J.nbins + cs - 1) / cs;
    const long long i0 = min((long long)rank * per, (long long)J.nbins);
    const int rows = (int)(min(i0 + per, (long long)J.nbins) - i0);
    extern __shared__ __align__(16) uint8_t mh_sm[];
    double* const sZ = reinterpret_cast<double*>(mh_sm);   // ln Z of the iteration's start
    double* const sNew = sZ + nt;
    double* const sA = sNew + nt;       // a0 (log-domain iteration: a)
    double* const sB = sA + nt;
    double* x = sB + nt;
    double* xnew = x + nt;
    double* const sT = xnew + nt;
    double* const part = sT + nt;       // column sums of the row groups
    double* const inbox = part + max(nt, T);   // [2][cs][nt]: every CTA's column sums
    float* const sAf = reinterpret_cast<float*>(inbox + 2 * cs * nt);
    float* const sBf = sAf + nt;
    const size_t fixed = mh_fixed_bytes(nt, cs);
    // the slice in shared memory when it fits, else in the cluster's slot of
    // device memory (L2); without one every iteration is made in the log domain
    const bool in_smem = fixed + mh_slice_bytes(per, nt) <= smem_bytes, matrix = in_smem || work != nullptr;
    uint8_t* const slice = in_smem ? mh_sm + fixed
                           : matrix ? work + (size_t)mine * slot + (size_t)rank * mh_slice_bytes(per, nt) : nullptr;
    double* const K = reinterpret_cast<double*>(slice);
    double* const c = K + (size_t)per * p;
    double* const g = c + per;
    double* const m = g + per;
    int2* const range = reinterpret_cast<int2*>(m + per);
    __shared__ int s_flag[2];   // done, what the next iteration needs
    __shared__ float4 s_vote[kMhThreads / 32];
    const int nt4 = (4 * nt + 31) & ~31, voters = min(nt4, T) >> 5;   // four lanes per temperature, whole warps
    enum : int { NEXT_PLAIN = 0, NEXT_REF = 1, NEXT_LOG = 2 };
    const uint64_t* ho = hoff + J.row0;
    const uint64_t* hl = hlen + J.row0;
    const double* em = emin + J.row0;
    double* ld = logdos + J.bin0;
    double* lc = logc + J.bin0;
    float* lf = ldf + J.bin0;
    for (int j = tid; j < nt; j += T) {
        sZ[j] = 0.0;
        sB[j] = beta[J.row0 + j];
        sBf[j] = (float)sB[j];
        x[j] = 1.0;
    }
    // summed counts per bin (constant over the iterations)
    for (int r = tid; r < rows; r += T) {
        const long long i = i0 + r;
        const double e = J.min_emin + (double)i * J.estep;
        unsigned long long count = 0;
        for (int j = 0; j < nt; j++) {
            if (e < em[j]) continue;
            const double idx = floor((e - em[j]) / J.estep);
            if (idx >= (double)hl[j]) continue;
            count += hist[ho[j] + (uint64_t)idx];
        }
        if (matrix) c[r] = (double)count;
        lc[i] = count ? log((double)count) : -DBL_MAX;
    }
    __threadfence();
    cluster.sync();
    long long it = 0;
    int next = NEXT_LOG, parity = 0;
    bool last_log = true;
    while (it < max_iters) {
        if (next == NEXT_LOG) {
            // log domain, by the first CTA; every CTA then holds its ln Z
            cluster.sync();   // (no CTA still reads its inbox)
            if (rank == 0) {
                mh_log_iteration(J, sZ, sA, sB, sAf, sBf, lc, ld, lf, sNew);
                for (int q = tid; q < cs * nt; q += T) cluster.map_shared_rank(inbox, q / nt)[q % nt] = sNew[q % nt];
            }
            cluster.sync();
            if (tid == 0) {
                float far = 0.f;
                bool finite = true;
                for (int j = 0; j < nt; j++) {
                    sNew[j] = inbox[j];
                    const float dz = (float)fabs(sNew[j] - sZ[j]);
                    finite = finite && dz < FLT_MAX;
                    far = fmaxf(far, dz);
                }
                s_flag[0] = mh_converged(sZ, sNew, nt);
                s_flag[1] = matrix && finite && far < kFarNats ? NEXT_REF : NEXT_LOG;
                for (int j = 0; j < nt; j++) sZ[j] = sNew[j];
            }
            cluster.sync();   // the inbox is read before anyone writes it again
            it++;
            last_log = true;
            next = s_flag[1];
            if (s_flag[0]) break;
            continue;
        }
        if (next == NEXT_REF) {
            // K of the current ln Z
            for (int j = tid; j < nt; j += T) {
                sA[j] = J.logn - sZ[j];
                x[j] = 1.0;
            }
            __syncthreads();
            for (int r = tid; r < rows; r += T) {
                double* const Kr = K + (size_t)r * p;
                const double e = J.min_emin + (double)(i0 + r) * J.estep;
                int k = 0;
                double mx = -DBL_MAX;
                for (int j = 0; j < nt; j++) {
                    const double t = sA[j] - sB[j] * e;
                    if (t > mx) { mx = t; k = j; }
                }
                // exponents as differences to temperature k's: their rounding
                // is relative to the exponent, not to a_j and beta_j e (it
                // stays the same while the reference does, and would add up)
                const double ak = sA[k], bk = sB[k];
                int lo = nt, hi = 0;
                for (int j = 0; j < nt; j++) {
                    const double t = (sA[j] - ak) - (sB[j] - bk) * e;
                    double v = 0.0;
                    if (t >= -kZeroNats && c[r] > 0.0) {
                        v = exp(t);
                        lo = min(lo, j);
                        hi = j + 1;
                    }
                    Kr[j] = v;
                }
                m[r] = mx;
                range[r] = make_int2(lo, hi);
            }
            __syncthreads();
        }
        // S_i and c_i / S_i, a thread per bin
        for (int r = tid; r < rows; r += T) {
            const int2 q = range[r];
            const double* const Kr = K + (size_t)r * p;
            double s0 = 0.0, s1 = 0.0;
            int j = q.x;
            for (; j + 1 < q.y; j += 2) {
                s0 += Kr[j] * x[j];
                s1 += Kr[j + 1] * x[j + 1];
            }
            if (j < q.y) s0 += Kr[j] * x[j];
            g[r] = q.x < q.y ? c[r] / (s0 + s1) : 0.0;
        }
        __syncthreads();
        // T_j: groups of threads take the rows in turn, then a thread per
        // temperature adds the groups and hands the sum to every CTA
        const int groups = max(1, T / nt);
        for (int q = tid; q < groups * nt; q += T) {
            const int gr = q / nt, j = q - gr * nt;
            double s0 = 0.0, s1 = 0.0;
            int r = gr;
            for (; r + groups < rows; r += 2 * groups) {
                s0 += K[(size_t)r * p + j] * g[r];
                s1 += K[(size_t)(r + groups) * p + j] * g[r + groups];
            }
            if (r < rows) s0 += K[(size_t)r * p + j] * g[r];
            part[q] = s0 + s1;
        }
        __syncthreads();
        // four lanes per temperature add the groups, then the sum goes to
        // every CTA, a thread per copy
        for (int q = tid; q < nt4; q += T) {
            const int j = min(q >> 2, nt - 1);
            double t = 0.0;
            for (int gr = q & 3; gr < groups; gr += 4) t += part[gr * nt + j];
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            if ((q & 3) == 0 && (q >> 2) < nt) sT[j] = t;
        }
        __syncthreads();
        for (int q = tid; q < cs * nt; q += T) {
            const int d = q / nt, j = q - d * nt;
            cluster.map_shared_rank(inbox, d)[(parity * cs + rank) * nt + j] = sT[j];
        }
        cluster.sync();
        // every CTA adds the same sums in the same order and decides alike.
        // ln Z'_j - ln Z_j = ln(x_j / x'_j): in FP32, unless the convergence
        // sum or a |ln Z'_j| is too close to call
        float metric = 0.f, off = 0.f;
        bool bad = false, close = false;
        for (int q = tid; q < nt4; q += T) {
            const int j = min(q >> 2, nt - 1);
            double t = 0.0;
            for (int d = q & 3; d < cs; d += 4) t += inbox[(parity * cs + d) * nt + j];
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            if ((q & 3) != 0 || (q >> 2) >= nt) continue;
            const double xn = J.n / t;
            const float tf = (float)t, xf = (float)xn;
            bad = bad || !(t > 0.0) || !(t < DBL_MAX) || !(xn > 0.0);
            const float u = (float)(x[j] - xn) / xf;
            const float dz = fabsf(u) < 0.5f ? log1pf(u) : logf((float)x[j] / xf);
            const float z = (float)((double)logf(tf) - sA[j]);
            close = close || !(fabsf(z) > 1.f) || !(tf >= FLT_MIN && tf <= FLT_MAX);
            const float w = dz / z;
            metric += w * w;
            bad = bad || !(fabsf(dz) < kFarNats);
            off = fmaxf(off, fabsf(logf(xf)));
            sT[j] = t;
            xnew[j] = xn;
        }
        for (int o = 16; o > 0; o >>= 1) {
            metric += __shfl_xor_sync(0xffffffffu, metric, o);
            off = fmaxf(off, __shfl_xor_sync(0xffffffffu, off, o));
        }
        bad = __any_sync(0xffffffffu, bad);
        close = __any_sync(0xffffffffu, close);
        if ((tid & 31) == 0) s_vote[tid >> 5] = make_float4(metric, off, bad ? 1.f : 0.f, close ? 1.f : 0.f);
        __syncthreads();
        metric = off = 0.f;
        for (int w = 0; w < voters; w++) {
            const float4 v = s_vote[w];
            metric += v.x;
            off = fmaxf(off, v.y);
            bad = bad || v.z != 0.f;
            close = close || v.w != 0.f;
        }
        close = close || !(fabsf(metric - 1e-7f) > 1e-9f);
        bool done = !(metric > 1e-7f);
        const bool moved = !(off <= kRefNats);
        parity ^= 1;
        if (bad) {
            // made again in the log domain, from this iteration's ln Z
            for (int j = tid; j < nt; j += T) sZ[j] = J.logn - sA[j] - log(x[j]);
            __syncthreads();
            next = NEXT_LOG;
            continue;
        }
        if (close || done || moved) {
            // FP64 ln Z before and after: for the decision, the result, or
            // the next reference
            for (int j = tid; j < nt; j += T) {
                sZ[j] = J.logn - sA[j] - log(x[j]);
                sNew[j] = log(sT[j]) - sA[j];
            }
            __syncthreads();
            if (close) {
                if (tid == 0) s_flag[0] = mh_converged(sZ, sNew, nt);
                __syncthreads();
                done = s_flag[0] != 0;
            }
            __syncthreads();
            for (int j = tid; j < nt; j += T) sZ[j] = sNew[j];
            __syncthreads();
        }
        it++;
        last_log = false;
        next = moved ? NEXT_REF : NEXT_PLAIN;
        if (done) break;   // (ln g comes from the last iteration's x)
        double* const y = x;
        x = xnew;
        xnew = y;
    }
    if (!last_log) {
        // ln g of the last iteration: its S_i again
        for (int r = tid; r < rows; r += T) {
            const int2 q = range[r];
            double s = 0.0;
            for (int j = q.x; j < q.y; j++) s += K[(size_t)r * p + j] * x[j];
            ld[i0 + r] = q.x < q.y ? lc[i0 + r] - (m[r] + log(s)) : -DBL_MAX;
        }
    }
    if (rank == 0) {
        for (int j = tid; j < nt; j += T) logZ[J.row0 + j] = sZ[j];
        if (tid == 0) iters[job] = (unsigned long long)it;
    }
    if (!MANY) break;
    if (rank == 0 && tid == 0) {
        const int next = clusters + atomicAdd(taken, 1);
        for (int q = 0; q < cs; q++) *cluster.map_shared_rank(&s_job, q) = next;
    }
    cluster.sync();
    job = s_job;
    cluster.sync();   // (read before it is written again)
    }
    cluster.sync();   // no CTA leaves while another may still write to its shared memory
}

// CTAs per instance: enough instances fill the GPU with one or two each; a few
// are spread over up to 16 SMs, as long as a CTA keeps about 2000 terms (below
// that the cluster's barrier costs more than the work it spreads).
static int mh_cluster_size(const std::vector<MhJob>& jobs, int max_nt, int sms) {
    long long terms = 1;
    for (const MhJob& J : jobs) terms = std::max(terms, (long long)J.nt * (long long)J.nbins);
    int cs = 1;
    while (cs < 16 && (long long)jobs.size() * cs * 2 <= sms && terms / (cs * 2) >= 2000 &&
           mh_fixed_bytes(max_nt, cs * 2) <= kMhSmem)
        cs *= 2;
    return cs;
}

static void mhist_config(int clusters, int cs, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
    cfg.gridDim = dim3((unsigned)clusters * (unsigned)cs);
    cfg.blockDim = dim3(kMhThreads);
    cfg.dynamicSmemBytes = kMhSmem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

template <class Kernel>
static cudaError_t mhist_allow(Kernel kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMhSmem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

// The launch of a solve: CTAs per instance, clusters and, for slices that do
// not fit shared memory, a slot of device memory for each cluster (0: all fit).
// A slot holds the largest such instance and its cluster's next instances use
// it again, so a launch with slots has only as many clusters as the GPU runs at
// once and `most` bytes of slots (but one slot); the clusters take the instances
// in turn.  (A matrix per instance, 8 bytes a bin and temperature each, grew with
// the number of instances: 1000 of 20000 bins and 128 temperatures 21 GB.)
cudaError_t mhist_plan(const std::vector<MhJob>& jobs, int max_nt, size_t most, int& cs, int& clusters, size_t& slot) {
    // (more temperatures than a launch has ever taken)
    if ((size_t)max_nt * (4 * sizeof(double) + 2 * sizeof(float)) > 48 * 1024) return cudaErrorInvalidValue;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = mhist_allow(mh_solve_kernel<false>);
    if (e != cudaSuccess) return e;
    cs = mh_cluster_size(jobs, max_nt, sms);
    int resident = sms / cs;
    while (cs > 8) {   // (above the portable size: when the GPU can place one)
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        mhist_config((int)jobs.size(), cs, nullptr, cfg, attr);
        int placed = 0;
        if (cudaOccupancyMaxActiveClusters(&placed, mh_solve_kernel<false>, &cfg) == cudaSuccess && placed > 0) {
            resident = placed;
            break;
        }
        cudaGetLastError();
        cs /= 2;
        resident = sms / cs;
    }
    clusters = (int)jobs.size();
    slot = 0;
    for (const MhJob& J : jobs) {
        const size_t slice = mh_slice_bytes((J.nbins + cs - 1) / cs, J.nt);
        if (mh_fixed_bytes(J.nt, cs) + slice > kMhSmem) slot = std::max(slot, (cs * slice + 127) & ~size_t(127));
    }
    if (slot) clusters = std::min<int>(std::min(clusters, resident), (int)std::max<size_t>(1, std::min(most / slot, (size_t)clusters)));
    return cudaSuccess;
}

cudaError_t mhist_solve(int njobs, int cs, int clusters, const MhJob* jobs, const uint32_t* hist, const uint64_t* hoff,
                        const uint64_t* hlen, const double* emin, const double* beta, double* logdos, double* logc,
                        float* ldf, double* logZ, unsigned long long* iters, long long max_iters, uint8_t* work,
                        size_t slot, int* taken, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    mhist_config(clusters, cs, st, cfg, attr);
    const auto kernel = clusters < njobs ? mh_solve_kernel<true> : mh_solve_kernel<false>;
    const cudaError_t e = mhist_allow(kernel);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, kernel, njobs, jobs, hist, hoff, hlen, emin, beta, logdos, logc, ldf, logZ,
                              iters, max_iters, work, slot, taken, kMhSmem);
}

}  // namespace pticm
