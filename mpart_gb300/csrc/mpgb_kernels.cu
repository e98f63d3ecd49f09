// Dispatch of the fused/inverse kernels and the small helper kernels.
#include <algorithm>
#include <atomic>

#include "mpgb_types.h"
#include "mpgb_launch.h"
#include "mpgb_sigmoid.cuh"

namespace mpgb {

template <int BASIS, int POS, int PMAX>
cudaError_t launchFusedP(const FusedParams& prm, int nItems, int needJ, int needE, cudaStream_t stream);
template <int BASIS, int POS>
cudaError_t launchBatchP(const FusedParams& prm, int nItems, int pmaxClass, int* counter, cudaStream_t stream);
template <int BASIS, int POS, int PMAX>
cudaError_t launchInverseP(const InverseParams& prm, int nBlocks, cudaStream_t stream);

// --------------------------------------------------------------------------
// Coefficient gather: cm[slot] = coeffs[component offset + slotTerm[slot]].
// --------------------------------------------------------------------------
__global__ void gatherKernel(const int32_t* slotGlobalTerm, int nSlots, const double* coeffs, double* cm) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < nSlots) {
        const int t = slotGlobalTerm[s];
        cm[s] = (t >= 0) ? coeffs[t] : 0.0;
    }
}

// Fixed-order reduction of partial rows: out[t] = scale * sum_r part[base_r + t].
// Block = 32 terms x kRowGroups row groups, whose sums are added in order.
// (Eight groups of 300 rows one load after another took 153 us at the end of a
// 6-D KL step, 6 % of it.)
constexpr int kRowGroups = 32;

__device__ __forceinline__ double sumRowGroup(const double* part, const long long* rowBase, int nRows, int t, int g) {
    double s = 0.0;
    int r = g;
    for (; r + 3 * kRowGroups < nRows; r += 4 * kRowGroups) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = part[rowBase[r + q * kRowGroups] + t];
#pragma unroll
        for (int q = 0; q < 4; ++q) s += v[q];
    }
    for (; r < nRows; r += kRowGroups) s += part[rowBase[r] + t];
    return s;
}

__global__ void reduceRowsKernel(const double* part, const long long* rowBase, int nRows, int nTerms,
                                 double scale, double* out, int accumulate) {
    __shared__ double red[kRowGroups][33];
    const int t = blockIdx.x * 32 + threadIdx.x;
    const int g = threadIdx.y;
    red[g][threadIdx.x] = t < nTerms ? sumRowGroup(part, rowBase, nRows, t, g) : 0.0;
    __syncthreads();
    if (g == 0 && t < nTerms) {
        double v = 0.0;
        for (int q = 0; q < kRowGroups; ++q) v += red[q][threadIdx.x];
        v *= scale;
        out[t] = accumulate ? out[t] + v : v;
    }
}

// ---------------------------------------------------------------------------
// Stable counting sort of points by |x_D| (the 256 buckets of sortBucket).
// The per-point cost of the adaptive quadrature grows with |x_D|; grouping
// points of similar cost keeps a warp's lanes busy.
// Deterministic: bucket-major, original order within a bucket.
// ---------------------------------------------------------------------------
constexpr int kSortBuckets = 256;
constexpr int kSortChunk = 1024;

__device__ __forceinline__ int sortKey(double x) { return sortBucket(x); }

// Segment blockIdx.y of a multi-segment sort: keys at xd + y * keySeg, counts
// at hist + y * histSeg (bucket-major, [bucket][chunk], then the 256 bucket
// totals), permutation at perm + y * permSeg.
__global__ void keyHistKernel(const double* xd, long long stride, long long N, int* hist, long long keySeg,
                              long long histSeg) {
    xd += blockIdx.y * keySeg;
    hist += blockIdx.y * histSeg;
    __shared__ int h[kSortBuckets];
    for (int t = threadIdx.x; t < kSortBuckets; t += blockDim.x) h[t] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * kSortChunk;
    for (int j = threadIdx.x; j < kSortChunk; j += blockDim.x) {
        const long long i = base + j;
        if (i < N) atomicAdd(&h[sortKey(xd[i * stride])], 1);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kSortBuckets; t += blockDim.x) hist[(long long)t * gridDim.x + blockIdx.x] = h[t];
}

// One warp per bucket: its chunk counts -> exclusive sums over the chunks, and
// the bucket's total.  (One block walking all chunks of 256 buckets in turn
// took 62 of the sort's 104 us at 1M points.)
__global__ void keyScanKernel(int* hist, int nBlk, long long histSeg) {
    hist += blockIdx.y * histSeg;
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int* row = hist + (long long)b * nBlk;
    int run = 0;
    for (int k0 = 0; k0 < nBlk; k0 += 32) {
        const int k = k0 + lane;
        const int v = k < nBlk ? row[k] : 0;
        int s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += x;
        }
        if (k < nBlk) row[k] = run + s - v;
        run += __shfl_sync(0xffffffffu, s, 31);
    }
    if (lane == 0) hist[(long long)kSortBuckets * nBlk + b] = run;
}

// One warp per chunk, chunk order kept within each bucket.  The chunk's keys
// are loaded together (a lane's loads one after another left the warp waiting
// for memory 32 times: 30 us at any size).
__global__ void keyScatterKernel(const double* xd, long long stride, long long N, const int* off, int* perm,
                                 long long keySeg, long long histSeg, long long permSeg) {
    xd += blockIdx.y * keySeg;
    off += blockIdx.y * histSeg;
    perm += blockIdx.y * permSeg;
    __shared__ int cnt[kSortBuckets];
    const int lane = threadIdx.x;
    const int nBlk = gridDim.x;
    const long long base = (long long)blockIdx.x * kSortChunk;
    double x[kSortChunk / 32];
#pragma unroll
    for (int c = 0; c < kSortChunk / 32; ++c) {
        const long long i = base + c * 32 + lane;
        x[c] = i < N ? xd[i * stride] : 0.0;
    }
    // First slot of (bucket, this chunk): eight buckets per lane.
    {
        int t[kSortBuckets / 32], s = 0;
#pragma unroll
        for (int q = 0; q < kSortBuckets / 32; ++q) {
            t[q] = off[(long long)kSortBuckets * nBlk + lane * (kSortBuckets / 32) + q];
            s += t[q];
        }
        int incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        int run = incl - s;
#pragma unroll
        for (int q = 0; q < kSortBuckets / 32; ++q) {
            const int b = lane * (kSortBuckets / 32) + q;
            cnt[b] = run + off[(long long)b * nBlk + blockIdx.x];
            run += t[q];
        }
    }
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int c = 0; c < kSortChunk / 32; ++c) {
        const long long i = base + c * 32 + lane;
        const bool active = i < N;
        const int key = active ? sortKey(x[c]) : kSortBuckets + lane;
        const unsigned grp = __match_any_sync(0xffffffffu, key);
        const int rank = __popc(grp & lt);
        int slot = 0;
        if (active) slot = cnt[key];
        __syncwarp();
        if (active) {
            perm[slot + rank] = (int)i;
            if (rank == 0) cnt[key] = slot + __popc(grp);
        }
        __syncwarp();
    }
}

// The per-component reductions of a KL step in one launch (blockIdx.y =
// component): gradient rows exactly as reduceRowsKernel with scale 1, the
// loss exactly as sumLossKernel, so results equal the per-component launches.
__global__ void klReduceKernel(const double* part, const long long* rowBase, const KLReduceDesc* descs,
                               double* grad, const double* lossPart, const int* lossSlots, double lossScale,
                               double* loss) {
    __shared__ double red[kRowGroups][33];
    const KLReduceDesc q = descs[blockIdx.y];
    const int t = blockIdx.x * 32 + threadIdx.x;
    const int g = threadIdx.y;
    const long long* rb = rowBase + q.rowOff;
    red[g][threadIdx.x] = t < q.nTerms ? sumRowGroup(part, rb, q.nRows, t, g) : 0.0;
    __syncthreads();
    if (g == 0 && t < q.nTerms) {
        double v = 0.0;
        for (int k = 0; k < kRowGroups; ++k) v += red[k][threadIdx.x];
        grad[q.outOff + t] = v;
    }
    if (loss && blockIdx.x == 0) {
        // The loss partials likewise: one group each, its lanes' sums in order.
        __shared__ double ls[32];
        if (g == kRowGroups - 1) {
            double l = 0.0;
            for (int j = threadIdx.x; j < q.nLoss; j += 32) l += lossPart[lossSlots[q.lossOff + j]];
            ls[threadIdx.x] = l;
            __syncwarp();
            if (threadIdx.x == 0) {
                l = 0.0;
                for (int k = 0; k < 32; ++k) l += ls[k];
                loss[q.comp] = l * lossScale;
            }
        }
    }
}

__global__ void sumLossKernel(const double* lossPart, const int* slots, int n, double scale, double* out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double s = 0.0;
        for (int j = 0; j < n; ++j) s += lossPart[slots[j]];
        *out = s * scale;
    }
}

// The reference objective's reductions over dense per-point outputs
// (FastGaussianReverseKLObjective, src/MapObjective.cpp:185-234): block b < nTerms
// sums grad_b = invN sum_i (sT(b,i) - sL(b,i)); block nTerms sums the loss
// invN sum_i (0.5 T_i^2 - ld_i).  Fixed-order (strided, then tree) sums.
__global__ void denseKLReduceKernel(const double* T, const double* ld, const double* dT, const double* dL, int nTerms,
                                    long long N, double invN, double* loss, double* grad) {
    __shared__ double red[256];
    const int b = blockIdx.x;
    double s = 0.0;
    if (b < nTerms) {
        const double* a = dT + (long long)b * N;
        const double* c = dL + (long long)b * N;
        for (long long i = threadIdx.x; i < N; i += blockDim.x) s += a[i] - c[i];
    } else {
        for (long long i = threadIdx.x; i < N; i += blockDim.x) s += 0.5 * T[i] * T[i] - ld[i];
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (b < nTerms) grad[b] = red[0] * invN;
        else *loss = red[0] * invN;
    }
}

// Per term, the mean over points of the squared per-point KL gradient,
// (dT_j - dL_j)^2 with the dense outputs of denseKLReduceKernel.
__global__ void denseKLSquaresKernel(const double* dT, const double* dL, long long N, double invN, double* out) {
    __shared__ double red[256];
    const int b = blockIdx.x;
    const double* a = dT + (long long)b * N;
    const double* c = dL + (long long)b * N;
    double s = 0.0;
    for (long long i = threadIdx.x; i < N; i += blockDim.x) {
        const double g = a[i] - c[i];
        s = fma(g, g, s);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[b] = red[0] * invN;
}

// FP64 peak probe: independent DFMA chains (8 per thread).
__global__ void dfmaPeakKernel(double* out, int iters, double seed) {
    double x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = seed + j * 1e-3 + threadIdx.x * 1e-9;
    const double m = 0.999999, c = 1e-7;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = fma(x[j], m, c);
    }
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += x[j];
    if (s == 12345.678) out[0] = s;
}

// --------------------------------------------------------------------------
// Dispatch.
// --------------------------------------------------------------------------
template <int BASIS, int POS>
static cudaError_t launchFusedBP(const FusedParams& prm, int pmax, int nItems, int needJ, int needE,
                                 cudaStream_t stream) {
    switch (pmax) {
        case 1: return launchFusedP<BASIS, POS, 1>(prm, nItems, needJ, needE, stream);
        case 2: return launchFusedP<BASIS, POS, 2>(prm, nItems, needJ, needE, stream);
        case 3: return launchFusedP<BASIS, POS, 3>(prm, nItems, needJ, needE, stream);
        case 4: return launchFusedP<BASIS, POS, 4>(prm, nItems, needJ, needE, stream);
        case 5: return launchFusedP<BASIS, POS, 5>(prm, nItems, needJ, needE, stream);
        case 6: return launchFusedP<BASIS, POS, 6>(prm, nItems, needJ, needE, stream);
        case 8: return launchFusedP<BASIS, POS, 8>(prm, nItems, needJ, needE, stream);
        case 12: return launchFusedP<BASIS, POS, 12>(prm, nItems, needJ, needE, stream);
        default: return cudaErrorInvalidValue;
    }
}

template <int BASIS, int POS>
static cudaError_t launchInverseBP(const InverseParams& prm, int pmax, int nBlocks, cudaStream_t stream) {
    switch (pmax) {
        case 1: return launchInverseP<BASIS, POS, 1>(prm, nBlocks, stream);
        case 2: return launchInverseP<BASIS, POS, 2>(prm, nBlocks, stream);
        case 3: return launchInverseP<BASIS, POS, 3>(prm, nBlocks, stream);
        case 4: return launchInverseP<BASIS, POS, 4>(prm, nBlocks, stream);
        case 5: return launchInverseP<BASIS, POS, 5>(prm, nBlocks, stream);
        case 6: return launchInverseP<BASIS, POS, 6>(prm, nBlocks, stream);
        case 8: return launchInverseP<BASIS, POS, 8>(prm, nBlocks, stream);
        case 12: return launchInverseP<BASIS, POS, 12>(prm, nBlocks, stream);
        default: return cudaErrorInvalidValue;
    }
}

int instantiatedPmax(int p) {
    if (p <= 6) return p < 1 ? 1 : p;
    if (p <= 8) return 8;
    if (p <= 12) return 12;
    return -1;
}

cudaError_t launchFused(int basis, int pos, int pmax, const FusedParams& prm, int nItems, int needJ, int needE,
                        cudaStream_t stream) {
    if (basis == kBasisSigmoid) {
        if (pos == kPosSoftPlus) return launchFusedBP<kBasisSigmoid, kPosSoftPlus>(prm, pmax, nItems, 0, 0, stream);
        return launchFusedBP<kBasisSigmoid, kPosExp>(prm, pmax, nItems, 0, 0, stream);
    }
    if (basis == kBasisProbHermite) {
        if (pos == kPosSoftPlus) return launchFusedBP<kBasisProbHermite, kPosSoftPlus>(prm, pmax, nItems, needJ, needE, stream);
        return launchFusedBP<kBasisProbHermite, kPosExp>(prm, pmax, nItems, needJ, needE, stream);
    }
    if (pos == kPosSoftPlus) return launchFusedBP<kBasisHermiteFunctions, kPosSoftPlus>(prm, pmax, nItems, needJ, needE, stream);
    return launchFusedBP<kBasisHermiteFunctions, kPosExp>(prm, pmax, nItems, needJ, needE, stream);
}

int batchOrderClass(int p) {
    if (p <= 2) return 2;
    if (p <= 4) return 4;
    if (p <= 6) return 6;
    if (p <= 8) return 8;
    return -1;
}

cudaError_t launchBatch(int basis, int pos, const FusedParams& prm, int nItems, int pmaxClass, int* counter,
                        cudaStream_t stream) {
    if (basis == kBasisSigmoid) return cudaErrorNotSupported;
    if (basis == kBasisProbHermite) {
        if (pos == kPosSoftPlus)
            return launchBatchP<kBasisProbHermite, kPosSoftPlus>(prm, nItems, pmaxClass, counter, stream);
        return launchBatchP<kBasisProbHermite, kPosExp>(prm, nItems, pmaxClass, counter, stream);
    }
    if (pos == kPosSoftPlus)
        return launchBatchP<kBasisHermiteFunctions, kPosSoftPlus>(prm, nItems, pmaxClass, counter, stream);
    return launchBatchP<kBasisHermiteFunctions, kPosExp>(prm, nItems, pmaxClass, counter, stream);
}

cudaError_t launchInverse(int basis, int pos, int pmax, const InverseParams& prm, int nBlocks, cudaStream_t stream) {
    if (basis == kBasisSigmoid) {
        if (pos == kPosSoftPlus) return launchInverseBP<kBasisSigmoid, kPosSoftPlus>(prm, pmax, nBlocks, stream);
        return launchInverseBP<kBasisSigmoid, kPosExp>(prm, pmax, nBlocks, stream);
    }
    if (basis == kBasisProbHermite) {
        if (pos == kPosSoftPlus) return launchInverseBP<kBasisProbHermite, kPosSoftPlus>(prm, pmax, nBlocks, stream);
        return launchInverseBP<kBasisProbHermite, kPosExp>(prm, pmax, nBlocks, stream);
    }
    if (pos == kPosSoftPlus) return launchInverseBP<kBasisHermiteFunctions, kPosSoftPlus>(prm, pmax, nBlocks, stream);
    return launchInverseBP<kBasisHermiteFunctions, kPosExp>(prm, pmax, nBlocks, stream);
}

static std::atomic<long long> g_launches{0};

void countLaunches(cudaStream_t stream, long long n) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess) {
        cudaGetLastError();  // the query's own error; the launch error was read before
        return;
    }
    if (cs == cudaStreamCaptureStatusNone) g_launches.fetch_add(n, std::memory_order_relaxed);
}

long long launchCount() { return g_launches.load(std::memory_order_relaxed); }

size_t fusedSmemBytes(int tpb, int dmax, int nBmax, int depthMax, int pmax, bool input) {
    size_t n = (size_t)dmax * tpb + (size_t)nBmax * (tpb + 1) + 1 + (size_t)(depthMax + 1) * tpb +
               (size_t)(pmax + 1) * tpb;
    if (input) {
        n += (size_t)nBmax * (tpb + 1) + (size_t)dmax * tpb +
             (size_t)((depthMax + 1) * (depthMax + 2) / 2) * tpb;
    }
    return n * sizeof(double);
}

cudaError_t launchGather(const int32_t* slotGlobalTerm, int nSlots, const double* coeffs, double* cm,
                         cudaStream_t stream) {
    if (nSlots <= 0) return cudaSuccess;
    gatherKernel<<<(nSlots + 255) / 256, 256, 0, stream>>>(slotGlobalTerm, nSlots, coeffs, cm);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

cudaError_t launchReduceRows(const double* part, const long long* rowBase, int nRows, int nTerms, double scale,
                             double* out, int accumulate, cudaStream_t stream) {
    if (nTerms <= 0) return cudaSuccess;
    dim3 blk(32, kRowGroups);
    reduceRowsKernel<<<(nTerms + 31) / 32, blk, 0, stream>>>(part, rowBase, nRows, nTerms, scale, out, accumulate);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

cudaError_t launchKLReduce(const double* part, const long long* rowBase, const KLReduceDesc* descs, int nComps,
                           int maxTerms, double* grad, const double* lossPart, const int* lossSlots, double lossScale,
                           double* loss, cudaStream_t stream) {
    if (nComps <= 0) return cudaSuccess;
    dim3 grid((unsigned)std::max(1, (maxTerms + 31) / 32), (unsigned)nComps), blk(32, kRowGroups);
    klReduceKernel<<<grid, blk, 0, stream>>>(part, rowBase, descs, grad, lossPart, lossSlots, lossScale, loss);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

cudaError_t launchSumLoss(const double* lossPart, const int* slots, int n, double scale, double* out,
                          cudaStream_t stream) {
    sumLossKernel<<<1, 32, 0, stream>>>(lossPart, slots, n, scale, out);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

size_t sortScratchInts(long long N) { return (size_t)((N + kSortChunk - 1) / kSortChunk + 1) * kSortBuckets; }

cudaError_t launchSortByLast(const double* xd, long long stride, long long N, int* hist, int* perm,
                             cudaStream_t stream) {
    return launchSortByLastSegments(xd, stride, 0, 1, N, hist, perm, 0, stream);
}

cudaError_t launchSortByLastSegments(const double* keys, long long stride, long long keySeg, int nSeg, long long N,
                                     int* hist, int* perm, long long permSeg, cudaStream_t stream) {
    if (N <= 0 || nSeg <= 0) return cudaSuccess;
    const int nBlk = (int)((N + kSortChunk - 1) / kSortChunk);
    const long long histSeg = (long long)sortScratchInts(N);
    keyHistKernel<<<dim3(nBlk, nSeg), 256, 0, stream>>>(keys, stride, N, hist, keySeg, histSeg);
    keyScanKernel<<<dim3(kSortBuckets / 8, nSeg), 256, 0, stream>>>(hist, nBlk, histSeg);
    keyScatterKernel<<<dim3(nBlk, nSeg), 32, 0, stream>>>(keys, stride, N, hist, perm, keySeg, histSeg, permSeg);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 3);
    return e;
}

cudaError_t launchDenseKLSquares(const double* dT, const double* dL, int nTerms, long long N, double* out,
                                 cudaStream_t stream) {
    if (nTerms <= 0 || N <= 0) return cudaSuccess;
    denseKLSquaresKernel<<<nTerms, 256, 0, stream>>>(dT, dL, N, 1.0 / (double)N, out);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

cudaError_t launchDenseKLReduce(const double* T, const double* ld, const double* dT, const double* dL, int nTerms,
                                long long N, double* loss, double* grad, cudaStream_t stream) {
    denseKLReduceKernel<<<nTerms + 1, 256, 0, stream>>>(T, ld, dT, dL, nTerms, N, 1.0 / (double)N, loss, grad);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

__global__ void sigmoidEvalKernel(const CompDesc c, int maxOrder, const double* x, long long n, long long stride,
                                  double* out, double* d1, double* d2) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v[kMaxLastOrder + 1], g1[kMaxLastOrder + 1], g2[kMaxLastOrder + 1];
    sigmoidBasis<kMaxLastOrder, true>(x[i * stride], maxOrder, c, v, g1, g2);
    for (int k = 0; k <= maxOrder; ++k) {
        out[k * n + i] = v[k];
        if (d1) d1[k * n + i] = g1[k];
        if (d2) d2[k * n + i] = g2[k];
    }
}

cudaError_t launchSigmoidEval(const CompDesc& c, int maxOrder, const double* x, long long n, long long stride,
                              double* out, double* d1, double* d2, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    if (maxOrder < 0 || maxOrder > kMaxLastOrder) return cudaErrorInvalidValue;
    sigmoidEvalKernel<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(c, maxOrder, x, n, stride, out, d1, d2);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

cudaError_t launchDfmaPeak(double* out, int blocks, int threads, int iters, cudaStream_t stream) {
    dfmaPeakKernel<<<blocks, threads, 0, stream>>>(out, iters, 1.0);
    const cudaError_t e = cudaGetLastError();
    countLaunches(stream, 1);
    return e;
}

}  // namespace mpgb
