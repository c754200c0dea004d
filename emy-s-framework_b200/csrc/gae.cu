// GAE over a flat rollout buffer on the device.
//
// Same results, element for element, as the reference's device GAE,
// rsc::ComputeGAEOnDevice (RocketSimCuda/src/GAECuda.cu:247-300): the buffer splits at every
// nonzero terminal into independent segments, each segment runs the backward recurrence of
// GAECuda.cu:71-115 from its end with zero carries, and targetValues = valPreds + advantages
// (GAECuda.cu:120-129).  Compiled with --fmad=false, so each multiply and add rounds as the
// reference's --fmad=false build does.
//
// Layout of the work (two launches, no host round trip):
//   gaeSummaryKernel  truncations in each 4,096-element chunk (left out when there are none);
//   gaeScanKernel     their exclusive prefix, for buffers of more than kGaeDirect chunks; in
//                     smaller ones each block adds up the counts before its own;
//   gaeSegmentKernel  one block per chunk, for the segments that END in it: see there.
// The last block to finish (a ticket counter, no waiting) adds the blocks' sums of |r/std| and
// of what clipping took of it in block order and writes rewClipPortion.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "rsb.h"

namespace rsb {
void setGlobalError(const std::string& msg);
}

namespace {

constexpr int kGaeThreads = 256;
constexpr int kGaePerThread = 16;
constexpr int kGaeChunk = kGaeThreads * kGaePerThread;  // elements per block
constexpr int8_t kTermNormal = 1;
constexpr int8_t kTermTruncated = 2;
// largest T: chunk arithmetic stays inside int32
constexpr int32_t kGaeMaxT = INT32_MAX - 2 * kGaeChunk;

// Shared rows are padded by one word per 32 elements, so that lanes walking segments whose lengths
// are multiples of 32 (one trajectory of a 32-step rollout per lane) fall into different banks.
constexpr int kPadded = kGaeChunk + kGaeChunk / 32;
__host__ __device__ constexpr int padIdx(int i) { return i + (i >> 5); }
constexpr int kGaeWords = kGaeChunk / 32;
constexpr int kGaeHalo = 4 * kGaeThreads;
// Up to this many chunks (16.8 million elements) a block adds up the counts of the chunks before
// its own, at most 16 loads a thread beside those of its elements; a scan of its own costs a launch
// and a single block's pass, 4 us at 3,072 chunks.
constexpr int kGaeDirect = 4096;

struct GaeArgs {
    const float* rews;
    const int8_t* term;
    const float* vals;
    const float* truncVals;
    int numTruncs;
    float* adv;
    float* tgt;
    float* ret;
    float* clipPortion;
    int T;
    int nChunks;
    float gamma, lambda, returnStd, clipRange;
    const int* count;  // truncations of each chunk, or before each chunk (counted)
    bool counted;
    float2* part;
    unsigned* ticket;
};

__device__ __forceinline__ int warpSum(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ int warpMax(int v) { return __reduce_max_sync(0xffffffffu, v); }

// Truncations of each chunk.  Thread t reads bytes [16 t, 16 t + 16) of its chunk, as one 16-byte
// load when the row is 16-byte aligned.  The first block clears the ticket.
template <bool kVec>
__global__ void __launch_bounds__(kGaeThreads) gaeSummaryKernel(const int8_t* __restrict__ term, int T,
                                                                int* __restrict__ count, unsigned* ticket) {
    const int base = blockIdx.x * kGaeChunk;
    const int len = min(kGaeChunk, T - base);
    const int j0 = threadIdx.x * kGaePerThread;
    cudaTriggerProgrammaticLaunchCompletion();
    if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
    int tr = 0;
    if (kVec && j0 + kGaePerThread <= len) {
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(term + base + j0));
        const unsigned words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int k = 0; k < kGaePerThread; ++k) tr += (int8_t)(words[k >> 2] >> (8 * (k & 3))) == kTermTruncated;
    } else {
        for (int k = 0; k < kGaePerThread && j0 + k < len; ++k) tr += __ldg(term + base + j0 + k) == kTermTruncated;
    }
    tr = __syncthreads_count(tr & 1) + 2 * __syncthreads_count(tr >> 1 & 1) + 4 * __syncthreads_count(tr >> 2 & 1) +
         8 * __syncthreads_count(tr >> 3 & 1) + 16 * __syncthreads_count(tr >> 4 & 1);
    if (threadIdx.x == 0) count[blockIdx.x] = tr;
}

// Exclusive prefix over chunks, in place: truncations before the chunk.
__global__ void __launch_bounds__(1024) gaeScanKernel(int* __restrict__ count, int n) {
    __shared__ int wSum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += 1024) {
        const int i = base + (int)threadIdx.x;
        const int v = i < n ? count[i] : 0;
        int s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int s2 = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += s2;
        }
        if (lane == 31) wSum[warp] = s;
        __syncthreads();
        const int w = wSum[lane];
        const int before = warpSum(lane < warp ? w : 0), all = warpSum(w);
        if (i < n) count[i] = carry + before + s - v;
        carry += all;
        __syncthreads();
    }
}

__device__ __forceinline__ int8_t termOf(unsigned w, int c) { return (int8_t)(w >> (8 * c)); }
// Bit c of the result: byte c of a comparison's mask (0 or 255).
__device__ __forceinline__ unsigned bytesToBits(unsigned mask) { return (mask & 0x01010101u) * 0x01020408u >> 24 & 15u; }

// The reward as the advantages use it.  Adds its magnitude and what clipping took of it; summed
// apart, the small excess keeps the digits that the difference of two large sums would lose.
template <bool kScaled>
__device__ __forceinline__ float gaeReward(const GaeArgs& a, float rew, float& sum, float& excess) {
    if (!kScaled) {
        sum += fabsf(rew);
        return rew;
    }
    const float r = rew / a.returnStd;
    float used = r;
    if (a.clipRange > 0.0f) used = fminf(fmaxf(r, -a.clipRange), a.clipRange);
    sum += fabsf(r);
    excess += fabsf(r) - fabsf(used);
    return used;
}

// The recurrence of GAECuda.cu:77-113 over rows [stop, end], backward.  Its rows hold what does not
// depend on later steps (sD the delta, sR the reward), an aligned four of them read ahead of the
// chain; they take the advantages and the returns.  A segment's last step starts from zero carries,
// so that the factors (1 - done)(1 - trunc), which are 1 at every other step, need not be applied.
__device__ __forceinline__ void gaeWalk(float* sD, float* sR, int end, int stop, float gl, float gamma, float& adv,
                                        float& ret) {
    auto one = [&](int at) {
        ret = sR[at] + ret * gamma;
        adv = sD[at] + gl * adv;
        sD[at] = adv;
        sR[at] = ret;
    };
    int rel = end;
    for (; rel >= stop && (rel & 3) != 3; --rel) one(padIdx(rel));
    for (; rel - 3 >= stop; rel -= 4) {
        const int at = padIdx(rel - 3);
        float d[4], r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            d[k] = sD[at + k];
            r[k] = sR[at + k];
        }
#pragma unroll
        for (int k = 3; k >= 0; --k) {
            ret = r[k] + ret * gamma;
            adv = d[k] + gl * adv;
            sD[at + k] = adv;
            sR[at + k] = ret;
        }
    }
    for (; rel >= stop; --rel) one(padIdx(rel));
}

// Elements j .. j + 3 of a row, zero from len on.
template <bool kVec>
__device__ __forceinline__ void gaeLoad4(const float* __restrict__ p, int j, int len, float* v) {
    if (kVec && j + 4 <= len) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(p + j));
        v[0] = x.x;
        v[1] = x.y;
        v[2] = x.z;
        v[3] = x.w;
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = j + c < len ? __ldg(p + j + c) : 0.0f;
    }
}
template <bool kVec>
__device__ __forceinline__ unsigned gaeTerm4(const int8_t* __restrict__ p, int j, int len) {
    if (kVec && j + 4 <= len) return __ldg(reinterpret_cast<const unsigned*>(p + j));
    unsigned w = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (j + c < len) w |= (unsigned)(uint8_t)__ldg(p + j + c) << (8 * c);
    return w;
}
// Results of elements j .. j + 3 that lie in [from, to).
template <bool kVec>
__device__ __forceinline__ void gaeStore4(const GaeArgs& a, int base, int j, int from, int to, const float* sD,
                                          const float* sR, const float* val) {
    if (j >= to || j + 4 <= from) return;
    const int at = padIdx(j);
    float d[4], r[4], g[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        d[c] = sD[at + c];
        r[c] = sR[at + c];
        g[c] = val[c] + d[c];
    }
    if (kVec && j >= from && j + 4 <= to) {
        *reinterpret_cast<float4*>(a.adv + base + j) = make_float4(d[0], d[1], d[2], d[3]);
        *reinterpret_cast<float4*>(a.ret + base + j) = make_float4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<float4*>(a.tgt + base + j) = make_float4(g[0], g[1], g[2], g[3]);
        return;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (j + c >= from && j + c < to) {
            a.adv[base + j + c] = d[c];
            a.ret[base + j + c] = r[c];
            a.tgt[base + j + c] = g[c];
        }
}

// One block per chunk.  What a step needs besides the carries (reward, delta) is computed for every
// element in parallel, in the threads that loaded it, four elements to a load; a thread then walks
// each segment that ends among 32 elements of its own, two multiplies and two adds a step; the
// threads that hold the values write the results.  A segment that began in an earlier chunk goes on
// through windows of kGaeHalo elements, staged and written by the whole block and walked by one
// thread.
//
// What bounds it: 393,216 x 32 elements (266 MB, 41 us at the rate of a copy) take 64 us in calls
// side by side, against 77 us with bounds, terminals and padding worked out for every element and 81
// us with the arithmetic in the walk as well; the rest is instructions and the waits between the
// phases.  More blocks on a multiprocessor do not shorten it (five or six of 48 or 40 registers: 77
// and 81 us before those instructions went).  257 episodes of 400 uneven steps: 10 us, against 23 us
// when a segment went on through global memory step by step.
template <bool kVec, bool kScaled>
__global__ void __launch_bounds__(kGaeThreads, 4) gaeSegmentKernel(GaeArgs a) {
    __shared__ float sD[kPadded], sR[kPadded];
    __shared__ unsigned sEnd[kGaeWords], sTrunc[kGaeWords];  // a bit per element: ends of segments, truncations
    __shared__ int sBefore[kGaeWords], sCount[kGaeThreads / 32], sMax[kGaeThreads / 32];
    __shared__ float2 sWarpSum[kGaeThreads / 32], sCarry;
    __shared__ bool sLastBlock;

    const uint32_t all = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = blockIdx.x * kGaeChunk;
    const int len = min(kGaeChunk, a.T - base);
    const bool lastChunk = base + len == a.T;
    // past the buffer the reference reads valPreds[T] only for a non-terminal final step
    // (GAECuda.cu:101-102)
    const int lenVal = len + (!lastChunk || __ldg(a.term + a.T - 1) == 0);

    // 1. the chunk's elements; bits of the segments' ends (nonzero terminals, and the buffer's last
    //    element) and of the truncations; truncations before the chunk
    float rew[4][4], val[4][4], after[4];
    unsigned term[4];
    if (tid < kGaeWords) sEnd[tid] = sTrunc[tid] = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j = 4 * (k * kGaeThreads + tid);
        term[k] = gaeTerm4<kVec>(a.term + base, j, len);
        gaeLoad4<kVec>(a.rews + base, j, len, rew[k]);
        if (kVec && j + 4 <= len) gaeLoad4<true>(a.vals + base, j, len, val[k]);
        else gaeLoad4<false>(a.vals + base, j, lenVal, val[k]);
        after[k] = lane == 31 && j + 4 < lenVal ? __ldg(a.vals + base + j + 4) : 0.0f;
    }
    cudaGridDependencySynchronize();  // from here on the counts and the ticket
    int before = 0;
    if (a.count) {
        if (a.counted) before = tid == 0 ? __ldcg(a.count + blockIdx.x) : 0;
        else
            for (int i = tid; i < (int)blockIdx.x; i += kGaeThreads) before += __ldcg(a.count + i);
    }
    before = warpSum(before);
    if (lane == 0) sCount[warp] = before;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j = 4 * (k * kGaeThreads + tid);
        const float first = __shfl_down_sync(all, val[k][0], 1);
        if (lane != 31) after[k] = first;
        // elements past the buffer have terminals of 0
        unsigned ends = bytesToBits(__vcmpne4(term[k], 0));
        if (lastChunk && j >> 2 == (len - 1) >> 2) ends |= 1u << ((len - 1) & 3);
        if (ends) {
            atomicOr(&sEnd[j >> 5], ends << (j & 31));
            const unsigned truncs = bytesToBits(__vcmpeq4(term[k], 0x01010101u * kTermTruncated));
            if (truncs) atomicOr(&sTrunc[j >> 5], truncs << (j & 31));
        }
    }
    __syncthreads();
    before = 0;
#pragma unroll
    for (int w = 0; w < kGaeThreads / 32; ++w) before += sCount[w];
    if (warp == 0) {
        // truncations before each word
        for (int w0 = 0; w0 < kGaeWords; w0 += 32) {
            const int n = __popc(sTrunc[w0 + lane]);
            int s = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int s2 = __shfl_up_sync(all, s, o);
                if (lane >= o) s += s2;
            }
            sBefore[w0 + lane] = before + s - n;
            before += __shfl_sync(all, s, 31);
        }
    }
    __syncthreads();

    // 2. reward and delta of every element (past the buffer: zeros)
    float accRew = 0.0f, accExcess = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j = 4 * (k * kGaeThreads + tid), at = padIdx(4 * tid) + k * padIdx(4 * kGaeThreads);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int8_t t = termOf(term[k], c);
            float next = c < 3 ? val[k][c < 3 ? c + 1 : 3] : after[k];
            if (t == kTermNormal) next = 0.0f;
            if (t == kTermTruncated) {
                const int bit = (j + c) & 31;
                const int idx = a.numTruncs - (sBefore[j >> 5] + __popc(sTrunc[j >> 5] & ((1u << bit) - 1u))) - 1;
                // a count that does not match the truncated steps reads nothing out of range
                next = idx >= 0 && idx < a.numTruncs ? __ldg(a.truncVals + idx) : 0.0f;
            }
            const float r = gaeReward<kScaled>(a, rew[k][c], accRew, accExcess);
            sD[at + c] = (r + a.gamma * next) - val[k][c];
            sR[at + c] = rew[k][c];
        }
    }
    if (!kScaled) accExcess = accRew;
    __syncthreads();

    // 3. a thread per 32 elements, backward from each end among them
    const float gl = a.gamma * a.lambda;
    for (unsigned ends = tid < kGaeWords ? sEnd[tid] : 0u; ends; ends &= ends - 1u) {
        const int end = 32 * tid + __ffs((int)ends) - 1;
        int w = end >> 5;
        unsigned earlier = sEnd[w] & ((1u << (end & 31)) - 1u);
        while (!earlier && w > 0) earlier = sEnd[--w];
        const int start = earlier ? 32 * w + 32 - __clz((int)earlier) : 0;
        float adv = 0.0f, ret = 0.0f;
        gaeWalk(sD, sR, end, start, gl, a.gamma, adv, ret);
        if (!earlier) sCarry = make_float2(adv, ret);
    }
    __syncthreads();

    // 4. the elements of the segments that end here
    int owned = 0;
    for (int w0 = 0; w0 < kGaeWords; w0 += 32) {
        const unsigned e = sEnd[w0 + lane];
        owned = max(owned, e ? 32 * (w0 + lane) + 32 - __clz((int)e) : 0);
    }
    owned = warpMax(owned);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        gaeStore4<kVec>(a, base, 4 * (k * kGaeThreads + tid), 0, owned, sD, sR, val[k]);

    // 5. the part of the first of them in earlier chunks
    for (int lo = base; owned > 0 && lo > 0;) {
        const int hi = lo;
        lo -= kGaeHalo;
        const int j = 4 * tid;
        const unsigned t = gaeTerm4<kVec>(a.term + lo, j, kGaeHalo);
        int last = -1;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (termOf(t, c) != 0) last = j + c;
        last = warpMax(last);
        __syncthreads();  // the rows and sMax are read until here
        if (lane == 0) sMax[warp] = last;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kGaeThreads / 32; ++w) last = max(last, sMax[w]);
        const int start = last + 1;
        if (start == hi - lo) break;
        const bool mine = j + 4 > start;
        float r[4], v[5], sum = 0.0f;
        if (mine) {
            gaeLoad4<kVec>(a.rews + lo, j, kGaeHalo, r);
            gaeLoad4<kVec>(a.vals + lo, j, kGaeHalo, v);
            v[4] = __ldg(a.vals + lo + j + 4);  // lo + j + 4 <= base
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                sD[padIdx(j) + c] = (gaeReward<kScaled>(a, r[c], sum, sum) + a.gamma * v[c + 1]) - v[c];
                sR[padIdx(j) + c] = r[c];
            }
        }
        __syncthreads();
        if (tid == 0) {
            float2 carry = sCarry;
            gaeWalk(sD, sR, kGaeHalo - 1, start, gl, a.gamma, carry.x, carry.y);
            sCarry = carry;
        }
        __syncthreads();
        if (mine) gaeStore4<kVec>(a, lo, j, start, kGaeHalo, sD, sR, v);
        if (start > 0) break;
    }

    // 6. clip-portion sums: block partial, then the last block adds the partials in order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        accRew += __shfl_xor_sync(all, accRew, o);
        accExcess += __shfl_xor_sync(all, accExcess, o);
    }
    if (lane == 0) sWarpSum[warp] = make_float2(accRew, accExcess);
    __syncthreads();
    if (tid == 0) {
        float r = 0.0f, cl = 0.0f;
        for (int w = 0; w < kGaeThreads / 32; ++w) {
            r += sWarpSum[w].x;
            cl += sWarpSum[w].y;
        }
        a.part[blockIdx.x] = make_float2(r, cl);
        __threadfence();
        sLastBlock = atomicAdd(a.ticket, 1u) == (unsigned)(a.nChunks - 1);
    }
    __syncthreads();
    if (!sLastBlock) return;
    __threadfence();
    float r = 0.0f, cl = 0.0f;
    for (int i = tid; i < a.nChunks; i += kGaeThreads) {
        const float2 p = __ldcg(a.part + i);
        r += p.x;
        cl += p.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_xor_sync(0xffffffffu, r, o);
        cl += __shfl_xor_sync(0xffffffffu, cl, o);
    }
    __syncthreads();
    if (lane == 0) sWarpSum[warp] = make_float2(r, cl);
    __syncthreads();
    if (tid == 0) {
        float tr = 0.0f, tc = 0.0f;
        for (int w = 0; w < kGaeThreads / 32; ++w) {
            tr += sWarpSum[w].x;
            tc += sWarpSum[w].y;
        }
        *a.clipPortion = tc / fmaxf(tr, 1e-7f);
    }
}

// What a call works in: a row of counts, a row of partial sums and a ticket, in one allocation.
struct GaeRows {
    int capacity = 0;  // chunks
    int* count = nullptr;
    float2* part = nullptr;
    unsigned* ticket = nullptr;
};
// `sets` of them, one after another; `first` is the first one.
bool allocRows(int nChunks, int sets, GaeRows& first) {
    const size_t cap = (size_t)(nChunks < 64 ? 64 : nChunks);
    if (cudaMalloc(&first.part, ((sizeof(float2) + sizeof(int)) * cap + sizeof(unsigned)) * sets) != cudaSuccess) return false;
    first.capacity = (int)cap;
    first.count = reinterpret_cast<int*>(first.part + cap * sets);
    first.ticket = reinterpret_cast<unsigned*>(first.count + cap * sets);
    return true;
}

// Allocations that this thread makes while a stream is captured are not part of the capture.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The rows of a captured call belong to the graph it is captured into: replays of two graphs, or of
// two calls in one, may run side by side, and at any time while the graph lives.  The graph and its
// executables give them back when the last of them is gone; a later capture takes them again, and
// what is more than kGaeReturned is freed by the next call that is not captured.
constexpr size_t kGaeReturned = 16;
struct GaeGraphRows {
    int dev;
    GaeRows rows;
};
struct GaeReturnedRows {
    std::mutex mu;
    std::vector<GaeGraphRows*> list;
};
GaeReturnedRows& gaeReturned() {
    static GaeReturnedRows* r = new GaeReturnedRows;  // graphs may be destroyed as late as at exit
    return *r;
}
void CUDART_CB gaeGiveBack(void* p) {  // may call nothing of CUDA
    GaeReturnedRows& r = gaeReturned();
    std::lock_guard<std::mutex> lock(r.mu);
    r.list.push_back(static_cast<GaeGraphRows*>(p));
}
rsb_status rowsForGraph(int dev, int nChunks, cudaGraph_t graph, GaeRows& out) {
    GaeReturnedRows& r = gaeReturned();
    GaeGraphRows* g = nullptr;
    {
        std::lock_guard<std::mutex> lock(r.mu);
        for (size_t i = 0; i < r.list.size() && !g; ++i)
            if (r.list[i]->dev == dev && r.list[i]->rows.capacity >= nChunks) {
                g = r.list[i];
                r.list.erase(r.list.begin() + (ptrdiff_t)i);
            }
    }
    if (!g) {
        RelaxedCapture relaxed;
        g = new GaeGraphRows{dev, {}};
        if (!allocRows(nChunks, 1, g->rows)) {
            delete g;
            return RSB_ERR_NOMEM;
        }
    }
    out = g->rows;
    cudaUserObject_t owner = nullptr;
    if (cudaUserObjectCreate(&owner, g, gaeGiveBack, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        gaeGiveBack(g);
        return RSB_ERR_CUDA;
    }
    if (cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaUserObjectRelease(owner, 1);
        return RSB_ERR_CUDA;
    }
    return RSB_OK;
}
void freeReturnedRows() {
    GaeReturnedRows& r = gaeReturned();
    std::vector<GaeGraphRows*> over;
    {
        std::lock_guard<std::mutex> lock(r.mu);
        while (r.list.size() > kGaeReturned) {
            over.push_back(r.list.back());
            r.list.pop_back();
        }
    }
    for (GaeGraphRows* g : over) {
        RelaxedCapture relaxed;
        cudaFree(g->rows.part);
        delete g;
    }
}

// Per-device scratch of the other calls, never waited for on the host: rows for each stream that
// calls, so that calls on several streams run side by side.  The first kGaeOwn streams keep theirs.
// Beyond them a stream takes, of kGaeShared rows, those used longest ago, and its work waits on the
// device for the call that had them (an event is recorded after each call in these).  The rows of all
// are allocated together; a longer buffer makes new ones at least twice as long, which a slot takes
// when it needs them, and the old ones stay, since work may still use them (all together are at most
// twice the last).
constexpr int kGaeOwn = 16, kGaeShared = 8;
struct GaeSlot {
    unsigned long long stream = 0, used = 0;  // id of the stream, number of its last call (0: none)
    GaeRows rows;
    cudaEvent_t done = nullptr;  // shared slots
};
struct GaeScratch {
    GaeSlot slot[kGaeOwn + kGaeShared];
    GaeRows rows;  // the first slot's of the last allocation
    unsigned long long calls = 0;
};

std::mutex g_gaeMu;
std::vector<GaeScratch> g_gaeScratch;

// Host-buffer staging for rsb_compute_gae_host, per device.
struct GaeHostStage {
    size_t capT = 0, capTrunc = 0;
    float *rews = nullptr, *vals = nullptr, *trunc = nullptr, *adv = nullptr, *tgt = nullptr, *ret = nullptr,
          *clip = nullptr;
    int8_t* term = nullptr;
    cudaStream_t stream = nullptr;
};
std::vector<GaeHostStage> g_gaeHost;

rsb_status slotForStream(int dev, int nChunks, cudaStream_t st, GaeSlot*& out) {
    freeReturnedRows();
    if ((int)g_gaeScratch.size() <= dev) g_gaeScratch.resize(dev + 1);
    GaeScratch& s = g_gaeScratch[dev];
    unsigned long long id = 0;
    if (cudaStreamGetId(st, &id) != cudaSuccess) return RSB_ERR_CUDA;
    GaeSlot *slot = nullptr, *oldest = &s.slot[kGaeOwn];
    for (int k = 0; k < kGaeOwn + kGaeShared && !slot; ++k) {
        GaeSlot& c = s.slot[k];
        if ((c.used && c.stream == id) || (!c.used && k < kGaeOwn)) slot = &c;
        else if (k >= kGaeOwn && c.used < oldest->used) oldest = &c;
    }
    if (!slot) {
        slot = oldest;
        if (!slot->done && cudaEventCreateWithFlags(&slot->done, cudaEventDisableTiming) != cudaSuccess) return RSB_ERR_CUDA;
        if (slot->used && cudaStreamWaitEvent(st, slot->done, 0) != cudaSuccess) return RSB_ERR_CUDA;
    }
    if (slot->rows.capacity < nChunks) {
        if (s.rows.capacity < nChunks) {
            RelaxedCapture relaxed;
            GaeRows rows;
            if (!allocRows(nChunks > 2 * s.rows.capacity ? nChunks : 2 * s.rows.capacity, kGaeOwn + kGaeShared, rows))
                return RSB_ERR_NOMEM;
            s.rows = rows;
        }
        const size_t k = (size_t)(slot - s.slot), at = k * s.rows.capacity;
        slot->rows = GaeRows{s.rows.capacity, s.rows.count + at, s.rows.part + at, s.rows.ticket + k};
    }
    slot->stream = id;
    slot->used = ++s.calls;
    out = slot;
    return RSB_OK;
}

rsb_status launchGae(const float* rews, const int8_t* terminals, const float* valPreds, const float* truncValPreds,
                     int32_t numTruncs, float* advantages, float* targetValues, float* returns,
                     float* rewClipPortion, int32_t T, const rsb_gae_params& p, cudaStream_t st) {
    if (T == 0) {
        // no element: the sums are zero, so the portion is 0 / 1e-7 = 0
        return cudaMemsetAsync(rewClipPortion, 0, sizeof(float), st) == cudaSuccess ? RSB_OK : RSB_ERR_CUDA;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return RSB_ERR_CUDA;
    const int nChunks = (T + kGaeChunk - 1) / kGaeChunk;
    GaeRows rows;
    GaeSlot* slot = nullptr;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo(st, &capture, nullptr, &graph) != cudaSuccess ||
        capture == cudaStreamCaptureStatusInvalidated)
        return RSB_ERR_CUDA;
    const rsb_status rc = capture == cudaStreamCaptureStatusActive ? rowsForGraph(dev, nChunks, graph, rows)
                                                                   : slotForStream(dev, nChunks, st, slot);
    if (rc != RSB_OK) return rc;
    if (slot) rows = slot->rows;
    GaeArgs a;
    a.rews = rews;
    a.term = terminals;
    a.vals = valPreds;
    a.truncVals = truncValPreds;
    a.numTruncs = numTruncs;
    a.adv = advantages;
    a.tgt = targetValues;
    a.ret = returns;
    a.clipPortion = rewClipPortion;
    a.T = T;
    a.nChunks = nChunks;
    a.gamma = p.gamma;
    a.lambda = p.lambda;
    a.returnStd = p.return_std;
    a.clipRange = p.clip_range;
    int* const count = rows.count;
    a.part = rows.part;
    a.ticket = rows.ticket;
    a.count = numTruncs > 0 ? count : nullptr;
    a.counted = nChunks > kGaeDirect;
    auto aligned = [](const void* p, uintptr_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; };
    if (a.count) {
        if (aligned(terminals, 16)) gaeSummaryKernel<true><<<nChunks, kGaeThreads, 0, st>>>(terminals, T, count, a.ticket);
        else gaeSummaryKernel<false><<<nChunks, kGaeThreads, 0, st>>>(terminals, T, count, a.ticket);
        if (a.counted) gaeScanKernel<<<1, 1024, 0, st>>>(count, nChunks);
    } else if (cudaMemsetAsync(a.ticket, 0, sizeof(unsigned), st) != cudaSuccess) {
        return RSB_ERR_CUDA;
    }
    // four elements to a load and a store where every row allows it
    const bool vec = aligned(terminals, 4) && aligned(rews, 16) && aligned(valPreds, 16) && aligned(advantages, 16) &&
                     aligned(targetValues, 16) && aligned(returns, 16);
    const auto kernel = p.return_std > 0.0f ? (vec ? gaeSegmentKernel<true, true> : gaeSegmentKernel<false, true>)
                                            : (vec ? gaeSegmentKernel<true, false> : gaeSegmentKernel<false, false>);
    // it may start while the kernel before it runs: that kernel's results are read after a wait
    cudaLaunchAttribute overlap;
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nChunks);
    cfg.blockDim = dim3(kGaeThreads);
    cfg.stream = st;
    cfg.attrs = &overlap;
    cfg.numAttrs = a.count ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kernel, a) != cudaSuccess)
        return RSB_ERR_CUDA;
    if (slot && slot->done && cudaEventRecord(slot->done, st) != cudaSuccess) return RSB_ERR_CUDA;
    return cudaGetLastError() == cudaSuccess ? RSB_OK : RSB_ERR_CUDA;
}

bool validArgs(const void* rews, const void* terminals, const void* valPreds, const void* truncValPreds,
               int32_t numTruncs, const void* advantages, const void* targetValues, const void* returns,
               const void* rewClipPortion, int32_t T, const rsb_gae_params* params) {
    if (!params || !rewClipPortion || T < 0 || T > kGaeMaxT || numTruncs < 0) return false;
    if (numTruncs > 0 && !truncValPreds) return false;
    if (T > 0 && (!rews || !terminals || !valPreds || !advantages || !targetValues || !returns)) return false;
    return true;
}

}  // namespace

extern "C" {

rsb_status rsb_gae_default_params(rsb_gae_params* out) {
    if (!out) return RSB_ERR_INVALID;
    out->gamma = 0.99f;
    out->lambda = 0.95f;
    out->return_std = 0.0f;
    out->clip_range = 0.0f;
    return RSB_OK;
}

rsb_status rsb_compute_gae(const float* rews, const int8_t* terminals, const float* val_preds,
                           const float* trunc_val_preds, int32_t num_truncs, float* advantages, float* target_values,
                           float* returns, float* rew_clip_portion, int32_t T, const rsb_gae_params* params,
                           void* stream) {
    std::lock_guard<std::mutex> lock(g_gaeMu);
    if (!validArgs(rews, terminals, val_preds, trunc_val_preds, num_truncs, advantages, target_values, returns,
                   rew_clip_portion, T, params)) {
        rsb::setGlobalError("rsb_compute_gae: invalid argument");
        return RSB_ERR_INVALID;
    }
    const rsb_status rc = launchGae(rews, terminals, val_preds, trunc_val_preds, num_truncs, advantages,
                                    target_values, returns, rew_clip_portion, T, *params,
                                    reinterpret_cast<cudaStream_t>(stream));
    if (rc != RSB_OK) rsb::setGlobalError("rsb_compute_gae: CUDA launch or allocation failed");
    return rc;
}

rsb_status rsb_compute_gae_host(const float* rews, const int8_t* terminals, const float* val_preds,
                                int32_t num_val_preds, const float* trunc_val_preds, int32_t num_truncs,
                                float* advantages, float* target_values, float* returns, float* rew_clip_portion,
                                int32_t T, const rsb_gae_params* params) {
    std::lock_guard<std::mutex> lock(g_gaeMu);
    if (!validArgs(rews, terminals, val_preds, trunc_val_preds, num_truncs, advantages, target_values, returns,
                   rew_clip_portion, T, params) ||
        num_val_preds < T || (T > 0 && terminals[T - 1] == 0 && num_val_preds < T + 1)) {
        rsb::setGlobalError("rsb_compute_gae_host: invalid argument (a non-terminal final step needs T + 1 values)");
        return RSB_ERR_INVALID;
    }
    auto fail = [&](rsb_status rc, const char* what) {
        rsb::setGlobalError(std::string("rsb_compute_gae_host: ") + what);
        return rc;
    };
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return fail(RSB_ERR_CUDA, "no CUDA device");
    if ((int)g_gaeHost.size() <= dev) g_gaeHost.resize(dev + 1);
    GaeHostStage& h = g_gaeHost[dev];
    if (!h.stream && cudaStreamCreateWithFlags(&h.stream, cudaStreamNonBlocking) != cudaSuccess)
        return fail(RSB_ERR_CUDA, "stream creation failed");
    const size_t needT = (size_t)T + 1;
    if (h.capT < needT) {
        cudaFree(h.rews);
        cudaFree(h.vals);
        cudaFree(h.adv);
        cudaFree(h.tgt);
        cudaFree(h.ret);
        cudaFree(h.term);
        h.rews = h.vals = h.adv = h.tgt = h.ret = nullptr;
        h.term = nullptr;
        h.capT = 0;
        if (cudaMalloc(&h.rews, needT * 4) != cudaSuccess || cudaMalloc(&h.vals, needT * 4) != cudaSuccess ||
            cudaMalloc(&h.adv, needT * 4) != cudaSuccess || cudaMalloc(&h.tgt, needT * 4) != cudaSuccess ||
            cudaMalloc(&h.ret, needT * 4) != cudaSuccess || cudaMalloc(&h.term, needT) != cudaSuccess)
            return fail(RSB_ERR_NOMEM, "device allocation failed");
        h.capT = needT;
    }
    if (!h.clip && cudaMalloc(&h.clip, sizeof(float)) != cudaSuccess) return fail(RSB_ERR_NOMEM, "allocation failed");
    if (h.capTrunc < (size_t)num_truncs || !h.trunc) {
        cudaFree(h.trunc);
        h.trunc = nullptr;
        const size_t n = num_truncs > 0 ? (size_t)num_truncs : 1;
        if (cudaMalloc(&h.trunc, n * 4) != cudaSuccess) return fail(RSB_ERR_NOMEM, "device allocation failed");
        h.capTrunc = n;
    }
    cudaStream_t st = h.stream;
    const size_t nv = (size_t)(num_val_preds < T + 1 ? num_val_preds : T + 1);
    if (T > 0 && (cudaMemcpyAsync(h.rews, rews, (size_t)T * 4, cudaMemcpyHostToDevice, st) != cudaSuccess ||
                  cudaMemcpyAsync(h.term, terminals, (size_t)T, cudaMemcpyHostToDevice, st) != cudaSuccess ||
                  cudaMemcpyAsync(h.vals, val_preds, nv * 4, cudaMemcpyHostToDevice, st) != cudaSuccess))
        return fail(RSB_ERR_CUDA, "host to device copy failed");
    if (num_truncs > 0 &&
        cudaMemcpyAsync(h.trunc, trunc_val_preds, (size_t)num_truncs * 4, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return fail(RSB_ERR_CUDA, "host to device copy failed");
    rsb_status rc = launchGae(h.rews, h.term, h.vals, h.trunc, num_truncs, h.adv, h.tgt, h.ret, h.clip, T, *params, st);
    if (rc != RSB_OK) return fail(rc, "launch failed");
    if (T > 0 && (cudaMemcpyAsync(advantages, h.adv, (size_t)T * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                  cudaMemcpyAsync(target_values, h.tgt, (size_t)T * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                  cudaMemcpyAsync(returns, h.ret, (size_t)T * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess))
        return fail(RSB_ERR_CUDA, "device to host copy failed");
    if (cudaMemcpyAsync(rew_clip_portion, h.clip, sizeof(float), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return fail(RSB_ERR_CUDA, "device to host copy failed");
    return cudaStreamSynchronize(st) == cudaSuccess ? RSB_OK : fail(RSB_ERR_CUDA, "stream synchronize failed");
}

}  // extern "C"
