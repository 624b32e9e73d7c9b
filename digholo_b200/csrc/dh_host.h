// Host-side launch helpers shared by the kernel launchers: cached
// shared-memory attributes, SM counts and TMA tensor maps, so that a launch
// costs one cudaLaunchKernel and no driver queries.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "dh_params.h"

namespace dh {

inline std::mutex& hostCacheLock() {
    static std::mutex m;
    return m;
}

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize, and the maximal shared
// memory carveout) once per kernel, device and size (raised when a larger
// size is asked for).
inline cudaError_t setSmemOnce(const void* func, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    static std::map<std::pair<const void*, int>, int> done;
    std::lock_guard<std::mutex> g(hostCacheLock());
    auto it = done.find({func, dev});
    if (it != done.end() && it->second >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    // every kernel of the pipeline asks for the same L1 / shared split, so
    // consecutive launches need no reconfiguration of the SMs
    e = cudaFuncSetAttribute(func, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) done[{func, dev}] = bytes;
    return e;
}

// Multiprocessors of the current device.
inline int smCountCached() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    static std::map<int, int> counts;
    std::lock_guard<std::mutex> g(hostCacheLock());
    auto it = counts.find(dev);
    if (it != counts.end()) return it->second;
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n < 1) n = 1;
    counts[dev] = n;
    return n;
}

// A launch that, where `early`, may start its blocks before the kernel ahead of
// it in the stream has ended (the kernel waits by dependentWait).
template <typename... Par, typename... Arg>
inline cudaError_t launchDependent(void (*kern)(Par...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, bool early,
                                   const Arg&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Registers per thread of a kernel.
inline int regsCached(const void* func) {
    static std::map<const void*, int> regs;
    std::lock_guard<std::mutex> g(hostCacheLock());
    auto it = regs.find(func);
    if (it != regs.end()) return it->second;
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, func) != cudaSuccess) return 255;
    return regs[func] = a.numRegs;
}

// Blocks `b` that fit an SM beside n blocks `a` (sm_100: 2048 threads, 64 K
// registers in units of 8 per thread, 228 KB of shared memory with 1 KB a block).
inline int roomBeside(const DhFollower& a, int n, const DhFollower& b) {
    auto regs = [](const DhFollower& k) { return (k.threads + 31) / 32 * 32 * ((k.regs + 7) / 8 * 8); };
    const int byThreads = (2048 - n * a.threads) / b.threads, byRegs = (65536 - n * regs(a)) / regs(b);
    const int bySmem = (228 * 1024 - n * (a.smem + 1024)) / (b.smem + 1024);
    const int r = byThreads < byRegs ? byThreads : byRegs;
    return r < bySmem ? (r > 0 ? r : 0) : (bySmem > 0 ? bySmem : 0);
}

// Whether all small blocks `f` find room beside the blocks `own`, spread evenly:
// beside every SM's, or no more than two on each of the SMs that have any.
inline bool fitsBeside(const DhFollower& own, const DhFollower& f) {
    const int sms = smCountCached(), n = own.blocks / sms, more = own.blocks % sms;   // `more` SMs have n + 1
    const int r0 = roomBeside(own, n, f), r1 = more ? roomBeside(own, n + 1, f) : 0;
    const int places = (r0 > 0 ? sms - more : 0) + (r1 > 0 ? more : 0);
    return f.blocks <= (long long)(sms - more) * r0 + (long long)more * r1 && (places == sms || f.blocks <= 2 * places);
}

// Whether two kernels' small blocks may start together under the blocks `own`
// (averaging and the inverse behind it): each fits by itself, and the SMs that
// have room for them are all, or half of the GPU is free.  Frame averaging, 50
// items of two 640 x 512 uint16 frames, 32-pixel windows (100 forward blocks
// that leave no room): 32.3 us together, 28.9 without the attribute; four items
// of eight (32 blocks): 26.1 and 42.3, 29.6 with the inverse after.
inline bool bothFitBeside(const DhFollower& own, const DhFollower& a, const DhFollower& b) {
    if (a.blocks <= 0 || b.blocks <= 0 || !fitsBeside(own, a) || !fitsBeside(own, b)) return false;
    const int sms = smCountCached(), most = (own.blocks + sms - 1) / sms;
    return 2 * own.blocks <= sms || (roomBeside(own, most, a) > 0 && roomBeside(own, most, b) > 0);
}

// Whether a persistent forward kernel of blocks `own` (own.blocks launched, at
// most perSM on each SM) lets the kernel behind it start its blocks at once,
// instead of when its own blocks have ended:
// - where those blocks fill an SM each (k_field128): they go where forward
//   blocks end first, and nowhere else;
// - where they are small (low-resolution fields, averaging) and all fit beside
//   the forward blocks; or, when the forward blocks take several turns, in the
//   places of those that have no unit in a nearly empty last turn, no more than
//   two each; or when they are so many (twelve units per SM) that they take
//   several turns themselves.  Otherwise those that found room crowd there or on
//   the few free SMs, the others wait for them, and all end late.
// 640 x 512 frames, us without the attribute / at the blocks' ends / at once.
// uint16, 32-pixel windows (forward blocks that leave no room), one
// polarisation: 75 frames 21.5 / 20.1 / 19.6, 147 frames 22.0 / 20.1 / 31.8, 300
// frames 25.9 / 24.1 / 33.9; two: 500 frames 37.3 / 35.8 / 43.5, 1200 frames
// 74.2 / 73.2 / 70.4.  float, 32-pixel windows (room for three small blocks
// beside each forward block): 300 frames 27.6 / 25.2 / 23.6.  float, 16-pixel
// windows (296 forward blocks): 400 frames 17.9 / 17.4 / 19.9, 600 frames 23.4 /
// 21.5 / 19.9.
inline bool releasesEarly(const DhFwdParams& p, const DhFollower& own, int perSM) {
    if (p.wideFollower) return true;
    const DhFollower& f = p.follower;
    if (f.blocks <= 0) return false;
    if (fitsBeside(own, f) || p.followerUnits >= 12 * smCountCached()) return true;
    const int units = p.frameCount * p.polCount, last = units % own.blocks;
    const int freed = roomBeside(own, perSM - 1, f) - roomBeside(own, perSM, f);   // in one forward block's place
    return units > own.blocks && 8 * last <= own.blocks && freed <= 2 && f.blocks <= (long long)(own.blocks - last) * freed;
}

inline PFN_cuTensorMapEncodeTiled_v12000 tensorMapEncoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    });
    return fn;
}

// 2-D tiled tensor map over a batch of frames ([rows][width] elements,
// 128-byte swizzle, 64-byte L2 promotion), cached by its arguments: the
// batch buffers a caller rotates through are encoded once each.  A window
// row starts on a 32-byte boundary inside a 128-byte line; with 64-byte
// promotion the DRAM reads equal the window bytes (measured 67.2 MB per
// 1024-frame launch against 100.8 MB without promotion).
inline bool frameTensorMap(CUtensorMap& out, const void* base, CUtensorMapDataType type, int elemBytes,
                           unsigned long long width, unsigned long long rows, unsigned boxX, unsigned boxY) {
    struct Key {
        const void* base;
        int type, es;
        unsigned long long width, rows;
        unsigned boxX, boxY;
        bool operator<(const Key& o) const { return memcmp(this, &o, sizeof(Key)) < 0; }
    };
    static std::map<Key, CUtensorMap> cache;
    Key k;
    memset(&k, 0, sizeof(k));
    k.base = base;
    k.type = (int)type;
    k.es = elemBytes;
    k.width = width;
    k.rows = rows;
    k.boxX = boxX;
    k.boxY = boxY;
    {
        std::lock_guard<std::mutex> g(hostCacheLock());
        auto it = cache.find(k);
        if (it != cache.end()) {
            out = it->second;
            return true;
        }
    }
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensorMapEncoder();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)width * elemBytes};
    const cuuint32_t box[2] = {boxX, boxY};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&out, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_64B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return false;
    std::lock_guard<std::mutex> g(hostCacheLock());
    if (cache.size() >= 64) cache.clear();
    cache[k] = out;
    return true;
}

}  // namespace dh
