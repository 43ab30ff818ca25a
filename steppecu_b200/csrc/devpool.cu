// steppecu_b200/csrc/devpool.cu
//
// The per-device store of released device blocks behind DevBuf (stpf2_internal.cuh).
#include <algorithm>
#include <mutex>

#include "stpf2_internal.cuh"

namespace stpf2 {

namespace {

struct Block {
    void* p;
    size_t bytes;
};
constexpr int kMaxDevices = 64;

struct Store {
    std::mutex mu;
    std::vector<Block> blocks[kMaxDevices];
    size_t held[kMaxDevices] = {};
    size_t limit[kMaxDevices] = {};  // of held, from the last look at the device's memory
    int contexts[kMaxDevices] = {};
};

// Never destroyed: buffers of objects that live to the end of the process come back late.
Store& store() {
    static Store* s = new Store;
    return *s;
}

bool known(int device) { return device >= 0 && device < kMaxDevices; }

// Under 1 MiB powers of two (few sizes, so tables of one call fit the next one's), above it
// whole 2 MiB pages.
size_t rounded(size_t n) {
    if (n > (size_t(1) << 20)) return (n + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);
    size_t r = 512;
    while (r < n) r *= 2;
    return r;
}

// The blocks released longest ago go until at most `bytes` are held: those of earlier calls of
// other sizes would otherwise fill the store and every later call allocate anew.
void trim(Store& s, int device, size_t bytes) {
    std::vector<Block>& v = s.blocks[device];
    size_t old = 0;
    while (s.held[device] > bytes) {
        s.held[device] -= v[old].bytes;
        cudaFree(v[old++].p);
    }
    v.erase(v.begin(), v.begin() + static_cast<std::ptrdiff_t>(old));
}

void empty(Store& s, int device) {
    for (const Block& b : s.blocks[device]) cudaFree(b.p);
    s.blocks[device].clear();
    s.held[device] = 0;
}

}  // namespace

void* pool_alloc(size_t& bytes, int& device) {
    STPF2_CUDA(cudaGetDevice(&device));
    bytes = rounded(bytes);
    Store& s = store();
    if (known(device)) {
        std::lock_guard<std::mutex> lock(s.mu);
        std::vector<Block>& v = s.blocks[device];
        size_t best = v.size();
        for (size_t k = 0; k < v.size(); ++k)  // the smallest that fits, and wastes at most a quarter
            if (v[k].bytes >= bytes && v[k].bytes <= bytes + bytes / 4 && (best == v.size() || v[k].bytes < v[best].bytes))
                best = k;
        if (best < v.size()) {
            void* p = v[best].p;
            bytes = v[best].bytes;
            s.held[device] -= bytes;
            v.erase(v.begin() + static_cast<std::ptrdiff_t>(best));  // the rest stay in order of their release
            return p;
        }
    }
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation && known(device)) {
        (void)cudaGetLastError();
        std::lock_guard<std::mutex> lock(s.mu);
        empty(s, device);
        e = cudaMalloc(&p, bytes);
    }
    cuda_check(e, "cudaMalloc");
    if (known(device)) {
        // The store holds blocks only while they are a small part of what the device has left
        // for others: what is held can only grow by a block that was allocated here, so this is
        // where to look (the query costs less than the allocation it follows).
        size_t free_b = 0, total = 0;
        if (cudaMemGetInfo(&free_b, &total) != cudaSuccess) {
            (void)cudaGetLastError();
            free_b = 0;
        }
        std::lock_guard<std::mutex> lock(s.mu);
        s.limit[device] = std::min(kPoolBytes, (free_b + s.held[device]) / kPoolShare);
        trim(s, device, s.limit[device]);
    }
    return p;
}

size_t pool_held(int device) {
    if (!known(device)) return 0;
    Store& s = store();
    std::lock_guard<std::mutex> lock(s.mu);
    return s.held[device];
}

void pool_free(void* p, size_t bytes, int device) noexcept {
    int cur = -1;
    // Work on the block may still run on any stream of the device: wait for it, as cudaFree
    // does. A failed wait (a lost context) leaves the block to cudaFree.
    if (known(device) && cudaGetDevice(&cur) == cudaSuccess && cur == device && bytes <= kPoolBytes / 2 &&
        cudaDeviceSynchronize() == cudaSuccess) {
        Store& s = store();
        std::lock_guard<std::mutex> lock(s.mu);
        const size_t limit = s.limit[device];
        if (s.contexts[device] > 0 && bytes <= limit / 2) {
            trim(s, device, limit - bytes);
            try {
                s.blocks[device].push_back(Block{p, bytes});
                s.held[device] += bytes;
                return;
            } catch (...) {
            }
        }
    }
    cudaFree(p);
}

void pool_open(int device) {
    if (!known(device)) return;
    Store& s = store();
    std::lock_guard<std::mutex> lock(s.mu);
    s.contexts[device]++;
}

void pool_close(int device) {
    if (!known(device)) return;
    Store& s = store();
    std::lock_guard<std::mutex> lock(s.mu);
    if (--s.contexts[device] == 0) empty(s, device);
}

}  // namespace stpf2
