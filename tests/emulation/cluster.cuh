// Host stand-in for cluster.cuh: one cluster, whose halo copies can be made as late as
// the kernel's own synchronisation allows.  A copy reads its source when it is delivered.
// What the kernel must never do is counted: arming a barrier whose phase still waits,
// and a copy from or into the memory of a block that has ended.
#pragma once
#include <cuda_runtime.h>

#include <chrono>
#include <cstdio>
#include <functional>
#include <list>
#include <map>
#include <mutex>
#include <thread>

struct HostBarrier {
    int phase = 0, arrived = 0;
    long pending = 0;
    void check() {
        if (arrived == 1 && pending == 0) {
            phase ^= 1;
            arrived = 0;
        }
    }
};
struct HostCopy {
    int to, from;
    unsigned dst, src, bytes, bar;
    double due;
};
struct HostCluster {
    std::mutex lock;
    std::vector<HostBlock> blocks;
    std::vector<int> running;   // threads of a block that have not ended
    std::unique_ptr<std::barrier<>> meet;
    std::map<std::pair<int, unsigned>, HostBarrier> bars;
    std::list<HostCopy> copies;
    std::vector<int> received;                            // copies issued to a block so far
    std::function<double(int to, int index)> delay;       // seconds; negative: never comes
    int faults = 0;
    void fault(const char* what) {
        if (faults++ < 5) std::printf("fault: %s\n", what);
    }
    void deliver(const HostCopy& c) {
        if (!running[c.to] || !running[c.from]) fault("a copy from or into a block that has ended");
        std::memcpy(blocks[c.to].smem + c.dst, blocks[c.from].smem + c.src, c.bytes);
        HostBarrier& b = bars[{c.to, c.bar}];
        b.pending -= c.bytes;
        b.check();
    }
};
inline HostCluster* cluster = nullptr;
inline double host_seconds() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}
// The kernel waits for a row for 4e9 clocks: two seconds.
inline long long clock64() { return (long long)(host_seconds() * 2e9); }

namespace tomo {

inline void cluster_arrive() {}
inline void cluster_wait() { cluster->meet->arrive_and_wait(); }
inline unsigned cluster_rank() { return blockIdx.x; }
inline unsigned cluster_blocks() { return (unsigned)cluster->blocks.size(); }
inline unsigned smem_addr(const void* p) { return (unsigned)((const unsigned char*)p - this_block->smem); }
inline unsigned remote_addr(unsigned local, unsigned rank) { return rank << 20 | local; }
inline int* remote_word(unsigned addr) { return (int*)(cluster->blocks[addr >> 20].smem + (addr & 0xfffff)); }
inline void remote_store(unsigned addr, int v) { __atomic_store_n(remote_word(addr), v, __ATOMIC_RELEASE); }
inline int remote_load(unsigned addr) { return __atomic_load_n(remote_word(addr), __ATOMIC_ACQUIRE); }
inline void mbar_init(unsigned bar) {
    std::lock_guard<std::mutex> g(cluster->lock);
    cluster->bars[{blockIdx.x, bar}] = HostBarrier{};
}
inline void mbar_arm(unsigned bar, unsigned bytes) {
    std::lock_guard<std::mutex> g(cluster->lock);
    HostBarrier& b = cluster->bars[{blockIdx.x, bar}];
    if (b.arrived) return cluster->fault("a barrier armed twice in a phase");
    b.arrived = 1;
    b.pending += bytes;
    b.check();
}
inline bool mbar_try(unsigned bar, unsigned parity) {
    {
        std::lock_guard<std::mutex> g(cluster->lock);
        for (auto c = cluster->copies.begin(); c != cluster->copies.end();)
            if (c->to == blockIdx.x && c->due <= host_seconds()) {
                cluster->deliver(*c);
                c = cluster->copies.erase(c);
            } else {
                ++c;
            }
        if (cluster->bars[{blockIdx.x, bar}].phase != (int)parity) return true;
    }
    std::this_thread::sleep_for(std::chrono::microseconds(50));
    return false;
}
inline void proxy_fence() {}
inline void copy_row(unsigned dst, unsigned src, unsigned bytes, unsigned bar) {
    std::lock_guard<std::mutex> g(cluster->lock);
    HostCopy c{(int)(dst >> 20), blockIdx.x, dst & 0xfffff, src, bytes, bar & 0xfffff, 0};
    const double wait = cluster->delay ? cluster->delay(c.to, cluster->received[c.to]++) : 0;
    if (wait < 0) return;
    if (wait == 0) return cluster->deliver(c);
    c.due = host_seconds() + wait;
    cluster->copies.push_back(c);
}
constexpr long long kHaloClocks = 4000000000ll;
inline bool mbar_wait(unsigned bar, unsigned parity, const volatile int* lost) {
    if (mbar_try(bar, parity)) return true;
    const long long start = clock64();
    while (clock64() - start < kHaloClocks && !(lost && *lost))
        if (mbar_try(bar, parity)) return true;
    return false;
}
template <typename T>
T* shared_at(size_t offset) {
    return reinterpret_cast<T*>(this_block->smem + offset);
}

}  // namespace tomo
