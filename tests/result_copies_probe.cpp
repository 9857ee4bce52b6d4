// Test probe (TEST INFRASTRUCTURE ONLY): csrc/result_copies.h over a fake of the CUDA runtime.  A copy is made when an event recorded after it is
// waited for, never earlier, so a slice that is emptied too soon, or filled again too soon, shows in the result.  The fake's n-th call fails on request.
#include "../turbogpt_b200/csrc/result_copies.h"
#include <cstdio>
#include <deque>
#include <map>

struct Copy {
    void *to;
    const void *from;
    size_t bytes;
};
static std::deque<Copy> queue;
static size_t made = 0, queued = 0;
static std::map<void *, size_t> recorded;
static int calls = 0, failing = 0, waits = 0, handles = 0;
static std::atomic<int> alive{0};
static bool fails() { return ++calls == failing; }
static void make(size_t until) {
    for (; made < until; ++made, queue.pop_front())
        memcpy(queue.front().to, queue.front().from, queue.front().bytes);
}
extern "C" {
cudaError_t cudaSetDevice(int) { return fails() ? cudaErrorInvalidDevice : cudaSuccess; }
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return fails() ? cudaErrorMemoryAllocation : (++alive, cudaSuccess); }
cudaError_t cudaHostUnregister(void *) { return --alive, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    if (fails())
        return cudaErrorMemoryAllocation;
    ++alive, *e = reinterpret_cast<cudaEvent_t>(uintptr_t(0x1000 + ++handles));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return --alive, cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    if (fails())
        return cudaErrorInvalidValue;
    queue.push_back({to, from, bytes}), ++queued;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return recorded[e] = queued, cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return make(recorded[e]), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return make(queued), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return ++waits, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
}

static bool ready(ResultCopies &c) { // once the ring has been made, or not
    while (c.making())
        std::this_thread::yield();
    return c.ready();
}

int main() {
    int wrong = 0;
    constexpr size_t Slice = ResultCopies::SliceBytes;
    const auto event = reinterpret_cast<cudaEvent_t>(uintptr_t(1));
    auto run = [&](ResultCopies &c, const std::vector<size_t> &sizes, unsigned seed, bool map) {
        std::vector<std::vector<uint8_t>> from, to;
        std::vector<ResultCopies::Segment> segments;
        for (size_t n : sizes) {
            from.emplace_back(n), to.emplace_back(n, uint8_t(0xee));
            for (size_t i = 0; i < n; ++i)
                from.back()[i] = uint8_t((seed = seed * 1664525u + 1013904223u) >> 24);
        }
        for (size_t i = 0; i < sizes.size(); ++i)
            segments.push_back({to[i].data(), from[i].data(), sizes[i], nullptr, i % 2 ? event : nullptr});
        c.run(segments.data(), segments.size(), segments.data(), map ? segments.size() : 0);
        wrong += from != to;
    };
    const std::vector<std::vector<size_t>> calls_of = {{1}, {Slice}, {Slice - 1, Slice + 1}, {0, 5, 0, 3 * Slice + 7},
                                                       {ResultCopies::Slices * Slice, 1}, {2 * ResultCopies::Slices * Slice + 13, Slice / 2, 40 * Slice + 1}};
    for (int threads = 1; threads <= ResultCopies::MostThreads; ++threads) {
        ResultCopies c;
        c.begin(threads, 0), c.begin(threads, 0);
        wrong += !ready(c) || !ready(c);
        for (int round = 0; round < 3; ++round)
            for (const auto &sizes : calls_of)
                run(c, sizes, unsigned(round * 7 + threads), round == 1);
        wrong += !queue.empty();
        for (int n : {1, 3, int(ResultCopies::Slices) + 5}) { // the n-th copy is refused: reported, and the next call is as ever
            calls = 0, failing = n;
            bool thrown = false;
            const int before = wrong;
            try {
                run(c, {30 * Slice}, 1, false);
            } catch (const std::exception &) {
                thrown = true;
            }
            wrong = before + !thrown + !queue.empty();
            failing = 0;
            run(c, {30 * Slice + 1, 17}, 2, false);
        }
    }
    for (int n = 1; n <= 2 + int(ResultCopies::Slices); ++n) { // the n-th creation is refused: nothing is left, and the next one serves
        ResultCopies c;
        calls = 0, failing = n;
        c.begin(2, 0);
        wrong += ready(c) || alive;
        failing = 0;
        c.begin(2, 0);
        wrong += !ready(c);
        run(c, {Slice + 3}, 5, false);
        c.destroy(), c.destroy();
        wrong += alive;
    }
    ResultCopies none;
    none.begin(0, 0);
    wrong += none.ready() || ResultCopies::threads_for(3) || ResultCopies::threads_for(4) != 1 || ResultCopies::threads_for(200) != ResultCopies::MostThreads;
    printf("wrong %d alive %d waits %d\n", wrong, alive.load(), waits > 0);
    return 0;
}
