// Test probe (TEST INFRASTRUCTURE ONLY): csrc/result_copies.h over a fake of the CUDA runtime.  A copy is made when an event recorded after it is
// waited for, never earlier, so a slice that is emptied too soon, or filled again too soon, shows in the result.  The fake's n-th call fails on request.
#include "../turbogpt_b200/csrc/result_copies.h"
#include <cstdio>
#include <ctime>
#include <deque>
#include <map>
#include <sys/wait.h>
#include <utility>

struct Copy {
    void *to;
    const void *from;
    size_t bytes;
};
static std::deque<Copy> queue;
static size_t made = 0, queued = 0;
static std::map<void *, size_t> recorded;
static int calls = 0, failing = 0, stall = 0, waits = 0, handles = 0;
static std::atomic<int> wrong_at_once{0};
static std::atomic<int> alive{0};
static bool fails() { return ++calls == failing; }
static void make(size_t until) {
    for (; made < until; ++made, queue.pop_front())
        memcpy(queue.front().to, queue.front().from, queue.front().bytes);
}
extern "C" {
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
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::this_thread::sleep_for(std::chrono::milliseconds(std::exchange(stall, 0)));
    return make(recorded[e]), cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return make(queued), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return ++waits, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
}

int main(int count, char **) {
    if (count > 1)
        return printf("%u\n", ResultCopies::processors()), 0;
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
        const bool done = c.run(segments.data(), segments.size(), segments.data(), map ? segments.size() : 0);
        wrong += done && from != to;
        return done;
    };
    const std::vector<std::vector<size_t>> calls_of = {{1}, {Slice}, {Slice - 1, Slice + 1}, {0, 5, 0, 3 * Slice + 7},
                                                       {ResultCopies::Slices * Slice, 1}, {2 * ResultCopies::Slices * Slice + 13, Slice / 2, 40 * Slice + 1}};
    for (int threads = 1; threads <= ResultCopies::MostThreads; ++threads) {
        ResultCopies c;
        wrong += !c.create(threads);
        for (int round = 0; round < 3; ++round)
            for (const auto &sizes : calls_of)
                wrong += !run(c, sizes, unsigned(round * 7 + threads), round == 1);
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
    for (int n = 1; n <= 1 + int(ResultCopies::Slices); ++n) { // the n-th creation is refused: nothing is left, and the next one serves
        ResultCopies c;
        calls = 0, failing = n;
        wrong += c.create(2) || alive;
        failing = 0;
        wrong += !c.create(2);
        run(c, {Slice + 3}, 5, false);
        c.destroy(), c.destroy();
        wrong += alive;
    }
    { // made when it is worth it, shared, given back with its last owner; a call that finds it in use does without
        const auto of = [](int device, size_t bytes) { return ResultCopies::of(device, bytes, 2); };
        wrong += of(3, ResultCopies::Worth - 1) || of(4, 1) || of(3, 1);
        auto a = of(3, ResultCopies::Worth), b = of(3, 0), other = of(4, ResultCopies::Worth + 1);
        wrong += !a || a != b || !other || other == a;
        std::atomic<int> refused{0}, done{0};
        std::vector<std::thread> engines;
        for (int i = 0; i < 4; ++i)
            engines.emplace_back([&, i, ring = of(3, 0)] {
                std::vector<uint8_t> from(3 * Slice + i, uint8_t(i + 1)), to(from.size());
                const ResultCopies::Segment segment{to.data(), from.data(), from.size(), nullptr, nullptr};
                for (int call = 0; call < 50; ++call) {
                    std::fill(to.begin(), to.end(), uint8_t(0));
                    const bool ran = ring->run(&segment, 1, nullptr, 0);
                    ++(ran ? done : refused);
                    wrong_at_once += ran ? from != to : to != std::vector<uint8_t>(to.size());
                }
            });
        for (std::thread &t : engines)
            t.join();
        wrong += wrong_at_once || done + refused != 200 || !done;
        a.reset();
        wrong += of(3, 0) != b;
        const pid_t child = fork();
        if (!child) { // has no threads to wait for
            alarm(20);
            b.reset(), other.reset();
            _exit(0);
        }
        int status = -1;
        wrong += waitpid(child, &status, 0) != child || status;
        b.reset(), other.reset();
        wrong += alive || of(3, ResultCopies::Worth - 1);
        calls = 0, failing = 1; // refused for good
        wrong += of(3, ResultCopies::Worth) || of(3, ResultCopies::Worth) || calls != 1;
        failing = 0;
    }
    { // the threads sleep while the GPU computes: processor time, of this process
        ResultCopies c;
        wrong += !c.create(4);
        run(c, {Slice}, 6, false);
        const std::clock_t begin = std::clock();
        stall = 400;
        wrong += !run(c, {4 * Slice}, 7, true);
        wrong += double(std::clock() - begin) / CLOCKS_PER_SEC > .2;
    }
    wrong += ResultCopies::of(5, ResultCopies::Worth, 0) || ResultCopies::of(-1, ResultCopies::Worth, 1) || alive;
    wrong += ResultCopies::threads_for(3) || ResultCopies::threads_for(4) != 1 || ResultCopies::threads_for(200) != ResultCopies::MostThreads;
    printf("wrong %d alive %d waits %d\n", wrong, alive.load(), waits > 0);
    return 0;
}
