// How large results reach ordinary (pageable) host memory: through a ring of pinned slices that the copy engine fills and a few
// host threads empty into the caller's arrays, both while the GPU is still computing.  The driver's own copy into such memory does
// the two in turn on the calling thread (15 MB in 0.65 to 0.75 ms, 21 GB/s, of a call whose kernels take 0.48).  tg_batch, the driver's
// way and this: 2 MB of results 305 and 256 us, 6 MB 620 and 385, 15 MB 1290 and 600, 31 MB 2220 and 1080, 80 MB 13.3 and 4.2 ms, 345 MB 56 and
// 18.5 ms (from 32 MB on the C library maps an array afresh for every call, and the threads take its page faults).
//
// Making the ring takes 1.5 ms, giving it back 0.5, so that it is shared by a device's engines, belongs to those that have used it, and is made by the call that
// brings an engine's results to 32 MB, while that call's kernels run (made for every engine: second calls of 2 to 15 MB 1.0 -> 3.1 and
// 2.6 -> 4.2 ms).
#pragma once
#include "common.h"
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <sched.h>
#include <sys/mman.h>
#include <thread>
#include <unistd.h>

class ResultCopies {
  public:
    // A slice crosses in 10 us and a thread empties it in 50.  15 and 345 MB with 8 slices 720 us and 21.5 ms, 12 658 us and 18.5, 16 594 us and 18.4;
    // 24 and 32 of half the size 735 us and 20.1 ms, 680 us and 19.6.
    static constexpr size_t SliceBytes = size_t(1) << 19, Slices = 16;
    static constexpr int MostThreads = 4;
    static constexpr std::chrono::microseconds Patience{1000}; // without work; 300 is too short for evaluations of FP32 engines (500 -> 830 us after a pause), 3000 level
    static constexpr size_t Worth = size_t(32) << 20; // 40 us are saved for every megabyte

    struct Segment { // to[0, bytes) = from, device memory that is complete on `stream` after `ready` (null: after what `stream` holds)
        void *to;
        const void *from;
        size_t bytes;
        cudaStream_t stream;
        cudaEvent_t ready;
    };

    // Processors that the calling thread may run on (hardware_concurrency counts those it may not, too).
    static unsigned processors() {
        cpu_set_t set;
        return sched_getaffinity(0, sizeof(set), &set) == 0 ? unsigned(CPU_COUNT(&set)) : std::thread::hardware_concurrency(); // more than a set holds
    }
    // A quarter of them, or none: results then take the driver's way.
    static int threads_for(unsigned processors) { return int(processors / 4) < MostThreads ? int(processors / 4) : MostThreads; }

    ResultCopies() = default;
    ResultCopies(const ResultCopies &) = delete;
    ~ResultCopies() { destroy(); }

    // The ring of a device, which is the current one, for an engine whose results so far are `bytes`: made now where that is worth its time; null: results take
    // the driver's way.
    static std::shared_ptr<ResultCopies> of(int device, size_t bytes, int thread_count) {
        struct Entry {
            std::mutex mutex;
            std::weak_ptr<ResultCopies> ring;
            bool refused = false;
        };
        constexpr int Devices = 64;
        static Entry *const entries = new Entry[Devices]; // outlives every engine
        if (device < 0 || device >= Devices || thread_count < 1)
            return nullptr;
        Entry &entry = entries[device];
        std::unique_lock<std::mutex> lock(entry.mutex, std::try_to_lock);
        if (!lock) // another engine is making it
            return nullptr;
        if (std::shared_ptr<ResultCopies> ring = entry.ring.lock())
            return ring;
        if (entry.refused || bytes < Worth)
            return nullptr;
        // A forked child has the memory but not the threads: it leaves both alone, since nothing there would end a wait for them.
        std::shared_ptr<ResultCopies> ring(new ResultCopies, [owner = getpid()](ResultCopies *r) {
            if (getpid() == owner)
                delete r;
        });
        entry.refused = !ring->create(thread_count); // is not tried again
        if (entry.refused)
            return nullptr;
        entry.ring = ring;
        return ring;
    }
    // Ring, events and threads, or nothing.
    bool create(int thread_count) {
        bool made = make();
        try {
            while (made && int(threads.size()) < thread_count)
                threads.emplace_back([this] { work(); });
        } catch (const std::exception &) { // no thread, or no memory for one: those that run will do
        }
        made = !threads.empty();
        if (!made)
            destroy();
        return made;
    }
    void destroy() {
        {
            std::lock_guard<std::mutex> lock(mutex);
            stopping = true;
        }
        wake.notify_all();
        for (std::thread &t : threads)
            t.join();
        threads.clear();
        stopping = false;
        for (cudaEvent_t &e : landed) {
            if (e)
                cudaEventDestroy(e);
            e = nullptr;
        }
        if (pinned)
            cudaHostUnregister(ring);
        if (mapped)
            munmap(mapped, RingBytes + HugePage);
        ring = nullptr, mapped = nullptr, pinned = false;
    }

    // Has the kernel map pages before the copies into them need them.  Contents are left alone; where the call is not known, the copies take
    // the faults themselves.
    static void map_pages(void *to, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
        const uintptr_t page = uintptr_t(sysconf(_SC_PAGESIZE)), begin = (reinterpret_cast<uintptr_t>(to) + page - 1) / page * page,
                        end = (reinterpret_cast<uintptr_t>(to) + bytes) / page * page;
        if (begin < end)
            (void)madvise(reinterpret_cast<void *>(begin), end - begin, MADV_POPULATE_WRITE);
#endif
    }

    // Copies every segment, in order; returns when the last byte is in its place.  `map`: arrays whose pages the threads have the kernel map before
    // the first results arrive.  False: another engine's call has the ring, and nothing was done.
    bool run(const Segment *segments, size_t count, const Segment *map, size_t map_count) {
        std::unique_lock<std::mutex> lease(busy, std::try_to_lock);
        if (!lease)
            return false;
        try {
            copy(segments, count, map, map_count);
        } catch (...) { // nothing may be on its way into the ring when the next call uses it
            for (size_t i = 0; i < count; ++i)
                (void)cudaStreamSynchronize(segments[i].stream);
            throw;
        }
        return true;
    }

  private:
    // Huge pages, where there are any, are mapped and pinned in 1 ms; cudaHostAlloc takes 3.5 to 4.5 for eight megabytes.  Mapped here and not by the C library,
    // which when it got such a block back might give away the memory that it keeps for the caller's arrays.
    bool make() {
        void *memory = mmap(nullptr, RingBytes + HugePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        if (memory == MAP_FAILED)
            return false;
        mapped = memory;
        ring = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(mapped) + HugePage - 1) / HugePage * HugePage);
        (void)madvise(ring, RingBytes, MADV_HUGEPAGE);
        bool made = pinned = cudaHostRegister(ring, RingBytes, cudaHostRegisterDefault) == cudaSuccess;
        for (size_t i = 0; made && i < Slices; ++i)
            if (cudaEventCreateWithFlags(&landed[i], cudaEventDisableTiming) != cudaSuccess)
                landed[i] = nullptr, made = false;
        if (!made)
            (void)cudaGetLastError();
        return made;
    }
    void copy(const Segment *segments, size_t count, const Segment *map, size_t map_count) {
        size_t slices = 0;
        for (size_t i = 0; i < count; ++i)
            slices += (segments[i].bytes + SliceBytes - 1) / SliceBytes;
        size_t total = slices;
        for (size_t i = 0; i < map_count; ++i)
            total += (map[i].bytes + MapBytes - 1) / MapBytes;
        if (total > capacity)
            jobs.reset(new Job[total]), capacity = total;
        next.store(0, std::memory_order_relaxed);
        published.store(0, std::memory_order_relaxed);
        struct Active { // the threads take jobs while this lives; all have left the array when it is gone
            ResultCopies &c;
            explicit Active(ResultCopies &copies) : c(copies) {
                {
                    std::lock_guard<std::mutex> lock(c.mutex);
                    c.active.store(true);
                    ++c.call;
                }
                c.wake.notify_all();
            }
            ~Active() {
                {
                    std::lock_guard<std::mutex> lock(c.mutex);
                    c.active.store(false);
                }
                while (c.inside.load(std::memory_order_acquire))
                    std::this_thread::yield();
            }
        } active_now(*this);
        size_t at = 0; // jobs made
        auto publish = [&](void *to, const void *from, size_t bytes) {
            jobs[at].to = to, jobs[at].from = from, jobs[at].bytes = bytes;
            jobs[at].done.store(false, std::memory_order_relaxed);
            published.store(++at); // before `asleep` is read, which a thread counts up before it looks for jobs the last time
            if (asleep.load()) {
                std::lock_guard<std::mutex> lock(mutex);
                wake.notify_one();
            }
        };
        for (size_t i = 0; i < map_count; ++i) // the end first, as gradients arrive
            for (size_t end = map[i].bytes; end;) {
                const size_t begin = (end - 1) / MapBytes * MapBytes;
                publish(static_cast<char *>(map[i].to) + begin, nullptr, end - begin);
                end = begin;
            }
        // `issued` slices are on their way into the ring, the first `taken` of them have been handed to the threads.
        const size_t first_job = at;
        size_t issued = 0, taken = 0, segment = 0, offset = 0;
        struct {
            void *to;
            size_t bytes;
        } flying[Slices];
        while (taken < slices) {
            while (issued < slices && issued - taken < Slices &&
                   (issued < Slices || jobs[first_job + issued - Slices].done.load(std::memory_order_acquire))) {
                while (offset == segments[segment].bytes)
                    ++segment, offset = 0;
                const Segment &s = segments[segment];
                if (!offset && s.ready)
                    CHECK_CUDA(cudaStreamWaitEvent(s.stream, s.ready, 0));
                const size_t bytes = s.bytes - offset < SliceBytes ? s.bytes - offset : SliceBytes, slot = issued % Slices;
                CHECK_CUDA(cudaMemcpyAsync(ring + slot * SliceBytes, static_cast<const char *>(s.from) + offset, bytes, cudaMemcpyDeviceToHost, s.stream));
                CHECK_CUDA(cudaEventRecord(landed[slot], s.stream));
                flying[slot] = {static_cast<char *>(s.to) + offset, bytes};
                offset += bytes, ++issued;
            }
            if (taken == issued) { // every slice of the ring is still being emptied
                if (!take_one())
                    std::this_thread::yield();
                continue;
            }
            const size_t slot = taken % Slices;
            CHECK_CUDA(cudaEventSynchronize(landed[slot]));
            publish(flying[slot].to, ring + slot * SliceBytes, flying[slot].bytes);
            ++taken;
        }
        while (take_one())
            ;
        for (size_t i = 0; i < at; ++i)
            while (!jobs[i].done.load(std::memory_order_acquire))
                std::this_thread::yield();
    }

    static constexpr size_t MapBytes = size_t(4) << 20, RingBytes = SliceBytes * Slices, HugePage = size_t(2) << 20;
    struct Job { // a copy, or (from null) pages to be mapped
        void *to;
        const void *from;
        size_t bytes;
        std::atomic<bool> done;
    };
    void *mapped = nullptr;
    uint8_t *ring = nullptr;
    bool pinned = false;
    cudaEvent_t landed[Slices] = {};
    std::vector<std::thread> threads;
    std::unique_ptr<Job[]> jobs;
    size_t capacity = 0;
    std::atomic<size_t> next{0}, published{0};
    std::atomic<int> inside{0}, asleep{0};
    std::atomic<bool> active{false};
    std::mutex mutex, busy; // of the threads' state; for the length of a call
    std::condition_variable wake;
    bool stopping = false;
    unsigned call = 0;

    bool take_one() {
        size_t i = next.load(std::memory_order_relaxed);
        do
            if (i >= published.load(std::memory_order_acquire))
                return false;
        while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
        Job &job = jobs[i];
        if (job.from) {
            memcpy(job.to, job.from, job.bytes);
        } else {
            map_pages(job.to, job.bytes);
        }
        job.done.store(true, std::memory_order_release);
        return true;
    }
    // Awake from a call's beginning on, since waking takes 0.1 to 0.2 ms (woken for the first slice: 2 MB 270 -> 450 us a call), but a thread that finds nothing
    // to do for a while sleeps: polling through the kernels of a long call took four processors for all of it.
    void work() {
        std::unique_lock<std::mutex> lock(mutex);
        for (unsigned seen = 0;;) {
            ++asleep;
            wake.wait(lock, [&] { return stopping || (active.load() && (seen != call || next.load() < published.load())); });
            --asleep;
            if (stopping)
                return;
            seen = call;
            inside.fetch_add(1);
            lock.unlock();
            auto last = std::chrono::steady_clock::now();
            for (int idle = 0; active.load(std::memory_order_acquire);) {
                if (take_one()) {
                    idle = 0;
                } else if (++idle == 1) {
                    last = std::chrono::steady_clock::now();
                } else if (idle > 64) {
                    if (std::chrono::steady_clock::now() - last > Patience)
                        break;
                    std::this_thread::yield();
                }
            }
            inside.fetch_sub(1, std::memory_order_release);
            lock.lock();
        }
    }
};
