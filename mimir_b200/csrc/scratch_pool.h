// Cached scratch buffers, one per stream that has asked for one, and the right to use one for the length of a call. Host code only.
//
// A call that keeps intermediate results in such a buffer fills it by one launch and reads it by another. Calls on one stream are ordered by
// it, but only launch by launch: were the buffer free between two launches of a call, another host thread's call on the same stream could
// fill it again in between, or grow it and free the memory that the first call's launches name. So a buffer belongs to one call from
// `acquire` to `release`, and a second call on the stream waits for it; calls on other streams do not.
#pragma once

#include <condition_variable>
#include <cstddef>
#include <mutex>

namespace mimk {

// Memory: alloc(void**, size_t), free(void*) and wait(), which returns when no queued work uses any buffer; all give 0 if they succeed.
template <class Memory, int SLOTS>
class ScratchPool {
  public:
    struct Slot {
        void* stream = nullptr;
        void* ptr    = nullptr;
        size_t bytes = 0;
        unsigned long long last_use = 0;
        bool used = false, busy = false;  // it belongs to `stream`; a call has it
    };

    // A buffer of at least `bytes` for the calling thread's call on `stream`, until `release`. The stream's own one, grown if need be (they never
    // shrink); a new one while there are slots; else the one used longest ago that no call has, after a wait for its stream's work.
    int acquire(size_t bytes, void* stream, Slot** out) {
        std::unique_lock<std::mutex> lock(mutex_);
        Slot* e = nullptr;
        while (!(e = choose(stream))) released_.wait(lock);
        const bool mine = e->used && e->stream == stream;
        e->used = e->busy = true, e->stream = stream, e->last_use = ++clock_;
        lock.unlock();  // (what follows may wait for the device; nobody else touches a busy slot)
        int status = 0;
        if (e->ptr && (!mine || e->bytes < bytes)) {
            status = Memory::wait();
            if (!status) status = Memory::free(e->ptr);
            if (!status) e->ptr = nullptr, e->bytes = 0;
        }
        if (!status && e->bytes < bytes) {
            const size_t want = (bytes + (size_t(1) << 20) - 1) & ~((size_t(1) << 20) - 1);
            status            = Memory::alloc(&e->ptr, want);
            if (status) e->ptr = nullptr;
            else e->bytes = want;
        }
        if (status) {
            lock.lock();
            if (!mine) e->used = false;  // (a buffer that is still there is freed before the slot's next use)
            lock.unlock();
            release(e);
            return status;
        }
        *out = e;
        return 0;
    }

    void release(Slot* e) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            e->busy = false;
        }
        released_.notify_all();
    }

  private:
    // null: wait for a release
    Slot* choose(void* stream) {
        Slot *empty = nullptr, *oldest = nullptr;
        for (Slot& s : slots_) {
            if (s.used && s.stream == stream) return s.busy ? nullptr : &s;
            if (s.busy) continue;
            if (!s.used) empty = empty ? empty : &s;
            else if (!oldest || s.last_use < oldest->last_use) oldest = &s;
        }
        return empty ? empty : oldest;
    }

    std::mutex mutex_;
    std::condition_variable released_;
    Slot slots_[SLOTS];
    unsigned long long clock_ = 0;
};

}  // namespace mimk
