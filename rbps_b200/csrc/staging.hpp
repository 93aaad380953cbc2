// staging.hpp - page-locked blocks that pass from one batch to the next.
//
// Page-locking costs 2.5 ms and unlocking 0.4 ms whatever the size (4 KB to
// 1.7 MB measured), more than a step of a small batch, so a batch's block is
// kept when the batch ends: no more blocks than batches are alive, one at
// least and kKeep at most.  A block belongs to the context it was locked in
// and is gone with it: cudaDeviceReset unlocks the memory and leaves the
// pointer dangling, so a block is only handed out (or unlocked) while its
// device's context is still the same, by the context's id, and is forgotten
// otherwise.
//
// Api: static uint64_t context(), the id of the current device's context, or
// 0 where there is none to ask for (no block is then kept);
// static void *lock(size_t), null when it fails; static void unlock(void *).
// Callers have the block's device current.  No call throws.
#pragma once
#include <cstddef>
#include <cstdint>
#include <mutex>

namespace rbps_gpu
{
    struct StagingBlock
    {
        void *p = nullptr;
        int device = 0;
        uint64_t context = 0;
    };

    template <class Api>
    class StagingPool
    {
    public:
        static constexpr int kKeep = 8;

        explicit StagingPool(size_t bytes) : bytes_(bytes) {}

        void begin()
        {
            std::lock_guard<std::mutex> lock(m_);
            ++live_;
        }

        // A block for `device`; p is null when none can be locked.
        StagingBlock take(int device)
        {
            StagingBlock b;
            b.device = device;
            b.context = Api::context();
            {
                std::lock_guard<std::mutex> lock(m_);
                forget(device, b.context);
                for (int i = n_; i-- > 0;)
                    if (kept_[i].device == device)
                    {
                        b = kept_[i];
                        kept_[i] = kept_[--n_];
                        return b;
                    }
            }
            b.p = Api::lock(bytes_);
            return b;
        }

        // A batch ends, with the block it held (or none).
        void end(const StagingBlock &b)
        {
            const uint64_t now = Api::context();
            std::lock_guard<std::mutex> lock(m_);
            --live_;
            forget(b.device, now);
            const int limit = live_ < 1 ? 1 : live_ < kKeep ? live_ : kKeep;
            if (b.p && b.context == now)
            {
                if (now && n_ < limit)
                    kept_[n_++] = b;
                else
                    Api::unlock(b.p);
            }
            for (int i = n_; i-- > 0 && n_ > limit;)
                if (kept_[i].device == b.device)
                {
                    Api::unlock(kept_[i].p);
                    kept_[i] = kept_[--n_];
                }
        }

        int kept()
        {
            std::lock_guard<std::mutex> lock(m_);
            return n_;
        }

    private:
        // the device's blocks of an earlier context
        void forget(int device, uint64_t now)
        {
            for (int i = n_; i-- > 0;)
                if (kept_[i].device == device && kept_[i].context != now)
                    kept_[i] = kept_[--n_];
        }

        std::mutex m_;
        size_t bytes_;
        StagingBlock kept_[kKeep];
        int n_ = 0, live_ = 0;
    };
} // namespace rbps_gpu
