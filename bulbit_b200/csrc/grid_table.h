// Grid sizes of persistent kernels, asked of the runtime once per kernel,
// launch shape and device: a fixed table, so that queries that promise to
// allocate nothing keep that promise and no exception can leave a C entry
// point. (A std::map in its place allocated in the first call of each kernel.)
#pragma once

#include <cstddef>
#include <cstdint>
#include <mutex>

namespace bbg
{

struct GridKey
{
    const void* kernel;
    size_t smem;
    int block;
    int device;

    bool operator==(const GridKey&) const = default;
};

class GridTable
{
public:
    // The grid stored for the key, or 0.
    int Find(const GridKey& key)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        const Entry* e = Slot(key);
        return e && e->grid > 0 ? e->grid : 0;
    }
    // Stores a grid (> 0). A full table stores nothing more: those kernels
    // are asked about again each time.
    void Store(const GridKey& key, int grid)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        if (Entry* e = Slot(key))
        {
            e->key = key;
            e->grid = grid;
        }
    }
    // The library has some 120 such kernels; eight devices' worth.
    static constexpr int kCapacity = 1024;

private:
    struct Entry
    {
        GridKey key;
        int grid; // 0: free
    };
    // The key's entry, else the free one where it belongs, else null (full).
    Entry* Slot(const GridKey& key)
    {
        uint64_t h = uint64_t(reinterpret_cast<uintptr_t>(key.kernel)) + 31 * key.smem + 131 * uint64_t(key.block) +
                     1031 * uint64_t(key.device);
        h *= 0x9e3779b97f4a7c15ull;
        for (int i = 0; i < kCapacity; ++i)
        {
            Entry& e = entries_[((h >> 40) + uint64_t(i)) % kCapacity];
            if (e.grid == 0 || e.key == key)
            {
                return &e;
            }
        }
        return nullptr;
    }
    std::mutex mutex_;
    Entry entries_[kCapacity] = {};
};

} // namespace bbg
