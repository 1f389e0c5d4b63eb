// What a plan has already encoded for the buffers it is called with, keyed by what went into it.  Host code without CUDA, so that
// its replacement order is tested without a device.
#pragma once

#include <cstdint>

namespace eider {
namespace gemm {

struct MapKey {
    const void* base;
    uint64_t rows, row_bytes, pitch;
    uint32_t box_rows;
    bool operator==(const MapKey& o) const {
        return base == o.base && rows == o.rows && row_bytes == o.row_bytes && pitch == o.pitch && box_rows == o.box_rows;
    }
};

// The last kMapEntries values in the order they were made, zero-initialized with the plan.  A plan is driven by one host thread (the
// reference's contract), so the cache is not locked.  A value stays where it is until kMapEntries others have been made: what
// one call needs of one buffer is one value, so that no lookup of a call can replace what an earlier one returned.
constexpr int kMapEntries = 8;
template <typename Value> struct FifoCache {
    struct Entry {
        MapKey key;
        Value value;
    };
    Entry entries[kMapEntries];
    uint32_t next;

    // `make(Value*)` -> status, 0 = made; a value that could not be made is not kept.
    template <typename Make> auto get(const Value** out, const MapKey& key, Make make) -> decltype(make(static_cast<Value*>(nullptr))) {
        using Status = decltype(make(static_cast<Value*>(nullptr)));
        for (Entry& e : entries) {
            if (e.key == key) {
                *out = &e.value;
                return Status{};
            }
        }
        Entry& e = entries[next % kMapEntries];
        e.key = MapKey{};
        const Status status = make(&e.value);
        if (status != Status{}) return status;
        e.key = key;
        ++next;
        *out = &e.value;
        return status;
    }
};

}  // namespace gemm
}  // namespace eider
