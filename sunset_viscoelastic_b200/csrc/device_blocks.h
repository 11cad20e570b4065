// device_blocks.h -- the device memory of one handle, in blocks (host code, no CUDA in it).
//
// A set-up makes some 150 device arrays, and cudaMalloc and cudaFree take 0.36 and 0.30 ms each
// for 1 MB and for 128 MB alike (0.8 and 1.6 ms for 1.9 GB; up to a second where other processes
// keep the driver busy), so the handle takes its memory in blocks and cuts the arrays from them:
// first fit, freed neighbours joined.  A block is as large as what the handle holds already,
// between 4 and 64 MB; an array of 32 MB and more is a block of its own and is given back at
// once.  The smaller ones' blocks stay with the handle until it is destroyed, or until the device
// is out of memory: then the blocks that nothing is cut from go back first.  262,144 nodes at
// order 6, create to close: 135 -> 87 ms; 10,000 nodes at order 8: 30 -> 14 ms.
#pragma once

#include <algorithm>
#include <cstddef>
#include <iterator>
#include <map>
#include <vector>

namespace sunset {

class DeviceBlocks {
  public:
    static constexpr size_t kAlign = 256;
    static constexpr size_t kBlockMin = (size_t)4 << 20, kBlockMax = (size_t)64 << 20, kOwnBlock = (size_t)32 << 20;

    int (*acquire)(void **p, size_t bytes) = nullptr;  // 0 or an error code
    void (*release)(void *p) = nullptr;
    int error = 0;  // of the last acquire that failed

    // a 256-byte aligned piece, or null when there is no memory left
    void *take(size_t bytes) {
        bytes = (std::max(bytes, (size_t)1) + kAlign - 1) & ~(kAlign - 1);
        if (bytes < kOwnBlock) {
            if (char *q = cut(bytes)) return q;
            size_t held = 0;
            for (const Block &B : blocks_) held += B.size;
            if (add(std::max(bytes, std::min(kBlockMax, std::max(kBlockMin, held))))) return cut(bytes);
        }
        // memory is short: no more than asked for, then with the unused blocks given back, then
        // whatever range is left
        if (add(bytes)) return cut_last(bytes);
        if (give_back() > 0 && add(bytes)) return cut_last(bytes);
        return cut(bytes);
    }

    void give(void *p) {
        auto it = pieces_.find(p);
        if (it == pieces_.end()) return;
        const size_t bytes = it->second;
        pieces_.erase(it);
        for (size_t b = 0; b < blocks_.size(); b++) {
            Block &B = blocks_[b];
            if (p < B.base || p >= B.base + B.size) continue;
            if (bytes == B.size && bytes >= kOwnBlock) {
                release(B.base);
                blocks_.erase(blocks_.begin() + b);
                return;
            }
            size_t off = static_cast<char *>(p) - B.base, len = bytes;
            auto next = B.free.lower_bound(off);
            if (next != B.free.end() && off + len == next->first) {
                len += next->second;
                next = B.free.erase(next);
            }
            if (next != B.free.begin()) {
                auto prev = std::prev(next);
                if (prev->first + prev->second == off) {
                    prev->second += len;
                    return;
                }
            }
            B.free[off] = len;
            return;
        }
    }

    void clear() {
        for (Block &B : blocks_) release(B.base);
        blocks_.clear();
        pieces_.clear();
    }

  private:
    struct Block {
        char *base;
        size_t size;
        std::map<size_t, size_t> free;  // offset -> length
    };

    char *cut_from(Block &B, size_t bytes) {
        for (auto it = B.free.begin(); it != B.free.end(); ++it) {
            if (it->second < bytes) continue;
            const size_t off = it->first, len = it->second;
            B.free.erase(it);
            if (len > bytes) B.free[off + bytes] = len - bytes;
            pieces_[B.base + off] = bytes;
            return B.base + off;
        }
        return nullptr;
    }
    char *cut(size_t bytes) {
        for (Block &B : blocks_)
            if (char *q = cut_from(B, bytes)) return q;
        return nullptr;
    }
    char *cut_last(size_t bytes) { return cut_from(blocks_.back(), bytes); }

    bool add(size_t size) {
        void *q = nullptr;
        if (int e = acquire(&q, size)) {
            error = e;
            return false;
        }
        blocks_.push_back({static_cast<char *>(q), size, {{0, size}}});
        return true;
    }

    size_t give_back() {
        size_t n = 0;
        for (size_t b = blocks_.size(); b-- > 0;) {
            const Block &B = blocks_[b];
            if (B.free.size() != 1 || B.free.begin()->second != B.size) continue;
            release(B.base);
            blocks_.erase(blocks_.begin() + b);
            n++;
        }
        return n;
    }

    std::vector<Block> blocks_;
    std::map<void *, size_t> pieces_;
};

}  // namespace sunset
