// The unique-map's scratch and its stages, for callers that put the ids together and mark them in one kernel.
#pragma once
#include "common.cuh"

namespace ge2 {

constexpr int kScanThreads = 128;
constexpr int kWordsPerThread = 1;
constexpr int kTileWords = kScanThreads * kWordsPerThread;  // 128 words = 8192 ids per tile: a small domain still spreads over CTAs

struct UniqueWorkspace {
    uint32_t* tile_state;       // [num_tiles]   } control words: cleared together with the bitset by one memset
    uint32_t* ticket;           // [1]           }
    int32_t* status;            // [1]           } GE2_STATUS_* bits of this call
    unsigned long long* words;  // [num_words]  one bit per id that occurs   } cleared by the same memset
    unsigned long long* dup;    // [num_words]  ... that occurs again        } (null without out_shared)
    int32_t* word_offsets;      // [num_words]
    size_t clear_bytes;         // from tile_state on
};

constexpr int64_t kUniqueMaxIds = (1 << 30) - 1;  // a tile's packed state holds 30 bits

constexpr size_t align256c(size_t x) { return (x + 255) & ~(size_t)255; }
// control words (tile states, ticket, status, one spare), one bitset or (for out_shared) two, per-word offsets
constexpr size_t unique_ws_bytes(int64_t domain, int bitsets) {
    const int64_t nw = (domain + 63) >> 6;
    const int64_t tiles = (nw + kTileWords - 1) / kTileWords;
    return align256c((size_t)(tiles + 4) * 4) + bitsets * align256c((size_t)nw * 8) + align256c((size_t)nw * 4);
}

__host__ __device__ inline int64_t num_words_of(int64_t domain) { return (domain + 63) >> 6; }

inline UniqueWorkspace unique_carve(void* workspace, int64_t domain, bool shared) {
    const int64_t nw = num_words_of(domain), tiles = ceil_div<int64_t>(nw, kTileWords);
    char* p = (char*)workspace;
    UniqueWorkspace ws;
    ws.tile_state = (uint32_t*)p;
    ws.ticket = ws.tile_state + tiles;
    ws.status = (int32_t*)(ws.tile_state + tiles + 1);
    p += align256c((size_t)(tiles + 4) * 4);
    ws.words = (unsigned long long*)p;
    p += align256c((size_t)nw * 8);
    ws.dup = nullptr;
    if (shared) {
        ws.dup = (unsigned long long*)p;
        p += align256c((size_t)nw * 8);
    }
    ws.word_offsets = (int32_t*)p;
    ws.clear_bytes = (size_t)((char*)(shared ? ws.dup : ws.words) - (char*)ws.tile_state) + (size_t)nw * 8;
    return ws;
}

// an id below the domain is marked (and, where that is asked for, marked again)
__device__ __forceinline__ void mark_id(unsigned long long* words, unsigned long long* dup, int64_t key) {
    const unsigned long long bit = 1ull << (key & 63);
    if (dup == nullptr) atomicOr(&words[key >> 6], bit);
    else if ((atomicOr(&words[key >> 6], bit) & bit) != 0ull) atomicOr(&dup[key >> 6], bit);
}

// what follows the marking: the distinct ids in ascending order, the rank of every input id; counters[0 ... num_counters) + 1.  On as many CTAs as `sms`
// SMs hold
int unique_emit(const UniqueWorkspace& ws, const int64_t* ids, int64_t n, int64_t domain, int64_t* out_unique, int64_t* out_inverse, int32_t* out_count,
                uint8_t* out_shared, uint64_t* counters, int num_counters, int sms, cudaStream_t stream);

}  // namespace ge2
