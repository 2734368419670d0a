// The K-buffer of a pixel (HYBRID_BLEND, ALPHA_BLEND_FIRST_K): the K nearest core fragments seen so far.
//
// What it has to reproduce is the reference's insertion chain (hybrid_blend/kernels/inference.cuh:159-167)
//     for k: if (carried.depth < entry[k].depth) swap(carried, entry[k]);
// including which of several entries of EXACTLY equal depth comes first and which of them falls out of a full buffer.
// An entry is a depth and an 8-byte payload (alpha, word); the word is the Gaussian's index or its position in the tile's
// list, both ascending in the order in which fragments arrive.  The colour is not kept (COLOUR = false): it is read again from the
// Gaussian's outline record (in L1 or L2) for the entries that fall out and for the K that are composited, which leaves 12 bytes
// per entry and pixel in shared memory, and shared memory is what limits how many warps are resident.
//
// Both buffers announce the entry that the next insertion will push out (`last`), so that the caller can fetch what it needs of
// it long before it falls out; `replace` says whether the announced one is what fell out (it is, but for ties in depth).
// Exact copies of a Gaussian, which densification by cloning makes, are tied in depth at every pixel.
#pragma once

#include "common.cuh"

namespace htgs {

constexpr uint32_t kNoEntry = 0xffffffffu;      // payload word of an empty entry

// Which depths the keys of UnsortedCore can tell apart: see there.  `base` is passed to the kernel.
struct CoreKeyWindow { bool covers; int32_t base; };

constexpr int core_pos_bits(int K) { return K >= 32 ? 5 : K >= 16 ? 4 : K >= 8 ? 3 : 2; }

// Every fragment that reaches the buffer lies between the near and the far plane (Gaussians whose extent at the alpha
// threshold crosses one of them are culled: kernel_utils.cuh:110-116), so a window that starts a factor of two in front of the near plane and
// ends a factor of two behind the far plane holds all depths at full precision.
inline CoreKeyWindow core_key_window(int K, float near_plane, float far_plane) {
    int32_t near_bits, far_bits;
    __builtin_memcpy(&near_bits, &near_plane, 4);
    __builtin_memcpy(&far_bits, &far_plane, 4);
    const int binades = 1 << (9 - core_pos_bits(K));
    const int near_exp = near_bits >> 23, far_exp = far_bits >> 23;       // biased; negative for negative planes
    if (K < 4 || near_exp < 2 || far_exp < near_exp || far_exp >= 255) return {false, 0};
    const int lowest = near_exp - 1 < 255 - binades ? near_exp - 1 : 255 - binades;      // the largest key stays a finite float
    return {far_exp + 2 <= lowest + binades, int32_t(lowest) << 23};
}

// Entries stay where they were stored (shared memory, one column per thread); nothing is ever shifted.  Entry c has a 32-bit
// key, depth above position: the float's bits minus `base`, shifted up by log2 K bits, plus c.  Keys are distinct and ordered
// like the depths, the largest one names the entry that falls out next.  Keys are kept in rows of four (one 16-byte
// access) and registers hold the maximum of each row, so an insertion reads back one row: about 30 instructions whatever the
// K, where the chain takes 6 per level (K = 16: 96, K = 32: 192) and is run by the whole warp whenever one lane inserts.
template <int K, int THREADS, bool COLOUR>
struct UnsortedCore {
    static_assert(K >= 4, "rows of four keys");
    static constexpr int kPosBits = core_pos_bits(K), kRows = K / 4;
    static constexpr bool keeps_colour = COLOUR, unsorted = true;
    static constexpr size_t smem_bytes = size_t(K) * THREADS * (COLOUR ? 24 : 12);
    static constexpr uint32_t kEmpty = 0xffffffffu & ~uint32_t(K - 1);
    static constexpr int32_t kRelLimit = int32_t((1u << (32 - kPosBits)) - 2u);   // one below an empty entry

    uint32_t* keys;          // [kRows][THREADS][4]
    uint2* pay;              // [K][THREADS]
    float* rgb;              // COLOUR: [K][3][THREADS]
    int32_t base;
    uint32_t row_max[kRows];
    uint32_t kmax;
    uint32_t settled;        // depth key of the last depth whose entries have been put in order where they lie (settle_ties)
    float depth_limit;       // a fragment enters if it is nearer than this
    uint32_t order[K];       // after finish(): keys in ascending order

    __device__ __forceinline__ float decode(uint32_t key) const { return __int_as_float(int32_t(key >> kPosBits) + base); }

    __device__ __forceinline__ void init(unsigned char* smem, uint32_t tid, int32_t key_base) {
        keys = reinterpret_cast<uint32_t*>(smem) + 4 * tid;
        pay = reinterpret_cast<uint2*>(smem + size_t(K) * THREADS * 4) + tid;
        rgb = reinterpret_cast<float*>(smem + size_t(K) * THREADS * 12) + tid;
        base = key_base;
        #pragma unroll
        for (int q = 0; q < kRows; ++q) {
            *reinterpret_cast<uint4*>(keys + q * THREADS * 4) = make_uint4(kEmpty + 4 * q, kEmpty + 4 * q + 1, kEmpty + 4 * q + 2, kEmpty + 4 * q + 3);
            row_max[q] = kEmpty + 4 * q + 3;
        }
        #pragma unroll
        for (int c = 0; c < K; ++c) pay[c * THREADS] = make_uint2(0u, kNoEntry);
        if constexpr (COLOUR) {
            #pragma unroll
            for (int c = 0; c < 3 * K; ++c) rgb[c * THREADS] = 0.0f;
        }
        kmax = kEmpty + K - 1;
        settled = 0xffffffffu;               // no depth: depth keys have kPosBits fewer bits
        depth_limit = decode(kmax);
    }

    __device__ __forceinline__ float limit() const { return depth_limit; }

    // The entry that falls out next; false if it is an empty one.
    __device__ __forceinline__ bool last(uint2& payload) const {
        payload = pay[(kmax & uint32_t(K - 1)) * THREADS];
        return payload.y != kNoEntry;
    }

    // While there are empty entries nothing falls out, and the rows' maxima do not matter: a new entry takes the last empty place.
    __device__ __forceinline__ bool filling() const { return kmax >= kEmpty; }
    __device__ __forceinline__ void append(float depth, uint2 payload, float3& colour) {
        const uint32_t c = kmax & uint32_t(K - 1);
        pay[c * THREADS] = payload;
        if constexpr (COLOUR) swap_colour(c, colour);
        const int32_t rel = min(max(__float_as_int(depth) - base, 0), kRelLimit);
        keys[(c >> 2) * (THREADS * 4) + (c & 3u)] = uint32_t(rel) * uint32_t(K) + c;
        --kmax;
        if (c == 0) {
            #pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const uint4 row = *reinterpret_cast<const uint4*>(keys + i * (THREADS * 4));
                row_max[i] = max(__vimax3_u32(row.x, row.y, row.z), row.w);
            }
            kmax = row_max[0];
            #pragma unroll
            for (int i = 1; i < kRows; ++i) kmax = max(kmax, row_max[i]);
            depth_limit = decode(kmax);
        }
    }

    // One or the other; always the latter unless APPENDS.  `evicted` and `colour` of an empty entry are zero, as the caller set them in the beginning.
    template <bool APPENDS>
    __device__ __forceinline__ bool insert(float depth, uint2 payload, uint2& evicted, float3& colour) {
        if (!APPENDS || !filling()) return replace(depth, payload, evicted, colour);
        append(depth, payload, colour);
        if constexpr (COLOUR) { colour = make_float3(0.0f, 0.0f, 0.0f); evicted = make_uint2(0u, kNoEntry); }
        return true;
    }

    // Puts (depth, payload) in place of the last entry.  `evicted` holds the last entry's payload (from last()); if a tie in depth makes
    // another entry fall out, it receives that one's payload and the result is false.
    // COLOUR: `colour` is the new entry's on the way in and the evicted one's on the way out.
    __device__ __forceinline__ bool replace(float depth, uint2 payload, uint2& evicted, float3& colour) {
        const uint32_t old = kmax;
        const uint32_t c = old & uint32_t(K - 1), q = c >> 2;
        if constexpr (COLOUR) {
            evicted = pay[c * THREADS];
            swap_colour(c, colour);
        }
        pay[c * THREADS] = payload;
        uint32_t* row_ptr = keys + q * (THREADS * 4);
        const int32_t rel = min(max(__float_as_int(depth) - base, 0), kRelLimit);
        row_ptr[c & 3u] = uint32_t(rel) * uint32_t(K) + c;
        const uint4 row = *reinterpret_cast<const uint4*>(row_ptr);
        const uint32_t m = max(__vimax3_u32(row.x, row.y, row.z), row.w);
        #pragma unroll
        for (int i = 0; i < kRows; ++i) row_max[i] = (q == uint32_t(i)) ? m : row_max[i];
        uint32_t top = row_max[0];
        #pragma unroll
        for (int i = 1; i + 1 < kRows; i += 2) top = __vimax3_u32(top, row_max[i], row_max[i + 1]);
        if constexpr (kRows % 2 == 0) top = max(top, row_max[kRows - 1]);
        kmax = top;
        depth_limit = decode(top);
        if ((top ^ old) < uint32_t(K) && old < kEmpty && (old >> kPosBits) != settled) {
            // others of the depth stay: back into the slot with what was announced, and what the chain drops lies there afterwards
            settled = old >> kPosBits;
            const uint32_t announced = evicted.y;
            pay[c * THREADS] = evicted;
            if constexpr (COLOUR) swap_colour(c, colour);
            settle_ties(keys, pay, c, settled);
            if constexpr (COLOUR) swap_colour(c, colour);
            evicted = pay[c * THREADS];
            pay[c * THREADS] = payload;
            return evicted.y == announced;
        }
        return true;
    }

    // Sorts the keys (once per pixel) into `order` and puts entries of equal depth into the chain's order.
    __device__ __forceinline__ void finish() {
        #pragma unroll
        for (int q = 0; q < kRows; ++q) {
            const uint4 row = *reinterpret_cast<const uint4*>(keys + q * (THREADS * 4));
            order[4 * q] = row.x; order[4 * q + 1] = row.y; order[4 * q + 2] = row.z; order[4 * q + 3] = row.w;
        }
        #pragma unroll
        for (int k = 2; k <= K; k <<= 1) {
            #pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                #pragma unroll
                for (int i = 0; i < K; ++i) {
                    const int l = i ^ j;
                    if (l > i) {
                        const uint32_t lo = min(order[i], order[l]), hi = max(order[i], order[l]);
                        if ((i & k) == 0) { order[i] = lo; order[l] = hi; } else { order[i] = hi; order[l] = lo; }
                    }
                }
            }
        }
        bool tie = false;
        #pragma unroll
        for (int k = 0; k + 1 < K; ++k) tie |= (order[k] ^ order[k + 1]) < uint32_t(K) && order[k] < kEmpty;
        if (tie) order_ties(keys, pay, settled);
    }

    // After finish(): entry k from the front; false if there is none.
    __device__ __forceinline__ bool entry(int k, float& depth, uint2& payload) const {
        depth = decode(order[k]);
        payload = pay[(order[k] & uint32_t(K - 1)) * THREADS];
        return order[k] < kEmpty;
    }

private:
    __device__ __forceinline__ void swap_colour(uint32_t c, float3& colour) {
        float* at = rgb + c * (3 * THREADS);
        const float3 t = make_float3(at[0], at[THREADS], at[2 * THREADS]);
        at[0] = colour.x; at[THREADS] = colour.y; at[2 * THREADS] = colour.z;
        colour = t;
    }
    static __device__ __forceinline__ uint32_t key_at(const uint32_t* keys, uint32_t i) { return keys[(i >> 2) * (THREADS * 4) + (i & 3u)]; }

    static __device__ __forceinline__ uint32_t slot_key(const uint32_t* keys, uint32_t slot) { return keys[(slot >> 2) * (THREADS * 4) + (slot & 3u)]; }
    static __device__ __forceinline__ void exchange(uint2* pay, uint32_t a, uint32_t b) {
        const uint2 t = pay[a * THREADS];
        pay[a * THREADS] = pay[b * THREADS];
        pay[b * THREADS] = t;
        if constexpr (COLOUR) {
            float* rgb = reinterpret_cast<float*>(pay - threadIdx.x + K * THREADS) + threadIdx.x;
            #pragma unroll 1
            for (uint32_t i = 0; i < 3; ++i) {
                const float x = rgb[(3 * a + i) * THREADS];
                rgb[(3 * a + i) * THREADS] = rgb[(3 * b + i) * THREADS];
                rgb[(3 * b + i) * THREADS] = x;
            }
        }
    }

    // How the chain orders entries of exactly equal depth: a new one goes behind those that are there, and every later insertion in front
    // of them carries the first one past the others, to their end - or out of a full buffer, if no entry is farther.  Nothing nearer
    // than an entry falls out before it does, so the insertions in front are all still in the buffer, and as long as none of the tied
    // entries has fallen out their order can be replayed from the words, which ascend in the order of arrival.  That is done when the
    // first of them falls out (replace) or at the end (finish).  Once one has fallen out the order of the others is fixed: the depth is the
    // buffer's limit, so nothing is added to it, and every insertion takes away the first.

    // Exchanges the payloads of the entries of depth `depth_key` so that descending slots hold them in the chain's order, which is the order
    // in which their keys make them fall out.  Slot c counts as one of them, whatever its key (K: there is no such slot).
    static __device__ __noinline__ void settle_ties(const uint32_t* keys, uint2* pay, uint32_t c, uint32_t depth_key) {
        uint32_t words[K], n = 0;
        #pragma unroll 1
        for (uint32_t slot = 0; slot < uint32_t(K); ++slot) {         // in the order of arrival
            if (slot != c && (slot_key(keys, slot) >> kPosBits) != depth_key) continue;
            const uint32_t word = pay[slot * THREADS].y;
            uint32_t i = n++;
            #pragma unroll 1
            for (; i > 0 && words[i - 1] > word; --i) words[i] = words[i - 1];
            words[i] = word;
        }
        auto in_front_after = [&](uint32_t word) {                    // insertions in front of the depth since `word` arrived
            uint32_t count = 0;
            #pragma unroll 1
            for (uint32_t slot = 0; slot < uint32_t(K); ++slot)
                if (slot != c && (slot_key(keys, slot) >> kPosBits) < depth_key && pay[slot * THREADS].y > word) ++count;
            return count;
        };
        #pragma unroll 1
        for (uint32_t size = 2; size <= n; ++size) {                  // the first `size` that arrived, in the chain's order until the next one arrives
            uint32_t turns = in_front_after(words[size - 1]);
            if (size < n) turns -= in_front_after(words[size]);
            #pragma unroll 1
            for (turns %= size; turns > 0; --turns) {
                const uint32_t first = words[0];
                #pragma unroll 1
                for (uint32_t i = 1; i < size; ++i) words[i - 1] = words[i];
                words[size - 1] = first;
            }
        }
        uint32_t place = 0;
        #pragma unroll 1
        for (uint32_t slot = K; slot-- > 0 && place < n;) {
            if (slot != c && (slot_key(keys, slot) >> kPosBits) != depth_key) continue;
            const uint32_t word = words[place++];
            uint32_t other = slot;
            #pragma unroll 1
            while (other > 0 && pay[other * THREADS].y != word) --other;
            if (other != slot) exchange(pay, slot, other);
        }
    }

    // At the end: payloads of equal depth in the chain's order by ascending slot, as keys in ascending order name them.
    static __device__ __noinline__ void order_ties(const uint32_t* keys, uint2* pay, uint32_t settled) {
        #pragma unroll 1
        for (uint32_t first = 0; first < uint32_t(K); ++first) {
            const uint32_t key = slot_key(keys, first), depth_key = key >> kPosBits;
            if (key >= kEmpty) continue;
            uint32_t low = first, high = K;
            auto tied = [&](uint32_t slot) { return (slot_key(keys, slot) >> kPosBits) == depth_key; };
            bool seen = false;
            #pragma unroll 1
            for (uint32_t slot = 0; slot < first; ++slot) seen |= tied(slot);
            if (seen) continue;
            if (depth_key != settled) settle_ties(keys, pay, K, depth_key);
            #pragma unroll 1
            for (;;) {                                                // reverses them
                #pragma unroll 1
                do --high; while (high > low && !tied(high));
                if (high <= low) break;
                exchange(pay, low, high);
                #pragma unroll 1
                do ++low; while (low < high && !tied(low));
                if (low >= high) break;
            }
        }
    }
};

// The chain itself, on (depth, slot) pairs in registers; payloads in a shared-memory pool of K + 1 slots, one of them free.
// Serves K < 4, where it is shorter than a row update, and depth ranges that the keys above do not cover.
// Because kd is sorted, the DEPTH carried into level k is always max(depth, kd[k-1]) - with or without ties - so every level's
// comparison and new depth are computed from the old buffer in parallel; only the slot is passed from level to level.  Slot
// numbers travel as floats (0..K are exact): one add and two multiply-adds per level on the FMA pipes.
template <int K, int THREADS>
struct SortedCore {
    static constexpr bool keeps_colour = false, unsorted = false;
    static constexpr size_t smem_bytes = size_t(K + 1) * THREADS * 8;
    uint2* pay;              // [K + 1][THREADS]
    float kd[K];
    float ks[K];
    uint32_t free_slot;

    static __device__ __forceinline__ float less_than_as_float(float a, float b) {
        float r;
        asm("set.lt.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        return r;
    }
    __device__ __forceinline__ void init(unsigned char* smem, uint32_t tid, int32_t) {
        pay = reinterpret_cast<uint2*>(smem) + tid;
        #pragma unroll
        for (int k = 0; k < K; ++k) { kd[k] = FLT_MAX; ks[k] = float(k); pay[k * THREADS] = make_uint2(0u, kNoEntry); }
        free_slot = K;
    }
    __device__ __forceinline__ float limit() const { return kd[K - 1]; }
    __device__ __forceinline__ bool last(uint2& payload) const {
        if (kd[K - 1] == FLT_MAX) return false;
        payload = pay[uint32_t(__float2int_rz(ks[K - 1])) * THREADS];
        return true;
    }
    __device__ __forceinline__ bool replace(float depth, uint2 payload, uint2& evicted, float3&) {
        const float announced = ks[K - 1];
        pay[free_slot * THREADS] = payload;
        float slot = float(free_slot);
        float p[K], nd[K];
        #pragma unroll
        for (int k = 0; k < K; ++k) {
            const float carried = k == 0 ? depth : fmaxf(depth, kd[k - 1]);
            p[k] = less_than_as_float(carried, kd[k]);
            nd[k] = fminf(carried, kd[k]);   // = carried where carried < kd[k], else kd[k]
        }
        #pragma unroll
        for (int k = 0; k < K; ++k) {
            const float mine = ks[k];
            const float t = slot - mine;
            ks[k] = fmaf(t, p[k], mine);      // p ? slot : mine
            slot = fmaf(-t, p[k], slot);      // p ? mine : slot
            kd[k] = nd[k];
        }
        free_slot = uint32_t(__float2int_rz(slot));
        if (slot == announced) return true;
        evicted = pay[free_slot * THREADS];
        return evicted.y == kNoEntry;         // empty entries are all alike
    }
    __device__ __forceinline__ void finish() {}
    __device__ __forceinline__ bool entry(int k, float& depth, uint2& payload) const {
        depth = kd[k];
        payload = pay[uint32_t(__float2int_rz(ks[k])) * THREADS];
        return payload.y != kNoEntry;
    }
};

}  // namespace htgs
