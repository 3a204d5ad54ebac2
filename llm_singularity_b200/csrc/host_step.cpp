// Packing a step's metadata on the host: one pass over the entries writes, into one pinned buffer,
// everything the kernels read about the batch, so that one copy brings it to the device.
//
// The reference builds these arrays per request inside its forward pass and copies each on its own
// (models/llama/llama_model.cpp:560-615: positions, the block table row and the lengths of one
// request at a time).  Here a step has many requests with any number of tokens each.
#include <cstdint>

#define LSB_API extern "C" __attribute__((visibility("default")))

// Layout of `out`, in this order: token ids [T], positions [T], the entry of every token [T],
// q_start [R + 1], kv_len [R], block-table rows [R], wanted rows [W].  `offsets` gets the seven
// starts and the end (8 values), `summary` the total T, W, the longest entry and the longest
// sequence.  `tokens` are the entries' tokens one after another; `wants` the wanted places of the
// entries one after another, `want_count[r]` of them for entry r.
// Returns the number of ints written; -1 if `cap` is too small; -(r + 2) if entry r has no tokens
// or wants a place outside its tokens.
LSB_API long long lsbh_pack_step(int R, const int32_t* q_len, const int32_t* starts, const int32_t* rows,
                                 const int32_t* tokens, const int32_t* want_count, const int32_t* wants,
                                 int32_t* out, long long cap, long long* offsets, long long* summary) {
    long long T = 0, W = 0;
    int max_q = 0;
    long long max_kv = 0;
    for (int r = 0; r < R; ++r) {
        if (q_len[r] <= 0) return -(long long)(r + 2);
        T += q_len[r];
        W += want_count[r];
        if (q_len[r] > max_q) max_q = q_len[r];
        const long long kv = (long long)starts[r] + q_len[r];
        if (kv > max_kv) max_kv = kv;
    }
    const long long n = 3 * T + (R + 1) + 2 * (long long)R + W;
    if (n > cap) return -1;
    int32_t* tok = out;
    int32_t* pos = tok + T;
    int32_t* req = pos + T;
    int32_t* q_start = req + T;
    int32_t* kv_len = q_start + R + 1;
    int32_t* row = kv_len + R;
    int32_t* want = row + R;
    long long t = 0, w = 0;
    for (int r = 0; r < R; ++r) {
        q_start[r] = (int32_t)t;
        kv_len[r] = starts[r] + q_len[r];
        row[r] = rows[r];
        for (int i = 0; i < q_len[r]; ++i, ++t) {
            tok[t] = tokens[t];
            pos[t] = starts[r] + i;
            req[t] = r;
        }
        for (int i = 0; i < want_count[r]; ++i, ++w) {
            const int32_t place = wants[w];
            if (place < 0 || place >= q_len[r]) return -(long long)(r + 2);
            want[w] = q_start[r] + place;
        }
    }
    q_start[R] = (int32_t)t;
    offsets[0] = 0;
    offsets[1] = T;
    offsets[2] = 2 * T;
    offsets[3] = 3 * T;
    offsets[4] = offsets[3] + R + 1;
    offsets[5] = offsets[4] + R;
    offsets[6] = offsets[5] + R;
    offsets[7] = offsets[6] + W;
    summary[0] = T;
    summary[1] = W;
    summary[2] = max_q;
    summary[3] = max_kv;
    return n;
}

// A request's sampling settings as SamplingParams.packed lays them out.
struct SamplingRecord {
    double temperature, top_p, penalty;
    int64_t top_k;
    uint64_t seed;
};
static_assert(sizeof(SamplingRecord) == 40, "no padding");

// Per-row parameters of the sampling kernel: params[r] = {temperature, top_p, penalty, u}, top_k[r].  u is the request's
// draw number draws[r]: one splitmix64 scramble of seed + (draw + 1) * golden, its top 24 bits centred in their cell
// (0.5 for a greedy row).  Returns 1 if a row is not greedy, + 2 if one has a penalty; -(r + 1) if row r's top_k does
// not fit 32 bits.
LSB_API int lsbh_pack_sampling(int R, const void* records, const int64_t* draws, float* params, int32_t* top_k) {
    const SamplingRecord* rec = static_cast<const SamplingRecord*>(records);
    int flags = 0;
    for (int r = 0; r < R; ++r) {
        const SamplingRecord& p = rec[r];
        if (p.top_k != (int32_t)p.top_k) return -(r + 1);
        const bool greedy = p.temperature == 0.0;
        flags |= (greedy ? 0 : 1) | (p.penalty != 1.0 ? 2 : 0);
        uint64_t z = p.seed + ((uint64_t)draws[r] + 1u) * 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        params[4 * r] = (float)p.temperature;
        params[4 * r + 1] = (float)p.top_p;
        params[4 * r + 2] = (float)p.penalty;
        params[4 * r + 3] = greedy ? 0.5f : (float)(((double)(z >> 40) + 0.5) / (double)(1 << 24));
        top_k[r] = (int32_t)p.top_k;
    }
    return flags;
}
