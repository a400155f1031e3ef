// FLAC decoding of 16-bit mono RF captures (.ldf) on the GPU.
//
// The reference reads .ldf captures through libsndfile or ffmpeg
// (Core/Rf/LibsndfilePcm16SampleLoader.cs, Core/Rf/FfmpegPcm16SampleLoader.cs)
// and indexes their frames itself for seeking (Core/Rf/RawFlacFrameIndex.cs,
// Core/Rf/RawFlacStreamInfo.cs).  Here the decoding itself runs on the device,
// following the published format (IETF RFC 9639):
//
// * k_flac_sync scans every byte position of a chunk for a frame header
//   (the 14-bit sync code, valid field codes, a valid coded frame or sample
//   number and a matching CRC-8) and appends what it parsed;
// * the host sorts the candidates and chains them: a frame is accepted where
//   its number continues the stream's sequence, so a sync pattern inside
//   compressed data (which also needs a matching CRC-8) is skipped.  It looks
//   at no byte of the stream: parsing the headers again and sorting the frames
//   by a byte of each cost 2.1 ms of cache misses for 10,000 frames;
// * k_flac_frames decodes each frame with four lanes.  The residual is a
//   bit-serial Rice code and the prediction a recurrence, so a frame is
//   sequential work: what bounds it is the latency of a step, about 120
//   dependent instructions.  All four lanes read the residual (the same words
//   of the group's ring); the predictor runs in transposed form, its taps and
//   partial sums split over the lanes' registers, so a sample costs a lane
//   eight of the 32 multiply-adds at most, no history shifts and one
//   broadcast.  Frames are handed out sorted by subframe type so a warp's
//   eight run the same path.  It checks that the subframe ends where the next
//   frame begins and writes int16 samples (10,000 frames of 4096 samples 1.56
//   ms, 977 frames 1.1; with a thread a frame, history and CRC in it, 3.9 and
//   3.6);
// * k_flac_crc checks the frames' CRC-16, a warp per frame: each lane the
//   remainder of its 1/32 of the bytes, joined by multiplying with powers of x.
//
// Only what RF captures use is accepted: one channel of 16 bits per sample.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/vhsdecode_gb300.h"
#include "flac.hpp"
#include "session.hpp"

using namespace vhsd::detail;

namespace vhsd {

// A frame header k_flac_sync found.
struct FlacCand {
    int64_t at;
    uint64_t number;      // coded frame or (variable) sample number
    int32_t block;
    int16_t header_len;
    uint8_t type;         // subframe type bits of the byte after the header
    bool variable : 1;
    bool other : 1;       // not one channel of 16 bits
};

namespace {

__device__ __forceinline__ uint32_t bswap32(uint32_t v) { return __byte_perm(v, 0, 0x0123); }

constexpr int kGroup = 4;          // lanes of a frame
constexpr int kRing = 64;          // words of a frame's ring in shared memory
constexpr int kAhead = 16;         // words of it that a step outside the top-ups leaves
constexpr unsigned kWarp = 0xffffffffu;

// MSB-first bit reader over 32-bit big-endian words, by the four lanes of a
// group together.  Three words wait in registers, the first `bit` bits of the
// first consumed: the next 32 bits are one funnel shift and a step consumes at
// most 32.  The words behind them come from a ring in shared memory that the
// group tops up eight words at a time (two a lane, loaded from global memory
// one top-up before they enter the ring), at steps the whole warp takes
// together: a load of its own for every word made the warp wait for the
// latest load of any of its groups at every step.  A top-up every eight
// residual values, of a word at most each, keeps the ring ahead.  Loads never pass `limit`
// (words from the start): bits beyond it read as zero, and overrun() tells
// whether any were consumed.
struct BitReader {
    const uint32_t* w;      // the word the reader started in
    uint32_t* ring;
    int lane, limit;
    int next, filled;       // index of the word after w2; words in the ring
    int bit;                // 0 .. 31
    uint32_t w0, w1, w2;
    unsigned group;         // the group's lanes
    uint2 pending;          // this lane's words filled + 2 lane, + 1
    __device__ __forceinline__ uint32_t word(int i) const { return i < limit ? bswap32(__ldg(w + i)) : 0u; }
    __device__ __forceinline__ void load_pending() {
        pending = make_uint2(word(filled + 2 * lane), word(filled + 2 * lane + 1));
    }
    __device__ __forceinline__ void init(const uint32_t* words, int64_t byte_off, int64_t byte_limit, uint32_t* ring_,
                                         int lane_, unsigned group_) {
        w = words + (byte_off >> 2);
        limit = (int)(((byte_limit + 3) >> 2) - (byte_off >> 2));
        ring = ring_;
        lane = lane_;
        group = group_;
        seek(0, (int)(byte_off & 3) * 8);
    }
    __device__ __forceinline__ void push_pending() {
        *reinterpret_cast<uint2*>(ring + ((filled + 2 * lane) & (kRing - 1))) = pending;
        filled += 2 * kGroup;
        load_pending();
    }
    // the ring from word `next` on, at least kAhead words of it
    __device__ __forceinline__ void refill() {
        __syncwarp(group);
        filled = next & ~1;
        load_pending();
        push_pending();
        push_pending();
        push_pending();
        __syncwarp(group);
    }
    __device__ __forceinline__ void seek(int i, int bit_) {   // to bit `bit_` of word i
        bit = bit_;
        w0 = word(i);
        w1 = word(i + 1);
        w2 = word(i + 2);
        next = i + 3;
        refill();
    }
    // eight words more if there is room (by whole warps, at steps they take
    // together)
    __device__ __forceinline__ void top_up() {
        __syncwarp();
        if (filled - next <= kRing - 8) push_pending();
        __syncwarp();
    }
    __device__ __forceinline__ uint32_t top() const { return __funnelshift_l(w1, w0, bit); }
    // consumes 0 <= n <= 32 bits; the ring holds the next word
    __device__ __forceinline__ void skip_fast(int n) {
        bit += n;
        if (bit >= 32) {
            bit -= 32;
            w0 = w1;
            w1 = w2;
            w2 = ring[next & (kRing - 1)];
            next++;
        }
    }
    // the same from anywhere: leaves kAhead words in the ring
    __device__ __forceinline__ void skip(int n) {
        skip_fast(n);
        if (filled - next < kAhead) refill();
    }
    __device__ __forceinline__ uint32_t get(int n) {   // 0 <= n <= 32
        const uint32_t v = n == 0 ? 0u : top() >> (32 - n);
        skip(n);
        return v;
    }
    __device__ __forceinline__ int32_t sget(int n) {
        if (n == 0) return 0;
        const uint32_t v = get(n);
        return (int32_t)(v << (32 - n)) >> (32 - n);
    }
    // zeros before the next one bit (the bit is consumed); -1 past `cap` zeros
    __device__ __forceinline__ int32_t unary(int32_t cap) {
        int32_t q = 0;
        for (;;) {
            const uint32_t t = top();
            if (t) {
                const int z = __clz(t);
                skip(z + 1);
                q += z;
                return q <= cap ? q : -1;
            }
            skip(32);
            q += 32;
            if (q > cap || overrun()) return -1;
        }
    }
    // bits from the start of the reader's first word
    __device__ __forceinline__ int64_t bitpos() const { return (int64_t)(next - 3) * 32 + bit; }
    __device__ __forceinline__ bool overrun() const { return bitpos() > (int64_t)limit * 32; }
};

__device__ __forceinline__ bool utf8_number(const uint8_t* p, int64_t n, int64_t at, int& len, uint64_t& val) {
    if (at >= n) return false;
    uint8_t b0 = p[at];
    int extra;
    uint64_t v;
    if (b0 < 0x80) { extra = 0; v = b0; }
    else if ((b0 & 0xE0) == 0xC0) { extra = 1; v = b0 & 0x1F; }
    else if ((b0 & 0xF0) == 0xE0) { extra = 2; v = b0 & 0x0F; }
    else if ((b0 & 0xF8) == 0xF0) { extra = 3; v = b0 & 0x07; }
    else if ((b0 & 0xFC) == 0xF8) { extra = 4; v = b0 & 0x03; }
    else if ((b0 & 0xFE) == 0xFC) { extra = 5; v = b0 & 0x01; }
    else if (b0 == 0xFE) { extra = 6; v = 0; }
    else return false;
    if (at + extra >= n) return false;
    for (int i = 1; i <= extra; i++) {
        uint8_t b = p[at + i];
        if ((b & 0xC0) != 0x80) return false;
        v = (v << 6) | (b & 0x3F);
    }
    len = 1 + extra;
    val = v;
    return true;
}

__constant__ uint8_t c_crc8[256];
__constant__ uint16_t c_crc16[256];

// Frame header at byte `at` (RFC 9639 section 9.1): returns its length (0 if
// not a valid header), the coded number and the block size.
__device__ int parse_header(const uint8_t* p, int64_t n, int64_t at, uint64_t& number, int& block,
                            bool& variable) {
    if (at + 6 > n || p[at] != 0xFF || (p[at + 1] & 0xFE) != 0xF8) return 0;
    variable = p[at + 1] & 1;
    const int bcode = p[at + 2] >> 4, rcode = p[at + 2] & 15;
    const int chan = p[at + 3] >> 4, scode = (p[at + 3] >> 1) & 7, res = p[at + 3] & 1;
    if (bcode == 0 || rcode == 15 || chan > 10 || scode == 3 || res) return 0;
    int len = 0;
    uint64_t num = 0;
    if (!utf8_number(p, n, at + 4, len, num)) return 0;
    int64_t q = at + 4 + len;
    if (bcode == 6) {
        if (q + 1 > n) return 0;
        block = p[q] + 1;
        q += 1;
    } else if (bcode == 7) {
        if (q + 2 > n) return 0;
        block = ((p[q] << 8) | p[q + 1]) + 1;
        q += 2;
    } else if (bcode == 1) {
        block = 192;
    } else if (bcode <= 5) {
        block = 576 << (bcode - 2);
    } else {
        block = 256 << (bcode - 8);
    }
    if (rcode == 12) q += 1;
    else if (rcode == 13 || rcode == 14) q += 2;
    if (q + 1 > n) return 0;
    uint8_t c = 0;
    for (int64_t i = at; i < q; i++) c = c_crc8[c ^ p[i]];
    if (c != p[q]) return 0;
    number = num;
    return (int)(q + 1 - at);
}

// Candidate frame headers: one thread per byte position.
__global__ void k_flac_sync(const uint8_t* __restrict__ p, int64_t n, FlacCand* cand, int* count, int cap) {
    const int64_t at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (at + 1 >= n || p[at] != 0xFF || (p[at + 1] & 0xFE) != 0xF8) return;
    FlacCand c{};
    bool var;
    c.header_len = parse_header(p, n, at, c.number, c.block, var);
    if (!c.header_len) return;
    c.at = at;
    c.variable = var;
    c.other = (p[at + 3] >> 4) != 0 || ((p[at + 3] >> 1) & 7) != 4;
    c.type = p[at + c.header_len] & 0x7E;   // the buffer is padded
    const int k = atomicAdd(count, 1);
    if (k < cap) cand[k] = c;
}

// Residual of a subframe (RFC 9639 section 9.2.7), read one value at a time:
// partitions of Rice (4-bit parameters) or Rice2 (5-bit) codes, or escaped
// partitions of raw signed values.
struct Residual {
    int pbits, esc, porder, part, parts, left, k, width, order, block;
    bool escaped;
    __device__ __forceinline__ int init(BitReader& r, int block_, int order_) {
        block = block_;
        order = order_;
        const int method = (int)r.get(2);
        if (method > 1) return 1;
        pbits = method == 0 ? 4 : 5;
        esc = (1 << pbits) - 1;
        porder = (int)r.get(4);
        parts = 1 << porder;
        if ((block >> porder) < order || (block & (parts - 1))) return 2;
        part = -1;
        left = 0;
        return 0;
    }
    // next residual value; false on a malformed or overrunning stream
    __device__ __forceinline__ bool next(BitReader& r, int32_t& v) {
        while (left == 0) {
            if (++part >= parts) return false;
            left = (block >> porder) - (part == 0 ? order : 0);
            k = (int)r.get(pbits);
            escaped = k == esc;
            if (escaped) width = (int)r.get(5);
            if (r.overrun()) return false;
        }
        left--;
        if (escaped) {
            v = r.sget(width);
            return true;
        }
        const uint32_t top = r.top();
        const int z = __clz(top), len = z + 1 + k;
        uint32_t u;
        if (len <= 32) {
            // the whole code lies in the next 32 bits: z zeros, a one, k bits
            // (two shifts: k = 0 shifts everything out, z = 31 the one)
            u = (uint32_t)z << k | top << z << 1 >> 1 >> (31 - k);
            r.skip_fast(len);
        } else {
            const int32_t q = r.unary(1 << 20);
            if (q < 0) return false;
            u = ((uint32_t)q << k) | r.get(k);
        }
        v = (int32_t)(u >> 1) ^ -(int32_t)(u & 1);
        return true;
    }
};

// Output of one frame's samples by its four lanes: lane l keeps sample 4 m + l,
// and every fourth sample the group stores eight bytes side by side.
struct GroupOut {
    int16_t* o;   // this lane's next sample
    int i, lane;
    int16_t mine;
    __device__ __forceinline__ void init(int16_t* out, int lane_) {
        o = out + lane_;
        i = 0;
        lane = lane_;
        mine = 0;
    }
    __device__ __forceinline__ void put(int32_t x) {   // by every lane of the group
        if (i == lane) mine = (int16_t)x;
        i = (i + 1) & (kGroup - 1);
        if (i == 0) {
            *o = mine;
            o += kGroup;
        }
    }
    __device__ __forceinline__ void flush() {
        if (lane < i) *o = mine;
    }
};

// What a group knows of its predicted subframe (RFC 9639 sections 9.2.5,
// 9.2.6) before its samples.
struct Predicted {
    bool active;      // the frame has a predicted subframe and no error so far
    bool fixed;
    int order, block, bps, wasted;
};

// The samples of the predicted subframes of a warp's eight frames, of order
// <= 4 T, the group's lane l holding taps [T l, T l + T) in transposed form:
// s[t] is the sum, over the samples so far, of the products that the sample
// T l + t steps ahead will be predicted from (tap j of sample x goes into the
// sum of the sample j + 1 steps after it), accumulated in 64 bits.  The fixed
// predictors are the same with whole-number taps and no shift.  The whole warp
// takes every step together (a group that has ended or failed idles): with the
// groups on their own the shuffles of one group at a time ran the eight frames
// one after the other.  Returns the group's error.
template <int T>
__device__ __forceinline__ int predicted_samples(BitReader& r, Predicted f, int lane, GroupOut& o) {
    int err = 0;
    bool on = f.active;
    const int warm_word = r.next - 3, warm_bit = r.bit;   // the warm-up samples, read again once the taps are known
    int32_t c[T];
#pragma unroll
    for (int t = 0; t < T; t++) c[t] = 0;
    int shift = 0;
    Residual res;
    if (on) {
        for (int i = 0; i < f.order; i++) r.get(f.bps);
        if (f.fixed) {
            // taps of x[i-1], x[i-2], ...: 1; 2, -1; 3, -3, 1; 4, -6, 4, -1
            const int n = f.order;
            const int32_t tap[4] = {n, n == 1 ? 0 : n == 2 ? -1 : n == 3 ? -3 : n == 4 ? -6 : 0,
                                    n == 3 ? 1 : n == 4 ? 4 : 0, n == 4 ? -1 : 0};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (lane == j / T) c[j % T] = tap[j];
        } else {
            const int prec = (int)r.get(4) + 1;
            shift = r.sget(5);
            if (prec == 16) err = 6;
            else if (shift < 0) err = 7;
            if (!err)
#pragma unroll
                for (int j = 0; j < kGroup * T; j++)
                    if (j < f.order) {
                        const int32_t v = r.sget(prec);
                        if (lane == j / T) c[j % T] = v;
                    }
        }
        if (!err) err = res.init(r, f.block, f.order);
        if (err) on = false;
    }
    int64_t s[T];
#pragma unroll
    for (int t = 0; t < T; t++) s[t] = 0;
    // the sums move one sample on: the next lane's nearest sum (before x)
    // enters this lane's farthest slot
    auto next_sum = [&]() -> int64_t {
        const uint32_t lo = __shfl_down_sync(kWarp, (uint32_t)s[0], 1, kGroup);
        const uint32_t hi = __shfl_down_sync(kWarp, (uint32_t)((uint64_t)s[0] >> 32), 1, kGroup);
        return lane == kGroup - 1 ? 0 : (int64_t)((uint64_t)hi << 32 | lo);
    };
    auto feed = [&](int32_t x, int64_t from) {
#pragma unroll
        for (int t = 0; t < T; t++) s[t] = (t + 1 < T ? s[t + 1] : from) + (int64_t)c[t] * x;
    };
    const int res_word = r.next - 3, res_bit = r.bit;
    r.seek(warm_word, warm_bit);
    const int warm_steps = __reduce_max_sync(kWarp, on ? f.order : 0);
    for (int i = 0; i < warm_steps; i++) {
        const int64_t from = next_sum();
        if (on && i < f.order) {
            const int32_t x = r.sget(f.bps);
            feed(x, from);
            o.put(x << f.wasted);
        }
    }
    r.seek(res_word, res_bit);
    int n = on ? f.block - f.order : 0;
    const int steps = __reduce_max_sync(kWarp, n);
    for (int i = 0; i < steps; i++) {
        if ((i & 7) == 0) r.top_up();   // a step takes a word at most, save for very long codes
        const int64_t from = next_sum();
        const int32_t ahead = __shfl_sync(kWarp, (int32_t)__funnelshift_r((uint32_t)s[0], (uint32_t)((uint64_t)s[0] >> 32), shift), 0, kGroup);
        if (i < n) {
            int32_t e;
            if (res.next(r, e)) {
                const int32_t x = e + ahead;
                feed(x, from);
                o.put(x << f.wasted);
            } else {
                err = 5;
                n = 0;
            }
        }
    }
    return err;
}

// Four lanes per frame, frames taken in the order `order_idx` gives (sorted by
// subframe type, so the groups of a warp run the same predictor).  Every lane
// of a group reads the same bits and takes the same branches.
__global__ void __launch_bounds__(64) k_flac_frames(const uint32_t* __restrict__ words, const FlacFrame* frames,
                                                    const int* order_idx, int nframes, int16_t* out, int* status) {
    __shared__ __align__(8) uint32_t rings[64 / kGroup][kRing];
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) / kGroup;
    const bool valid = t < nframes;
    const int lane = threadIdx.x % kGroup;
    const int f = order_idx[valid ? t : nframes - 1];
    const FlacFrame fr = frames[f];
    GroupOut o;
    o.init(out + fr.sample0, lane);
    int err = 0;
    BitReader r;
    r.init(words, fr.off + fr.header_len, fr.end, rings[threadIdx.x / kGroup], lane,
           ((1u << kGroup) - 1) << (threadIdx.x % 32 / kGroup * kGroup));
    const int block = fr.block;
    Predicted p{};
    p.block = block;
    if (valid) {
        do {
            if (r.get(1) != 0) { err = 10; break; }
            const int type = (int)r.get(6);
            if (r.get(1)) {
                const int32_t z = r.unary(15);
                if (z < 0) { err = 11; break; }
                p.wasted = z + 1;
            }
            p.bps = 16 - p.wasted;
            if (p.bps <= 0) { err = 12; break; }
            if (type == 0) {
                const int32_t v = r.sget(p.bps);
                for (int i = 0; i < block; i++) o.put(v << p.wasted);
            } else if (type == 1) {
                for (int i = 0; i < block; i++) {
                    const int32_t v = r.sget(p.bps);
                    o.put(v << p.wasted);
                }
            } else if ((type >= 8 && type <= 12) || type >= 32) {
                p.fixed = type < 32;
                p.order = p.fixed ? type - 8 : type - 31;
                if (p.order > block) { err = p.fixed ? 13 : 14; break; }
                p.active = true;
            } else {
                err = 17;
            }
        } while (false);
    }
    const int most = __reduce_max_sync(kWarp, p.active ? p.order + 1 : 0);   // 0: no predicted frame
    if (most > 0) {
        int e;
        if (most <= kGroup + 1) e = predicted_samples<1>(r, p, lane, o);
        else if (most <= 2 * kGroup + 1) e = predicted_samples<2>(r, p, lane, o);
        else if (most <= 4 * kGroup + 1) e = predicted_samples<4>(r, p, lane, o);
        else e = predicted_samples<8>(r, p, lane, o);
        if (e) err = (p.fixed ? 20 : 30) + e;
    }
    if (valid && !err) {
        o.flush();
        const int64_t start = (fr.off + fr.header_len) & ~(int64_t)3;   // the reader's first word
        if (r.overrun()) err = 18;
        // byte alignment, then the frame's CRC-16 (k_flac_crc) must end the frame
        else if (start + ((r.bitpos() + 7) >> 3) + 2 != fr.end) err = 19;
    }
    if (valid && err && lane == 0) atomicCAS(status, 0, (f << 8) | err);
}

// a b mod x^16 + x^15 + x^2 + 1 over GF(2), the CRC-16's polynomial
__device__ __forceinline__ uint32_t gf16_mul(uint32_t a, uint32_t b) {
    uint32_t v = 0;
#pragma unroll
    for (int i = 15; i >= 0; i--) {
        v = v << 1 ^ (v & 0x8000u ? 0x18005u : 0u);
        if (b >> i & 1) v ^= a;
    }
    return v & 0xffffu;
}

// The frames' CRC-16, a warp per frame: bytes [off, end - 2) cut into 32 runs
// of equal length (the first one short), each lane the remainder of its own;
// two neighbouring remainders join as left x^(8 length of right) + right.
// A frame that failed already keeps its error.
__global__ void __launch_bounds__(128) k_flac_crc(const uint8_t* __restrict__ bytes, const FlacFrame* frames,
                                                  int nframes, int* status) {
    __shared__ uint16_t t16[256];   // per-thread table indices: shared, not constant, memory
    for (int i = threadIdx.x; i < 256; i += blockDim.x) t16[i] = c_crc16[i];
    __syncthreads();
    const int f = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
    if (f >= nframes) return;
    const int64_t off = frames[f].off, end = frames[f].end;
    const int64_t n = end - 2 - off;
    if (n <= 0) return;   // shorter than any frame: the decoder reports it
    const int64_t run = (n + 31) / 32, pad = 32 * run - n;
    const int64_t b = off + max(run * lane - pad, (int64_t)0), e = off + max(run * (lane + 1) - pad, (int64_t)0);
    uint32_t crc = 0;
    auto byte = [&](uint32_t v) { crc = (crc << 8 ^ t16[crc >> 8 ^ v]) & 0xffffu; };
    int64_t i = b;
    for (; i < e && (i & 3); i++) byte(bytes[i]);
    for (; i + 4 <= e; i += 4) {   // the buffer is word-aligned
        const uint32_t w = *reinterpret_cast<const uint32_t*>(bytes + i);
        byte(w & 0xffu);
        byte(w >> 8 & 0xffu);
        byte(w >> 16 & 0xffu);
        byte(w >> 24);
    }
    for (; i < e; i++) byte(bytes[i]);
    uint32_t x = 1;   // x^(8 run)
    for (int64_t k = 0; k < run; k++) x = (x << 8 ^ t16[x >> 8]) & 0xffffu;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t right = __shfl_down_sync(0xffffffffu, crc, d);
        crc = gf16_mul(crc, x) ^ right;   // kept by the lanes that are multiples of 2 d
        x = gf16_mul(x, x);
    }
    if (lane == 0 && crc != ((uint32_t)bytes[end - 2] << 8 | bytes[end - 1])) atomicCAS(status, 0, (f << 8) | 40);
}

std::vector<uint8_t> make_crc8() {
    std::vector<uint8_t> t(256);
    for (int b = 0; b < 256; b++) {
        uint8_t c = (uint8_t)b;
        for (int i = 0; i < 8; i++) c = (c & 0x80) ? (uint8_t)((c << 1) ^ 0x07) : (uint8_t)(c << 1);
        t[b] = c;
    }
    return t;
}
std::vector<uint16_t> make_crc16() {
    std::vector<uint16_t> t(256);
    for (int b = 0; b < 256; b++) {
        uint16_t c = (uint16_t)(b << 8);
        for (int i = 0; i < 8; i++) c = (c & 0x8000) ? (uint16_t)((c << 1) ^ 0x8005) : (uint16_t)(c << 1);
        t[b] = c;
    }
    return t;
}

}  // namespace

int32_t flac_stream_info(const uint8_t* p, uint64_t n, FlacInfo& info) {
    // "fLaC", then a first metadata block that is a 34-byte STREAMINFO
    // (the reference's loader rejects anything else: LibsndfilePcm16SampleLoaderTests.cs:1038-1047)
    if (n < 42 || std::memcmp(p, "fLaC", 4) != 0) return fail(VHSDECODE_GB300_STATUS_INPUT_ERROR, "not a FLAC stream");
    if ((p[4] & 0x7F) != 0 || ((p[5] << 16) | (p[6] << 8) | p[7]) != 34)
        return fail(VHSDECODE_GB300_STATUS_INPUT_ERROR, "first FLAC metadata block is not a 34-byte STREAMINFO");
    const uint8_t* si = p + 8;
    info.min_block = (si[0] << 8) | si[1];
    info.max_block = (si[2] << 8) | si[3];
    uint64_t packed = 0;
    for (int i = 10; i < 18; i++) packed = (packed << 8) | si[i];
    info.sample_rate = (uint32_t)(packed >> 44);
    info.channels = (uint32_t)((packed >> 41) & 7) + 1;
    info.bits_per_sample = (uint32_t)((packed >> 36) & 31) + 1;
    info.total_samples = packed & ((uint64_t(1) << 36) - 1);
    // metadata blocks up to the first frame
    uint64_t pos = 4;
    for (;;) {
        if (pos + 4 > n) return fail(VHSDECODE_GB300_STATUS_INPUT_ERROR, "truncated FLAC metadata");
        const bool last = p[pos] & 0x80;
        const uint64_t len = ((uint64_t)p[pos + 1] << 16) | ((uint64_t)p[pos + 2] << 8) | p[pos + 3];
        pos += 4 + len;
        if (last) break;
    }
    if (pos > n) return fail(VHSDECODE_GB300_STATUS_INPUT_ERROR, "truncated FLAC metadata");
    info.first_frame = pos;
    return VHSDECODE_GB300_STATUS_OK;
}

FlacStreamDecoder::~FlacStreamDecoder() {
    if (d_bytes) cudaFree(d_bytes);
    if (d_cand) cudaFree(d_cand);
    if (d_frames) cudaFree(d_frames);
    if (d_work) cudaFree(d_work);
    if (d_out) cudaFree(d_out);
    if (d_misc) cudaFree(d_misc);
    if (stream) cudaStreamDestroy(stream);
}

void FlacStreamDecoder::init(int device) {
    ck(cudaSetDevice(device), "cudaSetDevice");
    ck(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
    // the CRC tables live in this device's copy of the module's constant memory
    const std::vector<uint8_t> t8 = make_crc8();
    const std::vector<uint16_t> t16 = make_crc16();
    ck(cudaMemcpyToSymbol(c_crc8, t8.data(), 256), "crc table");
    ck(cudaMemcpyToSymbol(c_crc16, t16.data(), 512), "crc table");
    ck(cudaMalloc(&d_misc, 2 * sizeof(int)), "cudaMalloc");
}

void FlacStreamDecoder::reserve(size_t bytes, size_t samples, size_t frames) {
    auto grow = [](void** p, size_t& have, size_t want) {
        if (want <= have) return;
        if (*p) cudaFree(*p);
        *p = nullptr;
        ck(cudaMalloc(p, want), "cudaMalloc");
        have = want;
    };
    grow((void**)&d_bytes, cap_bytes, (bytes + 96) & ~(size_t)15);
    grow((void**)&d_cand, cap_cand, std::max<size_t>(frames, 1024) * sizeof(FlacCand));
    grow((void**)&d_frames, cap_frames, std::max<size_t>(frames + 16, 64) * sizeof(FlacFrame));
    grow((void**)&d_work, cap_work, std::max<size_t>(frames, 1) * sizeof(int32_t));   // frame order
    grow((void**)&d_out, cap_out, std::max<size_t>(samples, 1) * sizeof(int16_t));
}

size_t FlacStreamDecoder::decode(const uint8_t* p, size_t n, bool at_eof, std::vector<int16_t>& out) {
    return decode_to(p, n, at_eof, [&](size_t count) {
        const size_t old = out.size();
        out.resize(old + count);
        return out.data() + old;
    });
}

size_t FlacStreamDecoder::decode_to(const uint8_t* p, size_t n, bool at_eof,
                                    const std::function<int16_t*(size_t)>& dest) {
    if (n == 0) return 0;
    // header candidates: real frames of RF captures hold thousands of bytes; a
    // chunk may hold up to one candidate per 64 bytes (false sync patterns in
    // compressed data that also pass the CRC-8 are about 1 in 2^24 positions)
    const size_t max_frames = n / 64 + 1024;
    reserve(n, 0, max_frames);
    ck(cudaMemsetAsync(d_bytes + (n & ~(size_t)15), 0, 80, stream), "memset");   // zero pad after the data
    ck(cudaMemcpyAsync(d_bytes, p, n, cudaMemcpyHostToDevice, stream), "h2d flac");
    ck(cudaMemsetAsync(d_misc, 0, 2 * sizeof(int), stream), "memset");
    const bool timing = std::getenv("VHSD_STAGE_TIMING") != nullptr;
    cudaEvent_t ev[4] = {};
    if (timing)
        for (auto& e : ev) ck(cudaEventCreate(&e), "event");
    if (timing) ck(cudaEventRecord(ev[0], stream), "event");
    const int cap = (int)(cap_cand / sizeof(FlacCand));
    k_flac_sync<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(d_bytes, (int64_t)n, d_cand, d_misc, cap);
    ck(cudaGetLastError(), "flac sync launch");
    if (timing) ck(cudaEventRecord(ev[1], stream), "event");
    int count = 0;
    ck(cudaMemcpyAsync(&count, d_misc, sizeof(int), cudaMemcpyDeviceToHost, stream), "d2h");
    ck(cudaStreamSynchronize(stream), "sync");
    if (count > cap) throw Failure(VHSDECODE_GB300_STATUS_INPUT_ERROR, "too many FLAC frame candidates");
    std::vector<FlacCand> cand((size_t)count);
    if (count) ck(cudaMemcpy(cand.data(), d_cand, (size_t)count * sizeof(FlacCand), cudaMemcpyDeviceToHost), "d2h");
    std::sort(cand.begin(), cand.end(), [](const FlacCand& a, const FlacCand& b) { return a.at < b.at; });
    // chain: the chunk starts on a frame; accept headers that continue the sequence
    std::vector<FlacFrame> frames;
    std::vector<uint8_t> types;   // each frame's subframe type byte
    frames.reserve(cand.size());
    types.reserve(cand.size());
    int64_t expect_at = 0;
    for (size_t i = 0; i < cand.size(); i++) {
        const int64_t at = cand[i].at;
        if (at < expect_at) continue;
        const uint64_t num = cand[i].number;
        const int block = cand[i].block, hl = cand[i].header_len;
        const uint64_t want = cand[i].variable ? next_sample : next_frame;
        if (cand[i].other) {
            // a header of another sample format where this stream's next frame belongs
            if (num == want) throw Failure(VHSDECODE_GB300_STATUS_INPUT_ERROR, "FLAC stream is not 16-bit mono");
            continue;
        }
        if (num != want) {
            if (frames.empty() && at == 0)
                throw Failure(VHSDECODE_GB300_STATUS_INPUT_ERROR, "FLAC frame out of sequence");
            continue;
        }
        if (!frames.empty()) frames.back().end = at;
        else if (at != 0) throw Failure(VHSDECODE_GB300_STATUS_INPUT_ERROR, "FLAC data before the first frame");
        FlacFrame fr{};
        fr.off = at;
        fr.end = (int64_t)n;
        fr.header_len = hl;
        fr.block = block;
        fr.sample0 = (int64_t)(next_sample - sample_base);
        frames.push_back(fr);
        types.push_back(cand[i].type);
        next_frame++;
        next_sample += (uint64_t)block;
        expect_at = at + hl;
    }
    // the last frame of a chunk is complete only at the end of the stream
    if (!at_eof && !frames.empty()) {
        next_frame--;
        next_sample -= (uint64_t)frames.back().block;
        frames.pop_back();
    }
    if (frames.empty()) {
        if (at_eof && n > 0) throw Failure(VHSDECODE_GB300_STATUS_INPUT_ERROR, "no FLAC frame in the final data");
        return 0;
    }
    const size_t nsamp = (size_t)(next_sample - sample_base);
    reserve(n, nsamp, frames.size());
    // frames sorted by subframe type (the byte after the frame header), so the
    // lanes of a warp decode with the same predictor
    std::vector<int> idx(frames.size());
    {
        size_t first[257] = {};
        for (size_t i = 0; i < idx.size(); i++) first[types[i] + 1]++;
        for (int t = 0; t < 256; t++) first[t + 1] += first[t];
        for (size_t i = 0; i < idx.size(); i++) idx[first[types[i]]++] = (int)i;
    }
    ck(cudaMemcpyAsync(d_frames, frames.data(), frames.size() * sizeof(FlacFrame), cudaMemcpyHostToDevice, stream),
       "h2d frames");
    ck(cudaMemcpyAsync(d_work, idx.data(), idx.size() * sizeof(int), cudaMemcpyHostToDevice, stream), "h2d order");
    if (timing) ck(cudaEventRecord(ev[2], stream), "event");
    k_flac_frames<<<(unsigned)((frames.size() * kGroup + 63) / 64), 64, 0, stream>>>(
        reinterpret_cast<const uint32_t*>(d_bytes), d_frames, d_work, (int)frames.size(), d_out, d_misc + 1);
    k_flac_crc<<<(unsigned)((frames.size() + 3) / 4), 128, 0, stream>>>(d_bytes, d_frames, (int)frames.size(),
                                                                       d_misc + 1);
    if (timing) ck(cudaEventRecord(ev[3], stream), "event");
    ck(cudaGetLastError(), "flac decode launch");
    int st = 0;
    int16_t* dst = dest(nsamp);
    if (dst) ck(cudaMemcpyAsync(dst, d_out, nsamp * sizeof(int16_t), cudaMemcpyDeviceToHost, stream), "d2h");
    ck(cudaMemcpyAsync(&st, d_misc + 1, sizeof(int), cudaMemcpyDeviceToHost, stream), "d2h");
    ck(cudaStreamSynchronize(stream), "sync");
    if (timing) {
        float t_sync = 0, t_frames = 0;
        cudaEventElapsedTime(&t_sync, ev[0], ev[1]);
        cudaEventElapsedTime(&t_frames, ev[2], ev[3]);
        std::fprintf(stderr, "vhsd flac: %zu bytes, %zu frames, header scan %.3f ms, frame decode %.3f ms\n", n,
                     frames.size(), t_sync, t_frames);
        for (auto& e : ev) cudaEventDestroy(e);
    }
    if (st) {
        char msg[128];
        std::snprintf(msg, sizeof msg, "corrupt FLAC frame %lld (code %d)",
                      (long long)(next_frame - frames.size() + (st >> 8)), st & 255);
        throw Failure(VHSDECODE_GB300_STATUS_INPUT_ERROR, msg);
    }
    sample_base = next_sample;
    decoded_frames += frames.size();
    return (size_t)frames.back().end;
}

}  // namespace vhsd

using namespace vhsd;

extern "C" {

VHSDECODE_GB300_API int32_t VHSDECODE_GB300_CALL vhsdecode_gb300_flac_info(
    const uint8_t* data, uint64_t bytes, vhsdecode_gb300_flac_info_v1* info) {
    return guard([&]() -> int32_t {
        if (!data || !info) return fail(VHSDECODE_GB300_STATUS_NULL_POINTER, "null argument");
        if (info->struct_size != sizeof(vhsdecode_gb300_flac_info_v1))
            return fail(VHSDECODE_GB300_STATUS_INVALID_ARGUMENT, "flac_info struct_size mismatch");
        FlacInfo fi{};
        int32_t st = flac_stream_info(data, bytes, fi);
        if (st != VHSDECODE_GB300_STATUS_OK) return st;
        info->sample_rate = fi.sample_rate;
        info->channels = fi.channels;
        info->bits_per_sample = fi.bits_per_sample;
        info->min_block = fi.min_block;
        info->max_block = fi.max_block;
        info->total_samples = fi.total_samples;
        info->first_frame_offset = fi.first_frame;
        return VHSDECODE_GB300_STATUS_OK;
    });
}

VHSDECODE_GB300_API int32_t VHSDECODE_GB300_CALL vhsdecode_gb300_flac_decode(
    const uint8_t* data, uint64_t bytes, int16_t* out, uint64_t capacity, uint64_t* samples, int32_t device_id) {
    return guard([&]() -> int32_t {
        if (!data || !samples || (capacity && !out)) return fail(VHSDECODE_GB300_STATUS_NULL_POINTER, "null argument");
        FlacInfo fi{};
        int32_t st = flac_stream_info(data, bytes, fi);
        if (st != VHSDECODE_GB300_STATUS_OK) return st;
        if (fi.channels != 1 || fi.bits_per_sample != 16)
            return fail(VHSDECODE_GB300_STATUS_INPUT_ERROR, "FLAC stream is not 16-bit mono");
        // one decoder (device buffers, stream) per device, reused across calls;
        // calls on one device are serialised
        static std::mutex m;
        static FlacStreamDecoder* decoders[64] = {};
        if (device_id < 0 || device_id >= 64) return fail(VHSDECODE_GB300_STATUS_INVALID_ARGUMENT, "device_id out of range");
        std::lock_guard<std::mutex> lk(m);
        if (!decoders[device_id]) {
            auto* d = new FlacStreamDecoder();
            try {
                d->init(device_id);
            } catch (...) {
                delete d;
                throw;
            }
            decoders[device_id] = d;
        }
        FlacStreamDecoder& dec = *decoders[device_id];
        ck(cudaSetDevice(device_id), "cudaSetDevice");
        dec.reset();
        // the samples go straight to the caller's buffer when they fit
        std::vector<int16_t> spill;
        uint64_t produced = 0;
        dec.decode_to(data + fi.first_frame, bytes - fi.first_frame, true, [&](size_t count) -> int16_t* {
            produced = count;
            if (count <= capacity) return out;
            if (!capacity) return nullptr;
            spill.resize(count);
            return spill.data();
        });
        *samples = produced;
        if (!spill.empty()) std::memcpy(out, spill.data(), capacity * sizeof(int16_t));
        return VHSDECODE_GB300_STATUS_OK;
    });
}

}  // extern "C"
