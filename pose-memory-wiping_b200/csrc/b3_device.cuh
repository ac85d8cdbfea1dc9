/*
 * b3_device.cuh — register-resident BLAKE3 compression for sm_100a.
 *
 * Written from the BLAKE3 specification.  The 16-word state stays in
 * registers for the whole compression; the message schedule is resolved at
 * compile time (round r reads message word sched(r, i), the BLAKE3 message
 * permutation applied r times), so permuting costs no instructions.
 * Rotations by 16 and 8 are byte permutes, those by 12 and 7 funnel shifts;
 * the additions are split between the integer and the FMA pipe (g_mix).
 */
#ifndef PB_B3_DEVICE_CUH
#define PB_B3_DEVICE_CUH

#include <cstdint>

namespace pb {

/* BLAKE3 flags used by the node hash. */
constexpr uint32_t kFlagChunkStart = 1u << 0;
constexpr uint32_t kFlagChunkEnd = 1u << 1;
constexpr uint32_t kFlagRoot = 1u << 3;
constexpr uint32_t kFlagKeyed = 1u << 4;
constexpr uint32_t kFlagDeriveMaterial = 1u << 6;

/* Node message blocks: block 0 (node index) starts the chunk, block 2
 * (seed | descriptor) ends it and is the root (common/src/hash.c:136-140). */
constexpr uint32_t kFlagsBlock0 = kFlagKeyed | kFlagChunkStart;
constexpr uint32_t kFlagsBlock1 = kFlagKeyed;
constexpr uint32_t kFlagsBlock2 = kFlagKeyed | kFlagChunkEnd | kFlagRoot;

constexpr uint32_t kIV0 = 0x6A09E667u, kIV1 = 0xBB67AE85u, kIV2 = 0x3C6EF372u,
                   kIV3 = 0xA54FF53Au, kIV4 = 0x510E527Fu, kIV5 = 0x9B05688Cu,
                   kIV6 = 0x1F83D9ABu, kIV7 = 0x5BE0CD19u;

__host__ __device__ constexpr int perm16(int i)
{
    /* BLAKE3 message permutation */
    return i == 0 ? 2 : i == 1 ? 6 : i == 2 ? 3 : i == 3 ? 10 : i == 4 ? 7 : i == 5 ? 0
         : i == 6 ? 4 : i == 7 ? 13 : i == 8 ? 1 : i == 9 ? 11 : i == 10 ? 12
         : i == 11 ? 5 : i == 12 ? 9 : i == 13 ? 14 : i == 14 ? 15 : 8;
}

__host__ __device__ constexpr int sched(int r, int i)
{
    return r == 0 ? i : sched(r - 1, perm16(i));
}

__device__ __forceinline__ uint32_t rotr16(uint32_t x) { return __byte_perm(x, 0, 0x1032); }
__device__ __forceinline__ uint32_t rotr8(uint32_t x) { return __byte_perm(x, 0, 0x0321); }
__device__ __forceinline__ uint32_t rotr12(uint32_t x) { return __funnelshift_r(x, x, 12); }
__device__ __forceinline__ uint32_t rotr7(uint32_t x) { return __funnelshift_r(x, x, 7); }

/* 1, but not to the compiler: every kernel of this library is launched on a
 * grid one block deep. */
__device__ __forceinline__ uint32_t opaque_one() { return gridDim.z; }

__device__ __forceinline__ uint32_t madd(uint32_t a, uint32_t one, uint32_t b)
{
    uint32_t r;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(one), "r"(b));
    return r;
}

/* The G function.  Its xors and rotations (8 operations) go to the integer
 * ALU pipe, which then bounds both one warp and a full SM, so its additions
 * are kept off that pipe: a + b + m is a plain a + m, off the dependent chain
 * since a and m are known before b, then an integer multiply-add b * 1 + that
 * (`one`, opaque to the compiler, keeps it a multiply-add, which goes to the
 * FMA pipe); c + d is left to the compiler.
 * The best of 145 mixes of the four additions (plain, multiply-add, either
 * order, alternating between columns) in latency and in throughput: 964
 * clocks a compression for one warp and 40.0 G compressions/s with every SM
 * full (39.7 in k_compress_bench), against 1162 clocks and 32.7 G/s with all
 * additions plain, and at most 36.9 G/s with all of them multiply-adds. */
__device__ __forceinline__ void g_mix(uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d,
                                      uint32_t x, uint32_t y, uint32_t one)
{
    a = madd(b, one, a + x);
    d = rotr16(d ^ a);
    c = c + d;
    b = rotr12(b ^ c);
    a = madd(b, one, a + y);
    d = rotr8(d ^ a);
    c = c + d;
    b = rotr7(b ^ c);
}

template <int R>
__device__ __forceinline__ void round_fn(uint32_t (&v)[16], const uint32_t (&m)[16], uint32_t one)
{
    g_mix(v[0], v[4], v[8], v[12], m[sched(R, 0)], m[sched(R, 1)], one);
    g_mix(v[1], v[5], v[9], v[13], m[sched(R, 2)], m[sched(R, 3)], one);
    g_mix(v[2], v[6], v[10], v[14], m[sched(R, 4)], m[sched(R, 5)], one);
    g_mix(v[3], v[7], v[11], v[15], m[sched(R, 6)], m[sched(R, 7)], one);
    g_mix(v[0], v[5], v[10], v[15], m[sched(R, 8)], m[sched(R, 9)], one);
    g_mix(v[1], v[6], v[11], v[12], m[sched(R, 10)], m[sched(R, 11)], one);
    g_mix(v[2], v[7], v[8], v[13], m[sched(R, 12)], m[sched(R, 13)], one);
    g_mix(v[3], v[4], v[9], v[14], m[sched(R, 14)], m[sched(R, 15)], one);
}

/* One compression with counter 0: cv <- first 8 output words (the chaining
 * value; for a ROOT block these are the first 32 output bytes). */
__device__ __forceinline__ void compress(uint32_t (&cv)[8], const uint32_t (&m)[16],
                                         uint32_t block_len, uint32_t flags)
{
    const uint32_t one = opaque_one();
    uint32_t v[16] = {cv[0], cv[1], cv[2], cv[3], cv[4], cv[5], cv[6], cv[7],
                      kIV0,  kIV1,  kIV2,  kIV3,  0u,    0u,    block_len, flags};
    round_fn<0>(v, m, one);
    round_fn<1>(v, m, one);
    round_fn<2>(v, m, one);
    round_fn<3>(v, m, one);
    round_fn<4>(v, m, one);
    round_fn<5>(v, m, one);
    round_fn<6>(v, m, one);
#pragma unroll
    for (int i = 0; i < 8; i++) cv[i] = v[i] ^ v[i + 8];
}

/* ── four lanes per compression ──────────────────────────────────────────── */

/* One compression spread over four neighbouring lanes (a quad): lane i holds
 * column i of the state, so a column step is one G per lane and a diagonal
 * step one more after three of the four rows have moved.  Row b, which G
 * finishes last, stays in place; rows a, c and d, finished earlier, move
 * (a by one lane down, c one up, d two across), so most of their shuffle
 * latency (26 clocks) passes behind the rest of G.  A rotated word is added
 * to the next row straight from the unrotated one (rotl_add), beside the
 * rotation that keeps the row, so that the chain need not pass through it.
 * Measured: 755 clocks a compression for 1 to 4 warps of an SM (8 nodes each)
 * and 824 for 8 warps, against 964 for one lane a node; a full SM does only
 * 24 G compressions/s this way against 40.0, so it is for narrow levels. */
struct QuadLane {
    uint32_t i;       /* lane within the quad */
    int below, above; /* lanes i - 1 and i + 1 of the quad, modulo 4 */
    bool b0, b1;      /* bits of i */
    __device__ __forceinline__ explicit QuadLane(uint32_t lane)
    {
        /* opaque to the compiler, so that it keeps them for a level's 84
         * shuffles and selections in place of computing them anew */
        asm volatile("and.b32 %0, %1, 3;" : "=r"(i) : "r"(lane));
        asm volatile("add.s32 %0, %1, 3;" : "=r"(below) : "r"(i));
        asm volatile("add.s32 %0, %1, 1;" : "=r"(above) : "r"(i));
        b0 = (i & 1u) != 0;
        b1 = (i & 2u) != 0;
    }
    __device__ __forceinline__ uint32_t pick(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) const
    {
        return b1 ? (b0 ? w3 : w2) : (b0 ? w1 : w0);
    }
};

/* shf.l written out, apart from the rotation that produces the row itself,
 * so that the compiler may fold it into the addition. */
template <int N>
__device__ __forceinline__ uint32_t rotl_add(uint32_t x, uint32_t y)
{
    uint32_t r;
    asm("shf.l.wrap.b32 %0, %1, %1, %2;" : "=r"(r) : "r"(x), "n"(N));
    return y + r;
}

/* Half a round: G with message words x and y, then the rows' move.  COLUMN:
 * the step just done was the column step (a goes to the lane above's place,
 * that is, each lane reads a from the lane below). */
template <bool COLUMN>
__device__ __forceinline__ void quad_half(uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d, uint32_t x,
                                          uint32_t y, const QuadLane &q)
{
    a = a + b + x;
    uint32_t t = d ^ a;
    const uint32_t d1 = rotr16(t);
    c = rotl_add<16>(t, c);
    uint32_t u = b ^ c;
    a = rotl_add<20>(u, a + y);
    const uint32_t b1 = rotr12(u);
    t = d1 ^ a;
    d = rotr8(t);
    c = rotl_add<24>(t, c);
    u = b1 ^ c;
    a = __shfl_sync(0xFFFFFFFFu, a, COLUMN ? q.below : q.above, 4);
    d = __shfl_xor_sync(0xFFFFFFFFu, d, 2);
    c = __shfl_sync(0xFFFFFFFFu, c, COLUMN ? q.above : q.below, 4);
    b = rotr7(u);
}

/* Message words of lane i in round R: column step m[2i], m[2i+1]; diagonal
 * step m[8+2j], m[9+2j] with j = i-1, since b stays and row a moved up by
 * one (permuted by the round's schedule). */
template <int R>
__device__ __forceinline__ void quad_round(uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d,
                                           const uint32_t (&m)[16], const QuadLane &q)
{
    quad_half<true>(a, b, c, d, q.pick(m[sched(R, 0)], m[sched(R, 2)], m[sched(R, 4)], m[sched(R, 6)]),
                    q.pick(m[sched(R, 1)], m[sched(R, 3)], m[sched(R, 5)], m[sched(R, 7)]), q);
    quad_half<false>(a, b, c, d, q.pick(m[sched(R, 14)], m[sched(R, 8)], m[sched(R, 10)], m[sched(R, 12)]),
                     q.pick(m[sched(R, 15)], m[sched(R, 9)], m[sched(R, 11)], m[sched(R, 13)]), q);
}

/* compress() by a quad, block length 64: lane i has chaining words i (a) and
 * 4 + i (b), and every lane the whole message.  step.at<R>() runs after round
 * R: independent work of the caller, for the issue slots that the quad's
 * dependent chain leaves empty. */
template <class Step>
__device__ __forceinline__ void quad_compress(uint32_t &a, uint32_t &b, const uint32_t (&m)[16], uint32_t flags,
                                              const QuadLane &q, Step &step)
{
    uint32_t c = q.pick(kIV0, kIV1, kIV2, kIV3), d = q.pick(0u, 0u, 64u, flags);
    quad_round<0>(a, b, c, d, m, q);
    step.template at<0>();
    quad_round<1>(a, b, c, d, m, q);
    step.template at<1>();
    quad_round<2>(a, b, c, d, m, q);
    step.template at<2>();
    quad_round<3>(a, b, c, d, m, q);
    step.template at<3>();
    quad_round<4>(a, b, c, d, m, q);
    step.template at<4>();
    quad_round<5>(a, b, c, d, m, q);
    step.template at<5>();
    quad_round<6>(a, b, c, d, m, q);
    a ^= c;
    b ^= d;
}

/* The same with the message words of every round laid out per lane
 * (quad_table_entry): words[4 * r] is this lane's of round r, and the caller
 * has those of round 0 in `first`. */
__device__ __forceinline__ void quad_compress_table(uint32_t &a, uint32_t &b, uint4 first, const uint4 *words,
                                                    uint32_t flags, const QuadLane &q)
{
    uint32_t c = q.pick(kIV0, kIV1, kIV2, kIV3), d = q.pick(0u, 0u, 64u, flags);
    uint4 w = first;
#pragma unroll
    for (int r = 0; r < 7; r++) {
        uint4 next = w;
        if (r < 6) next = words[4 * (r + 1)];
        quad_half<true>(a, b, c, d, w.x, w.y, q);
        quad_half<false>(a, b, c, d, w.z, w.w, q);
        w = next;
    }
    a ^= c;
    b ^= d;
}

/* Message word index of position p in round r, with r known at run time. */
__device__ __forceinline__ uint32_t sched_rt(uint32_t r, uint32_t p)
{
    for (; r > 0; r--) p = (uint32_t)(0x8FE95CB1D407A362ull >> (4 * p)) & 15u; /* perm16, a nibble each */
    return p;
}

/* Entry k (round k >> 2, lane k & 3) of a message's quad table. */
__device__ __forceinline__ uint4 quad_table_entry(const uint32_t *msg, uint32_t k)
{
    const uint32_t r = k >> 2, i = k & 3u, j = (i + 3u) & 3u;
    return make_uint4(msg[sched_rt(r, 2 * i)], msg[sched_rt(r, 2 * i + 1)], msg[sched_rt(r, 8 + 2 * j)],
                      msg[sched_rt(r, 9 + 2 * j)]);
}

/* Block 0 of a node message: node index big-endian in bytes 0..7, the rest
 * zero.  As little-endian words: w0 = bswap(index >> 32), w1 = bswap(index). */
__device__ __forceinline__ void block0_words(uint32_t (&m)[16], uint64_t node_index)
{
    m[0] = __byte_perm((uint32_t)(node_index >> 32), 0, 0x0123);
    m[1] = __byte_perm((uint32_t)node_index, 0, 0x0123);
#pragma unroll
    for (int i = 2; i < 16; i++) m[i] = 0;
}

} /* namespace pb */

#endif
