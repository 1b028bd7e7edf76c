// pk_exchange.cuh -- exchanges between blocks by tagged packets, and the row updates that
// owners and copies of a row share (pk_pcg_res.cu, pk_pcg_part.cu).
//
// Every value of an exchange travels in a 16-byte packet with a tag (the exchange's number),
// written and read whole, so that no fence orders it.
#pragma once

#include "pk_device.cuh"

namespace pk {
namespace {

struct Packet {
    unsigned long long lo, hi;
};
__device__ __forceinline__ void st_packet(void* p, Packet v)
{
    asm volatile(
        "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p), "l"(v.lo),
        "l"(v.hi)
        : "memory");
}
__device__ __forceinline__ Packet ld_packet(const void* p)
{
    Packet v;
    asm volatile(
        "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
        : "=l"(v.lo), "=l"(v.hi)
        : "l"(p)
        : "memory");
    return v;
}
__device__ __forceinline__ unsigned packet_tag(Packet v) { return (unsigned)(v.hi >> 32); }

// A row of q with its tag: one packet in FP32; two in FP64 (96 bits of data and a tag each).
__device__ __forceinline__ void st_row(unsigned char* p, V3<float> q, unsigned tag)
{
    st_packet(p, {(unsigned long long)__float_as_uint(q.x) | ((unsigned long long)__float_as_uint(q.y) << 32),
                  (unsigned long long)__float_as_uint(q.z) | ((unsigned long long)tag << 32)});
}
__device__ __forceinline__ void st_row(unsigned char* p, V3<double> q, unsigned tag)
{
    const unsigned long long x = __double_as_longlong(q.x), y = __double_as_longlong(q.y),
                             z = __double_as_longlong(q.z), t = (unsigned long long)tag << 32;
    st_packet(p, {x, (y & 0xffffffffull) | t});
    st_packet(p + 16, {(y >> 32) | (z << 32), (z >> 32) | t});
}
__device__ __forceinline__ bool ld_row(const unsigned char* p, unsigned tag, V3<float>& q)
{
    const Packet a = ld_packet(p);
    q = V3<float>{__uint_as_float((unsigned)a.lo), __uint_as_float((unsigned)(a.lo >> 32)),
                  __uint_as_float((unsigned)a.hi)};
    return packet_tag(a) == tag;
}
__device__ __forceinline__ bool ld_row(const unsigned char* p, unsigned tag, V3<double>& q)
{
    const Packet a = ld_packet(p), b = ld_packet(p + 16);
    q = V3<double>{__longlong_as_double((long long)a.lo),
                   __longlong_as_double((long long)((a.hi & 0xffffffffull) | (b.lo << 32))),
                   __longlong_as_double((long long)((b.lo >> 32) | (b.hi << 32)))};
    return packet_tag(a) == tag && packet_tag(b) == tag;
}

// The row updates, with every rounding spelled out: owners and halo copies must agree.
template <class Real>
__device__ __forceinline__ V3<Real> fma3(Real a, V3<Real> b, V3<Real> c)
{
    return V3<Real>{fma(a, b.x, c.x), fma(a, b.y, c.y), fma(a, b.z, c.z)};
}
__device__ __forceinline__ V3<float> fma3(float a, V3<float> b, V3<float> c)
{
    return V3<float>{__fmaf_rn(a, b.x, c.x), __fmaf_rn(a, b.y, c.y), __fmaf_rn(a, b.z, c.z)};
}
template <class Real>
__device__ __forceinline__ V3<Real> apply_minv(const Real (&m)[9], V3<Real> v)
{
    V3<Real> r{m[0] * v.x, m[1] * v.x, m[2] * v.x};
    r = V3<Real>{fma(m[3], v.y, r.x), fma(m[4], v.y, r.y), fma(m[5], v.y, r.z)};
    return V3<Real>{fma(m[6], v.z, r.x), fma(m[7], v.z, r.y), fma(m[8], v.z, r.z)};
}
// c + a b with the FP64 scalar a: in FP32 a is split into two floats (see SplitAlpha in
// pk_pcg_slab.cu: within an ulp of the FP64 update, without conversions).
template <class Real>
struct Scale;
template <>
struct Scale<float> {
    float hi, lo;
    __device__ __forceinline__ explicit Scale(double a) : hi(float(a)), lo(float(a - double(float(a)))) {}
    __device__ __forceinline__ Scale(float h, float l) : hi(h), lo(l) {}
    __device__ __forceinline__ Scale negated() const { return Scale(-hi, -lo); }
    __device__ __forceinline__ V3<float> axpy(V3<float> b, V3<float> c) const { return fma3(lo, b, fma3(hi, b, c)); }
};
template <>
struct Scale<double> {
    double a;
    __device__ __forceinline__ explicit Scale(double v) : a(v) {}
    __device__ __forceinline__ Scale negated() const { return Scale(-a); }
    __device__ __forceinline__ V3<double> axpy(V3<double> b, V3<double> c) const { return fma3(a, b, c); }
};

// An FP32 system's sums are added in double here and judged as floats, so that a solve whose
// sums a float does not hold ends as it does where they are added in float (the other kernels,
// the reference): from 2^128 infinite, below 2^-150 zero.
__device__ __forceinline__ double as_float_sum(double v)
{
    const int m = __double2hiint(v) & 0x7fffffff;
    return m >= 0x47f00000 ? (double)INFINITY : m < 0x36900000 ? 0.0 : v;
}
// What alpha and beta may reach: the largest finite value of the sums' type.
template <bool FS>
constexpr double scalar_max()
{
    return FS ? 3.4028234663852886e38 : 1.7976931348623157e308;
}

// The exchange of a group of blocks through global memory: sums of four doubles and the OR
// of a word.  A block pushes its sums into the inbox of every member (kTagSlotBytes a
// sender), so that a reader polls lines nobody else reads.  The inbox of member j has
// 2 x size slots at inbox + 2 x size x j x kTagSlotBytes, two buffers by the parity of the
// exchange number gen = 1, 2, ...: a block overwrites exchange g's packets in g + 2, after
// it has seen every member's sums of g + 1, which each sends only when it has read all of
// g.  The inboxes are zero before the first exchange.  All sums keep one fixed order (warp
// shuffles, the block's warps, the group's blocks), the same in every block.
constexpr int kTagSums = 4;
constexpr int kTagSlotBytes = 16 * kTagSums;
constexpr int kTagMaxGroup = 160;
constexpr int kTagPoll = kTagMaxGroup / 32;
struct TagShared {
    double part[2][kTagSums * 16];  // the warps' partials, by exchange parity
    double sum[2][kTagSums];
    unsigned bits[3], gbits[3];     // by exchange number
    int fail;
};
// The warps of the block that take part: the first `warps`, which meet at named barrier `id`.
struct TagTeam {
    int warps;
    unsigned id;
    __device__ __forceinline__ void sync() const
    {
        asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(32 * warps) : "memory");
    }
};
__device__ __forceinline__ void tag_init(TagShared& sh)  // one thread; then a block barrier
{
    for (int i = 0; i < 3; ++i) sh.bits[i] = sh.gbits[i] = 0u;
    sh.fail = 0;
}
// Reduces the block's v (of the first `value_warps` warps) and sends them.
__device__ __forceinline__ void tag_publish(unsigned char* inbox, int size, int me, unsigned gen, double (&v)[kTagSums],
                                            unsigned& bits, int value_warps, TagTeam team, TagShared& sh)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = team.warps;
    // The warps' four sums, each in one butterfly: two steps that halve the values a lane
    // carries, then (lane >> 3) holds its own sum.
    if (warp < value_warps) {
        const bool up = (lane & 16) != 0, right = (lane & 8) != 0;
        double k0 = up ? v[2] : v[0], k1 = up ? v[3] : v[1];
        k0 += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
        k1 += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
        double t = right ? k1 : k0;
        t += __shfl_xor_sync(0xffffffffu, right ? k0 : k1, 8);
        t += __shfl_xor_sync(0xffffffffu, t, 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        if ((lane & 7) == 0) sh.part[gen & 1u][(lane >> 3) * 16 + warp] = t;
    }
    if (bits) atomicOr(&sh.bits[gen % 3u], bits);
    team.sync();
    if (threadIdx.x == 0) sh.bits[(gen + 2u) % 3u] = 0u;
    if (size > 1 && 8 * warp >= size) return;
    // The block's sums: lane (k, i) takes the partials of sum k of warps i and i + 8.  Warps
    // that send do it each for itself; a group of one block needs nothing else.
    const double* q = sh.part[gen & 1u] + (lane >> 3) * 16 + (lane & 7);
    double t = (lane & 7) < value_warps ? q[0] : 0.0;
    if (value_warps > 8) t += (lane & 7) + 8 < value_warps ? q[8] : 0.0;
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    const unsigned w = sh.bits[gen % 3u];
    if (size <= 1) {
#pragma unroll
        for (int k = 0; k < kTagSums; ++k) v[k] = __shfl_sync(0xffffffffu, t, 8 * k);
        bits = w;
        return;
    }
    // warp w's lane (k, i) sends sum k to the members 8 w + i, + 8 nw, ...
    unsigned char* out = inbox + ((size_t)(gen & 1u) * size + me) * kTagSlotBytes + 16 * (lane >> 3);
    for (int d = 8 * warp + (lane & 7); d < size; d += 8 * nw)
        st_packet(out + (size_t)2 * size * d * kTagSlotBytes,
                  {(unsigned long long)__double_as_longlong(t), (unsigned long long)w | ((unsigned long long)gen << 32)});
}
// Waits (bounded: `limit` polls) for the group's sums; false when a wait gave up.  The last
// four of eight or more warps (all of four) read one sum each, lane i of them the members i, i + 32, ...
__device__ __forceinline__ bool tag_finish(const unsigned char* inbox, int size, int me, unsigned gen,
                                           double (&v)[kTagSums], unsigned& bits, unsigned* flags, TagTeam team,
                                           TagShared& sh, unsigned limit = kTagSpinLimit)
{
    if (size <= 1) return sh.fail == 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = team.warps;
    const int sum = nw >= 8 ? warp - (nw - kTagSums) : warp;
    if (sum >= 0 && sum < kTagSums) {
        const unsigned char* in = inbox + ((size_t)2 * size * me + (size_t)(gen & 1u) * size) * kTagSlotBytes + 16 * sum;
        Packet pk[kTagPoll];
        unsigned todo = 0;
#pragma unroll
        for (int j = 0; j < kTagPoll; ++j) {
            pk[j] = Packet{0ull, 0ull};
            if (lane + 32 * j < size) todo |= 1u << j;
        }
        for (unsigned long long spins = 0; todo; ++spins) {
#pragma unroll
            for (int j = 0; j < kTagPoll; ++j)
                if ((todo >> j) & 1u) pk[j] = ld_packet(in + (size_t)(lane + 32 * j) * kTagSlotBytes);
#pragma unroll
            for (int j = 0; j < kTagPoll; ++j)
                if (((todo >> j) & 1u) && packet_tag(pk[j]) == gen) todo &= ~(1u << j);
            if (spins > limit) {
                atomicOr(flags, kFlagBarrierTimeout);
                sh.fail = 1;
                break;
            }
            if ((spins & 1023u) == 1023u && (*(volatile unsigned*)flags & kFlagBarrierTimeout)) {
                sh.fail = 1;
                break;
            }
        }
        __syncwarp();
        double t = 0.0;
        unsigned w = 0;
#pragma unroll
        for (int j = 0; j < kTagPoll; ++j)
            if (lane + 32 * j < size) {
                t += __longlong_as_double((long long)pk[j].lo);
                w |= (unsigned)pk[j].hi;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) sh.sum[gen & 1u][sum] = t;
        if (w) atomicOr(&sh.gbits[gen % 3u], w);
    }
    team.sync();
#pragma unroll
    for (int k = 0; k < kTagSums; ++k) v[k] = sh.sum[gen & 1u][k];
    bits = sh.gbits[gen % 3u];
    if (threadIdx.x == 0) sh.gbits[(gen + 2u) % 3u] = 0u;
    return sh.fail == 0;
}
__device__ __forceinline__ bool tag_exchange(unsigned char* inbox, int size, int me, unsigned gen, double (&v)[kTagSums],
                                             unsigned& bits, int value_warps, unsigned* flags, TagTeam team, TagShared& sh,
                                             unsigned limit = kTagSpinLimit)
{
    tag_publish(inbox, size, me, gen, v, bits, value_warps, team, sh);
    return tag_finish(inbox, size, me, gen, v, bits, flags, team, sh, limit);
}

// Waits (bounded) until the shared-memory word holds `want`; false when it gave up.
__device__ __forceinline__ bool wait_shared(const int* flag, int want, unsigned long long limit = kBarrierSpinLimit)
{
    for (unsigned long long spins = 0; *(const volatile int*)flag != want; ++spins) {
        if (spins > limit) return false;
        __nanosleep(32);
    }
    __threadfence_block();
    return true;
}

}  // namespace
}  // namespace pk
