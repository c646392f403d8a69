/*
 * engine.cuh -- the typed superstep engine: sm_100a kernels instantiated with
 * the application's IP_* types, its ip_compute and its ip_combine.
 *
 * Versions (selected as in src/iPregel_preamble.h:319-331):
 *   combiner (push)                src/combiner_postamble.h:123-199
 *   single_broadcast (pull)        src/combiner_single_broadcast_postamble.h:125-259
 *   spread (frontier push)         src/combiner_spread_postamble.h:160-431
 *   spread + single_broadcast      src/combiner_spread_single_broadcast_postamble.h:145-399
 *
 * Device layout (structure of arrays, all resident in HBM):
 *   value[V]                       IP_VALUE_TYPE
 *   CSR row[V+1] (u64), adj[E]     the loader's layout; in-CSR for pulls
 *   active / has_message           bitmaps (combiner, written by warp ballot)
 *                                  or bytes (pulls, written by any thread)
 *   mailbox[2][V]                  push: combined message of the superstep,
 *                                  double-buffered by superstep parity
 *   received[2]                    push: bitmap of mailboxes that got mail
 *   outbox[V] + broadcaster bitmap push: ip_broadcast records here; delivery
 *                                  is a separate edge-parallel kernel
 *   bslot[V]                       pull: the externalised broadcast slot of
 *                                  combiner_single_broadcast_preamble.h:42-50,
 *                                  {message, superstep stamp} in 8 or 16 bytes
 * Messages become visible only at the next superstep in every version
 * (combiner_postamble.h:168-183), so recording broadcasts in an outbox and
 * delivering them after the compute kernel gives the reference's results;
 * ip_combine is associative and commutative by contract
 * (iPregel_preamble.h:256-262), so combining in a different order is allowed.
 */
#ifndef IPREGEL_B200_ENGINE_CUH
#define IPREGEL_B200_ENGINE_CUH

#include <cuda_runtime.h>

#include <limits>
#include <type_traits>

typedef IP_VERTEX_ID_TYPE ipx_vid;
typedef IP_MESSAGE_TYPE ipx_msg;
typedef IP_VALUE_TYPE ipx_val;

#ifdef IP_NEEDS_OUT_NEIGHBOUR_WEIGHTS
#define IPX_OUT_WEIGHTS 1
#else
#define IPX_OUT_WEIGHTS 0
#endif
#ifdef IP_NEEDS_IN_NEIGHBOUR_WEIGHTS
#define IPX_IN_WEIGHTS 1
#else
#define IPX_IN_WEIGHTS 0
#endif
#if IPX_OUT_WEIGHTS || IPX_IN_WEIGHTS
typedef IP_EDGE_WEIGHT_TYPE ipx_wgt;
#define IPX_WEIGHT_BYTES ((int)sizeof(IP_EDGE_WEIGHT_TYPE))
#else
typedef unsigned int ipx_wgt;
#define IPX_WEIGHT_BYTES 0
#endif

/* Weighted broadcast (extension, no reference counterpart): an application
 * that defines IP_BROADCAST_EDGE_MESSAGE(m, w) before including iPregel.h
 * makes ip_broadcast deliver IP_BROADCAST_EDGE_MESSAGE(m, weight) along each
 * out-edge (e.g. m + w for SSSP).  The transform must distribute over
 * ip_combine, because two broadcasts of one vertex in one superstep are
 * combined before delivery. */
#ifdef IP_BROADCAST_EDGE_MESSAGE
#define IPX_EDGE_MSG 1
#if !IPX_OUT_WEIGHTS
#error "IP_BROADCAST_EDGE_MESSAGE needs IP_NEEDS_OUT_NEIGHBOUR_WEIGHTS"
#endif
#if IPX_PULL
#error "IP_BROADCAST_EDGE_MESSAGE applies to the combiner and spread versions"
#endif
#else
#define IPX_EDGE_MSG 0
#endif

static_assert(sizeof(ipx_msg) <= 8, "iPregel-B200: IP_MESSAGE_TYPE must be at most 8 bytes");

#define IPX_FULL 0xffffffffu
/* Largest CTA the kernels are compiled for; the launch size is a runtime
 * tuning parameter (a multiple of 32 up to this). */
#define IPX_THREADS 256
/* CTA of the target marking kernel, its shared memory the bits of the most
 * often visited targets (bitmap words of the lowest, that is best connected,
 * vertices). */
#define IPX_MARK_THREADS 1024
#ifndef IPX_MARK_WORDS
#define IPX_MARK_WORDS 1024
#endif
#define IPX_ERR_SEND_IN_BROADCAST 1u
#define IPX_ERR_COMBINE_HINT 2u
#define IPX_ERR_SUPERSTEP_LIMIT 4u
#define IPX_ERR_COPY_TIMEOUT 8u
#define IPX_ERR_RESERVED_MESSAGE 16u
#define IPX_HIST 65536
/* Supersteps the host-driven loop enqueues before it waits for the device. */
#define IPX_BATCH 8

/* Default thresholds of the rows' classes (runtime tuning parameters,
 * ipg_app_set_tuning). */
#ifndef IPX_T0
#define IPX_T0 16
#endif
#ifndef IPX_T1
#define IPX_T1 4096
#endif

/* ------------------------------------------------------------------------ */
/* Mailbox policies: how a push delivers a message into mailbox[w].          */
/* deliver() returns true when the received bit of w may still be clear      */
/* (the CAS policies know exactly: this call filled an empty mailbox; the    */
/* hardware-atomic ones return true whenever they issued an update), and the */
/* caller then sets the bit with a fire-and-forget atomic OR.  Policies with */
/* kPeek let a push look at the slot first: a message that does not win is   */
/* dropped, and only a push that saw the slot empty sets the bit (the first  */
/* to deliver in a superstep always does).                                   */
/* ------------------------------------------------------------------------ */
template <class T>
struct ipx_word {
    typedef typename std::conditional<(sizeof(T) <= 4), unsigned int, unsigned long long>::type type;
};

template <class T>
__device__ __forceinline__ typename ipx_word<T>::type ipx_to_word(const T& x)
{
    typename ipx_word<T>::type w = 0;
    memcpy(&w, &x, sizeof(T));
    return w;
}

template <class T>
__device__ __forceinline__ T ipx_from_word(typename ipx_word<T>::type w)
{
    T x;
    memcpy(&x, &w, sizeof(T));
    return x;
}

/* Bitwise equality: a compute kernel writes a vertex's value back only when
 * ip_compute changed it (unchanged receivers are common in min-propagation
 * supersteps; each skipped store is a dirty sector less). */
template <class T>
__device__ __forceinline__ bool ipx_same_bits(const T& a, const T& b)
{
    if constexpr (sizeof(T) <= 8) {
        return ipx_to_word(a) == ipx_to_word(b);
    } else {
        const unsigned char* p = reinterpret_cast<const unsigned char*>(&a);
        const unsigned char* q = reinterpret_cast<const unsigned char*>(&b);
        for (size_t k = 0; k < sizeof(T); k++)
            if (p[k] != q[k]) return false;
        return true;
    }
}

template <class T>
__device__ __forceinline__ T ipx_shfl_down(T x, int o)
{
    typedef typename ipx_word<T>::type W;
    W w = ipx_to_word(x);
    w = __shfl_down_sync(IPX_FULL, w, o);
    return ipx_from_word<T>(w);
}

/* Read-modify-write by compare-and-swap on the message's bits, for operand
 * types without a hardware atomic of the operator. */
template <class T, class Op>
__device__ __forceinline__ void ipx_atomic_cas_op(T* a, T v, Op op)
{
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "combiner hints need a 4- or 8-byte message type");
    typedef typename std::conditional<sizeof(T) == 4, unsigned int, unsigned long long>::type W;
    W* p = reinterpret_cast<W*>(a);
    W old = *p;
    for (;;) {
        T cur;
        memcpy(&cur, &old, sizeof(T));
        T nv = op(cur, v);
        W nw;
        memcpy(&nw, &nv, sizeof(T));
        if (nw == old) return;
        W prev = atomicCAS(p, old, nw);
        if (prev == old) return;
        old = prev;
    }
}

template <class T>
__device__ __forceinline__ void ipx_atomic_min(T* a, T v)
{
    if constexpr (std::is_unsigned<T>::value && sizeof(T) == 4) atomicMin((unsigned int*)a, (unsigned int)v);
    else if constexpr (std::is_unsigned<T>::value && sizeof(T) == 8) atomicMin((unsigned long long*)a, (unsigned long long)v);
    else if constexpr (std::is_signed<T>::value && std::is_integral<T>::value && sizeof(T) == 4) atomicMin((int*)a, (int)v);
    else if constexpr (std::is_signed<T>::value && std::is_integral<T>::value && sizeof(T) == 8) atomicMin((long long*)a, (long long)v);
    else ipx_atomic_cas_op(a, v, [](T x, T y) { return y < x ? y : x; });
}

template <class T>
__device__ __forceinline__ void ipx_atomic_max(T* a, T v)
{
    if constexpr (std::is_unsigned<T>::value && sizeof(T) == 4) atomicMax((unsigned int*)a, (unsigned int)v);
    else if constexpr (std::is_unsigned<T>::value && sizeof(T) == 8) atomicMax((unsigned long long*)a, (unsigned long long)v);
    else if constexpr (std::is_signed<T>::value && std::is_integral<T>::value && sizeof(T) == 4) atomicMax((int*)a, (int)v);
    else if constexpr (std::is_signed<T>::value && std::is_integral<T>::value && sizeof(T) == 8) atomicMax((long long*)a, (long long)v);
    else ipx_atomic_cas_op(a, v, [](T x, T y) { return y > x ? y : x; });
}

template <class T>
__device__ __forceinline__ void ipx_atomic_add(T* a, T v)
{
    if constexpr (std::is_same<T, double>::value || std::is_same<T, float>::value) atomicAdd(a, v);
    else if constexpr (std::is_integral<T>::value && sizeof(T) == 4) atomicAdd((unsigned int*)a, (unsigned int)v);
    else if constexpr (std::is_integral<T>::value && sizeof(T) == 8) atomicAdd((unsigned long long*)a, (unsigned long long)v);
    else ipx_atomic_cas_op(a, v, [](T x, T y) { return x + y; });
}

/* Read of a mailbox for the precheck of a monotone combiner.  Within a
 * superstep a min (max) mailbox only falls (rises), so a stale read can only
 * let a redundant atomic through, never drop a message: the read may come
 * from L1 (IPX_PRECHECK_L1 = 1, each SM keeps its own copy of hot mailboxes
 * such as the hubs') or from L2 (0, fresher but every read of a hot mailbox
 * lands on one L2 slice). */
#ifndef IPX_PRECHECK_L1
#define IPX_PRECHECK_L1 1
#endif
template <class T>
__device__ __forceinline__ T ipx_peek(const T* p)
{
#if IPX_PRECHECK_L1
    return *p;
#else
    return __ldcg(p);
#endif
}

/* 128-bit compare-and-swap (sm_90+ atom.cas.b128) for the generic 8-byte path. */
struct __align__(16) ipx_slot128 {
    unsigned long long flag;
    unsigned long long bits;
};

__device__ __forceinline__ void ipx_cas128(ipx_slot128* addr, unsigned long long cmp_f, unsigned long long cmp_b,
                                           unsigned long long new_f, unsigned long long new_b,
                                           unsigned long long& old_f, unsigned long long& old_b)
{
    asm volatile(
        "{\n\t"
        ".reg .b128 c, n, o;\n\t"
        "mov.b128 c, {%2, %3};\n\t"
        "mov.b128 n, {%4, %5};\n\t"
        "atom.global.cas.b128 o, [%6], c, n;\n\t"
        "mov.b128 {%0, %1}, o;\n\t"
        "}"
        : "=l"(old_f), "=l"(old_b)
        : "l"(cmp_f), "l"(cmp_b), "l"(new_f), "l"(new_b), "l"(addr)
        : "memory");
}

template <int KIND, int MSGBYTES>
struct ipx_mailbox;

/* Hardware min / max on the message itself (4 or 8 bytes).  The slot holds
 * no flag: whether a vertex received mail is its received bit, which the
 * caller sets whenever deliver/commit return true.  A message equal to the
 * empty value still passes the precheck and so still sets the bit.  Keeping
 * the slot at the message's width halves the mailboxes of 4-byte messages
 * (V x 4 bytes per parity), which then stay in L2 at larger scales. */
struct ipx_mailbox_min {
    typedef ipx_msg slot;
    static constexpr bool kPeek = true;
    __device__ static slot empty() { return std::numeric_limits<ipx_msg>::max(); }
    __device__ static bool fresh(slot c) { return c == empty(); }
    __device__ static bool wins(slot c, ipx_msg m) { return m < c || (m == c && fresh(c)); }
    __device__ static void commit(slot* s, ipx_msg m) { ipx_atomic_min(s, m); }
    __device__ static bool deliver(slot* s, ipx_msg m)
    {
        if (m < __ldcg(s)) ipx_atomic_min(s, m);
        return true;
    }
    __device__ static bool merge(slot* s, ipx_msg m)
    {
        if (m < *s) *s = m;
        return true;
    }
    __device__ static ipx_msg message(const slot& c) { return c; }
};

struct ipx_mailbox_max {
    typedef ipx_msg slot;
    static constexpr bool kPeek = true;
    __device__ static slot empty() { return std::numeric_limits<ipx_msg>::lowest(); }
    __device__ static bool fresh(slot c) { return c == empty(); }
    __device__ static bool wins(slot c, ipx_msg m) { return m > c || (m == c && fresh(c)); }
    __device__ static void commit(slot* s, ipx_msg m) { ipx_atomic_max(s, m); }
    __device__ static bool deliver(slot* s, ipx_msg m)
    {
        if (m > __ldcg(s)) ipx_atomic_max(s, m);
        return true;
    }
    __device__ static bool merge(slot* s, ipx_msg m)
    {
        if (m > *s) *s = m;
        return true;
    }
    __device__ static ipx_msg message(const slot& c) { return c; }
};

template <>
struct ipx_mailbox<IP_COMBINE_MIN, 4> : ipx_mailbox_min {};
template <>
struct ipx_mailbox<IP_COMBINE_MIN, 8> : ipx_mailbox_min {};
template <>
struct ipx_mailbox<IP_COMBINE_MAX, 4> : ipx_mailbox_max {};
template <>
struct ipx_mailbox<IP_COMBINE_MAX, 8> : ipx_mailbox_max {};

template <int MSGBYTES>
struct ipx_mailbox<IP_COMBINE_SUM, MSGBYTES> {
    typedef ipx_msg slot;
    static constexpr bool kPeek = false;
    __device__ static slot empty() { return (ipx_msg)0; }
    __device__ static bool deliver(slot* s, ipx_msg m)
    {
        ipx_atomic_add(s, m);
        return true;
    }
    __device__ static bool merge(slot* s, ipx_msg m)
    {
        *s = *s + m;
        return true;
    }
    __device__ static ipx_msg message(const slot& c) { return c; }
};

/* Generic, up to 4 bytes: {flag, bits} in one 64-bit word, CAS loop around
 * the user's ip_combine with the early exit of ip_cas (combiner_postamble.h:
 * 41-52): no write when combining leaves the mailbox unchanged. */
template <int MSGBYTES>
struct ipx_mailbox_generic32 {
    typedef unsigned long long slot;
    static constexpr bool kPeek = false;
    __device__ static slot empty() { return 0ULL; }
    __device__ static bool deliver(slot* s, ipx_msg m)
    {
        unsigned long long old = __ldcg(s);
        for (;;) {
            unsigned long long nw;
            if (old >> 32) {
                ipx_msg cur = ipx_from_word<ipx_msg>((unsigned int)old);
                ipx_msg nv = cur;
                ip_combine(&nv, m);
                unsigned int nb = ipx_to_word(nv);
                if (nb == (unsigned int)old) return false;
                nw = (1ULL << 32) | nb;
            } else {
                nw = (1ULL << 32) | ipx_to_word(m);
            }
            unsigned long long prev = atomicCAS(s, old, nw);
            if (prev == old) return (old >> 32) == 0;
            old = prev;
        }
    }
    __device__ static bool merge(slot* s, ipx_msg m)
    {
        const unsigned long long old = *s;
        ipx_msg v = m;
        if (old >> 32) {
            v = ipx_from_word<ipx_msg>((unsigned int)old);
            ip_combine(&v, m);
        }
        *s = (1ULL << 32) | ipx_to_word(v);
        return true;
    }
    __device__ static ipx_msg message(const slot& c) { return ipx_from_word<ipx_msg>((unsigned int)c); }
};

template <>
struct ipx_mailbox<IP_COMBINE_GENERIC, 1> : ipx_mailbox_generic32<1> {};
template <>
struct ipx_mailbox<IP_COMBINE_GENERIC, 2> : ipx_mailbox_generic32<2> {};
template <>
struct ipx_mailbox<IP_COMBINE_GENERIC, 4> : ipx_mailbox_generic32<4> {};

/* Generic, 8 bytes: {flag, bits} in a 16-byte slot with a 128-bit CAS. */
template <>
struct ipx_mailbox<IP_COMBINE_GENERIC, 8> {
    typedef ipx_slot128 slot;
    static constexpr bool kPeek = false;
    __device__ static slot empty() { return slot{0ULL, 0ULL}; }
    __device__ static bool deliver(slot* s, ipx_msg m)
    {
        unsigned long long of = __ldcg(&s->flag), ob = __ldcg(&s->bits);
        for (;;) {
            unsigned long long nb;
            if (of) {
                ipx_msg cur = ipx_from_word<ipx_msg>(ob);
                ipx_msg nv = cur;
                ip_combine(&nv, m);
                nb = ipx_to_word(nv);
                if (nb == ob) return false;
            } else {
                nb = ipx_to_word(m);
            }
            unsigned long long pf, pb;
            ipx_cas128(s, of, ob, 1ULL, nb, pf, pb);
            if (pf == of && pb == ob) return of == 0;
            of = pf;
            ob = pb;
        }
    }
    __device__ static bool merge(slot* s, ipx_msg m)
    {
        ipx_msg v = m;
        if (s->flag) {
            v = ipx_from_word<ipx_msg>(s->bits);
            ip_combine(&v, m);
        }
        s->bits = ipx_to_word(v);
        s->flag = 1ULL;
        return true;
    }
    __device__ static ipx_msg message(const slot& c) { return ipx_from_word<ipx_msg>(c.bits); }
};

template <>
struct ipx_mailbox<IP_COMBINE_MIN, 1> : ipx_mailbox_generic32<1> {};
template <>
struct ipx_mailbox<IP_COMBINE_MIN, 2> : ipx_mailbox_generic32<2> {};
template <>
struct ipx_mailbox<IP_COMBINE_MAX, 1> : ipx_mailbox_generic32<1> {};
template <>
struct ipx_mailbox<IP_COMBINE_MAX, 2> : ipx_mailbox_generic32<2> {};

typedef ipx_mailbox<IP_COMBINE_KIND, (int)sizeof(ipx_msg)> ipx_mb;
typedef typename ipx_mb::slot ipx_slot;

/* ------------------------------------------------------------------------ */
/* Pull broadcast slot.  The reference keeps {has_broadcast, message} per    */
/* vertex (combiner_single_broadcast_preamble.h:42-50) and clears the flags  */
/* every superstep.  Here a slot holds the message's bits and the superstep  */
/* in which it was broadcast: it counts in superstep s iff its stamp is s,   */
/* so no slot is ever cleared, and a gathered edge costs one 8-byte (message */
/* up to 4 bytes) or 16-byte (up to 8 bytes) load -- one L2 request -- where */
/* a flag bitmap costs a dependent bitmap-word load before the value.        */
/* ------------------------------------------------------------------------ */
typedef typename std::conditional<(sizeof(ipx_msg) <= 4), uint2, uint4>::type ipx_bslot;
/* Stamp of a slot that holds no broadcast (all bytes 0xff after a reset);
 * supersteps stay below it (ipx_max_supersteps). */
#define IPX_NO_STAMP 0xffffffffu

__device__ __forceinline__ void ipx_bslot_store(uint2* p, unsigned long long w, uint32_t stamp)
{
    *p = make_uint2((uint32_t)w, stamp);
}
__device__ __forceinline__ void ipx_bslot_store(uint4* p, unsigned long long w, uint32_t stamp)
{
    *p = make_uint4((uint32_t)w, (uint32_t)(w >> 32), stamp, 0u);
}
__device__ __forceinline__ unsigned long long ipx_bslot_bits(const uint2& w) { return w.x; }
__device__ __forceinline__ unsigned long long ipx_bslot_bits(const uint4& w)
{
    return ((unsigned long long)w.y << 32) | w.x;
}
__device__ __forceinline__ uint32_t ipx_bslot_stamp(const uint2& w) { return w.y; }
__device__ __forceinline__ uint32_t ipx_bslot_stamp(const uint4& w) { return w.z; }

/* A slot that holds no broadcast. */
__device__ __forceinline__ ipx_bslot make_ipx_nobslot()
{
    ipx_bslot w;
    memset(&w, 0xff, sizeof w);
    return w;
}

__device__ __forceinline__ void ipx_bslot_put(ipx_bslot* p, const ipx_msg& m, uint32_t stamp)
{
    ipx_bslot_store(p, (unsigned long long)ipx_to_word(m), stamp);
}

/* The message of a loaded slot; true when it was broadcast in superstep
 * `stamp`. */
__device__ __forceinline__ bool ipx_bslot_take(const ipx_bslot& w, uint32_t stamp, ipx_msg& m)
{
    m = ipx_from_word<ipx_msg>((typename ipx_word<ipx_msg>::type)ipx_bslot_bits(w));
    return ipx_bslot_stamp(w) == stamp;
}

/* The single_broadcast version with FP64 messages (PageRank) keeps 8-byte
 * slots without a stamp: its fused kernel visits every vertex each
 * superstep and writes every slot of the next buffer -- the broadcast, or
 * IPX_ABSENT64 when the vertex does not broadcast -- so a slot never holds
 * a message of an older superstep.  IPX_ABSENT64 (all bits set) is a NaN
 * that FP64 arithmetic does not produce; a broadcast of exactly that bit
 * pattern is reported as an error (IPX_ERR_RESERVED_MESSAGE).  Half the
 * bytes of a stamped 16-byte slot: twice as many vertices' slots fit in the
 * L2.  Other message types keep stamped slots. */
#ifndef IPX_SB_DENSE
#define IPX_SB_DENSE 1
#endif
#define IPX_ABSENT64 0xffffffffffffffffULL
typedef typename std::conditional<(IPX_SB_DENSE && std::is_same<ipx_msg, double>::value), unsigned long long,
                                  ipx_bslot>::type ipx_sbslot;

__device__ __forceinline__ bool ipx_slot_take(const ipx_bslot& w, uint32_t stamp, ipx_msg& m)
{
    return ipx_bslot_take(w, stamp, m);
}
__device__ __forceinline__ bool ipx_slot_take(const unsigned long long& w, uint32_t, ipx_msg& m)
{
    m = ipx_from_word<ipx_msg>((typename ipx_word<ipx_msg>::type)w);
    return w != IPX_ABSENT64;
}
template <class S>
__device__ __forceinline__ S ipx_no_slot()
{
    S w;
    memset(&w, 0xff, sizeof w);
    return w;
}

/* ---- L2 eviction policies for the gathered slots ----
 * The slots of a few million often-gathered vertices would fit the L2, but
 * the gather's cold accesses (most vertices are gathered a few times per
 * superstep) evict them.  The single_broadcast version can gather from a
 * copy of the in-lists whose ids carry a flag in bit 31 for the vertices
 * gathered most often (ipx_consts::in_adj_hot, built at attach): their
 * slots are loaded evict-last, all others evict-first. */
#define IPX_HOT_BIT 0x80000000u
__device__ __forceinline__ uint64_t ipx_policy(bool hot)
{
    uint64_t p;
    if (hot) asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    else asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ unsigned long long ipx_ld_policy(const unsigned long long* p, uint64_t pol)
{
    unsigned long long r;
    asm volatile("ld.global.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(pol));
    return r;
}
__device__ __forceinline__ uint2 ipx_ld_policy(const uint2* p, uint64_t pol)
{
    uint2 r;
    asm volatile("ld.global.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;" : "=r"(r.x), "=r"(r.y) : "l"(p), "l"(pol));
    return r;
}
__device__ __forceinline__ uint4 ipx_ld_policy(const uint4* p, uint64_t pol)
{
    uint4 r;
    asm volatile("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p), "l"(pol));
    return r;
}
/* The slot of the in-neighbour whose id word is w: HOT ids carry the flag.
 * Slots, mailboxes, messages, bitmaps and lists are written by the kernel before,
 * which may still run when this one's CTAs come onto the SMs (ipx_done): they are
 * read by ordinary loads, not through the read-only path (__ldg, ld.global.nc),
 * which is for what nothing writes while the grid exists, and their pointers are
 * not declared __restrict__. */
template <bool HOT, class S>
__device__ __forceinline__ S ipx_slot_ld(const S* bs, uint64_t w)
{
    if constexpr (HOT) {
        return ipx_ld_policy(&bs[w & (IPX_HOT_BIT - 1u)], ipx_policy((w & IPX_HOT_BIT) != 0));
    } else {
        return bs[w];
    }
}

/* ------------------------------------------------------------------------ */
/* Device-resident engine state, read through the constant bank.            */
/* ------------------------------------------------------------------------ */
/* What a superstep's kernels count: zeroed by the superstep's end.  n:
 * broadcasters listed in the three row classes and the chunks of the hubs;
 * tn: spread+single_broadcast's targets by class; edges / tedges: the degree
 * sums (hubs last). */
struct ipx_stat {
    unsigned long long count;
    unsigned long long edges[4];
    unsigned long long tedges[3];
    uint32_t n[4];
    uint32_t tn[4];
};

struct ipx_consts {
    uint64_t V, E, W;  /* W = bitmap words */
    const uint64_t* row;
    const ipx_vid* adj;
    const ipx_wgt* wgt;
    const uint64_t* in_row;
    const ipx_vid* in_adj;
    const ipx_wgt* in_wgt;
    ipx_val* value;
    /* combiner */
    uint32_t* active_bm;
    uint32_t* hasmsg_bm;
    /* pulls */
    uint8_t* active_b;
    uint8_t* hasmsg_b;
    ipx_msg* msg;
    /* push mail */
    ipx_slot* mbox[2];
    uint32_t* recv[2];
    ipx_msg* outbox;
    uint32_t* bcaster; /* pulling push versions only */
    /* pull broadcast slots: single_broadcast alternates bslot[s & 1] (its
     * fused kernel reads superstep s's slots while writing s+1's);
     * spread+single_broadcast uses bslot[0] */
    ipx_bslot* bslot[2];
    ipx_sbslot* sbslot[2];
    uint32_t* bt;
    /* this superstep's counts, and a copy of the last one's */
    ipx_stat* stat;
    ipx_stat* last;
    /* control words (IPX_CTL_*) */
    unsigned long long* ctl;
    uint32_t* err;
    /* direction optimisation (push versions on symmetric graphs): pull when
     * the broadcasters' out-edges exceed pull_threshold */
    int pull_ok;
    unsigned long long pull_threshold;
    /* broadcasters by row length, and the hubs' chunks {vertex, chunk}: rows
     * up to push_t[0] take a thread, up to push_t[1] 8 lanes, up to push_t[2]
     * 32 lanes, longer ones a warp per push_chunk edges */
    uint32_t* blist[3];
    uint2* bchunk;
    uint64_t push_t[3];
    uint32_t push_chunk;
    /* ids (and 4-byte weights) can be read in whole aligned groups of four */
    int out_quads, in_quads;
    /* spread+single_broadcast: targets by in-degree class */
    uint32_t* tlist[3];
    /* per superstep a record of hist[s % IPX_HIST]: active count, edges
     * traversed, direction | error word << 32, nanoseconds */
    unsigned long long* hist;
    /* single_broadcast, and pulling push versions: the vertices by in-degree
     * class (short, middle and long rows, the hubs among the long ones; their
     * numbers in class_n), and the hubs (rows above hub_min, ipg_graph_hubs)
     * {vertex, first chunk, chunks} with, per chunk, the index of its hub;
     * single_broadcast also per chunk the partial fold ({message, has} in a
     * slot, has in the stamp word) and per hub the chunks arrived */
    const uint32_t* class_list[3];
    uint32_t class_n[3];
    const uint4* hub;
    ipx_bslot* hub_part;
    uint32_t* hub_arrived;
    uint64_t hub_min;
    uint32_t chunks, hub_chunk;
    const uint32_t* hub_owner;
    /* the in-lists with the flag of the most gathered vertices (null: none) */
    const uint32_t* in_adj_hot;
    /* The kernels run on a degree-ordered copy of the graph: vid_of[v] is
     * the id of vertex v in the caller's numbering, vindex_of its inverse
     * (both null when the graph is not renamed). */
    const uint32_t* vid_of;
    const uint32_t* vindex_of;
    /* the caller's graph, whose row vid_of[v] holds the same edges in the
     * same order as row v of the copy: the neighbour ids ip_compute reads
     * (null when not renamed) */
    const uint64_t* user_row;
    const ipx_vid* user_adj;
    const uint64_t* user_in_row;
    const ipx_vid* user_in_adj;
};

__constant__ ipx_consts ipx_c;

/* The id ip_compute sees for vertex v (the caller's numbering). */
__device__ __forceinline__ ipx_vid ipx_user_id(uint64_t v)
{
    return (ipx_vid)(ipx_c.vid_of ? (uint64_t)__ldg(&ipx_c.vid_of[v]) : v);
}

/* The current superstep, from device memory: each superstep's last kernel
 * advances it, so every kernel of a superstep reads the same value.  A plain
 * load, like the end flag's below: a kernel may have started before the value
 * was written (ipx_done). */
__device__ __forceinline__ uint64_t ipx_step() { return (uint64_t)ipd_superstep; }
__device__ __forceinline__ int ipx_parity() { return (int)(ipx_step() & 1); }

/* Control words: the error word, "the program has ended" (the kernels of
 * supersteps enqueued beyond it return at once), CTAs of the last kernel
 * that are done, and the time stamp of the last superstep's end. */
enum { IPX_CTL_ERR, IPX_CTL_DONE, IPX_CTL_ARRIVED, IPX_CTL_STAMP, IPX_NCTL };
/* step: the kernel runs functions of the application (ip_compute, ip_combine,
 * the edge's message), which may ask for the superstep. */
__device__ __forceinline__ bool ipx_done(bool step = true)
{
    /* lets the next kernel's CTAs onto the SMs as this one's leave them, and
     * waits for the one before; each kernel of a superstep begins with it */
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
    const bool done = ipx_c.ctl[IPX_CTL_DONE] != 0ULL;
    if (step) {
        if (threadIdx.x == 0) ipx_step_word() = ipd_compute_superstep;
        __syncthreads();
    }
    return done;
}

/* Kernel ids for launch counting and per-kernel profiling. */
enum {
    IPX_K_COMPUTE,
    IPX_K_PUSH,
    IPX_K_COMPACT_T,
    IPX_K_GATHER,
    IPX_K_GATHER_HUBS,
    IPX_K_MARK,
    IPX_K_COUNT,
    IPX_K_PULLD,
    IPX_K_N
};
static const char* const ipx_kname[IPX_K_N] = {
    "compute", "push", "compact_targets", "gather", "gather_hubs", "mark", "count_active",
    "pull_deliver"};

__device__ __forceinline__ uint64_t ipx_gtid() { return blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint64_t ipx_gstride() { return (uint64_t)gridDim.x * blockDim.x; }
__device__ __forceinline__ bool ipx_test(const uint32_t* bm, uint64_t v) { return (bm[v >> 5] >> (v & 31)) & 1u; }

/* Load of an edge stream element (neighbour id, weight).  A superstep reads
 * each edge once, and the streams are gigabytes, so they are loaded
 * evict-first (ld.global.cs): the L2 stays with the vertex arrays that edges
 * read at random (mailboxes, broadcast values, bitmaps). */
template <class T>
__device__ __forceinline__ T ipx_ld_stream(const T* p)
{
    T r;
    if constexpr (sizeof(T) == 8) {
        const unsigned long long w = __ldcs(reinterpret_cast<const unsigned long long*>(p));
        memcpy(&r, &w, 8);
    } else if constexpr (sizeof(T) == 4) {
        const unsigned int w = __ldcs(reinterpret_cast<const unsigned int*>(p));
        memcpy(&r, &w, 4);
    } else if constexpr (sizeof(T) == 2) {
        const unsigned short w = __ldcs(reinterpret_cast<const unsigned short*>(p));
        memcpy(&r, &w, 2);
    } else if constexpr (sizeof(T) == 1) {
        const unsigned char w = __ldcs(reinterpret_cast<const unsigned char*>(p));
        memcpy(&r, &w, 1);
    } else {
        r = *p;
    }
    return r;
}

/* Edge element read by a loop whose lanes take every lanes-th edge: evict-
 * first only when a warp reads consecutive edges in one instruction (lanes
 * >= 32).  A thread walking a short row alone (lanes = 1) comes back to the
 * same line in its next steps, and an evict-first line is often gone by
 * then (measured: more DRAM traffic and a slower thread class). */
template <class T>
__device__ __forceinline__ T ipx_ld_edge(const T* p, uint64_t lanes)
{
    return lanes >= 32 ? ipx_ld_stream(p) : *p;
}

/* Sets bit v of a shared bitmap; lanes that hit the same word combine first. */
__device__ __forceinline__ void ipx_set_bit_agg(uint32_t* bm, uint64_t v)
{
    const unsigned act = __activemask();
    const unsigned long long word = v >> 5;
    const unsigned peers = __match_any_sync(act, word);
    const unsigned bits = __reduce_or_sync(peers, 1u << (v & 31));
    if ((threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) atomicOr(&bm[word], bits);
}

/* Warp + block sum into a global counter (all threads of the block call). */
__device__ __forceinline__ void ipx_block_count(unsigned long long c, unsigned long long* dst)
{
    __shared__ unsigned long long s_part[IPX_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(IPX_FULL, c, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s_part[w];
        if (t) atomicAdd(dst, t);
    }
}

/* The loop the kernels run in: a captured one continues by its condition.
 * starts: the superstep is the first that the host enqueued after a wait, and is
 * timed from its own first kernel, not from the end of the one before. */
struct ipx_loop {
    cudaGraphConditionalHandle handle;
    int captured;
    int starts;
    unsigned long long max_supersteps;
};

/* True in one CTA, the last of the grid to get here, with every other CTA's
 * writes visible (all threads of every CTA call it, after their last write). */
__device__ __forceinline__ bool ipx_last_cta()
{
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned int n = atomicInc((unsigned int*)&ipx_c.ctl[IPX_CTL_ARRIVED], gridDim.x - 1);
        s_last = n == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    return s_last;
}

__device__ __forceinline__ unsigned long long ipx_now()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void ipx_start_clock(bool starts)
{
    if (starts && blockIdx.x == 0 && threadIdx.x == 0) ipx_c.ctl[IPX_CTL_STAMP] = ipx_now();
}

/* Direction of the superstep's delivery (push versions). */
__device__ __forceinline__ bool ipx_pulls()
{
    if (!ipx_c.pull_ok) return false;
    unsigned long long m = 0;
    for (int k = 0; k < 4; k++) m += __ldcg(&ipx_c.stat->edges[k]);
    return m > ipx_c.pull_threshold;
}

/* End of a superstep, by one thread after everything else of it: records
 * the superstep in the history, advances to the next and decides whether
 * the program goes on: while the count is nonzero (combiner_postamble.h:134;
 * spread versions test it after superstep 0, combiner_spread_postamble.h:
 * 212), no kernel reported an error and the superstep bound is not reached. */
__device__ __forceinline__ void ipx_end_of_superstep(const ipx_loop& loop, unsigned long long count)
{
    const uint64_t s = ipx_step();
    ipx_stat* st = ipx_c.stat;
    ipx_stat x;
    x.count = count;
    unsigned long long edges = 0;
    for (int k = 0; k < 4; k++) edges += x.edges[k] = __ldcg(&st->edges[k]);
    bool pulled = false;
#if IPX_VERSION == IPX_SINGLE_BROADCAST
    edges = ipx_c.E;
#else
    pulled = ipx_c.pull_ok && edges > ipx_c.pull_threshold;
    if (pulled) edges = ipx_c.E; /* a pulled superstep reads every row */
#endif
    for (int k = 0; k < 3; k++) edges += x.tedges[k] = __ldcg(&st->tedges[k]);
    for (int k = 0; k < 4; k++) {
        x.n[k] = __ldcg(&st->n[k]);
        x.tn[k] = __ldcg(&st->tn[k]);
    }
    *ipx_c.last = x;
    memset(st, 0, sizeof *st);
    bool go = count != 0 && __ldcg(ipx_c.err) == 0;
    if (go && s + 1 >= loop.max_supersteps) {
        atomicOr(ipx_c.err, IPX_ERR_SUPERSTEP_LIMIT);
        go = false;
    }
    const unsigned long long now = ipx_now(), then = __ldcg(&ipx_c.ctl[IPX_CTL_STAMP]);
    ipx_c.ctl[IPX_CTL_STAMP] = now;
    unsigned long long* h = ipx_c.hist + (s % IPX_HIST) * 4;
    h[0] = count;
    h[1] = edges;
    h[2] = (pulled ? 1ULL : 0ULL) | ((unsigned long long)__ldcg(ipx_c.err) << 32);
    h[3] = now > then ? now - then : 0ULL;
    ipd_superstep = s + 1;
#if IPX_VERSION == IPX_SINGLE_BROADCAST
    /* the fused kernel of superstep s + 1 runs the compute phase of s + 2 */
    ipd_compute_superstep = s + 2;
#else
    ipd_compute_superstep = s + 1;
#endif
    if (!go) ipx_c.ctl[IPX_CTL_DONE] = 1ULL;
    if (loop.captured) cudaGraphSetConditional(loop.handle, go ? 1u : 0u);
}

/* Delivery of one message into mailbox parity p of vertex w. */
__device__ __forceinline__ void ipx_deliver(int p, uint64_t w, ipx_msg m)
{
    if (ipx_mb::deliver(&ipx_c.mbox[p][w], m)) atomicOr(&ipx_c.recv[p][w >> 5], 1u << (w & 31));
}

/* Edges per chunk of a hub's row at most (fewer on small graphs) in push, mark
 * and pull delivery, where a warp takes a chunk: one hub does not leave a single warp working after the
 * others have finished. */
#ifndef IPX_HUB_CHUNK
#define IPX_HUB_CHUNK 2048
#endif
/* Lanes per row of the middle and the long class of push and mark, and the
 * longest middle row.  CC / weighted SSSP, undirected R-MAT scale 24, ms of
 * push a run: 8 and 32 lanes 4.6 / 6.9, 8 and 16 5.0 / 8.0, 16 and 32 4.5 / 6.6
 * against 4.4 / 6.4 for 8 and 32 with the compute kernel's later lists; middle
 * rows up to 32 or 128 edges within 2 % of 64. */
#ifndef IPX_PUSH_GROUP
#define IPX_PUSH_GROUP 8
#endif
#ifndef IPX_PUSH_LONG
#define IPX_PUSH_LONG 32
#endif
#ifndef IPX_PUSH_MID
#define IPX_PUSH_MID 64
#endif
/* 1: the hub class of the fused pull kernel takes a warp per chunk instead
 * of a CTA (no CTA-wide barriers per chunk); 0: a CTA per chunk, its ids
 * staged in shared memory (IPX_HUB_SMEM).  On directed R-MAT scale 25
 * (FP64 PageRank, 30 rounds) a warp per 4,096-edge chunk took 109 ms (8,192:
 * 105.9 ms), a CTA per 2,048-edge chunk, staged or not, 118.7 ms: the CTA
 * version waits at two barriers per chunk. */
#ifndef IPX_HUB_WARP
#define IPX_HUB_WARP 1
#endif
/* Most in-edges per chunk of the single_broadcast gather's hubs (a warp's
 * with IPX_HUB_WARP, fewer on small graphs; 2,048 for a CTA's: the staging
 * buffers of larger chunks do not fit the 48 KB of static shared memory). */
#ifndef IPX_GATHER_CHUNK
#if IPX_HUB_WARP
#define IPX_GATHER_CHUNK 8192
#else
#define IPX_GATHER_CHUNK 2048
#endif
#endif
#ifndef IPX_UNROLL
#define IPX_UNROLL 4
#endif
template <class T>
__device__ __forceinline__ T ipx_shfl_idx(T x, int src)
{
    typedef typename ipx_word<T>::type W;
    W w = ipx_to_word(x);
    w = __shfl_sync(IPX_FULL, w, src);
    return ipx_from_word<T>(w);
}

/* ------------------------------------------------------------------------ */
/* Row walks: G lanes per row, each lane four consecutive edges per step.    */
/* ------------------------------------------------------------------------ */

/* Edges of a row; no row but a hub's comes near the limit. */
__device__ __forceinline__ uint32_t ipx_row_edges(uint64_t r0, uint64_t r1)
{
    return r1 - r0 < 0x7fffffffull ? (uint32_t)(r1 - r0) : 0x7fffffffu;
}

/* The aligned four words at position rel (a multiple of 4) from row start r0
 * rounded down to one: which of them belong to the row of deg edges is
 * decided when they are used, so that nothing waits for the load before. */
__device__ __forceinline__ uint4 ipx_ld_quad(const uint32_t* __restrict__ a, uint64_t r0, uint32_t deg, uint32_t rel)
{
    const uint32_t off = (uint32_t)r0 & 3u;
    return __ldcs(reinterpret_cast<const uint4*>(a + (rel < off + deg ? r0 - off + rel : 0)));
}

/* A visitor gets up to four edges at once: edge index e + k, target w[k],
 * ok[k] (the lane holds an edge), the source's message m. */

/* Push: looks at four mailboxes before committing to any. */
struct ipx_push_visit {
    static constexpr bool kNeedsMessage = true;
    int p;
    template <class MB = ipx_mb>
    __device__ __forceinline__ void deliver(const ipx_vid* w, const bool* ok, const ipx_msg* mk) const
    {
        ipx_slot* box = ipx_c.mbox[p];
        if constexpr (MB::kPeek) {
            ipx_slot c[4];
#pragma unroll
            for (int k = 0; k < 4; k++) c[k] = ok[k] ? ipx_peek(&box[(uint64_t)w[k]]) : MB::empty();
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (ok[k] && MB::wins(c[k], mk[k])) {
                    const uint64_t t = (uint64_t)w[k];
                    MB::commit(&box[t], mk[k]);
                    if (MB::fresh(c[k])) atomicOr(&ipx_c.recv[p][t >> 5], 1u << (t & 31));
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint64_t t = (uint64_t)w[k];
                if (ok[k] && MB::deliver(&box[t], mk[k])) atomicOr(&ipx_c.recv[p][t >> 5], 1u << (t & 31));
            }
        }
    }
    /* Weighted broadcasts take the quad's weights the way its ids came. */
    __device__ __forceinline__ void unpack(const uint4& q, uint64_t r0, uint32_t deg, uint32_t rel, const ipx_msg& m,
                                           ipx_vid* w, bool* ok, ipx_msg* mk) const
    {
        const uint32_t t = rel - ((uint32_t)r0 & 3u); /* edge of the row; before its first: wraps */
        const uint32_t id[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            w[k] = (ipx_vid)id[k];
            ok[k] = t + k < deg;
            mk[k] = m;
        }
#if IPX_EDGE_MSG
        if constexpr (sizeof(ipx_wgt) == 4) {
            const uint4 x = ipx_ld_quad(reinterpret_cast<const uint32_t*>(ipx_c.wgt), r0, deg, rel);
            const uint32_t xk[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                ipx_wgt y;
                memcpy(&y, &xk[k], 4);
                mk[k] = IP_BROADCAST_EDGE_MESSAGE(m, y);
            }
        } else {
            const uint64_t e = r0 - ((uint32_t)r0 & 3u) + rel;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (ok[k]) mk[k] = IP_BROADCAST_EDGE_MESSAGE(m, ipx_ld_stream(&ipx_c.wgt[e + k]));
        }
#endif
    }
    __device__ __forceinline__ void quad(const uint4& q, uint64_t r0, uint32_t deg, uint32_t rel, const ipx_msg& m) const
    {
        ipx_vid w[4];
        bool ok[4];
        ipx_msg mk[4];
        unpack(q, r0, deg, rel, m, w, ok, mk);
        deliver(w, ok, mk);
    }
    __device__ __forceinline__ void edges(const ipx_vid* w, const bool* ok, uint64_t e, uint64_t lanes, const ipx_msg& m) const
    {
        ipx_msg mk[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
#if IPX_EDGE_MSG
            mk[k] = ok[k] ? IP_BROADCAST_EDGE_MESSAGE(m, ipx_ld_edge(&ipx_c.wgt[e + k * lanes], lanes)) : m;
#else
            (void)e;
            (void)lanes;
            mk[k] = m;
#endif
        }
        deliver(w, ok, mk);
    }
};

/* Target marking (spread+single_broadcast).  Targets below `bits` have a bit
 * in the CTA's shared memory too, set at the CTA's first visit: a hub is hit
 * by a large part of all edges, and without it every hit would read (or, from
 * a stale L1 line, set) the same word of the L2.  Few targets are hubs: with
 * the bits of 1.3 M vertices (160 KiB, which leaves room for one CTA and little
 * L1) CC at R-MAT scale 22 / 24 took 3.74 / 13.0 ms, with 512 k 3.67 / 12.9,
 * with 32 k 3.50 / 12.7, and with 32 k and two CTAs per SM 3.13 / 10.8, the
 * latency of the other targets' words being what is left.  16 k bits do as
 * well; CTAs of 256 or 512 threads take 1 to 3 % more. */
struct ipx_mark_visit {
    static constexpr bool kNeedsMessage = false;
    uint32_t* seen;
    uint64_t bits;
    __device__ __forceinline__ void four(const ipx_vid* w, const bool* ok) const
    {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (!ok[k]) continue;
            const uint64_t t = (uint64_t)w[k];
            const uint32_t bit = 1u << (t & 31);
            if (t < bits) {
                if (seen[t >> 5] & bit) continue;
                if (atomicOr(&seen[t >> 5], bit) & bit) continue;
            }
            if (!(ipx_c.bt[t >> 5] & bit)) atomicOr(&ipx_c.bt[t >> 5], bit);
        }
    }
    __device__ __forceinline__ void quad(const uint4& q, uint64_t r0, uint32_t deg, uint32_t rel, const ipx_msg&) const
    {
        const uint32_t t = rel - ((uint32_t)r0 & 3u);
        const ipx_vid w[4] = {(ipx_vid)q.x, (ipx_vid)q.y, (ipx_vid)q.z, (ipx_vid)q.w};
        const bool ok[4] = {t < deg, t + 1 < deg, t + 2 < deg, t + 3 < deg};
        four(w, ok);
    }
    __device__ __forceinline__ void edges(const ipx_vid* w, const bool* ok, uint64_t, uint64_t, const ipx_msg&) const
    {
        four(w, ok);
    }
};

/* Edges [e0, e1) of one source, lane-strided: ids without 128-bit loads
 * (64-bit ids; a caller's unaligned or unpadded array). */
template <class Visit>
__device__ __forceinline__ void ipx_edges_strided(const ipx_vid* __restrict__ adj, uint64_t e0, uint64_t e1,
                                                  uint64_t lane, uint64_t lanes, const ipx_msg& m, const Visit& visit)
{
    for (uint64_t e = e0 + lane; e < e1; e += 4 * lanes) {
        ipx_vid w[4];
        bool ok[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            ok[k] = e + k * lanes < e1;
            w[k] = ok[k] ? ipx_ld_edge(&adj[e + k * lanes], lanes) : (ipx_vid)0;
        }
        visit.edges(w, ok, e, lanes, m);
    }
}

/* The out-edges of a list's sources, G lanes each.  The chain list entry ->
 * row bounds and message -> ids -> mailboxes is pipelined over the group's
 * next sources, as in the pull gather. */
template <int G, class Visit>
__device__ __forceinline__ void ipx_walk_rows(const uint32_t* list, uint32_t n, const Visit& visit)
{
    const uint32_t gl = threadIdx.x & (G - 1);
    const uint64_t* __restrict__ row = ipx_c.row;
    const uint64_t step = ipx_gstride() / G;
    uint64_t i = ipx_gtid() / G;
    if (i >= n) return;
    if (!ipx_c.out_quads) {
        for (; i < n; i += step) {
            const uint64_t u = list[i];
            ipx_msg m = ipx_msg();
            if constexpr (Visit::kNeedsMessage) m = ipx_c.outbox[u];
            ipx_edges_strided(ipx_c.adj, row[u], row[u + 1], gl, G, m, visit);
        }
        return;
    }
    if constexpr (sizeof(ipx_vid) == 4) {
        const uint32_t* __restrict__ adj = reinterpret_cast<const uint32_t*>(ipx_c.adj);
        /* a: the row being walked, b: the next, c: the one after it; past the
         * list's end vertex 0 stands in: loaded, never walked */
        uint32_t ua = list[i], ub = i + step < n ? list[i + step] : 0u, uc = i + 2 * step < n ? list[i + 2 * step] : 0u;
        uint64_t a0 = row[ua], b0 = row[ub];
        uint32_t ad = ipx_row_edges(a0, row[ua + 1]), bd = ipx_row_edges(b0, row[ub + 1]);
        ipx_msg ma = ipx_msg(), mb = ipx_msg(), mc = ipx_msg();
        if constexpr (Visit::kNeedsMessage) {
            ma = ipx_c.outbox[ua];
            mb = ipx_c.outbox[ub];
        }
        uint4 qa = ipx_ld_quad(adj, a0, ad, 4 * gl);
        for (; i < n; i += step) {
            const uint32_t ud = i + 3 * step < n ? list[i + 3 * step] : 0u;
            const uint64_t c0 = row[uc], c1 = row[uc + 1];
            if constexpr (Visit::kNeedsMessage) mc = ipx_c.outbox[uc];
            const uint4 qb = ipx_ld_quad(adj, b0, bd, 4 * gl);
            const uint32_t len = ((uint32_t)a0 & 3u) + ad;
            for (uint32_t rel = 4 * gl;;) {
                const uint4 next = ipx_ld_quad(adj, a0, ad, rel + 4 * G);
                visit.quad(qa, a0, ad, rel, ma);
                rel += 4 * G;
                if (rel >= len) break;
                qa = next;
            }
            uc = ud;
            a0 = b0;
            ad = bd;
            ma = mb;
            b0 = c0;
            bd = ipx_row_edges(c0, c1);
            mb = mc;
            qa = qb;
        }
    }
}

/* The chunks of the hubs among the sources, a warp each. */
template <class Visit>
__device__ __forceinline__ void ipx_walk_chunks(uint32_t n, const Visit& visit)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = ipx_gstride() >> 5, chunk = ipx_c.push_chunk;
    for (uint64_t c = ipx_gtid() >> 5; c < n; c += warps) {
        const uint2 h = ipx_c.bchunk[c];
        const uint64_t e0 = ipx_c.row[h.x] + h.y * chunk, end = ipx_c.row[h.x + 1];
        const uint64_t e1 = e0 + chunk < end ? e0 + chunk : end;
        ipx_msg m = ipx_msg();
        if constexpr (Visit::kNeedsMessage) m = ipx_c.outbox[h.x];
        if (!ipx_c.out_quads) {
            ipx_edges_strided(ipx_c.adj, e0, e1, lane, 32, m, visit);
            continue;
        }
        if constexpr (sizeof(ipx_vid) == 4) {
            const uint32_t* __restrict__ adj = reinterpret_cast<const uint32_t*>(ipx_c.adj);
            const uint32_t deg = (uint32_t)(e1 - e0), len = ((uint32_t)e0 & 3u) + deg;
            uint4 q = ipx_ld_quad(adj, e0, deg, 4 * lane);
            for (uint32_t rel = 4 * lane; rel < len; rel += 128) {
                const uint4 next = ipx_ld_quad(adj, e0, deg, rel + 128);
                visit.quad(q, e0, deg, rel, m);
                q = next;
            }
        }
    }
}

/* All of a superstep's broadcasters, the longest work items first. */
template <class Visit>
__device__ __forceinline__ void ipx_walk_broadcasters(const Visit& visit)
{
    const ipx_stat* st = ipx_c.stat;
    ipx_walk_chunks(__ldcg(&st->n[3]), visit);
    ipx_walk_rows<IPX_PUSH_LONG>(ipx_c.blist[2], __ldcg(&st->n[2]), visit);
    ipx_walk_rows<IPX_PUSH_GROUP>(ipx_c.blist[1], __ldcg(&st->n[1]), visit);
    ipx_walk_rows<1>(ipx_c.blist[0], __ldcg(&st->n[0]), visit);
}

/* ---- the flagged in-lists of the single_broadcast gather (attach time) ---- */
/* cnt[u] += 1 for every occurrence of u in the in-lists. */
__global__ void ipx_k_count_occurrences(const uint32_t* __restrict__ adj, uint64_t E, uint32_t* __restrict__ cnt)
{
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(&cnt[adj[e]], 1u);
}

/* hist[b] = vertices whose occurrence count has b significant bits. */
__global__ void ipx_k_count_hist(const uint32_t* __restrict__ cnt, uint64_t V, unsigned long long* __restrict__ hist)
{
    __shared__ unsigned int h[33];
    if (threadIdx.x < 33) h[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(&h[32 - __clz(cnt[v])], 1u);
    __syncthreads();
    if (threadIdx.x < 33 && h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], (unsigned long long)h[threadIdx.x]);
}

/* out[e] = adj[e], with IPX_HOT_BIT set when that vertex occurs at least
 * `threshold` times in the in-lists. */
__global__ void ipx_k_flag_hot(const uint32_t* __restrict__ adj, uint64_t E, const uint32_t* __restrict__ cnt,
                               uint32_t threshold, uint32_t* __restrict__ out)
{
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t u = adj[e];
        out[e] = u | (cnt[u] >= threshold ? IPX_HOT_BIT : 0u);
    }
}

/* ---- the vertex functions that depend on the version ---- */
__device__ inline void ip_broadcast(struct ip_vertex_t* v, IP_MESSAGE_TYPE message)
{
#if IPX_PULL
    /* single_broadcast: write the vertex's own slot (combiner_single_broadcast_
     * postamble.h:51-55); spread+single_broadcast also flags the out-neighbours
     * as targets (combiner_spread_single_broadcast_postamble.h:64-76), which the
     * engine does after the compute kernel. */
    v->ipx_has_out = true;
    v->ipx_out = message;
#else
    /* combiner / spread: every out-neighbour receives the message
     * (combiner_postamble.h:81-87); two broadcasts in one call are combined. */
    if (v->ipx_has_out) {
        ip_combine(&v->ipx_out, message);
    } else {
        v->ipx_has_out = true;
        v->ipx_out = message;
    }
#endif
}

__device__ inline void ip_send_message(IP_VERTEX_ID_TYPE id, IP_MESSAGE_TYPE message)
{
#if IPX_PULL
    /* Fatal in the single-broadcast versions (combiner_single_broadcast_
     * postamble.h:42-49): flagged here, reported and exited on the host. */
    (void)id;
    (void)message;
    atomicOr(ipx_c.err, IPX_ERR_SEND_IN_BROADCAST);
#else
    uint64_t w = (uint64_t)id;
    if (ipx_c.vindex_of && w < ipx_c.V) w = ipx_c.vindex_of[w]; /* the caller's id -> the copy's vertex */
    ipx_deliver((int)(ip_get_superstep() & 1), w, message);
#endif
}

__device__ inline void ip_vote_to_halt(struct ip_vertex_t* v)
{
#if IPX_VERSION == IPX_COMBINER || IPX_VERSION == IPX_SINGLE_BROADCAST
    v->active = false;
#else
    (void)v; /* spread versions ignore it (combiner_spread_postamble.h:433-436) */
#endif
}

/* Fills the neighbour fields of the proxy (loads the compiler drops when
 * ip_compute does not read them). */
__device__ __forceinline__ void ipx_fill_topology(struct ip_vertex_t& x, uint64_t v)
{
#if defined(IP_NEEDS_OUT_NEIGHBOUR_IDS) || defined(IP_NEEDS_OUT_NEIGHBOUR_COUNT) || IPX_OUT_WEIGHTS
    const uint64_t r0 = ipx_c.row[v], r1 = ipx_c.row[v + 1];
#endif
#ifdef IP_NEEDS_OUT_NEIGHBOUR_IDS
    x.out_neighbours = const_cast<ipx_vid*>(ipx_c.user_adj ? ipx_c.user_adj + ipx_c.user_row[ipx_c.vid_of[v]]
                                                           : ipx_c.adj + r0);
#endif
#ifdef IP_NEEDS_OUT_NEIGHBOUR_COUNT
    x.out_neighbour_count = (IP_NEIGHBOUR_COUNT_TYPE)(r1 - r0);
#endif
#if IPX_OUT_WEIGHTS
    x.out_neighbour_weights = const_cast<ipx_wgt*>(ipx_c.wgt + r0);
#endif
#if defined(IP_NEEDS_IN_NEIGHBOUR_IDS) || defined(IP_NEEDS_IN_NEIGHBOUR_COUNT) || IPX_IN_WEIGHTS
    const uint64_t q0 = ipx_c.in_row[v], q1 = ipx_c.in_row[v + 1];
#endif
#ifdef IP_NEEDS_IN_NEIGHBOUR_IDS
    x.in_neighbours = const_cast<ipx_vid*>(ipx_c.user_in_adj ? ipx_c.user_in_adj + ipx_c.user_in_row[ipx_c.vid_of[v]]
                                                             : ipx_c.in_adj + q0);
#endif
#ifdef IP_NEEDS_IN_NEIGHBOUR_COUNT
    x.in_neighbour_count = (IP_NEIGHBOUR_COUNT_TYPE)(q1 - q0);
#endif
#if IPX_IN_WEIGHTS
    x.in_neighbour_weights = const_cast<ipx_wgt*>(ipx_c.in_wgt + q0);
#endif
}

/* ------------------------------------------------------------------------ */
/* Push delivery of the superstep's broadcasts.                             */
/* ------------------------------------------------------------------------ */
/* Bound by the random mailbox reads: 283 G edges/s for CC, 226 for weighted
 * SSSP (which reads weights and commits more) on undirected R-MAT scale 24,
 * where the same ids gathered flat, without rows, messages or commits, reach
 * 376 G/s from the L2.  A run's pushes took 5.1 / 7.6 ms with a launch per row
 * class, sources by 1 and 16 lanes and hubs by a CTA per chunk, without the
 * pipeline; 4.4 / 6.7 now.  64 registers: with 5 CTAs a few spills and the same
 * time, with 6 5.8 / 8.6 (16 lanes), 8 mailbox reads in flight a lane instead
 * of 4 no faster. */
#ifndef IPX_PUSH_CTAS
#define IPX_PUSH_CTAS 4
#endif
__global__ void __launch_bounds__(IPX_THREADS, IPX_PUSH_CTAS) ipx_k_push()
{
    if (ipx_done() || ipx_pulls()) return;
    ipx_walk_broadcasters(ipx_push_visit{ipx_parity()});
}

#if IPX_VERSION == IPX_SPREAD_SINGLE_BROADCAST
/* Marks the out-neighbours of broadcasters as targets.  CTAS per SM: two on
 * 2^23 edges and more; below, where there is less to wait for, one with twice
 * the registers (561 against 575 us, SSSP at R-MAT scale 18). */
extern __shared__ uint32_t ipx_seen[];
template <int CTAS>
__global__ void __launch_bounds__(IPX_MARK_THREADS, CTAS) ipx_k_mark(uint32_t words)
{
    if (ipx_done(false)) return;
    for (uint32_t k = threadIdx.x; k < words; k += blockDim.x) ipx_seen[k] = 0u;
    __syncthreads();
    ipx_walk_broadcasters(ipx_mark_visit{ipx_seen, 32ULL * words});
}
#endif

/* ------------------------------------------------------------------------ */
/* Pull gather (ip_fetch_broadcast_messages, combiner_single_broadcast_      */
/* postamble.h:57-89): fold ip_combine over the in-neighbours that           */
/* broadcast.  A thread alone on a row folds in adjacency order, as the      */
/* reference does; several lanes fold their runs in order and then combine   */
/* the partial results in a tree.                                            */
/* ------------------------------------------------------------------------ */
__device__ __forceinline__ void ipx_fold(bool& has, ipx_msg& acc, bool oh, ipx_msg om)
{
    if (oh) {
        if (has) {
            ip_combine(&acc, om);
        } else {
            acc = om;
            has = true;
        }
    }
}

__device__ __forceinline__ void ipx_warp_fold(bool& has, ipx_msg& acc)
{
    for (int o = 16; o > 0; o >>= 1) {
        bool oh = __shfl_down_sync(IPX_FULL, has, o);
        ipx_msg om = ipx_shfl_down(acc, o);
        ipx_fold(has, acc, oh, om);
    }
}

/* Folds the broadcasts of the in-neighbours at edges e0 + lane, e0 + lane +
 * lanes, ... below e1, in that order.  IPX_UNROLL edges a step: their ids,
 * then their broadcast slots are each loaded for all IPX_UNROLL edges before
 * any is folded, so a lane has IPX_UNROLL independent slot loads in flight.
 * A warp or block (lanes >= 32) with 32-bit ids reads the ids 128 bits at a
 * time instead: four consecutive in-edges per lane and load instruction
 * (ipx_gather_fold_edges_v4). */
template <bool HOT = false, class S>
__device__ __forceinline__ void ipx_gather_fold_edges_v4(const uint32_t* __restrict__ adj,
                                                         const S* bs, uint32_t stamp,
                                                         uint64_t e0, uint64_t e1, uint64_t lane, uint64_t lanes,
                                                         bool& has, ipx_msg& acc)
{
    /* [e0, a): up to 3 edges before the first 16-byte boundary; [a, b): whole
     * groups of four; [b, e1): up to 3 edges after.  The 6 or fewer edges of
     * both ends take one lane each (lanes >= 8). */
    uint64_t a = (e0 + 3) & ~3ULL;
    if (a > e1) a = e1;
    const uint64_t b = a + ((e1 - a) & ~3ULL);
    {
        const uint64_t nh = a - e0, nt = e1 - b;
        uint64_t e = e1;
        if (lane < nh) e = e0 + lane;
        else if (lane < nh + nt) e = b + (lane - nh);
        if (e < e1) {
            const S w = ipx_slot_ld<HOT>(bs, adj[e]);
            ipx_msg m;
            if (ipx_slot_take(w, stamp, m)) ipx_fold(has, acc, true, m);
        }
    }
    const uint4* __restrict__ q = reinterpret_cast<const uint4*>(adj + a);
    const uint64_t groups = (b - a) >> 2;
    for (uint64_t g = lane; g < groups; g += lanes) {
        const uint4 id = __ldcs(q + g);
        S w[4];
        w[0] = ipx_slot_ld<HOT>(bs, id.x);
        w[1] = ipx_slot_ld<HOT>(bs, id.y);
        w[2] = ipx_slot_ld<HOT>(bs, id.z);
        w[3] = ipx_slot_ld<HOT>(bs, id.w);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            ipx_msg m;
            if (ipx_slot_take(w[k], stamp, m)) ipx_fold(has, acc, true, m);
        }
    }
}

template <bool HOT = false, class S>
__device__ __forceinline__ void ipx_gather_fold_edges(const ipx_vid* __restrict__ adj,
                                                      const S* bs, uint32_t stamp, uint64_t e0,
                                                      uint64_t e1, uint64_t lane, uint64_t lanes, bool& has,
                                                      ipx_msg& acc)
{
    if constexpr (sizeof(ipx_vid) == 4) {
        /* the vector path needs a 16-byte aligned id array (always so for
         * arrays the runtime allocates; a caller's array may not be) */
        if (lanes >= 8 && (reinterpret_cast<uintptr_t>(adj) & 15) == 0) {
            ipx_gather_fold_edges_v4<HOT>(reinterpret_cast<const uint32_t*>(adj), bs, stamp, e0, e1, lane, lanes, has,
                                          acc);
            return;
        }
    }
    for (uint64_t e = e0 + lane; e < e1; e += IPX_UNROLL * lanes) {
        uint64_t u[IPX_UNROLL];
        S w[IPX_UNROLL];
#pragma unroll
        for (int k = 0; k < IPX_UNROLL; k++)
            u[k] = (e + k * lanes < e1) ? (uint64_t)ipx_ld_edge(&adj[e + k * lanes], lanes) : 0;
#pragma unroll
        for (int k = 0; k < IPX_UNROLL; k++)
            w[k] = (e + k * lanes < e1) ? ipx_slot_ld<HOT>(bs, u[k]) : ipx_no_slot<S>();
#pragma unroll
        for (int k = 0; k < IPX_UNROLL; k++) {
            ipx_msg m;
            if (ipx_slot_take(w[k], stamp, m)) ipx_fold(has, acc, true, m);
        }
    }
}

/* The tree over the G lanes of one group (G a power of two <= 32); `mask`
 * holds the group's lanes. */
template <int G>
__device__ __forceinline__ void ipx_group_fold(bool& has, ipx_msg& acc, unsigned mask)
{
    typedef typename ipx_word<ipx_msg>::type W;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        const bool oh = __shfl_down_sync(mask, has, o, G);
        const ipx_msg om = ipx_from_word<ipx_msg>(__shfl_down_sync(mask, ipx_to_word(acc), o, G));
        ipx_fold(has, acc, oh, om);
    }
}

/* ------------------------------------------------------------------------ */
/* Pull delivery for the push versions (direction optimisation).  On a       */
/* symmetric graph a vertex's row lists exactly the vertices that would push */
/* to it, so folding the messages of its broadcasting row-neighbours gives   */
/* the message a push would have left in its mailbox (the fold order differs */
/* only as ip_combine's contract allows).  Used in dense supersteps: it      */
/* streams every row once and needs no atomics except for the hubs' chunks.  */
/* One launch, the longest work items first: a warp per chunk of a hub,      */
/* committed with the mailbox's atomic, then groups of 32, 8 and 1 lanes per */
/* row, pipelined over the group's next rows as in the push's walk.          */
/* ------------------------------------------------------------------------ */
#if IPX_VERSION == IPX_COMBINER || IPX_VERSION == IPX_SPREAD
/* The messages of up to four edges' sources, in edge order; ok[k]: the lane
 * holds an edge.  A source's bit is read first and its message only if it
 * broadcast: below one in 20 most would be read for nothing.  Rate bound: 240
 * G edges/s on random in-lists of 8 edges (256 graphs of 1,024 to 65,536
 * vertices in one union of 4.3 M) against 275 G/s for random reads that hit
 * the L2.  CC and weighted SSSP over that union took 2.26 and 3.93 ms with a
 * launch per class (a thread, a warp, a CTA a row) and no pipeline, 1.95 and
 * 3.39 now. */
__device__ __forceinline__ void ipx_pull_fold4(const uint64_t* u, const bool* ok, const ipx_wgt* x, bool& has, ipx_msg& acc)
{
    const uint32_t* bc = ipx_c.bcaster;
    const ipx_msg* ob = ipx_c.outbox;
    bool on[4];
    ipx_msg m[4];
#pragma unroll
    for (int k = 0; k < 4; k++) on[k] = ok[k] && ((bc[u[k] >> 5] >> (u[k] & 31)) & 1u);
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (on[k]) m[k] = ob[u[k]];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (!on[k]) continue;
#if IPX_EDGE_MSG
        ipx_fold(has, acc, true, IP_BROADCAST_EDGE_MESSAGE(m[k], x[k]));
#else
        (void)x;
        ipx_fold(has, acc, true, m[k]);
#endif
    }
}

/* A quad of ids (and of weights) of the row [r0, r0 + deg). */
__device__ __forceinline__ void ipx_pull_fold_quad(const uint4& q, uint64_t r0, uint32_t deg, uint32_t rel, bool& has,
                                                   ipx_msg& acc)
{
    const uint32_t t = rel - ((uint32_t)r0 & 3u); /* edge of the row; before its first: wraps */
    const uint64_t u[4] = {q.x, q.y, q.z, q.w};
    const bool ok[4] = {t < deg, t + 1 < deg, t + 2 < deg, t + 3 < deg};
    ipx_wgt x[4];
#if IPX_EDGE_MSG
    if constexpr (sizeof(ipx_wgt) == 4) {
        const uint4 w = ipx_ld_quad(reinterpret_cast<const uint32_t*>(ipx_c.in_wgt), r0, deg, rel);
        const uint32_t wk[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int k = 0; k < 4; k++) memcpy(&x[k], &wk[k], 4);
    } else {
        const uint64_t e = r0 - ((uint32_t)r0 & 3u) + rel;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (ok[k]) x[k] = ipx_ld_stream(&ipx_c.in_wgt[e + k]);
    }
#endif
    ipx_pull_fold4(u, ok, x, has, acc);
}

/* Edges [e0, e1) without 128-bit loads, lane-strided. */
__device__ __forceinline__ void ipx_pull_fold_edges(uint64_t e0, uint64_t e1, uint64_t lane, uint64_t lanes, bool& has,
                                                    ipx_msg& acc)
{
    const ipx_vid* __restrict__ adj = ipx_c.in_adj;
    for (uint64_t e = e0 + lane; e < e1; e += 4 * lanes) {
        uint64_t u[4];
        bool ok[4];
        ipx_wgt x[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            ok[k] = e + k * lanes < e1;
            u[k] = ok[k] ? (uint64_t)ipx_ld_edge(&adj[e + k * lanes], lanes) : 0;
#if IPX_EDGE_MSG
            if (ok[k]) x[k] = ipx_ld_edge(&ipx_c.in_wgt[e + k * lanes], lanes);
#endif
        }
        ipx_pull_fold4(u, ok, x, has, acc);
    }
}

/* The list's rows, G lanes each; SKIP: hubs are passed over. */
template <int G, bool SKIP>
__device__ __forceinline__ void ipx_pull_rows(const uint32_t* __restrict__ list, uint32_t n, int p)
{
    const int lane = threadIdx.x & 31, gl = lane & (G - 1);
    const unsigned mask = (G == 32) ? IPX_FULL : (((1u << (G & 31)) - 1u) << (lane & ~(G - 1)));
    const uint64_t* __restrict__ row = ipx_c.in_row;
    const uint64_t step = ipx_gstride() / G;
    uint64_t i = ipx_gtid() / G;
    auto done = [&](uint64_t v, bool has, ipx_msg acc) {
        if (G > 1) ipx_group_fold<G>(has, acc, mask);
        if (gl == 0 && has && ipx_mb::merge(&ipx_c.mbox[p][v], acc)) {
            if (G == 1) ipx_set_bit_agg(ipx_c.recv[p], v);
            else atomicOr(&ipx_c.recv[p][v >> 5], 1u << (v & 31));
        }
    };
    if (!ipx_c.in_quads) {
        for (; i < n; i += step) {
            const uint64_t v = list[i];
            if (SKIP && row[v + 1] - row[v] > ipx_c.hub_min) continue;
            bool has = false;
            ipx_msg acc;
            ipx_pull_fold_edges(row[v], row[v + 1], gl, G, has, acc);
            done(v, has, acc);
        }
        return;
    }
    if (i >= n) return;
    if constexpr (sizeof(ipx_vid) == 4) {
        const uint32_t* __restrict__ adj = reinterpret_cast<const uint32_t*>(ipx_c.in_adj);
        /* a: the row being folded, b: the next, c: the one after it; past the
         * list's end vertex 0 stands in: loaded, never folded */
        uint32_t va = list[i], vb = i + step < n ? list[i + step] : 0u, vc = i + 2 * step < n ? list[i + 2 * step] : 0u;
        uint64_t a0 = row[va], b0 = row[vb];
        uint32_t ad = ipx_row_edges(a0, row[va + 1]), bd = ipx_row_edges(b0, row[vb + 1]);
        uint4 qa = ipx_ld_quad(adj, a0, ad, 4 * gl);
        for (; i < n; i += step) {
            const uint32_t vd = i + 3 * step < n ? list[i + 3 * step] : 0u;
            const uint64_t c0 = row[vc], c1 = row[vc + 1];
            const uint4 qb = ipx_ld_quad(adj, b0, bd, 4 * gl);
            if (!SKIP || ad <= ipx_c.hub_min) {
                bool has = false;
                ipx_msg acc;
                const uint32_t len = ((uint32_t)a0 & 3u) + ad;
                for (uint32_t rel = 4 * gl;;) {
                    const uint4 next = ipx_ld_quad(adj, a0, ad, rel + 4 * G);
                    ipx_pull_fold_quad(qa, a0, ad, rel, has, acc);
                    rel += 4 * G;
                    if (rel >= len) break;
                    qa = next;
                }
                done(va, has, acc);
            }
            va = vb;
            vb = vc;
            vc = vd;
            a0 = b0;
            ad = bd;
            b0 = c0;
            bd = ipx_row_edges(c0, c1);
            qa = qb;
        }
    }
}

#ifndef IPX_PULL_CTAS
#define IPX_PULL_CTAS 4
#endif
__global__ void __launch_bounds__(IPX_THREADS, IPX_PULL_CTAS) ipx_k_pull_deliver()
{
    if (ipx_done() || !ipx_pulls()) return; /* this superstep pushes */
    const int p = ipx_parity(), lane = threadIdx.x & 31;
    const uint64_t warps = ipx_gstride() >> 5;
    for (uint64_t c = ipx_gtid() >> 5; c < ipx_c.chunks; c += warps) {
        const uint4 hub = ipx_c.hub[ipx_c.hub_owner[c]];
        const uint64_t v = hub.x, e0 = ipx_c.in_row[v] + (c - hub.y) * ipx_c.hub_chunk, end = ipx_c.in_row[v + 1];
        const uint64_t e1 = e0 + ipx_c.hub_chunk < end ? e0 + ipx_c.hub_chunk : end;
        bool has = false;
        ipx_msg acc;
        if (sizeof(ipx_vid) == 4 && ipx_c.in_quads) {
            const uint32_t* __restrict__ adj = reinterpret_cast<const uint32_t*>(ipx_c.in_adj);
            const uint32_t deg = (uint32_t)(e1 - e0), len = ((uint32_t)e0 & 3u) + deg;
            uint4 q = ipx_ld_quad(adj, e0, deg, 4 * lane);
            for (uint32_t rel = 4 * lane; rel < len; rel += 128) {
                const uint4 next = ipx_ld_quad(adj, e0, deg, rel + 128);
                ipx_pull_fold_quad(q, e0, deg, rel, has, acc);
                q = next;
            }
        } else {
            ipx_pull_fold_edges(e0, e1, lane, 32, has, acc);
        }
        ipx_warp_fold(has, acc);
        /* chunks of one hub meet in its mailbox: the atomic delivery */
        if (lane == 0 && has && ipx_mb::deliver(&ipx_c.mbox[p][v], acc)) atomicOr(&ipx_c.recv[p][v >> 5], 1u << (v & 31));
    }
    ipx_pull_rows<IPX_PUSH_LONG, true>(ipx_c.class_list[2], ipx_c.class_n[2], p);
    ipx_pull_rows<IPX_PUSH_GROUP, false>(ipx_c.class_list[1], ipx_c.class_n[1], p);
    ipx_pull_rows<1, false>(ipx_c.class_list[0], ipx_c.class_n[0], p);
}
#endif

/* ------------------------------------------------------------------------ */
/* Compute kernels.                                                         */
/* ------------------------------------------------------------------------ */
#if IPX_VERSION != IPX_SINGLE_BROADCAST
/* The compute phase of the push versions and of spread+single_broadcast, and
 * the lists of this superstep's broadcasters, in one pass over the bitmaps.
 *
 * Combiner (push): src/combiner_postamble.h:151-183, vertices that are
 * active, hold a message or received one; the mailbox swap of the previous
 * superstep (:168-183) happens here, for the vertex about to run.  Spread
 * (frontier push): src/combiner_spread_postamble.h:235-272 and the mailbox
 * update :331-342, the vertices that received mail (all at superstep 0).
 * Spread + single broadcast: combiner_spread_single_broadcast_postamble.h:
 * 228-237, the targets of the last superstep.
 *
 * A warp takes `words` bitmap words at a time (8 on a large graph, fewer when
 * that would leave warps with little to even out), a lane a word to load and write back
 * and, of the nonzero ones, a vertex of each of FRONT_W words to compute: a
 * dense frontier reads mailboxes, values and row bounds coalesced, a sparse
 * one costs a scan of the bitmap, and there are no atomics and no list of the
 * frontier.  Broadcasters go into the list of their row length through a
 * buffer per warp in shared memory, emptied in long runs behind
 * one reservation; hubs are listed by chunks.  No warp waits for another.
 * Latency bound (half of the warps wait on loads, issue slots 43 % busy).
 * Undirected R-MAT scale 24, CC / weighted SSSP, ms a run: 0.77 / 1.07 for what
 * a compute kernel over a frontier list (0.93 / 1.42), the compaction of the
 * broadcasters (0.35 / 0.48) and of the receivers (0.19 / 0.33) and the hubs'
 * chunk prefix (0.1 / 0.2) took.  A reservation per CTA step behind barriers
 * 0.82 / 1.33; 4, 16, 32 words a step 0.75 / 1.03, 0.84 / 1.16, 1.0 / 1.42;
 * 3 CTAs per SM 1.1 / 1.7, 5 (it spills) 1.1 / 1.8. */
#ifndef IPX_FRONT_CTAS
#define IPX_FRONT_CTAS 4
#endif
#define IPX_FRONT_W 4
#ifndef IPX_FRONT_BUF
#define IPX_FRONT_BUF 512 /* entries a warp buffers; a step adds at most 128 */
#endif

struct ipx_front_buf {
    uint32_t v[IPX_FRONT_BUF];
    uint8_t cls[IPX_FRONT_BUF];
};

/* The warp's buffered broadcasters go to the ends of their classes' lists;
 * n: how many of each class are among them. */
__device__ __forceinline__ void ipx_front_flush(const ipx_front_buf& buf, const uint32_t* n)
{
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u, total = n[0] + n[1] + n[2];
    const uint32_t mine = lane == 0 ? n[0] : (lane == 1 ? n[1] : n[2]);
    uint32_t at = 0;
    if (lane < 3 && mine) at = atomicAdd(&ipx_c.stat->n[lane], mine);
    uint32_t to[3];
#pragma unroll
    for (int j = 0; j < 3; j++) to[j] = __shfl_sync(IPX_FULL, at, j);
    __syncwarp();
    for (uint32_t q0 = 0; q0 < total; q0 += 32) {
        const uint32_t q = q0 + lane;
        const int c = q < total ? (int)buf.cls[q] : 3;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint32_t b = __ballot_sync(IPX_FULL, c == j);
            if (c == j) ipx_c.blist[j][to[j] + __popc(b & lt)] = buf.v[q];
            to[j] += __popc(b);
        }
    }
    __syncwarp();
}

__global__ void __launch_bounds__(IPX_THREADS, IPX_FRONT_CTAS) ipx_k_front(int words, bool starts)
{
    if (ipx_done()) return;
    __shared__ ipx_front_buf s_buf[IPX_THREADS / 32];
    const uint64_t s = ipx_step();
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    ipx_front_buf& buf = s_buf[threadIdx.x >> 5];
    const uint64_t W = ipx_c.W, step = (ipx_gstride() >> 5) * (uint64_t)words;
    [[maybe_unused]] const int pprev = (int)((s + 1) & 1); /* parity of superstep s-1 */
    unsigned long long es[4] = {0, 0, 0, 0};
    uint32_t n[3] = {0, 0, 0};
    ipx_start_clock(starts || s == 0);
    for (uint64_t base = (ipx_gtid() >> 5) * (uint64_t)words; base < W; base += step) {
        /* this lane's word */
        const uint64_t wl = base + lane;
        const bool mine = lane < words && wl < W;
        uint32_t word = 0;
        [[maybe_unused]] uint32_t act = 0, has = 0, rec = 0, out_word = 0;
        if (mine) {
#if IPX_VERSION == IPX_COMBINER
            act = ipx_c.active_bm[wl];
            has = ipx_c.hasmsg_bm[wl];
            rec = s ? ipx_c.recv[pprev][wl] : 0u;
            word = act | has | rec;
            if (rec) ipx_c.recv[pprev][wl] = 0u;
#else
#if IPX_VERSION == IPX_SPREAD
            uint32_t* from = ipx_c.recv[pprev];
#else
            uint32_t* from = ipx_c.bt;
#endif
            if (s) {
                word = from[wl];
                if (word) from[wl] = 0u;
            } else {
                /* the vertex count ends inside the last word */
                word = (wl == W - 1 && (ipx_c.V & 31)) ? (1u << (ipx_c.V & 31)) - 1u : IPX_FULL;
            }
#endif
        }
        [[maybe_unused]] const uint32_t act0 = act, has0 = has;
        uint32_t todo = __ballot_sync(IPX_FULL, word != 0u);
        while (todo) {
            /* the next FRONT_W nonzero words */
            int idx[IPX_FRONT_W];
            uint32_t run[IPX_FRONT_W];
            [[maybe_unused]] uint32_t hw[IPX_FRONT_W], rw[IPX_FRONT_W];
#pragma unroll
            for (int k = 0; k < IPX_FRONT_W; k++) {
                idx[k] = todo ? __ffs(todo) - 1 : 0;
                const uint32_t x = __shfl_sync(IPX_FULL, word, idx[k]);
                run[k] = todo ? x : 0u;
                todo &= todo - 1;
#if IPX_VERSION == IPX_COMBINER
                hw[k] = __shfl_sync(IPX_FULL, has0, idx[k]);
                rw[k] = __shfl_sync(IPX_FULL, rec, idx[k]);
#endif
            }
            /* every load of the warp's vertices before any of them computes */
            ipx_val v0[IPX_FRONT_W];
            [[maybe_unused]] ipx_slot box[IPX_FRONT_W];
            [[maybe_unused]] bool hm[IPX_FRONT_W];
            [[maybe_unused]] ipx_msg msg[IPX_FRONT_W];
#pragma unroll
            for (int k = 0; k < IPX_FRONT_W; k++) {
                const uint64_t v = (base + idx[k]) * 32 + lane;
                if ((run[k] >> lane) & 1u) {
                    v0[k] = ipx_c.value[v];
#if IPX_VERSION == IPX_COMBINER
                    if ((rw[k] >> lane) & 1u) box[k] = ipx_c.mbox[pprev][v];
                    else if ((hw[k] >> lane) & 1u) msg[k] = ipx_c.msg[v];
#elif IPX_VERSION == IPX_SPREAD
                    if (s) box[k] = ipx_c.mbox[pprev][v];
#else
                    hm[k] = ipx_c.hasmsg_b[v];
                    if (hm[k]) msg[k] = ipx_c.msg[v];
#endif
                }
            }
#pragma unroll
            for (int k = 0; k < IPX_FRONT_W; k++) {
                if (!run[k]) continue; /* warp-uniform */
                const uint64_t v = (base + idx[k]) * 32 + lane;
                uint64_t d = 0;
                bool out = false;
                [[maybe_unused]] bool na = false, nh = false;
                if ((run[k] >> lane) & 1u) {
                    struct ip_vertex_t x;
                    x.id = ipx_user_id(v);
                    x.active = true;
#if IPX_VERSION == IPX_COMBINER
                    const bool r = (rw[k] >> lane) & 1u;
                    x.has_message = r || ((hw[k] >> lane) & 1u);
                    if (r) {
                        x.message = ipx_mb::message(box[k]);
                        ipx_c.mbox[pprev][v] = ipx_mb::empty();
                    } else if (x.has_message) {
                        x.message = msg[k];
                    }
#elif IPX_VERSION == IPX_SPREAD
                    x.has_message = s != 0; /* a frontier vertex always has one */
                    if (s) {
                        x.message = ipx_mb::message(box[k]);
                        ipx_c.mbox[pprev][v] = ipx_mb::empty();
                    }
#else
                    x.has_message = hm[k];
                    if (hm[k]) x.message = msg[k];
#endif
                    x.value = v0[k];
                    x.ipx_has_out = false;
                    ipx_fill_topology(x, v);
                    ip_compute(&x);
                    if (!ipx_same_bits(x.value, v0[k])) ipx_c.value[v] = x.value;
                    out = x.ipx_has_out;
#if IPX_VERSION == IPX_COMBINER
                    na = x.active;
                    nh = x.has_message;
                    if (nh) ipx_c.msg[v] = x.message;
#endif
                    if (out) {
#if IPX_VERSION == IPX_SPREAD_SINGLE_BROADCAST
                        ipx_bslot_put(&ipx_c.bslot[0][v], x.ipx_out, (uint32_t)s);
#else
                        ipx_c.outbox[v] = x.ipx_out;
#endif
                        d = ipx_c.row[v + 1] - ipx_c.row[v];
                    }
                }
                const uint32_t nout = __ballot_sync(IPX_FULL, out);
                if (lane == idx[k]) out_word = nout;
#if IPX_VERSION == IPX_COMBINER
                const uint32_t aw = __ballot_sync(IPX_FULL, na), mw = __ballot_sync(IPX_FULL, nh);
                if (lane == idx[k]) {
                    act = aw;
                    has = mw;
                }
#endif
                if (!nout) continue;
                const int c = d == 0 ? -1 : (d <= ipx_c.push_t[0] ? 0 : (d <= ipx_c.push_t[1] ? 1 : (d <= ipx_c.push_t[2] ? 2 : 3)));
                const uint32_t in = __ballot_sync(IPX_FULL, c >= 0 && c < 3);
                if (c >= 0 && c < 3) {
                    const uint32_t q = n[0] + n[1] + n[2] + __popc(in & lt);
                    buf.v[q] = (uint32_t)v;
                    buf.cls[q] = (uint8_t)c;
                }
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    n[j] += __popc(__ballot_sync(IPX_FULL, c == j));
                    if (c == j) es[j] += d;
                }
                uint32_t hubs = __ballot_sync(IPX_FULL, c == 3);
                if (hubs) {
                    const uint32_t ch = c == 3 ? (uint32_t)((d + ipx_c.push_chunk - 1) / ipx_c.push_chunk) : 0u;
                    if (c == 3) es[3] += d;
                    uint32_t at = 0;
                    if (c == 3) at = atomicAdd(&ipx_c.stat->n[3], ch);
                    while (hubs) {
                        const int j = __ffs(hubs) - 1;
                        hubs &= hubs - 1;
                        const uint32_t aj = __shfl_sync(IPX_FULL, at, j), cj = __shfl_sync(IPX_FULL, ch, j);
                        const uint32_t u = __shfl_sync(IPX_FULL, (uint32_t)v, j);
                        for (uint32_t q = lane; q < cj; q += 32) ipx_c.bchunk[aj + q] = make_uint2(u, q);
                    }
                }
            }
            if (n[0] + n[1] + n[2] > IPX_FRONT_BUF - 32 * IPX_FRONT_W) {
                ipx_front_flush(buf, n);
                n[0] = n[1] = n[2] = 0;
            }
        }
        if (mine) {
#if IPX_VERSION == IPX_COMBINER
            if (act != act0) ipx_c.active_bm[wl] = act;
            if (has != has0) ipx_c.hasmsg_bm[wl] = has;
#endif
            if (ipx_c.pull_ok) ipx_c.bcaster[wl] = out_word;
        }
    }
    if (n[0] + n[1] + n[2]) ipx_front_flush(buf, n);
    __shared__ unsigned long long s_edges[4];
    if (threadIdx.x < 4) s_edges[threadIdx.x] = 0ULL;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++) {
        unsigned long long e = es[j];
        for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(IPX_FULL, e, o);
        if (lane == 0 && e) atomicAdd(&s_edges[j], e);
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_edges[threadIdx.x]) atomicAdd(&ipx_c.stat->edges[threadIdx.x], s_edges[threadIdx.x]);
}
#endif

/* The single_broadcast version's record of a vertex's broadcast (or of
 * none) for the superstep `stamp`: a stamped slot is written only for a
 * broadcast; a dense slot every time. */
__device__ __forceinline__ void ipx_sb_put(ipx_bslot* p, bool out, const ipx_msg& m, uint32_t stamp)
{
    if (out) ipx_bslot_put(p, m, stamp);
}
__device__ __forceinline__ void ipx_sb_put(unsigned long long* p, bool out, const ipx_msg& m, uint32_t)
{
    unsigned long long w = IPX_ABSENT64;
    if (out) {
        w = (unsigned long long)ipx_to_word(m);
        if (w == IPX_ABSENT64) atomicOr(ipx_c.err, IPX_ERR_RESERVED_MESSAGE);
    }
    *p = w;
}

/* Single broadcast (pull), superstep 0's compute phase
 * (combiner_single_broadcast_postamble.h:185-201): every vertex is active and
 * has no message.  A broadcast writes the vertex's slot in buffer 0 stamped
 * 0.  Later supersteps' compute phases run inside ipx_k_gather_compute; this
 * kernel returns at once after superstep 0, so the same launch sequence
 * serves every superstep of a captured loop.  The count of superstep 0 is
 * made by the gather that follows. */
__global__ void __launch_bounds__(IPX_THREADS) ipx_k_compute_sb0()
{
    if (ipx_step() != 0) return;
    if (threadIdx.x == 0) ipx_step_word() = ipd_compute_superstep;
    __syncthreads();
    ipx_start_clock(true);
    const uint64_t V = ipx_c.V;
    ipx_sbslot* __restrict__ out = ipx_c.sbslot[0];
    for (uint64_t v = ipx_gtid(); v < V; v += ipx_gstride()) {
        if (!ipx_c.active_b[v]) {
            ipx_sb_put(&out[v], false, ipx_msg(), 0u);
            continue;
        }
        struct ip_vertex_t x;
        x.id = ipx_user_id(v);
        x.active = true;
        x.has_message = false;
        const ipx_val v0 = ipx_c.value[v];
        x.value = v0;
        x.ipx_has_out = false;
        ipx_fill_topology(x, v);
        ip_compute(&x);
        if (!ipx_same_bits(x.value, v0)) ipx_c.value[v] = x.value;
        if (!x.active) ipx_c.active_b[v] = 0;
        ipx_sb_put(&out[v], x.ipx_has_out, x.ipx_out, 0u);
    }
    /* the fused kernel of superstep 0 runs the compute phase of superstep 1 */
    if (ipx_last_cta() && threadIdx.x == 0) ipd_compute_superstep = 1;
}

/* After vertex v's gather of superstep s: whether v is active (it was after
 * compute(s), or a message reactivates it, :65-71), and if so its compute
 * phase of superstep s+1 (:185-201) with the gathered message; a broadcast
 * goes to `out` stamped s+1.  a0 and v0: the vertex's activity and value.
 * Returns the activity that superstep s counts. */
__device__ __forceinline__ bool ipx_sb_compute_next(uint64_t v, bool has, const ipx_msg& acc, bool a0,
                                                    const ipx_val& v0, ipx_sbslot* out, uint32_t next_stamp)
{
    if (!a0 && !has) {
        ipx_sb_put(&out[v], false, acc, next_stamp);
        return false;
    }
    struct ip_vertex_t x;
    x.id = ipx_user_id(v);
    x.active = true;
    x.has_message = has;
    if (has) x.message = acc;
    x.value = v0;
    x.ipx_has_out = false;
    ipx_fill_topology(x, v);
    ip_compute(&x);
    if (!ipx_same_bits(x.value, v0)) ipx_c.value[v] = x.value;
    if (x.active != a0) ipx_c.active_b[v] = x.active ? 1 : 0;
    ipx_sb_put(&out[v], x.ipx_has_out, x.ipx_out, next_stamp);
    return true;
}

/* ---- bulk copies into shared memory (cp.async.bulk, completed on an
 * mbarrier; one CTA, no cluster, no multicast) ---- */
__device__ __forceinline__ uint32_t ipx_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ipx_mbar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ipx_smem(bar)) : "memory");
}

/* The issuing thread's arrival on `bar`, expecting `bytes` from a bulk copy
 * (0: a plain arrival, which completes the phase). */
__device__ __forceinline__ void ipx_mbar_arrive_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ipx_smem(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void ipx_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     ipx_smem(dst)),
                 "l"(src), "r"(bytes), "r"(ipx_smem(bar))
                 : "memory");
}

/* Waits for phase `parity` of `bar` to complete, at most `limit` polls. */
__device__ __forceinline__ bool ipx_mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit)
{
    for (uint32_t k = 0; k < limit; k++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(ipx_smem(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

/* Polls before a wait for a chunk's ids is given up (each try_wait may
 * suspend the thread for a while): an 8 KB copy lands in microseconds, so
 * this is reached only if the copy never completes. */
#define IPX_COPY_WAIT_LIMIT (1u << 22)

/* A hub chunk as thread 0 located it: the vertex, its hub index, the chunk's
 * edge range [e0, e1) and the 16-byte aligned range [a0, b) copied into
 * shared memory (b <= a0: nothing copied). */
struct ipx_hub_chunk {
    uint64_t v, e0, e1, a0, b;
    uint64_t i;
    uint32_t c, c0, nch, pad;
};

__device__ __forceinline__ void ipx_locate_chunk(const uint64_t* __restrict__ row, uint32_t c, ipx_hub_chunk& h)
{
    h.c = c;
    h.i = ipx_c.hub_owner[c];
    const uint4 hub = ipx_c.hub[h.i];
    h.v = hub.x;
    h.c0 = hub.y;
    h.nch = hub.z;
    const uint64_t chunk = ipx_c.hub_chunk;
    h.e0 = row[h.v] + (uint64_t)(c - h.c0) * chunk;
    const uint64_t end = row[h.v + 1];
    h.e1 = (h.e0 + chunk < end) ? h.e0 + chunk : end;
    h.a0 = h.e0 & ~3ULL;
    h.b = h.e1 & ~3ULL;
}

/* The CTA's fold of one hub chunk is done (thread 0 holds it in has/acc;
 * every thread of the CTA calls this).  The fold is stored; the CTA whose
 * chunk arrives last folds the hub's partials in chunk order -- each thread
 * a contiguous run of them, then the runs in order through the warps and
 * the CTA -- and thread 0 runs the vertex's compute phase of the next
 * superstep.  s_has / s_acc: the caller's per-warp shared scratch, free
 * again when this is called.  Returns the count (thread 0). */
__device__ __forceinline__ unsigned long long ipx_hub_chunk_done(const ipx_hub_chunk& h, bool has, ipx_msg acc,
                                                                 ipx_sbslot* out, uint32_t next_stamp,
                                                                 bool* s_has, ipx_msg* s_acc)
{
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        int last = 2; /* a hub of one chunk: its fold is the hub's */
        if (h.nch != 1) {
            ipx_bslot_put(&ipx_c.hub_part[h.c], acc, has ? 1u : 0u);
            __threadfence();
            last = atomicAdd(&ipx_c.hub_arrived[h.i], 1u) == h.nch - 1 ? 1 : 0;
        }
        s_last = last;
    }
    __syncthreads();
    const int last = s_last;
    if (last == 1) {
        __threadfence();
        const uint32_t nthr = blockDim.x, per = (h.nch + nthr - 1) / nthr;
        const uint32_t k0 = threadIdx.x * per, k1 = min(k0 + per, h.nch);
        bool hp = false;
        ipx_msg ap;
        for (uint32_t k = k0; k < k1; k++) {
            const ipx_bslot p = __ldcg(&ipx_c.hub_part[h.c0 + k]);
            ipx_msg m;
            if (ipx_bslot_take(p, 1u, m)) ipx_fold(hp, ap, true, m);
        }
        ipx_warp_fold(hp, ap);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane == 0) {
            s_has[warp] = hp;
            s_acc[warp] = ap;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            has = false;
            for (int w = 0; w < (int)(nthr >> 5); w++) ipx_fold(has, acc, s_has[w], s_acc[w]);
            ipx_c.hub_arrived[h.i] = 0; /* every chunk of the hub has arrived */
        }
    }
    if (threadIdx.x == 0 && last != 0)
        return (unsigned long long)ipx_sb_compute_next(h.v, has, acc, ipx_c.active_b[h.v] != 0, ipx_c.value[h.v], out,
                                                       next_stamp);
    return 0ULL;
}

#ifndef IPX_HUB_SMEM
#define IPX_HUB_SMEM 1
#endif
/* In-edges a thread of the staged hub gather loads per step. */
#ifndef IPX_HUB_UNROLL
#define IPX_HUB_UNROLL 4
#endif
#if !IPX_HUB_WARP
/* The hubs of ipx_k_gather_hubs with ids staged in shared memory: two id
 * buffers, each filled by one bulk copy per chunk and completed on its own
 * mbarrier.  Thread 0 locates chunk k+1 and starts its copy before
 * the CTA waits for chunk k's.  Each iteration thread 0 arrives once on the
 * barrier of the chunk it issues (with the copy's byte count, or alone when
 * the chunk has no whole 16-byte group), so buffer j's barrier completes its
 * u-th phase at its u-th use.  Edges outside the copied range are read from
 * global memory.  A wait that gives up (never expected) sets
 * IPX_ERR_COPY_TIMEOUT, and the CTA reads ids from global memory for the
 * rest of the launch; results stay exact. */
template <bool HOT>
__device__ __forceinline__ unsigned long long ipx_gather_hubs_staged(
    const uint32_t* __restrict__ adj, const uint64_t* __restrict__ row, const ipx_sbslot* bs,
    uint32_t stamp, ipx_sbslot* __restrict__ out)
{
    const uint32_t chunks = ipx_c.chunks;
    __shared__ __align__(16) uint32_t s_ids[2][IPX_GATHER_CHUNK + 4];
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ ipx_hub_chunk s_h[2];
    __shared__ bool s_has[IPX_THREADS / 32];
    __shared__ ipx_msg s_acc[IPX_THREADS / 32];
    __shared__ int s_fail;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nthr = blockDim.x;
    unsigned long long cnt = 0;
    bool pending[2] = {false, false}; /* thread 0: a copy issued and not yet waited for */
    if (threadIdx.x == 0) {
        ipx_mbar_init(&s_bar[0]);
        ipx_mbar_init(&s_bar[1]);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    __syncthreads();
    auto issue = [&](uint32_t c, int buf) {
        ipx_hub_chunk& h = s_h[buf];
        ipx_locate_chunk(row, c, h);
        if (h.b > h.a0 && !s_fail) {
            const uint32_t bytes = (uint32_t)((h.b - h.a0) * 4);
            ipx_mbar_arrive_tx(&s_bar[buf], bytes);
            ipx_bulk_load(s_ids[buf], adj + h.a0, bytes, &s_bar[buf]);
            pending[buf] = true;
        } else {
            h.b = h.a0; /* nothing copied: every id from global memory */
            ipx_mbar_arrive_tx(&s_bar[buf], 0u);
        }
    };
    if (threadIdx.x == 0 && blockIdx.x < chunks) issue(blockIdx.x, 0);
    uint32_t it = 0;
    for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x, it++) {
        const int buf = (int)(it & 1);
        __syncthreads(); /* s_h[buf] is written; everyone is done with buffer buf ^ 1 */
        if (threadIdx.x == 0 && c + gridDim.x < chunks) issue(c + gridDim.x, buf ^ 1);
        bool staged = ipx_mbar_wait(&s_bar[buf], (it >> 1) & 1u, IPX_COPY_WAIT_LIMIT);
        if (!staged) {
            atomicOr(ipx_c.err, IPX_ERR_COPY_TIMEOUT);
            s_fail = 1;
        } else if (threadIdx.x == 0) {
            pending[buf] = false;
        }
        const ipx_hub_chunk h = s_h[buf];
        staged = staged && !s_fail;
        const uint64_t sb = staged ? h.b : h.e0; /* ids of [e0, sb) from shared memory */
        bool has = false;
        ipx_msg acc;
        for (uint64_t e = h.e0 + threadIdx.x; e < h.e1; e += IPX_HUB_UNROLL * (uint64_t)nthr) {
            uint32_t u[IPX_HUB_UNROLL];
            ipx_sbslot w[IPX_HUB_UNROLL];
#pragma unroll
            for (int k = 0; k < IPX_HUB_UNROLL; k++) {
                const uint64_t ek = e + (uint64_t)k * nthr;
                u[k] = (ek < sb) ? s_ids[buf][ek - h.a0] : (ek < h.e1 ? __ldcs(&adj[ek]) : 0u);
            }
#pragma unroll
            for (int k = 0; k < IPX_HUB_UNROLL; k++) {
                w[k] = (e + (uint64_t)k * nthr < h.e1) ? ipx_slot_ld<HOT>(bs, u[k]) : ipx_no_slot<ipx_sbslot>();
            }
#pragma unroll
            for (int k = 0; k < IPX_HUB_UNROLL; k++) {
                ipx_msg m;
                if (ipx_slot_take(w[k], stamp, m)) ipx_fold(has, acc, true, m);
            }
        }
        ipx_warp_fold(has, acc);
        if (lane == 0) {
            s_has[warp] = has;
            s_acc[warp] = acc;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            has = false;
            for (int w = 0; w < (int)(nthr >> 5); w++) ipx_fold(has, acc, s_has[w], s_acc[w]);
        }
        cnt += ipx_hub_chunk_done(h, has, acc, out, stamp + 1, s_has, s_acc);
    }
    /* a copy given up on may still be in flight: wait for it (bounded)
     * before the CTA's shared memory is released */
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; b++)
            if (pending[b]) {
                /* the phase in progress is the copy's: one of the two
                 * parities is the completed phase before it and returns at
                 * once, the other waits for the copy */
                ipx_mbar_wait(&s_bar[b], 0u, IPX_COPY_WAIT_LIMIT);
                ipx_mbar_wait(&s_bar[b], 1u, IPX_COPY_WAIT_LIMIT);
            }
    }
    __syncthreads();
    return cnt;
}
#endif /* !IPX_HUB_WARP */

/* ---- the rows of the fused pull kernel ----
 *
 * G lanes fold one row at a time, each lane four consecutive in-edges per
 * step: one 128-bit load of their ids (aligned down; edges of the rows before
 * and after are masked out), then four slot loads in flight, folded in edge
 * order, and the lanes' folds meet in a tree.  What bounds a row is the chain
 * list entry -> row bounds -> ids -> slots, four dependent loads for a few
 * dozen edges, so the chain is pipelined over the group's next rows: while
 * the slots of one row are in flight, the ids of the next row, the bounds of
 * the one after it and the list entry of the one after that are loaded.
 * Measured (FP64 PageRank, directed R-MAT scale 25, 31 supersteps; ms with
 * one launch per class and no pipeline -> with it): 88 -> 74; FP64
 * personalised PageRank, undirected, 4 M vertices: 11.7 -> 9.8.  The rows of
 * 17 and more edges go from 203 to 263 G edges/s; the same ids gathered flat,
 * without rows, reach 314 G/s, which the L2 bounds. */

/* Folds the broadcasts of the row's edges among a quad's ids, in order. */
template <bool HOT, class S>
__device__ __forceinline__ void ipx_fold_quad(const S* bs, uint32_t stamp, const uint4& q, uint64_t r0,
                                              uint32_t deg, uint32_t rel, bool& has, ipx_msg& acc)
{
    const uint32_t t = rel - ((uint32_t)r0 & 3u); /* edge of the row; before its first: wraps */
    const uint32_t id[4] = {q.x, q.y, q.z, q.w};
    S w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = t + k < deg ? ipx_slot_ld<HOT>(bs, (uint64_t)id[k]) : ipx_no_slot<S>();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        ipx_msg m;
        if (ipx_slot_take(w[k], stamp, m)) ipx_fold(has, acc, true, m);
    }
}

/* Lanes per row of the middle and the long class, and the longest middle
 * row (rows up to t0 take a thread each): about as many lanes as a row has
 * quads.  PageRank at scale 25 / personalised PageRank at 4 M vertices took
 * 74.1 / 9.8 ms with 8 lanes up to 64 edges and 16 beyond, 77.6 / 10.3 with 16
 * for both, 73.5 / 10.9 with 8 for both, 75.9 / 10.2 with 32 beyond 64. */
#ifndef IPX_GATHER_GROUP
#define IPX_GATHER_GROUP 8
#endif
#ifndef IPX_GATHER_LONG
#define IPX_GATHER_LONG 16
#endif
#ifndef IPX_GATHER_MID
#define IPX_GATHER_MID 64
#endif

#if IPX_VERSION == IPX_SINGLE_BROADCAST
typedef ipx_sbslot ipx_gslot;
#else
typedef ipx_bslot ipx_gslot;
#endif

/* What becomes of vertex v's fold: single_broadcast runs its compute phase
 * of the next superstep (with its activity and value, loaded before the
 * fold) and returns the activity that this superstep counts;
 * spread+single_broadcast stores it for the next superstep's. */
struct ipx_vertex_state {
    bool active;
    ipx_val value;
};
__device__ __forceinline__ void ipx_gather_ahead(uint64_t v, bool mine, ipx_vertex_state& x)
{
#if IPX_VERSION == IPX_SINGLE_BROADCAST
    x.active = mine ? ipx_c.active_b[v] != 0 : false;
    x.value = mine ? ipx_c.value[v] : ipx_val();
#else
    (void)v;
    (void)mine;
    (void)x;
#endif
}
__device__ __forceinline__ bool ipx_gather_done(uint64_t v, bool has, const ipx_msg& acc, const ipx_vertex_state& x,
                                                ipx_gslot* out, uint32_t stamp)
{
#if IPX_VERSION == IPX_SINGLE_BROADCAST
    return ipx_sb_compute_next(v, has, acc, x.active, x.value, out, stamp + 1);
#else
    (void)x;
    (void)out;
    (void)stamp;
    ipx_c.hasmsg_b[v] = has;
    if (has) ipx_c.msg[v] = acc;
    return false;
#endif
}

/* Gathers the list's vertices, G lanes each; SKIP: hubs are passed over. */
template <int G, bool SKIP, bool HOT>
__device__ __forceinline__ unsigned long long ipx_gather_rows(const uint32_t* list, uint32_t n,
                                                              const ipx_vid* __restrict__ ids,
                                                              const uint64_t* __restrict__ row,
                                                              const ipx_gslot* bs, uint32_t stamp,
                                                              ipx_gslot* __restrict__ out)
{
    const int lane = threadIdx.x & 31, gl = lane & (G - 1);
    const unsigned mask = (G == 32) ? IPX_FULL : (((1u << (G & 31)) - 1u) << (lane & ~(G - 1)));
    const uint64_t step = ipx_gstride() / G;
    uint64_t i = ipx_gtid() / G;
    unsigned long long cnt = 0;
    if (!ipx_c.in_quads) {
        for (; i < n; i += step) {
            const uint64_t v = list[i];
            if (SKIP && row[v + 1] - row[v] > ipx_c.hub_min) continue;
            ipx_vertex_state x;
            ipx_gather_ahead(v, gl == 0, x);
            bool has = false;
            ipx_msg acc;
            ipx_gather_fold_edges<HOT>(ids, bs, stamp, row[v], row[v + 1], gl, G, has, acc);
            if (G > 1) ipx_group_fold<G>(has, acc, mask);
            if (gl == 0) cnt += ipx_gather_done(v, has, acc, x, out, stamp);
        }
        return cnt;
    }
    const uint32_t* __restrict__ adj = reinterpret_cast<const uint32_t*>(ids);
    if (i >= n) return cnt;
    /* a: the row being folded, b: the next, c: the one after it.  Past the
     * list's end vertex 0 stands in: loaded, never folded. */
    uint32_t va = list[i], vb = i + step < n ? list[i + step] : 0u, vc = i + 2 * step < n ? list[i + 2 * step] : 0u;
    uint64_t a0 = row[va], b0 = row[vb];
    uint32_t ad = ipx_row_edges(a0, row[va + 1]), bd = ipx_row_edges(b0, row[vb + 1]);
    uint4 qa = ipx_ld_quad(adj, a0, ad, 4 * gl);
    for (; i < n; i += step) {
        ipx_vertex_state x;
        ipx_gather_ahead(va, gl == 0, x);
        const uint32_t vd = i + 3 * step < n ? list[i + 3 * step] : 0u;
        const uint64_t c0 = row[vc], c1 = row[vc + 1];
        const uint4 qb = ipx_ld_quad(adj, b0, bd, 4 * gl);
        bool has = false;
        ipx_msg acc;
        const bool skip = SKIP && ad > ipx_c.hub_min;
        if (skip) ad = 0;
        ipx_fold_quad<HOT>(bs, stamp, qa, a0, ad, 4 * gl, has, acc);
        const uint32_t len = ((uint32_t)a0 & 3u) + ad;
        for (uint32_t rel = 4 * gl + 4 * G; rel < len; rel += 4 * G)
            ipx_fold_quad<HOT>(bs, stamp, ipx_ld_quad(adj, a0, ad, rel), a0, ad, rel, has, acc);
        if (G > 1) ipx_group_fold<G>(has, acc, mask);
        if (gl == 0 && !skip) cnt += ipx_gather_done(va, has, acc, x, out, stamp);
        va = vb;
        vb = vc;
        vc = vd;
        a0 = b0;
        ad = bd;
        b0 = c0;
        bd = ipx_row_edges(c0, c1);
        qa = qb;
    }
    return cnt;
}

#if IPX_VERSION == IPX_SINGLE_BROADCAST
/* The hub class with a warp per chunk: the warp folds its chunk, lane 0
 * stores the fold, and the warp whose chunk arrives last folds the hub's
 * partials -- each lane a contiguous run of them, then the runs in order by
 * shuffles -- and lane 0 runs the vertex's compute phase. */
template <bool HOT>
__device__ __forceinline__ unsigned long long ipx_gather_hubs_warp(
    const ipx_vid* __restrict__ ids, const uint64_t* __restrict__ row, const ipx_sbslot* bs,
    uint32_t stamp, ipx_sbslot* __restrict__ out)
{
    const int lane = threadIdx.x & 31;
    const uint64_t nwarps = ipx_gstride() >> 5;
    unsigned long long cnt = 0;
    for (uint64_t c = ipx_gtid() >> 5; c < ipx_c.chunks; c += nwarps) {
        ipx_hub_chunk h;
        ipx_locate_chunk(row, (uint32_t)c, h);
        bool has = false;
        ipx_msg acc;
        if (ipx_c.in_quads) {
            const uint32_t* __restrict__ adj = reinterpret_cast<const uint32_t*>(ids);
            const uint32_t deg = (uint32_t)(h.e1 - h.e0), len = ((uint32_t)h.e0 & 3u) + deg;
            uint4 q = ipx_ld_quad(adj, h.e0, deg, 4 * lane);
            for (uint32_t rel = 4 * lane; rel < len; rel += 128) {
                const uint4 next = ipx_ld_quad(adj, h.e0, deg, rel + 128);
                ipx_fold_quad<HOT>(bs, stamp, q, h.e0, deg, rel, has, acc);
                q = next;
            }
        } else {
            ipx_gather_fold_edges<HOT>(ids, bs, stamp, h.e0, h.e1, lane, 32, has, acc);
        }
        ipx_warp_fold(has, acc);
        int last = 2; /* a hub of one chunk: its fold is the hub's */
        if (lane == 0 && h.nch != 1) {
            ipx_bslot_put(&ipx_c.hub_part[h.c], acc, has ? 1u : 0u);
            __threadfence();
            last = atomicAdd(&ipx_c.hub_arrived[h.i], 1u) == h.nch - 1 ? 1 : 0;
        }
        last = __shfl_sync(IPX_FULL, last, 0);
        if (last == 1) {
            __threadfence();
            const uint32_t per = (h.nch + 31) / 32;
            const uint32_t k0 = (uint32_t)lane * per, k1 = min(k0 + per, h.nch);
            has = false;
            for (uint32_t k = k0; k < k1; k++) {
                const ipx_bslot p = __ldcg(&ipx_c.hub_part[h.c0 + k]);
                ipx_msg m;
                if (ipx_bslot_take(p, 1u, m)) ipx_fold(has, acc, true, m);
            }
            ipx_warp_fold(has, acc);
            if (lane == 0) ipx_c.hub_arrived[h.i] = 0; /* every chunk of the hub has arrived */
        }
        if (lane == 0 && last != 0)
            cnt += ipx_sb_compute_next(h.v, has, acc, ipx_c.active_b[h.v] != 0, ipx_c.value[h.v], out, stamp + 1);
    }
    return cnt;
}

/* Resident CTAs per SM the fused pull kernel is compiled for: it carries
 * ip_compute and the pipeline's registers besides the gather (64 a thread, with
 * 36 bytes of spills for PageRank; many more with 48 or 40: PageRank at scale 25
 * 78.0 ms with 4 CTAs, 83.4 with 5, 95.0 with 6, 80 with 3). */
#ifndef IPX_GATHER_CTAS
#define IPX_GATHER_CTAS 4
#endif

/* Single broadcast (pull), one superstep s >= 0 after its compute phase:
 * ip_fetch_broadcast_messages (combiner_single_broadcast_postamble.h:57-89)
 * and then, vertex by vertex, the compute phase of superstep s+1.  The
 * gather reads buffer s & 1 (slots stamped s) and the compute writes buffer
 * (s+1) & 1, which no gather of superstep s reads, so the two phases need no
 * grid-wide barrier between them and the message goes from the fold to
 * ip_compute in registers.  Count of superstep s: the vertices active after
 * the gather.  When it is 0 no vertex was active or received a message, so
 * no compute phase of superstep s+1 ran, and the loop ends (:164).  All
 * degree classes in one launch, the longest rows first: three launches of
 * 16 k to 500 k threads each end in a tail of their own, which on a graph of
 * 65,536 vertices was half of the superstep. */
template <bool HOT>
__global__ void __launch_bounds__(IPX_THREADS, IPX_GATHER_CTAS) ipx_k_gather_compute(ipx_loop loop)
{
    if (ipx_done()) return;
    const uint64_t s = ipx_step();
    /* superstep 0 starts with its compute phase, others may with the hubs */
    ipx_start_clock((IPX_HUB_WARP || !ipx_c.chunks) && loop.starts && s != 0);
    const uint32_t stamp = (uint32_t)s;
    /* HOT: ids of the in-lists carry the flag of the most gathered vertices */
    const ipx_vid* __restrict__ adj = HOT ? reinterpret_cast<const ipx_vid*>(ipx_c.in_adj_hot) : ipx_c.in_adj;
    const uint64_t* __restrict__ row = ipx_c.in_row;
    const ipx_sbslot* bs = ipx_c.sbslot[s & 1];
    ipx_sbslot* __restrict__ out = ipx_c.sbslot[(s + 1) & 1];
    unsigned long long cnt = 0;
    /* the longest work items first */
    if constexpr (IPX_HUB_WARP) cnt += ipx_gather_hubs_warp<HOT>(adj, row, bs, stamp, out);
    cnt += ipx_gather_rows<IPX_GATHER_LONG, true, HOT>(ipx_c.class_list[2], ipx_c.class_n[2], adj, row, bs, stamp,
                                                       out);
    cnt += ipx_gather_rows<IPX_GATHER_GROUP, false, HOT>(ipx_c.class_list[1], ipx_c.class_n[1], adj, row, bs, stamp,
                                                         out);
    cnt += ipx_gather_rows<1, false, HOT>(ipx_c.class_list[0], ipx_c.class_n[0], adj, row, bs, stamp, out);
    ipx_block_count(cnt, &ipx_c.stat->count);
    if (ipx_last_cta() && threadIdx.x == 0) ipx_end_of_superstep(loop, __ldcg(&ipx_c.stat->count));
}

#if !IPX_HUB_WARP
/* The hub chunks of the fused pull kernel in a launch of their own, a CTA
 * per chunk (IPX_HUB_WARP = 0): each chunk's fold is stored, and the CTA
 * whose chunk arrives last folds the partials in chunk order, then runs the
 * compute phase (ipx_hub_chunk_done).  No CTA waits for another.  With
 * 32-bit ids the chunk's ids are staged through shared memory: while the CTA
 * gathers one chunk, a bulk copy brings the ids of its next chunk, so the
 * slot loads are issued from shared memory instead of behind a global id
 * load each. */
template <bool HOT>
__global__ void __launch_bounds__(IPX_THREADS, IPX_GATHER_CTAS) ipx_k_gather_hubs(bool starts)
{
    if (ipx_done()) return;
    const uint64_t s = ipx_step();
    ipx_start_clock(starts && s != 0);
    const uint32_t stamp = (uint32_t)s;
    const ipx_vid* __restrict__ adj = HOT ? reinterpret_cast<const ipx_vid*>(ipx_c.in_adj_hot) : ipx_c.in_adj;
    const uint64_t* __restrict__ row = ipx_c.in_row;
    const ipx_sbslot* bs = ipx_c.sbslot[s & 1];
    ipx_sbslot* __restrict__ out = ipx_c.sbslot[(s + 1) & 1];
    unsigned long long cnt = 0;
    if constexpr (sizeof(ipx_vid) == 4 && IPX_HUB_SMEM) {
        if ((reinterpret_cast<uintptr_t>(adj) & 15) == 0) {
            cnt += ipx_gather_hubs_staged<HOT>(reinterpret_cast<const uint32_t*>(adj), row, bs, stamp, out);
            ipx_block_count(cnt, &ipx_c.stat->count);
            return;
        }
    }
    __shared__ bool s_has[IPX_THREADS / 32];
    __shared__ ipx_msg s_acc[IPX_THREADS / 32];
    __shared__ ipx_hub_chunk s_h;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t c = blockIdx.x; c < ipx_c.chunks; c += gridDim.x) {
        if (threadIdx.x == 0) ipx_locate_chunk(row, c, s_h);
        __syncthreads();
        const ipx_hub_chunk h = s_h;
        bool has = false;
        ipx_msg acc;
        ipx_gather_fold_edges<HOT>(adj, bs, stamp, h.e0, h.e1, threadIdx.x, blockDim.x, has, acc);
        ipx_warp_fold(has, acc);
        if (lane == 0) {
            s_has[warp] = has;
            s_acc[warp] = acc;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            has = false;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) ipx_fold(has, acc, s_has[w], s_acc[w]);
        }
        cnt += ipx_hub_chunk_done(h, has, acc, out, stamp + 1, s_has, s_acc);
        __syncthreads();
    }
    ipx_block_count(cnt, &ipx_c.stat->count);
}
#endif /* !IPX_HUB_WARP */
#endif /* IPX_SINGLE_BROADCAST */

#if IPX_VERSION == IPX_SPREAD_SINGLE_BROADCAST
/* Spread + single broadcast: the targets' fetch (combiner_spread_single_
 * broadcast_postamble.h:249-309): a thread a target up to t0 in-edges, 16 lanes up to
 * t1, a CTA beyond; then the end of the superstep. */
#ifndef IPX_TARGET_CTAS
#define IPX_TARGET_CTAS 4
#endif
__global__ void __launch_bounds__(IPX_THREADS, IPX_TARGET_CTAS) ipx_k_gather_targets(ipx_loop loop)
{
    if (ipx_done()) return;
    __shared__ bool s_has[IPX_THREADS / 32];
    __shared__ ipx_msg s_acc[IPX_THREADS / 32];
    const uint32_t stamp = (uint32_t)ipx_step();
    const ipx_vid* __restrict__ adj = ipx_c.in_adj;
    const uint64_t* __restrict__ row = ipx_c.in_row;
    const ipx_bslot* bs = ipx_c.bslot[0];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t n2 = __ldcg(&ipx_c.stat->tn[2]);
    for (uint32_t i = blockIdx.x; i < n2; i += gridDim.x) {
        const uint64_t v = ipx_c.tlist[2][i];
        bool has = false;
        ipx_msg acc;
        ipx_gather_fold_edges(adj, bs, stamp, row[v], row[v + 1], threadIdx.x, blockDim.x, has, acc);
        ipx_warp_fold(has, acc);
        if (lane == 0) {
            s_has[warp] = has;
            s_acc[warp] = acc;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            has = false;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) ipx_fold(has, acc, s_has[w], s_acc[w]);
            ipx_gather_done(v, has, acc, ipx_vertex_state(), nullptr, stamp);
        }
        __syncthreads();
    }
    ipx_gather_rows<IPX_GATHER_LONG, false, false>(ipx_c.tlist[1], __ldcg(&ipx_c.stat->tn[1]), adj, row, bs, stamp, nullptr);
    ipx_gather_rows<1, false, false>(ipx_c.tlist[0], __ldcg(&ipx_c.stat->tn[0]), adj, row, bs, stamp, nullptr);
    if (ipx_last_cta() && threadIdx.x == 0) {
        unsigned long long n = 0;
        for (int k = 0; k < 3; k++) n += __ldcg(&ipx_c.stat->tn[k]);
        ipx_end_of_superstep(loop, n);
    }
}
#endif

/* ------------------------------------------------------------------------ */
/* Initialisation kernels (ip_init_vertex_range of each version).           */
/* ------------------------------------------------------------------------ */
__global__ void ipx_k_init_values(uint64_t first, uint64_t last)
{
    /* [first, last] are ids in the caller's numbering: on a renamed graph
     * every vertex checks its own id */
    const bool renamed = ipx_c.vid_of != nullptr;
    const uint64_t lo = renamed ? 0 : first, hi = renamed ? ~0ULL : last;
    for (uint64_t v = lo + ipx_gtid(); v <= hi && v < ipx_c.V; v += ipx_gstride()) {
        if (renamed) {
            const uint64_t id = ipx_c.vid_of[v];
            if (id < first || id > last) continue;
        }
        ipx_c.value[v] = ipx_val();
#if IPX_VERSION == IPX_SINGLE_BROADCAST
        ipx_c.active_b[v] = 1;
#endif
#if IPX_VERSION == IPX_COMBINER || IPX_VERSION == IPX_SPREAD
        ipx_c.mbox[0][v] = ipx_mb::empty();
        ipx_c.mbox[1][v] = ipx_mb::empty();
#endif
    }
}

/* out[i] = value of the vertex whose id is i in the caller's numbering. */
__global__ void ipx_k_values_by_id(ipx_val* __restrict__ out)
{
    for (uint64_t i = ipx_gtid(); i < ipx_c.V; i += ipx_gstride()) out[i] = ipx_c.value[ipx_c.vindex_of[i]];
}

__global__ void ipx_k_fill_bits(uint32_t* bm, uint64_t V, uint64_t W)
{
    for (uint64_t w = ipx_gtid(); w < W; w += ipx_gstride()) {
        uint32_t x = IPX_FULL;
        if (w == W - 1 && (V & 31)) x = (1u << (V & 31)) - 1u;
        bm[w] = x;
    }
}

#if IPX_VERSION == IPX_COMBINER || IPX_VERSION == IPX_SPREAD
/* Active count of the superstep and its end: the vertices that received mail
 * (spread), or that are active or did (combiner_postamble.h:151-183). */
__global__ void __launch_bounds__(IPX_THREADS) ipx_k_count(ipx_loop loop)
{
    if (ipx_done(false)) return;
    /* four words at a time: the bitmaps' last words of four are padding */
    const uint4* r = reinterpret_cast<const uint4*>(ipx_c.recv[ipx_parity()]);
    unsigned long long c = 0;
    for (uint64_t i = ipx_gtid(); i < (ipx_c.W + 3) / 4; i += ipx_gstride()) {
        uint4 x = r[i];
#if IPX_VERSION == IPX_COMBINER
        const uint4 a = reinterpret_cast<const uint4*>(ipx_c.active_bm)[i];
        x.x |= a.x;
        x.y |= a.y;
        x.z |= a.z;
        x.w |= a.w;
#endif
        c += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
    }
    ipx_block_count(c, &ipx_c.stat->count);
    if (ipx_last_cta() && threadIdx.x == 0) ipx_end_of_superstep(loop, __ldcg(&ipx_c.stat->count));
}
#endif

/* Checks an IP_COMBINE_KIND hint against the user's ip_combine on sample
 * pairs before the hint is trusted. */
__global__ void ipx_k_check_hint(int kind)
{
    if (threadIdx.x == 0) ipx_step_word() = ipd_compute_superstep;
    __syncthreads();
    for (uint64_t i = ipx_gtid(); i < 4096; i += ipx_gstride()) {
        unsigned long long ra = (i * 0x9E3779B97F4A7C15ULL) ^ (i >> 3), rb = (i * 0xC2B2AE3D27D4EB4FULL) + 7;
        ipx_msg a, b;
        if constexpr (std::is_floating_point<ipx_msg>::value) {
            a = (ipx_msg)((double)(ra >> 11) * (1.0 / 9007199254740992.0));
            b = (ipx_msg)((double)(rb >> 11) * (1.0 / 9007199254740992.0));
        } else if constexpr (std::is_integral<ipx_msg>::value) {
            a = (ipx_msg)((i & 1) ? (ra & 0xFFFF) : ra);
            b = (ipx_msg)((i & 2) ? (rb & 0xFFFF) : rb);
        } else {
            return;
        }
        ipx_msg c = a;
        ip_combine(&c, b);
        ipx_msg e;
        if (kind == IP_COMBINE_MIN) e = (b < a) ? b : a;
        else if (kind == IP_COMBINE_MAX) e = (b > a) ? b : a;
        else e = a + b;
        if (!(c == e)) atomicOr(ipx_c.err, IPX_ERR_COMBINE_HINT);
    }
}

#endif /* IPREGEL_B200_ENGINE_CUH */
