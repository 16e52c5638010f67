// Pieces shared by the transfer engines (kv_transfer.cu, kv_transfer_tma.cu): the way pages are handed out, when progress is
// published in the credit page, the end of a launch, and the fp8 packing of eight elements.
#pragma once
#include <cuda_fp8.h>

#include <cstddef>

#include "common.cuh"
#include "kv_transfer.h"

namespace sky {

// Work is handed out in units: a chunk of `pages_per_chunk` pages (the granularity of credit, cursor and accounting) cut into
// `subs` parts, so that a short transfer still reaches every CTA (17 tokens are 144 pages, 18 chunks). All units of a chunk ask for
// the chunk's credit, so they are granted or refused together.
struct KvUnits {
    long long n_pages, n_units, pages_per_pair;
    int per;                                           // pages per unit
    __device__ explicit KvUnits(const KvTransferParams& p) {
        pages_per_pair = 2LL * p.layers;
        n_pages = pages_per_pair * p.n_pairs;
        const long long n_chunks = (n_pages + p.pages_per_chunk - 1) / p.pages_per_chunk;
        n_units = n_chunks * p.subs;
        per = (p.pages_per_chunk + p.subs - 1) / p.subs;
    }
    __device__ void pages_of(const KvTransferParams& p, long long unit, long long& page0, long long& page1) const {
        const long long chunk = unit / p.subs;
        const int sub = (int)(unit - chunk * p.subs);
        const long long end = min((chunk + 1) * (long long)p.pages_per_chunk, n_pages);
        page0 = min(chunk * (long long)p.pages_per_chunk + (long long)sub * per, end);
        page1 = min(page0 + per, end);
    }
};

// Every CTA starts on the unit of its own index; later units come from the launch's counter. A ticket that was taken is always
// resolved (moved, or refused and recorded in the cursor), so it may be taken ahead of time. All of them in order of need.
__device__ __forceinline__ long long kv_next_unit(const KvTransferParams& p, const KvUnits& u) {
    const long long first = (long long)p.first_chunk * p.subs + gridDim.x;
    if (first >= u.n_units) return u.n_units;
    return first + atomicAdd(&p.status->work_counter, 1u);
}

// Credit and progress of one driving thread. How often progress goes into the page: every chunk while the flow is paced, every
// SKY_PUBLISH_CHUNKS-th chunk of the flow while it is not (8 MB between two publications are 10 us at link rate, a control window
// is a millisecond or more).
// The page is host memory. Reads of it take about 0.7 us each and do not overlap: when every CTA read it for itself (three or four
// words, again after every 256 MB of the flow), 64k tokens took 12.3 ms, 10 of them these reads, and 17 tokens 98 us. So the CTAs share
// what is known of the grant (SkyGrantCache) and whoever holds its lock reads the page for all; a flow that is not paced is looked
// at again while half of the last look is still unused, so that nobody waits for that read.
constexpr unsigned long long SKY_PUBLISH_CHUNKS = 32;

struct KvCredit {
    unsigned long long grant_cache = 0, stall_ns = 0, my_bytes = 0, my_chunks = 0, last_need = 0;
    bool unlimited = false;

    // Waits (bounded) until the flow's grant covers `need`. On refusal `code` says why.
    __device__ bool wait_grant(const KvTransferParams& p, unsigned long long need, unsigned long long max_wait_ns, unsigned detail, unsigned& code) {
        SkyGrantCache* gc = p.grant;
        unsigned long long t0 = 0;
        unsigned ns = 64;
        for (;;) {
            const unsigned long long g = *(volatile unsigned long long*)&gc->granted;
            const unsigned unl = *(volatile unsigned int*)&gc->unlimited;
            if (need <= g) {
                unlimited = unl != 0;
                const unsigned long long half = SKY_UNLIMITED_RECHECK_BYTES / 2;
                if (!unl || need + half < g) { grant_cache = unl ? g - half : g; break; }
                if (atomicCAS(&gc->lock, 0u, 1u) != 0u) { grant_cache = need; break; }     // somebody is looking already
                unsigned long long cache = 0, none = 0;
                bool stopped, lost;
                const bool ok = credit_acquire(p.page, need, &cache, 0ull, &none, &stopped, &lost, gc);
                __threadfence();
                atomicExch(&gc->lock, 0u);
                if (!ok && stopped) { code = SKY_STATUS_STOPPED; return false; }
                grant_cache = need;
                break;
            }
            const unsigned long long now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            if (atomicCAS(&gc->lock, 0u, 1u) == 0u) {
                bool stopped, lost;
                const unsigned long long left = now - t0 < max_wait_ns ? max_wait_ns - (now - t0) : 0ull;
                const bool ok = credit_acquire(p.page, need, &grant_cache, left, &stall_ns, &stopped, &lost, gc);
                unlimited = *(volatile unsigned int*)&gc->unlimited != 0;
                if (ok && unlimited) grant_cache -= SKY_UNLIMITED_RECHECK_BYTES / 2;
                code = stopped ? SKY_STATUS_STOPPED : lost ? SKY_STATUS_CONTROL_LOST : SKY_STATUS_YIELD_CREDIT;
                if (!ok) set_status(p.status, code, detail);              // before the lock is free: the others shall not start over
                __threadfence();
                atomicExch(&gc->lock, 0u);
                return ok;
            }
            const unsigned st = *(volatile unsigned int*)&p.status->status;
            if (st != SKY_STATUS_OK || now - t0 > max_wait_ns) {
                code = st != SKY_STATUS_OK ? st : SKY_STATUS_YIELD_CREDIT;
                stall_ns += now - t0;
                return false;
            }
            __nanosleep(ns);
            if (ns < 1024) ns <<= 1;
        }
        if (t0) stall_ns += globaltimer_ns() - t0;
        return true;
    }

    // True: the pages of `unit` may be sent. False: refused, and the cursor and the status say why.
    __device__ bool acquire(const KvTransferParams& p, const KvUnits& u, long long unit, unsigned long long page_link_bytes) {
        const unsigned long long k = (unsigned long long)(unit / p.subs);
        const bool first_sub = unit == (long long)k * p.subs;
        const long long chunk_end = min((long long)(k + 1) * p.pages_per_chunk, u.n_pages);
        const unsigned long long need = p.consumed_base + (unsigned long long)(chunk_end - (long long)p.first_chunk * p.pages_per_chunk) * page_link_bytes;
        // A launch that is to end: a bad block id or a lost barrier ends it for good; a stop is obeyed at once; and once a chunk has
        // been refused, later ones are not begun (a resumed launch would move them again) and earlier ones do not wait.
        const unsigned st = *(volatile unsigned int*)&p.status->status;
        if (st != SKY_STATUS_OK) {
            if (st == SKY_STATUS_BAD_INDEX || st == SKY_STATUS_TIMEOUT_MBAR) return false;
            if (st != SKY_STATUS_YIELD_CREDIT || k > *(volatile unsigned long long*)&p.status->cursor) {
                atomicMin(&p.status->cursor, k);
                return false;
            }
        }
        if (p.page && need > grant_cache) {
            unsigned code = SKY_STATUS_YIELD_CREDIT;
            if (!wait_grant(p, need, st == SKY_STATUS_OK ? p.max_wait_ns : 0ull, (unsigned)k, code)) {
                if (code == SKY_STATUS_BAD_INDEX || code == SKY_STATUS_TIMEOUT_MBAR) return false;
                atomicMin(&p.status->cursor, k);
                set_status(p.status, code, (unsigned)k);
                return false;
            }
        }
        // granted, but perhaps after a wait that an earlier chunk did not outlast
        if (p.page && !unlimited && *(volatile unsigned int*)&p.status->status == SKY_STATUS_YIELD_CREDIT && k > *(volatile unsigned long long*)&p.status->cursor)
            return false;
        if (p.usage && first_sub && (!unlimited || k % SKY_PUBLISH_CHUNKS == 0)) {
            // chunks are ticketed in order, so `need` is within a few chunks of the true cumulative count
            st_sys_u64((unsigned long long*)&p.usage->consumed_bytes, need);
            if (last_need) st_sys_u64((unsigned long long*)&p.usage->completed_bytes, last_need);
        }
        last_need = need;
        long long page0, page1;
        u.pages_of(p, unit, page0, page1);
        my_bytes += (unsigned long long)(page1 - page0) * page_link_bytes;
        my_chunks += first_sub ? 1 : 0;
        return true;
    }
};

// The end of a CTA's share, by one thread whose own and whose CTA's payload writes are complete or ordered before this call. The
// last CTA of the launch publishes the usage counters and the ready flags, hands the outcome to `result` and its host copy `mirror`,
// and leaves the working block as it found it, ready for the flow's next launch.
__device__ __forceinline__ void kv_finish(const KvTransferParams& p, const KvCredit& c) {
    if (c.my_chunks) atomicAdd(&p.status->chunks_done, c.my_chunks);
    if (c.my_bytes) atomicAdd(&p.status->bytes_done, c.my_bytes);
    if (c.stall_ns) atomicAdd(&p.status->stall_ns, c.stall_ns);
    __threadfence_system();
    const unsigned prev = atomicAdd(&p.status->ctas_done, 1u);
    if (prev != gridDim.x - 1) return;
    __threadfence();
    volatile LaunchStatus* w = p.status;
    LaunchStatus s;
    s.status = w->status; s.detail = w->detail; s.cursor = w->cursor; s.chunks_done = w->chunks_done; s.bytes_done = w->bytes_done;
    s.stall_ns = w->stall_ns; s.t_start_ns = w->t_start_ns; s.ctas_done = prev + 1; s.work_counter = w->work_counter;
    SkyCreditPage* u = p.usage;
    ulonglong2 stall_busy = make_ulonglong2(0, 0), ts_chunks = make_ulonglong2(0, 0);
    static_assert(offsetof(SkyCreditPage, stall_ns) % 16 == 0 && offsetof(SkyCreditPage, busy_ns) == offsetof(SkyCreditPage, stall_ns) + 8 &&
                  offsetof(SkyCreditPage, last_ts_ns) % 16 == 0 && offsetof(SkyCreditPage, chunks) == offsetof(SkyCreditPage, last_ts_ns) + 8, "pairs");
    if (u) {                                       // host memory: two reads for the three counters
        stall_busy = ld_sys_u64x2((const unsigned long long*)&u->stall_ns);
        ts_chunks = ld_sys_u64x2((const unsigned long long*)&u->last_ts_ns);
    }
    const bool complete = s.status == SKY_STATUS_OK;
    if (complete) {
        __threadfence_system();
        for (int g = 0; g < p.n_dst; ++g)
            if (p.done_flag[g]) st_release_sys_u32(p.done_flag[g], p.done_value);
    }
    const unsigned long long now = globaltimer_ns();
    s.t_end_ns = now;
    if (u) {
        st_sys_u64((unsigned long long*)&u->consumed_bytes, p.consumed_base + s.bytes_done);
        st_sys_u64((unsigned long long*)&u->completed_bytes, p.consumed_base + s.bytes_done);
        st_sys_u64((unsigned long long*)&u->stall_ns, stall_busy.x + s.stall_ns);
        st_sys_u64((unsigned long long*)&u->busy_ns, stall_busy.y + (now - s.t_start_ns));
        st_sys_u64((unsigned long long*)&u->chunks, ts_chunks.y + s.chunks_done);
        st_sys_u64((unsigned long long*)&u->last_ts_ns, now);
        if (!complete) st_sys_u64((unsigned long long*)&u->yields, ld_sys_u64((const unsigned long long*)&u->yields) + 1);
    }
    *p.mirror = s;
    *p.result = s;
    LaunchStatus z = {};
    z.cursor = ~0ull;
    z.t_start_ns = ~0ull;
    *p.status = z;
    *p.grant = SkyGrantCache{};
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// 8 bf16 -> 8 e4m3 with a shared scale 2^e chosen over 32 consecutive elements
// (4 neighbouring lanes). Returns the packed bytes; *scale_byte gets e + 127.
__device__ __forceinline__ uint2 pack_fp8_mx(uint4 v, bool valid, unsigned char* scale_byte) {
    float f[8] = {bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y), bf16_lo(v.z), bf16_hi(v.z), bf16_lo(v.w), bf16_hi(v.w)};
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(valid ? f[i] : 0.f));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    // Smallest power of two 2^e with amax / 2^e <= 448 = 1.75 * 2^8, from the float's own fields so
    // that the choice is exact: amax = m * 2^k with m in [1,2)  =>  e = k - 8 + (m > 1.75).
    const uint32_t bits = __float_as_uint(amax);
    int e = (int)(bits >> 23) - 127 - 8 + ((bits & 0x7fffffu) > 0x600000u ? 1 : 0);
    if (amax == 0.f) e = -127;
    e = max(-127, min(127, e));
    float inv = exp2f((float)-e);
    *scale_byte = (unsigned char)(e + 127);
    uint2 out;
    unsigned short p0 = __nv_cvt_float2_to_fp8x2(make_float2(f[0] * inv, f[1] * inv), __NV_SATFINITE, __NV_E4M3);
    unsigned short p1 = __nv_cvt_float2_to_fp8x2(make_float2(f[2] * inv, f[3] * inv), __NV_SATFINITE, __NV_E4M3);
    unsigned short p2 = __nv_cvt_float2_to_fp8x2(make_float2(f[4] * inv, f[5] * inv), __NV_SATFINITE, __NV_E4M3);
    unsigned short p3 = __nv_cvt_float2_to_fp8x2(make_float2(f[6] * inv, f[7] * inv), __NV_SATFINITE, __NV_E4M3);
    out.x = (uint32_t)p0 | ((uint32_t)p1 << 16);
    out.y = (uint32_t)p2 | ((uint32_t)p3 << 16);
    return out;
}

}  // namespace sky
