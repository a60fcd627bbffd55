// riv_rans.cuh -- the rANS batches of a coefficient stream on the GPU (com/rans.rs:215-292).
//
// Included by riv_kernels.cu inside namespace riv, after riv_symbols.cuh, whose stacks it codes: every
// batch of SYM_BATCH symbols starts from fresh states, so the batches are independent; inside one,
// the symbols alternate between two states, newest first, and a state that would grow too large
// gives up its low 16 bits before its symbol.
//
//   rans_cta         one warp per batch: 32 lanes prepare 64 symbols (frequency, reciprocal), lanes 0
//                    and 1 step the two states through them, 32 lanes write the words out, over the
//                    symbols already read
//   rans_gather_cta  the batches' words one behind the other, and the frame's side info, into the
//                    host's pinned buffers
//
// The frames of multi-clip steps are coded here, beside the next step's search: a step of 24 clips
// has some 575 batches, one per scheduler, and the host's threads took longer for them (75 million
// symbols in 8 steps) than the GPU for everything else.  One frame alone is coded faster by the
// host's threads: a batch takes 200 us here, about 60 us there, and there is nothing to hide it behind.
//
constexpr int RA_WARPS = 4;  // batches of a CTA, one on each scheduler

// floor(x / f) of any 32-bit x as (x * m + a) >> (32 + s), s = floor(log2 f): m = ceil(2^(32 + s) / f) and
// a = 0 where that exceeds the quotient by at most 2^s / f, else m = floor(2^(32 + s) / f) and a = m; one
// of the two is exact (A. Robison, N-bit unsigned division via N-bit multiply-add, 2005).  Powers of
// two: m = 2^31 and s one less; 1: m = 2^32 - 1 and a = m.
__device__ __forceinline__ uint2 ra_reciprocal(unsigned f) {
    if (f == 1u) return make_uint2(0xffffffffu, 1u << 8);
    const int s = 31 - __clz((int)f);
    if ((f & (f - 1u)) == 0u) return make_uint2(0x80000000u, (unsigned)(s - 1));
    const unsigned long long n = 1ull << (32 + s);
    const unsigned long long q = n / f, up = q + 1;
    const bool exact = up * f - n <= (1ull << s);
    return make_uint2((unsigned)(exact ? up : q), (unsigned)s | (exact ? 0u : 1u << 8));
}

struct RaSmem {
    // per state, its 32 symbols (4 more are read, not used): (m, f << 24, a, 0), (s, s + 16, start, 256 - f)
    uint4 sym[2][2 * 36 + 1];
    __align__(16) uint32_t state[2][32];  // before each symbol
};

// Bound by the serial steps of the two states, 8193 each in a full batch (200 us, 49 cycles each, for
// up to 592 batches; 255 us for 1184; 245 us with packed fields, found after the compare): their instructions, most of
// which the pipes take two cycles for, more than their latency.  So a step has nothing that another
// lane could do (its fields come unpacked; whether the state gave up 16 bits is worked out again from
// the states it leaves behind), and it multiplies before it knows whether 16 bits go, because
// floor((x >> 16) / f) = floor(x / f) >> 16.
__device__ __forceinline__ uint32_t rans_step(uint32_t x, const uint4 v, const uint4 q) {
    uint32_t y;
    asm("{\n\t.reg .pred p;\n\t.reg .u64 d, a;\n\t.reg .u32 l, h, s, r;\n\t"
        "mov.b64 a, {%4, %5};\n\t"
        "mad.wide.u32 d, %1, %2, a;\n\t"
        "setp.ge.u32 p, %1, %3;\n\t"
        "selp.u32 s, %7, %6, p;\n\t"
        "add.u32 r, %1, %8;\n\t"
        "@p shr.u32 r, %1, 16;\n\t"
        "@p add.u32 r, r, %8;\n\t"
        "mov.b64 {l, h}, d;\n\t"
        "shf.r.wrap.b32 h, h, 0, s;\n\t"
        "mad.lo.u32 %0, h, %9, r;\n\t}"
        : "=r"(y)
        : "r"(x), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w));
    return y;
}
__device__ __forceinline__ void rans_batch(uint16_t* __restrict__ st, int m, uint4* info, const uint2* rcp, RaSmem& S, int lane) {
    st += SYM_BATCH - (unsigned)m;  // newest symbol first; the words take the place of symbols that were read
    uint32_t x = 65536u;            // lane 0: the state of symbols 0, 2, ...; lane 1: of 1, 3, ...
    int base = 0;
    unsigned e0 = 2 * lane < m ? st[2 * lane] : 0x80u, e1 = 2 * lane + 1 < m ? st[2 * lane + 1] : 0x80u;
    for (int c = 0; c < m; c += 64) {
        uint32_t limit[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const unsigned e = h ? e1 : e0;
            const unsigned p = max(e & 255u, 1u), start = e & 256u ? p : 0u, f = e & 256u ? 256u - p : p;
            const uint2 r = rcp[f];
            limit[h] = f << 24;
            S.sym[h][2 * lane] = make_uint4(r.x, f << 24, r.y & 256u ? r.x : 0u, 0u);
            S.sym[h][2 * lane + 1] = make_uint4(r.y & 31u, (r.y & 31u) + 16u, start, 256u - f);
        }
        const int k = c + 64 + 2 * lane;  // the next 64 symbols, in flight meanwhile
        e0 = k < m ? st[k] : 0x80u;
        e1 = k + 1 < m ? st[k + 1] : 0x80u;
        __syncwarp();
        if (lane < 2) {
            const int n = min(32, (m - c + 1 - lane) >> 1);
            const uint4* q = S.sym[lane];
            uint32_t* o = S.state[lane];
            if (n == 32) {
                // 4 at a time, the next 4 on their way from shared memory (in a loop: unrolled, the
                // compiler moves each load to its use and every step waits for one)
                uint4 v[8], w[8];
                auto load = [&](uint4 (&b)[8], int g) {
#pragma unroll
                    for (int t = 0; t < 8; t++) b[t] = q[2 * g + t];
                };
                auto run = [&](const uint4 (&b)[8], int g) {
                    uint4 s;
                    s.x = x;
                    s.y = rans_step(s.x, b[0], b[1]);
                    s.z = rans_step(s.y, b[2], b[3]);
                    s.w = rans_step(s.z, b[4], b[5]);
                    x = rans_step(s.w, b[6], b[7]);
                    *(uint4*)(o + g) = s;
                };
                load(v, 0);
#pragma unroll 1
                for (int g = 0; g < 32; g += 8) {
                    load(w, g + 4);
                    run(v, g);
                    load(v, g + 8);
                    run(w, g + 4);
                }
            } else {
                for (int t = 0; t < n; t++) {
                    o[t] = x;
                    x = rans_step(x, q[2 * t], q[2 * t + 1]);
                }
            }
        }
        __syncwarp();
        const uint32_t x0 = S.state[0][lane], x1 = S.state[1][lane];
        const bool out0 = c + 2 * lane < m && x0 >= limit[0], out1 = c + 2 * lane + 1 < m && x1 >= limit[1];
        const uint32_t me = __ballot_sync(0xffffffffu, out0), mo = __ballot_sync(0xffffffffu, out1), lt = (1u << lane) - 1u;
        int at = base + __popc(me & lt) + __popc(mo & lt);  // in the order of the symbols, one word at most each
        if (out0) st[at++] = (uint16_t)x0;
        if (out1) st[at] = (uint16_t)x1;
        base += __popc(me) + __popc(mo);
        __syncwarp();
    }
    const uint32_t r0 = __shfl_sync(0xffffffffu, x, m & 1), r1 = __shfl_sync(0xffffffffu, x, ~m & 1);
    if (lane == 0) *info = make_uint4((uint32_t)base, r0, r1, 0u);
}

__device__ __forceinline__ void rans_cta(const RansFrame& f, int cta) {
    __shared__ uint2 rcp[256];
    __shared__ RaSmem S[RA_WARPS];
    const uint32_t n = f.info[0].x;
    if (n == SYM_FAIL || (uint32_t)cta * RA_WARPS * SYM_BATCH >= n) return;
    for (int i = threadIdx.x; i < 256; i += 32 * RA_WARPS) rcp[i] = ra_reciprocal((unsigned)max(i, 1));
    __syncthreads();
    const int w = threadIdx.x >> 5;
    const uint32_t b = (uint32_t)cta * RA_WARPS + w;
    if (b * SYM_BATCH >= n) return;
    rans_batch(f.stack + (size_t)b * SYM_BATCH, (int)min(SYM_BATCH, n - b * SYM_BATCH), f.info + 1 + b, rcp, S[w], threadIdx.x & 31);
}

// Batch b's words (the states, then its words backwards) behind those of the batches before it, as
// 32-bit stores; the CTA of the last batch writes the stream's size.  Further CTAs copy the side info.
constexpr int RA_GATHER = 256;
constexpr int RA_SIDE = 4096;  // side words of a CTA
__device__ __forceinline__ void rans_gather_cta(const RansFrame& f, int cta, int side_ctas) {
    __shared__ unsigned part[RA_GATHER / 32];
    if (cta < side_ctas) {
        for (int i = cta * RA_SIDE + (int)threadIdx.x; i < min(f.nside, (cta + 1) * RA_SIDE); i += RA_GATHER) f.side_out[i] = f.side[i];
        return;
    }
    const uint32_t n = f.info[0].x, b = (uint32_t)(cta - side_ctas);
    const uint32_t nb = n == SYM_FAIL ? 0u : (n + SYM_BATCH - 1u) / SYM_BATCH;
    if (nb == 0 && b == 0 && threadIdx.x == 0) *f.out_bytes = n == SYM_FAIL ? SYM_FAIL : 0u;
    if (b >= nb) return;
    unsigned sum = 0;
    for (uint32_t i = threadIdx.x; i < b; i += RA_GATHER) sum += f.info[1 + i].x + 4u;
    sum = __reduce_add_sync(0xffffffffu, sum);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    unsigned first = 0;
#pragma unroll
    for (int i = 0; i < RA_GATHER / 32; i++) first += part[i];
    const uint4 q = f.info[1 + b];
    const int size = (int)q.x + 4, odd = (int)(first & 1u);
    const bool fits = 2ull * (first + (unsigned)size) <= f.out_cap;
    if (b + 1 == nb && threadIdx.x == 0) *f.out_bytes = fits ? 2u * (first + (unsigned)size) : SYM_FAIL;
    if (!fits) return;
    const uint16_t* src = f.stack + (size_t)b * SYM_BATCH + (SYM_BATCH - min(SYM_BATCH, n - b * SYM_BATCH));
    uint16_t* dst = (uint16_t*)f.out + first;
    auto word = [&](int i) -> unsigned {
        if (i >= 4) return src[size - 1 - i];
        const uint32_t r = i < 2 ? q.z : q.y;
        return i & 1 ? r >> 16 : r & 0xffffu;
    };
    for (int i = 2 * (int)threadIdx.x - odd; i < size; i += 2 * RA_GATHER) {
        if (i < 0) dst[0] = (uint16_t)word(0);
        else if (i + 1 == size) dst[i] = (uint16_t)word(i);
        else *(uint32_t*)(dst + i) = word(i) | word(i + 1) << 16;
    }
}

static inline int rans_batches(unsigned cap) { return (int)((cap + SYM_BATCH - 1u) / SYM_BATCH); }
static inline int rans_side_ctas(int nside) { return (nside + RA_SIDE - 1) / RA_SIDE; }
size_t rans_info_bytes(unsigned cap) { return (size_t)(1 + rans_batches(cap)) * sizeof(uint4); }
// A symbol grows its state by 8 bits and log2(1 + 1 / 256) at most (a state is 2^8 f or more when its
// symbol of frequency f is coded).
size_t rans_max_bytes(unsigned cap) { return (size_t)cap + cap / 512 + 16 * (size_t)rans_batches(cap); }
