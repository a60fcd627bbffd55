// riv_symbols.cuh -- the DCT-coefficient coder's symbols and adaptive models on the GPU.
//
// Included by riv_kernels.cu inside namespace riv.  A frame's coefficient stream is a list of
// binary symbols (res/rans.rs:195-330), each coded either with a fixed probability (bypass) or
// with one of 427 adaptive models that start fresh every frame.  A model's probability at each
// of its symbols depends only on the bits it saw before, so the list can be made block-parallel
// and the models can run beside one another; what stays serial is the rANS state of each
// 16386-symbol batch, which riv_rans.cuh or the host codes from the (probability, bit) stacks left here.  The
// stacks are laid out as the host's writer fills them: batch k / 16386, newest symbol first.
//
//   k_sym_count   one warp per SY_MBS macroblocks: symbols per model, coded MBs, coefficients
//   k_sym_scan    exclusive scan of a CTA's counts over the CTAs, per row (model or total)
//   k_sym_emit    the same walk again: side info, every bypass symbol into its stack slot,
//                 every modelled symbol's (stack position, bit) into its model's list
//   k_sym_chain   one CTA per model: the model's counts at every 128th symbol of its list
//   k_sym_model   one warp per 128 symbols: their probabilities, into their stack slots
//
// 1080p P-frame of 662,000 symbols: 12 + 11 + 24 + 42 + 10 us.  On the host one thread takes about
// 2 ms to list and model such a frame, several threads 1.4 to 2.8 ms.
//
// A frame whose symbols exceed the stack, or that holds a magnitude class the reference cannot
// code, is marked in the header word instead and its coefficients are packed (pack_mb_at) for the
// host coder.
//
constexpr int SY_MBS = 2;         // macroblocks of a part (one warp)
constexpr int SY_WARPS = 8;       // parts of a CTA
constexpr int SY_MODELS = 427;    // adaptive models, in the host coder's numbering
constexpr int SY_SIG_Y = 0, SY_SIG_C = 256, SY_MAG_Y = 320, SY_MAG_C = 372, SY_EOB_Y = 411, SY_EOB_C = 420;
constexpr int SY_CODED = 427, SY_COEFS = 428, SY_SYMS = 429, SY_BAD = 430;  // further rows of the counts
static_assert(SY_EOB_C + 7 == SY_MODELS && SY_BAD < SYM_ROWS && SYM_ROWS % 32 == 0, "rows of the count table");
static_assert(SY_MBS * 384 * 27 < 65536, "a part's counts fit 16 bits (at most 27 symbols a coefficient)");
constexpr unsigned SY_BATCH = SYM_BATCH;
constexpr unsigned SY_UNIT = SYM_UNIT;

__device__ __forceinline__ unsigned sy_slot(unsigned k) {
    const unsigned b = k / SY_BATCH;
    return b * SY_BATCH + (SY_BATCH - 1u) - (k - b * SY_BATCH);
}
__device__ __forceinline__ int sy_len(unsigned v) { return 32 - __clz((int)v); }  // 0 -> 0

// Walks the symbols of one part (warp-collective).  Sink S:
//   mb(m, coded, e0, e1, e2)             start of a macroblock, all lanes
//   eob(model0, cls, maxc, last)         an EOB class, all lanes
//   chunk(i, act, v, cls, sig0, mag0, band)  up to 32 coefficients of a plane; v = 0 where !act,
//                                        band = the lanes of this lane's magnitude band
// A macroblock's coefficients (lane, lane + 32, ... of each plane, up to its last) are loaded
// while the one before is walked.
template <class S>
__device__ __forceinline__ void sy_walk(const SymFrame& f, int part, int lane, S& s) {
    const int m0 = part * SY_MBS, mn = min(SY_MBS, f.nmb - m0);
    int e = 0;
    bool cd = false;
    if (lane < mn) {
        const uint8_t* q = f.eobs + 3 * (m0 + lane);
        e = q[0] | (q[1] << 8) | (q[2] << 16);
        cd = f.intra || !f.opt_skip[m0 + lane];
    }
    const unsigned coded = __ballot_sync(0xffffffffu, cd);
    auto load = [&](int k, int (&v)[12]) {  // luma 0 .. 7, U 8, 9, V 10, 11
        const int ew = __shfl_sync(0xffffffffu, e, k);
        const int16_t* co = f.coeffs + (size_t)(m0 + k) * 384 + lane;
        if (!((coded >> k) & 1u)) return;
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = lane + 32 * j <= (ew & 255) ? (int)co[32 * j] : 0;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            v[8 + j] = lane + 32 * j <= ((ew >> 8) & 255) ? (int)co[256 + 32 * j] : 0;
            v[10 + j] = lane + 32 * j <= (ew >> 16) ? (int)co[320 + 32 * j] : 0;
        }
        if (f.intra && lane == 0 && m0 + k > 0) {  // DCs against the previous block's
            v[0] = (int16_t)(v[0] - (int)co[-384]);
            v[8] = (int16_t)(v[8] - (int)co[256 - 384]);
            v[10] = (int16_t)(v[10] - (int)co[320 - 384]);
        }
    };
    int nx[12];
    load(0, nx);
#pragma unroll 1
    for (int k = 0; k < mn; k++) {
        int v[12];
#pragma unroll
        for (int j = 0; j < 12; j++) v[j] = nx[j];
        if (k + 1 < mn) load(k + 1, nx);
        const int ew = __shfl_sync(0xffffffffu, e, k);
        const bool is = (coded >> k) & 1u;
        s.mb(m0 + k, is, ew & 255, (ew >> 8) & 255, ew >> 16);
        if (!is) continue;
#pragma unroll
        for (int pl = 0; pl < 3; pl++) {
            const int last = (ew >> (8 * pl)) & 255;
            s.eob(pl == 0 ? SY_EOB_Y : SY_EOB_C, sy_len((unsigned)last), pl == 0 ? 8 : 6, last);
#pragma unroll
            for (int b = 0; b < (pl == 0 ? 8 : 2); b++) {
                if (32 * b > last) break;
                const int i = 32 * b + lane, x = v[pl == 0 ? b : 6 + 2 * pl + b];
                const int cls = x != 0 ? sy_len((unsigned)abs(x) - 1u) : -1;
                int mag0;
                unsigned band;
                if (pl == 0) {
                    mag0 = SY_MAG_Y + 13 * (b > 1 ? 3 : b == 1 ? 2 : lane == 0 ? 0 : lane < 16 ? 1 : 2);
                    band = b > 0 ? 0xffffffffu : lane == 0 ? 1u : lane < 16 ? 0xfffeu : 0xffff0000u;
                } else {
                    mag0 = SY_MAG_C + 13 * (b == 1 ? 2 : lane == 0 ? 0 : lane < 8 ? 1 : 2);
                    band = b > 0 ? 0xffffffffu : lane == 0 ? 1u : lane < 8 ? 0xfeu : 0xffffff00u;
                }
                s.chunk(i, i <= last, x, cls, pl == 0 ? SY_SIG_Y : SY_SIG_C, mag0, band);
            }
        }
    }
}

// Symbols of a class code: cls continue bits, a stop bit below maxc, cls - 1 offset bits.
__device__ __forceinline__ int sy_class_syms(int cls, int maxc) { return cls + (cls < maxc ? 1 : 0) + max(cls - 1, 0); }

struct SyCount {
    unsigned* h;  // this warp's counts (shared, SYM_ROWS)
    int lane;
    unsigned coded = 0, coefs = 0, syms = 0, bad = 0;  // syms, bad: per lane
    __device__ __forceinline__ void mb(int, bool is, int e0, int e1, int e2) {
        if (is) {
            coded++;
            coefs += (unsigned)(e0 + e1 + e2 + 3);
        }
    }
    __device__ __forceinline__ void eob(int model0, int cls, int maxc, int) {
        if (lane < cls || (lane == cls && cls < maxc)) h[model0 + lane]++;
        if (lane == 0) syms += (unsigned)sy_class_syms(cls, maxc);
        __syncwarp();
    }
    __device__ __forceinline__ void chunk(int i, bool act, int, int cls, int sig0, int mag0, unsigned band) {
        if (act) {
            h[sig0 + i]++;
            syms++;
        }
        if (cls > 13) bad = 1;
        if (cls >= 0) syms += 1u + (unsigned)sy_class_syms(cls, 12);
        for (int c = 0; c < 13; c++) {
            const unsigned in = __ballot_sync(0xffffffffu, cls > c || (cls == c && c < 12));
            if (in == 0u) break;
            const unsigned mine = in & band;
            if (mine != 0u && lane == __ffs(mine) - 1) h[mag0 + c] += (unsigned)__popc(mine);
        }
        __syncwarp();
    }
};

// Counts of a CTA's parts.  Latency-bound: a warp walks its macroblocks one after another, every
// step a chain of ballots and shared-memory increments; four thousand warps at 1080p hide it.
// Per part 16-bit counts (read back by k_sym_emit), per CTA their sums (scanned by k_sym_scan: a
// scan over the parts themselves read and wrote eight times as much and took 20 us, not 11).
__device__ __forceinline__ void sym_count_cta(const SymFrame& f, int cta, unsigned (*h)[SYM_ROWS]) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, part = cta * SY_WARPS + w;
    unsigned* hw = h[w];
    for (int i = lane; i < SYM_ROWS; i += 32) hw[i] = 0u;
    __syncwarp();
    if (part * SY_MBS < f.nmb) {
        SyCount s;
        s.h = hw;
        s.lane = lane;
        sy_walk(f, part, lane, s);
        const unsigned syms = __reduce_add_sync(0xffffffffu, s.syms), bad = __reduce_max_sync(0xffffffffu, s.bad);
        if (lane == 0) {
            hw[SY_CODED] = s.coded;
            hw[SY_COEFS] = s.coefs;
            hw[SY_SYMS] = syms;
            hw[SY_BAD] = bad;
        }
        __syncwarp();
        uint32_t* o = (uint32_t*)(f.cnt + (size_t)part * SYM_ROWS);
        for (int i = lane; i < SYM_ROWS / 2; i += 32) o[i] = hw[2 * i] | (hw[2 * i + 1] << 16);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < SYM_ROWS; i += 32 * SY_WARPS) {
        unsigned t = 0;
#pragma unroll
        for (int q = 0; q < SY_WARPS; q++) t += h[q][i];
        f.tot[(size_t)cta * SYM_ROWS + i] = t;
    }
    if (cta == 0 && threadIdx.x == 0) f.work[0] = 0u;  // the list cursor k_sym_scan reserves from
}

// Exclusive scan over the CTAs' sums of 32 rows (lane = row, so loads and stores are whole lines)
// by the 32 warps of a CTA: each warp sums its share, then writes the running values.  A model's
// scan starts at the space it reserves in the symbol list.  The CTA of the totals
// writes the frame's header words.
__device__ __forceinline__ void sym_scan_rows(const SymFrame& f, int group) {
    __shared__ unsigned sums[32][33];
    __shared__ unsigned base[32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, row = group * 32 + lane;
    const int n = (f.nmb + SY_MBS * SY_WARPS - 1) / (SY_MBS * SY_WARPS), per = (n + 31) / 32;
    const int p0 = min(w * per, n), p1 = min(p0 + per, n);
    unsigned* c = f.tot + row;
    unsigned sum = 0;
#pragma unroll 16
    for (int p = p0; p < p1; p++) sum = sym_add(sum, c[(size_t)p * SYM_ROWS]);
    sums[w][lane] = sum;
    __syncthreads();
    if (w == 0) {
        unsigned run = 0;
        for (int q = 0; q < 32; q++) {
            const unsigned x = sums[q][lane];
            sums[q][lane] = run;
            run = sym_add(run, x);
        }
        unsigned b = 0;
        if (row < SY_MODELS) {
            b = atomicAdd(f.work, (run + SY_UNIT - 1u) / SY_UNIT * SY_UNIT);  // a list starts on a unit
            f.work[SYM_TAB + 2 * row] = b;
            f.work[SYM_TAB + 2 * row + 1] = run;
        }
        base[lane] = b;
        const unsigned coded = __shfl_sync(0xffffffffu, run, SY_CODED % 32), coefs = __shfl_sync(0xffffffffu, run, SY_COEFS % 32);
        const unsigned syms = __shfl_sync(0xffffffffu, run, SY_SYMS % 32), bad = __shfl_sync(0xffffffffu, run, SY_BAD % 32);
        if (group == SY_SYMS / 32 && lane == 0) {
            const bool ok = bad == 0u && syms <= f.cap;
            f.work[1] = ok ? 1u : 0u;
            f.hdr[0] = coded;
            f.hdr[1] = coefs;
            f.hdr[3] = ok ? syms : SYM_FAIL;
            f.hdr[5] = syms;
            if (f.nsym != nullptr) *f.nsym = ok ? syms : SYM_FAIL;
            if (f.status != nullptr) f.hdr[2] = *(volatile const unsigned*)f.status;
        }
    }
    __syncthreads();
    unsigned run = sums[w][lane] + base[lane];
#pragma unroll 16
    for (int p = p0; p < p1; p++) {
        const unsigned x = c[(size_t)p * SYM_ROWS];
        c[(size_t)p * SYM_ROWS] = run;
        run += x;
    }
}
static_assert(SY_CODED / 32 == SY_BAD / 32, "the totals share a CTA of the scan");

struct SyEmit {
    const SymFrame& f;
    unsigned* h;  // next list position of each model (shared)
    int lane;
    unsigned pos;  // stream position of the next symbol
    __device__ __forceinline__ void put(unsigned k, unsigned at, bool bit) { f.occ[k] = at | (bit ? 0x80000000u : 0u); }
    __device__ __forceinline__ void bypass(unsigned at, bool bit) { f.stack[sy_slot(at)] = (uint16_t)(bit ? 0x180 : 0x80); }
    __device__ __forceinline__ void mb(int m, bool, int, int, int) {
        if (lane == 0) f.side[m] = f.intra ? 0u : side_word(f.mb[m], f.opt_skip[m]);
    }
    __device__ __forceinline__ void eob(int model0, int cls, int maxc, int last) {
        const int n = cls + (cls < maxc ? 1 : 0);
        if (lane < n) put(h[model0 + lane]++, pos + (unsigned)lane, lane < cls);
        // offset bits, most significant first
        if (lane < cls - 1) bypass(pos + (unsigned)(n + lane), (((unsigned)last - (1u << (cls - 1))) >> (cls - 2 - lane)) & 1u);
        pos += (unsigned)sy_class_syms(cls, maxc);
        __syncwarp();
    }
    __device__ __forceinline__ void chunk(int i, bool act, int v, int cls, int sig0, int mag0, unsigned band) {
        unsigned n = act ? 1u : 0u;
        if (cls >= 0) n += 1u + (unsigned)sy_class_syms(cls, 12);
        unsigned x = n;  // inclusive scan of the lanes' symbol counts
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        unsigned at = pos + x - n;
        pos += __shfl_sync(0xffffffffu, x, 31);
        if (act) put(h[sig0 + i]++, at, v != 0);
        if (cls >= 0) bypass(at + 1u, v < 0);
        at += 2u;
        for (int c = 0; c < 13; c++) {
            const bool me = cls > c || (cls == c && c < 12);
            const unsigned in = __ballot_sync(0xffffffffu, me);
            if (in == 0u) break;
            const unsigned mine = in & band;
            unsigned k0 = 0;
            if (me) k0 = h[mag0 + c];
            __syncwarp();
            if (me) {
                put(k0 + (unsigned)__popc(mine & ((1u << lane) - 1u)), at + (unsigned)c, cls > c);
                if (lane == __ffs(mine) - 1) h[mag0 + c] = k0 + (unsigned)__popc(mine);
            }
        }
        if (cls >= 2) {
            at += (unsigned)(cls + (cls < 12 ? 1 : 0));
            const unsigned off = (unsigned)abs(v) - 1u - (1u << (cls - 1));
            for (int b = cls - 2; b >= 0; b--) bypass(at++, (off >> b) & 1u);
        }
        __syncwarp();
    }
};
__device__ __forceinline__ void sym_emit_cta(const SymFrame& f, int cta, unsigned (*hs)[SYM_ROWS]) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, part = cta * SY_WARPS + w;
    // each part's start: the CTA's, plus the parts before it
    const int np = min(SY_WARPS, (f.nmb - cta * SY_WARPS * SY_MBS + SY_MBS - 1) / SY_MBS);
    for (int i = threadIdx.x; i < SYM_ROWS; i += 32 * SY_WARPS) {
        unsigned run = f.tot[(size_t)cta * SYM_ROWS + i];
        for (int q = 0; q < np; q++) {
            hs[q][i] = run;
            run += f.cnt[((size_t)cta * SY_WARPS + q) * SYM_ROWS + i];
        }
    }
    __syncthreads();
    if (w >= np) return;
    unsigned* h = hs[w];
    if (f.work[1] != 0u) {
        SyEmit s{f, h, lane, h[SY_SYMS]};
        sy_walk(f, part, lane, s);
        return;
    }
    // the host coder takes this frame: side info, EOBs and truncated blocks
    unsigned k = h[SY_CODED], off = h[SY_COEFS];
    const int m1 = min((part + 1) * SY_MBS, f.nmb);
    for (int m = part * SY_MBS; m < m1; m++) {
        const bool is = f.intra || !f.opt_skip[m];
        const int e0 = f.eobs[3 * m], e1 = f.eobs[3 * m + 1], e2 = f.eobs[3 * m + 2];
        pack_mb_at(m, lane, is ? (int)k : -1, (int)off, f.opt_skip, f.mb, f.coeffs, e0, e1, e2, f.intra, f.side, f.packed,
                   f.peobs);
        if (is) {
            k++;
            off += (unsigned)(e0 + e1 + e2 + 3);
        }
    }
}

// BinProb after one bit (com/rans.rs:73-84): z zeros and o ones, both 1 .. 255; the count that
// would pass 255 instead halves both (the seen one to 129), except that 255 against 1 stays.
__device__ __forceinline__ void sy_observe(unsigned& a, unsigned& b) {  // a: the seen bit's count
    if (a < 255u) {
        a++;
    } else if (b != 1u) {
        a = 129u;
        b = (b + 1u) >> 1;
    }
}
// floor(256 z / (z + o)), at least 1 (com/rans.rs:30-44); the float quotient is off by at most one
__device__ __forceinline__ unsigned sy_prob(unsigned z, unsigned o) {
    const unsigned n = z << 8, d = z + o;
    int q = (int)__fdividef((float)n, (float)d);
    const int r = (int)n - q * (int)d;
    q += r < 0 ? -1 : r >= (int)d ? 1 : 0;
    return (unsigned)max(q, 1);
}
// The model's counts (z, o) at the start of each unit of 128 symbols of its list.  The counts
// only ever grow by the symbols seen until one of them would pass 255; at such an event (at least
// 126 symbols after the last that halved) they are halved, or stay where they are at 255 against
// 1.  So the CTA turns 4096 symbols at a time into bit words with running counts of ones, and its
// first warp steps from event to event: the event is the (256 - o)-th one or the (256 - z)-th
// zero from here, whichever comes first (at 255 against 1 the first other bit), found by two
// ballots over the words' counts and two inside a word.  Bound by that serial chain over the
// longest list, about 0.5 us an event: 42 us for the 19,400 symbols of a 1080p P-frame's longest
// list and 225 us for the 100,000 of its key frame.  Stepping 128 symbols at a time with their
// probabilities computed on the way took 112 and 622 us, 32 at a time 276 and 1434 us.
constexpr int SY_CHAIN_THREADS = 128, SY_CHAIN_SYMS = 4096;
__device__ __forceinline__ void sym_chain_cta(const SymFrame& f, int model) {
    __shared__ uint32_t word[2][SY_CHAIN_SYMS / 32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned b0 = f.work[SYM_TAB + 2 * model], n = f.work[SYM_TAB + 2 * model + 1];
    const unsigned* l = f.occ + b0;
    int z = 1, o = 1;
    for (unsigned c0 = 0, par = 0; c0 < n; c0 += SY_CHAIN_SYMS, par ^= 1) {
        // warp w: symbols 1024 w .. 1024 w + 1023 of the block, one word per ballot
        const unsigned cw = c0 + 1024u * w;
        uint32_t mine = 0;
        if (cw < n) {
            unsigned e[32];
#pragma unroll
            for (int k = 0; k < 32; k++) e[k] = cw + 32u * k + lane < n ? l[cw + 32u * k + lane] : 0u;
#pragma unroll
            for (int k = 0; k < 32; k++) {
                const uint32_t b = __ballot_sync(0xffffffffu, (e[k] >> 31) != 0u);
                if (lane == k) mine = b;
            }
        }
        word[par][32 * w + lane] = mine;
        __syncthreads();  // the other buffer is refilled while warp 0 walks this one
        if (w != 0) continue;
        for (unsigned c = c0; c < min(c0 + (unsigned)SY_CHAIN_SYMS, n); c += 1024u) {
            const int m = (int)min(1024u, n - c);
            const uint32_t x = word[par][((c - c0) >> 5) + lane];
            int ones = __popc(x);  // inclusive over the words
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, ones, d);
                if (lane >= d) ones += y;
            }
            const int end = min(32 * (lane + 1), m), zeros = end - ones;  // inclusive
            const int o_at = ones - __popc(x), z_at = 32 * lane - o_at;     // before this word
            const bool unit = (lane & 3) == 0 && 32 * lane < m;
            uint32_t* us = f.ustate + (b0 + c) / SY_UNIT + (lane >> 2);
            int s = 0, so = 0;  // symbols and ones behind us
            for (;;) {
                const bool sat = (z == 255 && o == 1) || (o == 255 && z == 1);
                const int to = sat ? (z == 255 ? so + 1 : 1 << 20) : so + 256 - o;        // the one
                const int tz = sat ? (o == 255 ? s - so + 1 : 1 << 20) : s - so + 256 - z;  // or zero it ends at
                const unsigned bo = __ballot_sync(0xffffffffu, ones >= to), bz = __ballot_sync(0xffffffffu, zeros >= tz);
                int t = m;  // the event's symbol
                bool bit = false;
                const unsigned below = (1u << lane) - 1u;
                if (bo != 0u) {
                    const int q = __ffs(bo) - 1;
                    const uint32_t xq = __shfl_sync(0xffffffffu, x, q);
                    const int r = to - __shfl_sync(0xffffffffu, o_at, q) - 1;  // ones before it in the word
                    t = 32 * q + __ffs(__ballot_sync(0xffffffffu, ((xq >> lane) & 1u) != 0u && __popc(xq & below) == r)) - 1;
                    bit = true;
                }
                if (bz != 0u) {
                    const int q = __ffs(bz) - 1;
                    const uint32_t xq = ~__shfl_sync(0xffffffffu, x, q);
                    const int r = tz - __shfl_sync(0xffffffffu, z_at, q) - 1;
                    const int t0 = 32 * q + __ffs(__ballot_sync(0xffffffffu, ((xq >> lane) & 1u) != 0u && __popc(xq & below) == r)) - 1;
                    if (t0 < t) {
                        t = t0;
                        bit = false;
                    }
                }
                // units that start at s .. t
                if (unit && 32 * lane >= s && 32 * lane <= t) {
                    const int uz = sat ? z : z + z_at - (s - so), uo = sat ? o : o + o_at - so;
                    *us = (uint32_t)uz | (uint32_t)uo << 8 | (uint32_t)model << 16;
                }
                if (t >= m) {  // no event in the rest of these symbols
                    const int all = __shfl_sync(0xffffffffu, ones, 31);
                    if (!sat) {
                        z += m - all - (s - so);
                        o += all - so;
                    }
                    break;
                }
                const int ot = bit ? to - 1 : t - (tz - 1);  // ones before t
                unsigned nz = (unsigned)(sat ? z : z + (t - ot) - (s - so)), no = (unsigned)(sat ? o : o + ot - so);
                if (bit) sy_observe(no, nz);
                else sy_observe(nz, no);
                z = (int)nz;
                o = (int)no;
                s = t + 1;
                so = ot + (bit ? 1 : 0);
                if (s >= m) break;
            }
        }
    }
}

// The probabilities of one unit of a list (four consecutive symbols a lane) from the counts at its
// start: in one step up to its first event, and on behind it.
__device__ __forceinline__ void sym_model_unit(const SymFrame& f, const uint4 q, int m, int lane, int z, int o) {
    const unsigned cur[4] = {q.x, q.y, q.z, q.w};
    const unsigned below = (1u << lane) - 1u;
    int op[5];  // ones of the chunk before symbol 4 lane + j
    op[0] = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const unsigned b = __ballot_sync(0xffffffffu, 4 * lane + j < m && (cur[j] >> 31) != 0u);
        op[0] += __popc(b & below);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) op[j + 1] = op[j] + (int)(cur[j] >> 31);
    int pz[4] = {1, 1, 1, 1}, po[4] = {1, 1, 1, 1};  // the counts before each symbol
    int Z = z, O = o;                                // counts of symbol k: Z + zeros before it, O + ones before it
    for (int s = 0;;) {  // symbols s .. m - 1 are left; (z, o) are the counts before s
        // the first symbol t >= s after which the line ends: the one that halves, or at 255
        // against 1 the first other bit
        const bool sat = (z == 255 && o == 1) || (o == 255 && z == 1);
        const unsigned other = z == 255 ? 1u : 0u;
        int first = 4;
#pragma unroll
        for (int j = 3; j >= 0; j--) {
            const int k = 4 * lane + j;
            const unsigned bit = cur[j] >> 31;
            const int zj = Z + k - op[j], oj = O + op[j];
            const bool in = k >= s && k < m;
            if (in) {  // rewritten behind t
                pz[j] = sat ? z : zj;
                po[j] = sat ? o : oj;
                if (sat ? bit == other : (bit ? oj : zj) == 255) first = j;
            }
        }
        const unsigned any = __ballot_sync(0xffffffffu, first < 4);
        if (any == 0u) break;
        const int tl = __ffs(any) - 1;
        // symbol t: its place in the lane, bit and counts
        const int zf = first == 0 ? pz[0] : first == 1 ? pz[1] : first == 2 ? pz[2] : pz[3];
        const int of = first == 0 ? po[0] : first == 1 ? po[1] : first == 2 ? po[2] : po[3];
        const int pf = first == 0 ? op[1] : first == 1 ? op[2] : first == 2 ? op[3] : op[4];
        const unsigned bf = (first == 0 ? cur[0] : first == 1 ? cur[1] : first == 2 ? cur[2] : cur[3]) >> 31;
        const unsigned w = __shfl_sync(0xffffffffu, (unsigned)first | bf << 2 | (unsigned)zf << 3 | (unsigned)of << 11 | (unsigned)pf << 19, tl);
        unsigned nz = (w >> 3) & 255u, no = (w >> 11) & 255u;
        if (w & 4u) sy_observe(no, nz);
        else sy_observe(nz, no);
        z = (int)nz;
        o = (int)no;
        s = 4 * tl + (int)(w & 3u) + 1;
        if (s >= m) break;
        const int ones = (int)(w >> 19);  // ones before s
        Z = z - (s - ones);
        O = o - ones;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (4 * lane + j < m)
            f.stack[sy_slot(cur[j] & 0x7fffffffu)] =
                (uint16_t)(sy_prob((unsigned)pz[j], (unsigned)po[j]) | (cur[j] >> 31) << 8);
}
// The units of a frame's lists, by warp `wi` of `nw`.
__device__ __forceinline__ void sym_model_units(const SymFrame& f, unsigned wi, unsigned nw, int lane) {
    if (f.work[1] == 0u) return;
    const unsigned nu = f.work[0] / SY_UNIT;
    for (unsigned u = wi; u < nu; u += nw) {
        const uint4 q = ((const uint4*)(f.occ + (size_t)u * SY_UNIT))[lane];  // what lies behind the list's end is not used
        const uint32_t st = f.ustate[u];
        const unsigned b0 = f.work[SYM_TAB + 2 * (st >> 16)], n = f.work[SYM_TAB + 2 * (st >> 16) + 1];
        sym_model_unit(f, q, (int)min(SY_UNIT, n - (u * SY_UNIT - b0)), lane, (int)(st & 255u), (int)((st >> 8) & 255u));
    }
}

__global__ void __launch_bounds__(32 * SY_WARPS, 4) k_sym_count(SymFrame f) {
    __shared__ unsigned h[SY_WARPS][SYM_ROWS];
    sym_count_cta(f, blockIdx.x, h);
}
__global__ void __launch_bounds__(1024) k_sym_scan(SymFrame f) { sym_scan_rows(f, blockIdx.x); }
__global__ void __launch_bounds__(32 * SY_WARPS, 4) k_sym_emit(SymFrame f) {
    __shared__ unsigned h[SY_WARPS][SYM_ROWS];
    sym_emit_cta(f, blockIdx.x, h);
}
__global__ void __launch_bounds__(SY_CHAIN_THREADS) k_sym_chain(SymFrame f) {
    if (f.work[1] != 0u) sym_chain_cta(f, blockIdx.x);
}
constexpr int SY_MODEL_THREADS = 128;
__global__ void __launch_bounds__(SY_MODEL_THREADS, 8) k_sym_model(SymFrame f) {
    sym_model_units(f, (blockIdx.x * SY_MODEL_THREADS + threadIdx.x) >> 5, gridDim.x * (SY_MODEL_THREADS / 32), threadIdx.x & 31);
}

static inline int sym_part_ctas(int nmb) { return (nmb + SY_MBS * SY_WARPS - 1) / (SY_MBS * SY_WARPS); }
// CTAs of the units of a frame: a warp takes about two when a macroblock has 64 modelled symbols.  Every
// model that occurs has a unit, however small the frame, so no fewer than a warp a model (by macroblocks
// alone a 64x48 key frame had one CTA for its 300 units, and 132 us a frame in flight went to 80).
static inline int sym_model_ctas(int nmb) {
    constexpr int warps = SY_MODEL_THREADS / 32;
    return std::max((SY_MODELS + warps - 1) / warps, std::min(8 * 148, nmb / 16));
}

size_t sym_workspace(SymFrame* f, int nmb, unsigned cap, void* p) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
        void* q = (uint8_t*)p + at;
        at += (bytes + 255) & ~(size_t)255;
        return q;
    };
    void* cnt = take((size_t)((nmb + SY_MBS - 1) / SY_MBS) * SYM_ROWS * sizeof(uint16_t));
    void* tot = take((size_t)sym_part_ctas(nmb) * SYM_ROWS * sizeof(unsigned));
    void* occ = take(((size_t)cap + SYM_OCC_SLACK) * sizeof(unsigned));
    void* us = take(((size_t)cap + SYM_OCC_SLACK) / SYM_UNIT * sizeof(uint32_t));
    void* work = take(SYM_WORK_WORDS * sizeof(unsigned));
    if (f != nullptr) {
        f->cnt = (uint16_t*)cnt;
        f->tot = (unsigned*)tot;
        f->occ = (unsigned*)occ;
        f->ustate = (uint32_t*)us;
        f->work = (unsigned*)work;
    }
    return at;
}
// With no room (cap 0) the blocks are packed for the host coder.
int launch_symbols(const SymFrame& f, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    k_sym_count<<<sym_part_ctas(f.nmb), 32 * SY_WARPS, 0, st>>>(f);
    k_sym_scan<<<SYM_ROWS / 32, 1024, 0, st>>>(f);
    k_sym_emit<<<sym_part_ctas(f.nmb), 32 * SY_WARPS, 0, st>>>(f);
    if (f.cap == 0) return (int)cudaGetLastError();
    k_sym_chain<<<SY_MODELS, SY_CHAIN_THREADS, 0, st>>>(f);
    k_sym_model<<<sym_model_ctas(f.nmb), SY_MODEL_THREADS, 0, st>>>(f);
    return (int)cudaGetLastError();
}
