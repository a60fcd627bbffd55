// riv_batch.cuh -- multi-clip (batched) launches of the P-frame encoder's stages.
//
// Included by riv_kernels.cu inside namespace riv (it uses that file's device functions).
// One step of a batch encodes one frame of every clip that has one; each stage below is ONE
// launch over all of them.  A stage's grid is the concatenation of per-clip CTA ranges
// (batch_ctas: prefix sums in BatchLaunch::start), so each CTA works for exactly one clip and
// runs the same per-MB / per-tile device code as the single-clip kernels: the results are those
// of a single-clip encode of the clip, bit for bit.
//
// The search is one cooperative launch whose grid is the concatenation of per-clip wavefront
// launches (SearchParams::cta0 = the clip's first CTA): each clip's row CTAs take its MB rows
// with a stride of its CTA count and wait only on rows of the same clip, all co-resident.

// The clip owning CTA b: the largest c with start[c] <= b (start holds n + 1 prefix sums).
__device__ __forceinline__ int batch_clip(const int* __restrict__ start, int n, int b) {
    int lo = 0, hi = n;  // start[lo] <= b < start[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(start + mid) <= b) lo = mid;
        else hi = mid;
    }
    return lo;
}

__host__ __device__ inline int batch_deblock_tiles(int W, int H, int tw) {
    const int ty = (H / 16) * ((W + tw - 1) / tw);
    const int tc = ((H / 2) / 8) * ((W / 2 + tw / 2 - 1) / (tw / 2));
    return ty + 2 * tc;
}

// CTAs of clip k in stage s.
inline int batch_ctas(int s, const BatchClip& k, const BatchTune& t) {
    const int nmb = k.NMB;
    switch (s) {
        case BS_CONVERT: return k.rgb != nullptr ? ((k.W / 2) * (k.H / 2) + 127) / 128 : 0;
        case BS_TABLE: return k.intra || k.tab == nullptr ? 0 : nmb;
        case BS_PREDICT: return k.intra || k.predicted ? 0 : nmb;
        case BS_AQSUM: return k.intra ? 0 : 1;
        case BS_RESIDUAL: return (nmb + t.res_mbs - 1) / t.res_mbs;
        case BS_DEBLOCK: return k.db_level > 0 ? batch_deblock_tiles(k.W, k.H, t.db_tw) : 0;
        case BS_SCAN: case BS_PACK: return sym_part_ctas(nmb);
        default: return 0;
    }
}

// ---- conversion: RGB24 (display size) -> planar YUV 4:2:0, one thread per 2x2 quad
__global__ void __launch_bounds__(128) kb_convert(BatchLaunch b) {
    const int* st = b.start + BS_CONVERT * (b.nclips + 1);
    const int c = batch_clip(st, b.nclips, blockIdx.x);
    const BatchClip& k = b.clips[c];
    const int W = k.W, H = k.H, cw = W / 2, nq = cw * (H / 2);
    const int q = ((int)blockIdx.x - st[c]) * 128 + (int)threadIdx.x;
    if (q >= nq) return;
    uint8_t* Y = k.cur;
    uint8_t* U = Y + (size_t)W * H;
    uint8_t* V = U + (size_t)cw * (H / 2);
    rgb_to_yuv_quad(k.rgb, k.dw, k.dh, Y, U, V, W, q % cw, q / cw);
}

// ---- exhaustive integer SAD table of every P-frame MB (sad_table_mb)
__global__ void __launch_bounds__(128) kb_table(BatchLaunch b) {
    extern __shared__ __align__(16) uint8_t sm[];
    const int* st = b.start + BS_TABLE * (b.nclips + 1);
    const int c = batch_clip(st, b.nclips, blockIdx.x);
    const BatchClip& k = b.clips[c];
    sad_table_mb(k.ref, k.cur, k.W, k.H, k.BW, k.sr, k.tab, k.tstride, (int)blockIdx.x - st[c], sm, threadIdx.x,
                 blockDim.x, 0);
}

// ---- motion-compensated prediction (predict_mb), then the MB's luma variance and its
// glibc-exact ln (k_aq_log's arithmetic) for the AQ mean
__global__ void __launch_bounds__(256) kb_predict(BatchLaunch b) {
    __shared__ unsigned ws[8], ws2[8];
    const int* st = b.start + BS_PREDICT * (b.nclips + 1);
    const int c = batch_clip(st, b.nclips, blockIdx.x);
    const BatchClip& k = b.clips[c];
    const int mb = (int)blockIdx.x - st[c];
    const uint2 vs = predict_mb(k.ref, k.mbo, k.pred, k.W, k.H, mb, ws, ws2);
    if (threadIdx.x == 0) {
        const unsigned long long N = 256ull * vs.y - (unsigned long long)vs.x * vs.x;
        float var = __fdiv_rn(__ull2float_rn(N), 65536.0f);
        var = var < 4.0f ? 4.0f : var;
        k.lnv[mb] = glibc_logf(var, k.logfix, k.nlog);
    }
}

// ---- the strictly sequential mean of a clip's ln variances (aq_sum_cta), one CTA per clip
__global__ void __launch_bounds__(1024) kb_aqsum(BatchLaunch b) {
    extern __shared__ float sl[];
    const int* st = b.start + BS_AQSUM * (b.nclips + 1);
    const BatchClip& k = b.clips[batch_clip(st, b.nclips, blockIdx.x)];
    aq_sum_cta(k.lnv, k.NMB, k.lnv + k.NMB, sl);
}

// ---- residual, transforms, quantisation and reconstruction (residual_pair), NM MBs per CTA
template <int NM>
__global__ void __launch_bounds__(16 * NM, 48 / NM) kb_residual(BatchLaunch b) {
    __shared__ ResPair S[NM / 2];
    const int* st = b.start + BS_RESIDUAL * (b.nclips + 1);
    const int c = batch_clip(st, b.nclips, blockIdx.x);
    const BatchClip& k = b.clips[c];
    const int w = threadIdx.x >> 5, mb = ((int)blockIdx.x - st[c]) * NM + 2 * w;
    if (mb < k.NMB) residual_pair(k.rp, k.NMB, mb, threadIdx.x & 31, S[w]);
}

// ---- out-of-place deblock (deblock_tile), TW luma columns per tile
template <int TW>
__global__ void __launch_bounds__(128) kb_deblock(BatchLaunch b) {
    __shared__ __align__(16) uint8_t tile[(16 + 8) * (TW + 8)];
    const int* st = b.start + BS_DEBLOCK * (b.nclips + 1);
    const int c = batch_clip(st, b.nclips, blockIdx.x);
    const BatchClip& k = b.clips[c];
    const int ty = (k.H / 16) * ((k.W + TW - 1) / TW);
    int t = (int)blockIdx.x - st[c];
    const int plane = t < ty ? 0 : (t - ty) % 2 + 1;
    if (plane > 0) t = (t - ty) / 2;
    deblock_tile<TW>(k.db_src, k.db_dst, k.W, k.H, k.BW, k.db_E, k.db_I, k.db_H, k.db_mask, plane, t, tile, threadIdx.x,
                     blockDim.x, 0);
}

// ---- coefficient symbols (riv_symbols.cuh): counts and their scan (which also copies the clip's
// status word to the mapped header, so no separate copy is needed), then symbols and models
__global__ void __launch_bounds__(32 * SY_WARPS, 4) kb_sym_count(BatchLaunch b) {
    __shared__ unsigned h[SY_WARPS][SYM_ROWS];
    const int* st = b.start + BS_SCAN * (b.nclips + 1);
    const int c = batch_clip(st, b.nclips, blockIdx.x);
    sym_count_cta(b.clips[c].sym, (int)blockIdx.x - st[c], h);
}
__global__ void __launch_bounds__(1024) kb_sym_scan(BatchLaunch b) {
    sym_scan_rows(b.clips[blockIdx.y].sym, blockIdx.x);
}
__global__ void __launch_bounds__(32 * SY_WARPS, 4) kb_sym_emit(BatchLaunch b) {
    __shared__ unsigned h[SY_WARPS][SYM_ROWS];
    const int* st = b.start + BS_PACK * (b.nclips + 1);
    const int c = batch_clip(st, b.nclips, blockIdx.x);
    sym_emit_cta(b.clips[c].sym, (int)blockIdx.x - st[c], h);
}
__global__ void __launch_bounds__(SY_CHAIN_THREADS) kb_sym_chain(BatchLaunch b) {
    const SymFrame& f = b.clips[blockIdx.y].sym;
    if (f.work[1] != 0u) sym_chain_cta(f, blockIdx.x);
}
constexpr int BATCH_MODEL_CTAS = 64;  // per clip; its warps share the clip's units
__global__ void __launch_bounds__(SY_MODEL_THREADS, 8) kb_sym_model(BatchLaunch b) {
    sym_model_units(b.clips[blockIdx.y].sym, (blockIdx.x * SY_MODEL_THREADS + threadIdx.x) >> 5,
                    BATCH_MODEL_CTAS * (SY_MODEL_THREADS / 32), threadIdx.x & 31);
}

// ---- rANS streams (riv_rans.cuh), a row of CTAs per clip
__global__ void __launch_bounds__(32 * RA_WARPS) kb_rans(const BatchClip* __restrict__ clips) {
    rans_cta(clips[blockIdx.y].rans, blockIdx.x);
}
__global__ void __launch_bounds__(RA_GATHER) kb_rans_gather(const BatchClip* __restrict__ clips) {
    const RansFrame& f = clips[blockIdx.y].rans;
    rans_gather_cta(f, blockIdx.x, (f.nside + RA_SIDE - 1) / RA_SIDE);
}
int launch_batch_rans(const BatchClip* clips, int nclips, unsigned max_cap, int max_nside, void* stream) {
    const int nb = rans_batches(max_cap);
    kb_rans<<<dim3((nb + RA_WARPS - 1) / RA_WARPS, nclips), 32 * RA_WARPS, 0, (cudaStream_t)stream>>>(clips);
    kb_rans_gather<<<dim3(nb + rans_side_ctas(max_nside), nclips), RA_GATHER, 0, (cudaStream_t)stream>>>(clips);
    return (int)cudaGetLastError();
}

// ---- the multi-clip search wavefront (per-MB reference windows; see the file comment).  96
// registers a thread: five 128-thread CTAs of the direct kind an SM (120: four, 1.68 ms a step of 24
// clips against 1.66; 80: six, 1.91).
template <bool TABLE, bool SMALL>
__global__ void __maxnreg__(96) k_search_multi(const SearchParams* __restrict__ ps, const int* __restrict__ start,
                                                int nclips) {
    search_body<false, TABLE, SMALL, true>(ps[batch_clip(start, nclips, blockIdx.x)]);
}

static const void* search_multi_fn(SearchKind k) {
    switch (k) {
        case SK_TABLE_SMALL: return (const void*)k_search_multi<true, true>;
        case SK_TABLE: return (const void*)k_search_multi<true, false>;
        case SK_DIRECT: return (const void*)k_search_multi<false, true>;
        default: return (const void*)k_search_multi<false, false>;
    }
}

static size_t batch_stage_smem(int s, int table_sr) {
    if (s == BS_TABLE) return sad_table_smem(table_sr);
    if (s == BS_AQSUM) return 8192 * sizeof(float);
    return 0;
}

static int batch_stage_threads(int s, const BatchTune& t) {
    switch (s) {
        case BS_CONVERT: case BS_TABLE: case BS_DEBLOCK: return 128;
        case BS_PREDICT: return 256;
        case BS_AQSUM: return 1024;
        case BS_RESIDUAL: return 16 * t.res_mbs;
        case BS_SCAN: case BS_PACK: return 32 * SY_WARPS;
        default: return 0;
    }
}

int batch_ctas_host(int s, const BatchClip& k, const BatchTune& t) { return batch_ctas(s, k, t); }

int launch_batch_stage(int s, const BatchLaunch& b, const BatchTune& t, int total, int table_sr, void* stream) {
    if (total <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t sm = batch_stage_smem(s, table_sr);
    const int nt = batch_stage_threads(s, t);
    switch (s) {
        case BS_CONVERT: kb_convert<<<total, nt, 0, st>>>(b); break;
        case BS_TABLE: kb_table<<<total, nt, sm, st>>>(b); break;
        case BS_PREDICT: kb_predict<<<total, nt, 0, st>>>(b); break;
        case BS_AQSUM: kb_aqsum<<<total, nt, sm, st>>>(b); break;
        case BS_RESIDUAL:
            if (t.res_mbs == 2) kb_residual<2><<<total, nt, 0, st>>>(b);
            else if (t.res_mbs == 4) kb_residual<4><<<total, nt, 0, st>>>(b);
            else if (t.res_mbs == 8) kb_residual<8><<<total, nt, 0, st>>>(b);
            else return (int)cudaErrorInvalidValue;
            break;
        case BS_DEBLOCK:
            if (t.db_tw == 64) kb_deblock<64><<<total, nt, 0, st>>>(b);
            else if (t.db_tw == 128) kb_deblock<128><<<total, nt, 0, st>>>(b);
            else if (t.db_tw == 256) kb_deblock<256><<<total, nt, 0, st>>>(b);
            else return (int)cudaErrorInvalidValue;
            break;
        case BS_SCAN:
            kb_sym_count<<<total, nt, 0, st>>>(b);
            kb_sym_scan<<<dim3(SYM_ROWS / 32, b.nclips), 1024, 0, st>>>(b);
            break;
        case BS_PACK:
            kb_sym_emit<<<total, nt, 0, st>>>(b);
            kb_sym_chain<<<dim3(SY_MODELS, b.nclips), SY_CHAIN_THREADS, 0, st>>>(b);
            kb_sym_model<<<dim3(BATCH_MODEL_CTAS, b.nclips), SY_MODEL_THREADS, 0, st>>>(b);
            break;
        default: return (int)cudaErrorInvalidValue;
    }
    return (int)cudaGetLastError();
}

int search_multi_kind(bool table, bool small, int sr) {
    return table ? (small ? SK_TABLE_SMALL : SK_TABLE) : untabled_kind(sr, 0, false, small);
}
bool search_multi_predicts(int kind) { return search_fast(false, (SearchKind)kind); }

int search_multi_capacity(int kind, int max_sr, int* per_sm, size_t* smem, int* threads) {
    const void* fn = search_multi_fn((SearchKind)kind);
    const size_t sm = search_smem(max_sr, 0, false, (SearchKind)kind);
    const int nt = search_threads(search_fast(false, (SearchKind)kind));
    int room = 0;
    cudaError_t e = open_smem(fn, &room);
    if (e == cudaSuccess && sm > (size_t)room) e = cudaErrorInvalidValue;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, fn, nt, sm);
    *smem = sm;
    *threads = nt;
    return (int)e;
}

int launch_search_multi(const SearchParams* dparams, const int* dstart, int nclips, int total, int kind, size_t smem,
                        int threads, void* stream) {
    if (total <= 0) return 0;
    void* args[] = {(void*)&dparams, (void*)&dstart, (void*)&nclips};
    // cooperative: every clip's row CTAs are co-resident, so each row's wait on the row above
    // (a CTA of the same clip) can always make progress
    return (int)cudaLaunchCooperativeKernel(search_multi_fn((SearchKind)kind), dim3(total), dim3(threads), args, smem,
                                            (cudaStream_t)stream);
}
