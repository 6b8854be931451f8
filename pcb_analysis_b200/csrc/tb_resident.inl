// Host side of the cooperative PCG kernel of small boards (tb_resident.cuh).
// Included by tb_system.cu inside its anonymous namespace.

constexpr int kResLimit = 512;      // iterations of one launch (a few milliseconds)
// The same beside a batch engine.  The kernel wants every SM, and gets in between
// two of the engine's kernels: with launches of 512 iterations one after another a
// thread of small solves left an engine a sixth of the device.  So each launch
// waits for what the engine has queued, a chunk or two, and is short.  Ten boards'
// batch (0.50 s alone) beside a thread of 96 x 80 x 8 two-level solves (0.029 s
// alone): 3.1 s and 0.033 s a solve before; 0.93 and 0.11 with 128 iterations, 0.84
// and 0.18 with 64, 0.70 and 0.30 with 32; 0.57 and 0.07 .. 0.20 with the
// graph-captured kernels.
constexpr int kResLimitShared = 64;
constexpr int kResMinChunk = 128;   // nodes of a block at least
// Longest node row: a block stages two rows beside its nodes on each of three
// planes, word by word.  Microseconds per iteration with Jacobi, this kernel /
// the graph-captured ones: 1 x 4000 x 12 elements 12.0 / 16.7, 1 x 5000 x 8 12.7 /
// 16.8, 2 x 5000 x 8 17.1 / 16.9, 1 x 6000 x 12 18.3 / 17.8, 1 x 7000 x 8 19.7 / 16.9.
constexpr int kResMaxRow = 4800;

using ResidentKernel = void (*)(const ResidentParams);
template <bool MUTE>
ResidentKernel resident_kernel(int nodes, bool tl) {
    if (nodes == 1) return tl ? resident_pcg<1, true, MUTE> : resident_pcg<1, false, MUTE>;
    return tl ? resident_pcg<2, true, MUTE> : resident_pcg<2, false, MUTE>;
}

// The chunks that this process's batch engines have queued, by engine: the device
// and the event behind the last one.  An engine is listed while any is in flight.
struct EngineQueues {
    std::mutex mu;
    std::map<const void*, std::pair<int, cudaEvent_t>> busy;
};
EngineQueues& engine_queues() {
    static EngineQueues* const q = new EngineQueues;  // outlives every engine
    return *q;
}
void engine_queued(const void* engine, int device, cudaEvent_t last) {
    std::lock_guard<std::mutex> lock(engine_queues().mu);
    engine_queues().busy[engine] = {device, last};
}
void engine_idle(const void* engine) {
    std::lock_guard<std::mutex> lock(engine_queues().mu);
    engine_queues().busy.erase(engine);
}
// Have `stream` wait for the chunks queued on the device; `any`: whether there are.
cudaError_t wait_for_engines(int device, cudaStream_t stream, bool* any) {
    std::lock_guard<std::mutex> lock(engine_queues().mu);
    *any = false;
    for (const auto& kv : engine_queues().busy) {
        if (kv.second.first != device) continue;
        *any = true;
        const cudaError_t e = cudaStreamWaitEvent(stream, kv.second.second, 0);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void free_resident(tb_system* s) {
    dev_free(s, s->res_rows);
    dev_free(s, s->res_words);
    s->res_state = 0;
}

// Whether the system's inner PCG runs as the cooperative kernel, and its
// buffers: thermal systems with the Jacobi or two-level preconditioner whose
// nodes fit the registers of one block per SM (two nodes a thread) and, with
// the coarse inverse's tile, its shared memory.  A launch plan set
// by the caller (tb_set_apply_plan) and event timing (tb_set_timing) ask for
// the graph-captured kernels.
int resident_setup(tb_system* s) {
    if (s->res_state != 0) return TB_OK;
    s->res_state = -1;  // not available
    const Layout& L = s->lay;
    const bool tl = s->precond == 1;
    if (s->physics != 0 || s->precond > 1 || s->sms > kResMaxBlocks) return TB_OK;
    if (L.L > (long long)s->sms * kResThreads * kResNodes || L.Xp > kResMaxRow) return TB_OK;
    int coop = 0;
    TB_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, s->device));
    if (!coop) return TB_OK;
    const int chunk = std::max(kResMinChunk, (int)round_up((L.L + s->sms - 1) / s->sms, 32));
    const int blocks = (int)((L.L + chunk - 1) / chunk);
    // tiles of the inverse: as square as the blocks allow
    const int tiles_y = tl ? std::max(1, (int)std::sqrt((double)blocks)) : 0;
    const int tiles_x = tl ? std::min(blocks / tiles_y, kResTileCols) : 0;
    const int trows = tl ? (int)round_up((s->cl.nc + tiles_y - 1) / tiles_y, 4) : 0;
    const int tcols = tl ? (int)round_up((s->cl.nc + tiles_x - 1) / tiles_x, 4) : 0;
    if (trows + tcols > kResThreads) return TB_OK;
    const int nodes = chunk <= kResThreads ? 1 : 2;
    const size_t smem = resident_smem(trows, tcols, chunk, L.Xp);
    int optin = 0;
    TB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device));
    for (const ResidentKernel kernel : {resident_kernel<false>(nodes, tl), resident_kernel<true>(nodes, tl)}) {
        cudaFuncAttributes fa{};
        TB_CUDA(cudaFuncGetAttributes(&fa, kernel));
        if (fa.sharedSizeBytes + smem > (size_t)optin) return TB_OK;
        TB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     optin - (int)fa.sharedSizeBytes));
        int per_sm = 0;
        TB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kResThreads, smem));
        if (per_sm < 1) return TB_OK;
    }
    int slots = 0;
    if (tl) {
        // blocks that touch one patch row: from the one that holds its first node on
        const int prows = s->cl.layers * s->cl.nby;
        for (int pr = 0; pr < prows; ++pr) {
            const int z = pr / s->cl.nby, y0 = (pr - z * s->cl.nby) * s->cl.b;
            const long long first = ((long long)z * (L.R + 1) + y0) * L.Xp;
            const long long last = first + (long long)std::min(s->cl.b, L.R + 1 - y0) * L.Xp - 1;
            slots = std::max(slots, (int)(last / chunk - first / chunk) + 1);
        }
        // patch rows one block touches: a chunk spans at most chunk / Xp + 2 lines,
        // and a patch row has b of them except at the end of a plane
        const int lines = chunk / L.Xp + 2;
        const int touched = std::min(prows, lines / s->cl.b + lines / (L.R + 1) + 3) * s->cl.nbx;
        if (slots > kResSlots || touched > kResTouched) return TB_OK;
    }
    // Without the memory for them the solve runs on the graph-captured kernels.
    const auto refused = [s]() {
        free_resident(s);
        s->res_state = -1;
        return TB_OK;
    };
    if (alloc_n(s, &s->res_rows, kResRow * L.L) != TB_OK) return refused();
    // tagged words: the direction, the sums, the patch sums, the coarse solution; and the next tag
    const long long sums = 8LL * kResCopies * blocks, parts = tl ? (long long)slots * s->cl.ld : 0, cs = (long long)tiles_x * s->cl.ld;
    s->res_word_count = L.L + sums + parts + cs + 1;  // L is a multiple of 4: the sums' pairs stay 16-byte aligned
    if (alloc_n(s, &s->res_words, s->test_refuse == 1 ? 1LL << 50 : s->res_word_count) != TB_OK) return refused();
    resident_rows<<<grid_for(L.L, 128, s->sms * 16), 128, 0, s->stream>>>(
        s->res_rows, s->kin64, s->kz64, s->rf64, s->dims64, s->dims64 + L.S, s->dims64 + L.S + L.C, L);
    TB_CUDA(cudaGetLastError());
    s->kernel_launches += 1;
    ResidentParams P{};
    P.p = s->p32;
    P.x = s->x32;
    P.r = s->r32;
    P.dinv = s->dinv32;
    P.halo = s->res_words;
    P.rows = s->res_rows;
    P.lay = L;
    P.pstride = (int)s->pstride;
    P.ctl = s->ctl;
    P.clock = s->clocks;
    P.posts = P.halo + L.L;
    P.part = P.posts + sums;
    P.c = P.part + parts;
    P.tag = reinterpret_cast<unsigned int*>(P.c + cs);
    P.err = s->stage_err;
    P.chunk = chunk;
    P.limit = s->test_slice > 0 ? s->test_slice : kResLimit;
    P.polls = kResPolls;
    P.cl = s->cl;
    P.minv = tl ? s->coarse_inv32 : nullptr;
    P.slots = slots;
    P.tiles_x = tiles_x;
    P.tiles_y = tiles_y;
    P.trows = trows;
    P.tcols = tcols;
    s->res_params = P;
    s->res_blocks = blocks;
    s->res_nodes = nodes;
    s->res_smem = smem;
    s->res_fresh = true;
    s->res_state = 1;
    return TB_OK;
}

bool resident_wanted(const tb_system* s) { return !s->timing && !s->plan_set && s->physics == 0 && s->precond <= 1; }

// The inner PCG from a prepared start (as run_pcg) on the cooperative kernel.
// A launch that the runtime refuses (the device's SMs shared out to several
// clients, say) leaves the vectors and the scalars as the last one left them,
// with `state` running: the caller goes on from there with the graph-captured
// kernels.
int run_resident(tb_system* s, SolveCtl* out) {
    if (s->res_fresh) {  // nothing exchanged yet, or a run that was given up: words without tags, the first tag 1
        TB_CUDA(cudaMemsetAsync(s->res_words, 0, sizeof(unsigned long long) * (size_t)s->res_word_count, s->stream));
        const unsigned int first = 1;
        TB_CUDA(cudaMemcpyAsync(s->res_params.tag, &first, sizeof(first), cudaMemcpyHostToDevice, s->stream));
        TB_CUDA(cudaStreamSynchronize(s->stream));
        s->res_fresh = false;
    }
    ResidentParams P = s->res_params;
    if (s->maps[0].test_polls > 0) {
        P.polls = s->maps[0].test_polls;
        P.mute = s->test_mute != 0 ? s->test_mute : ~0;
        P.mute_block = s->test_mute_block;
    }
    const bool tl = P.minv != nullptr;
    const ResidentKernel kernel = P.mute ? resident_kernel<true>(s->res_nodes, tl) : resident_kernel<false>(s->res_nodes, tl);
    void* args[] = {&P};
    for (long long n = 0;; ++n) {
        bool shared = false;
        TB_CUDA(wait_for_engines(s->device, s->stream, &shared));
        P.limit = shared ? std::min(s->res_params.limit, kResLimitShared) : s->res_params.limit;
        if (cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel),
                                        dim3(s->test_refuse == 2 ? 1 << 16 : s->res_blocks), dim3(kResThreads), args,
                                        s->res_smem, s->stream) != cudaSuccess) {
            cudaGetLastError();  // an error that outlives the launch meets the next call
            free_resident(s);
            s->res_state = -1;
            TB_CHECK(read_ctl(s, out));
            return TB_OK;
        }
        s->kernel_launches += 1;
        TB_CUDA(cudaMemcpyAsync(s->h_err, s->stage_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
        TB_CHECK(read_ctl(s, out));
        // The error word decides, whatever the state says: block 0, which writes
        // the scalars, may have had all it waited for when another block gave up.
        if (*s->h_err != 0) {
            s->res_fresh = true;
            TB_CUDA(cudaMemsetAsync(s->stage_err, 0, sizeof(int), s->stream));
            return fail(TB_ETIMEOUT, "a block of the PCG kernel gave up waiting for the others");
        }
        if (out->state != ST_RUNNING) return TB_OK;
        if (n > (1LL << 40)) return fail(TB_ETIMEOUT, "PCG did not stop");
    }
}
