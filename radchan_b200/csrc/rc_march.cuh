// rc_march.cuh -- the persistent march kernel (kernel_fluid + march_ray +
// kernel_surface of src/montecarlo/mc_gpu_noint.cu, restructured for SIMT).
#pragma once
#include "rc_device.cuh"

namespace rc {

// ---------------------------------------------------------------------------
// march: persistent warps over tiles of 32 work items
// ---------------------------------------------------------------------------
//
// A work item is one chunk of rays_per_thread consecutive bundles of one
// (cell, replicate).  A warp takes tiles of 32 items, i.e. pools of
// 32*rays_per_thread bundles:
//   * bundles are emitted in converged waves of 32 (all lanes decode their
//     item and run the Philox draws, direction, band/g search and OERM
//     weights together) into a per-warp ring in shared memory whenever the
//     ring holds fewer than kRefill bundles;
//   * every lane traces one ray; the warp steps all its rays until at least
//     kFeedIdle lanes are idle, then retires the rays that stopped and hands
//     those lanes the next emitted bundles (warp ballot + prefix count);
//   * two or three tiles can be in flight (tile_bufs): once every bundle of a
//     tile has been emitted, the warp fetches the next tile and keeps
//     emitting from it while the last rays of earlier tiles finish, so long
//     rays do not leave the other lanes idle;
//   * each bundle's FP64 tally goes to its own shared-memory slot; when a
//     tile's last bundle has finished, its slots are summed in bundle
//     order, so the result does not depend on which lane traced which
//     bundle.
// Shared memory per warp is the ring (42 emitted bundles of 32 bytes: the
// start position is rebuilt from the emitting cell when a lane takes the
// bundle) and the slot arrays; everything else stays in L1-cached global
// memory, so that most of the SM's 256 KB of L1/shared storage caches the
// temperature pyramid and the k / I_b tables (48-byte entries, an earlier
// layout, were 1.2% slower; 64-byte entries 4%).  The scattering variant
// keeps these entries and adds a small side array (see WarpShared).
//
// The kernel is bound by instruction issue (81-83% of the slots; DRAM idle):
// on the 64^3 narrow-band channel 607 warp instructions per emitted wave,
// about 330 per pass that retires and feeds, 120-140 per step-loop iteration
// at 23-24 lanes.  With two tiles in flight, four divergent paths per
// iteration and 64 registers it took 26.6 ms for photmax 256 there and 60 ms
// on the 192x128x128 channel; now 22 and 30-32 ms.

struct MarchArgs {
    const void *desc;            // DSolve<R> on the device (run-time fields patched)
    long long total_tiles;
    unsigned long long *tile_counter;
    int nbuf;  // tiles a warp has in flight (tile_bufs)
    // long-ray priority (NULL: tiles in natural order): the
    // first n_prio[0] claims take the head of prio_tiles[], the next
    // n_prio[1] its end (backwards), the rest take the natural order and skip
    // the tiles whose tile_prio byte is set
    const unsigned *prio_tiles;
    const unsigned char *tile_prio;
    const unsigned *n_prio;
};
// A launch carries its solve's descriptor in the kernel's parameters: what the
// march reads of it comes from constant memory (operands and uniform
// registers) instead of loads through L1 into registers.  The run-time values
// (Ibmax, table row) are read from the copy in device memory.  (A launch over
// several solves, with the descriptors in device memory, ran 30% slower per
// step: several solves are several launches, side by side.)
template <typename R>
struct MarchParams {
    MarchArgs m;
    DSolve<R> one;
};

// Long-ray priority list.  A bundle whose path is long -- nearly parallel
// to the x walls, so that it runs between the periodic y/z boundaries, and
// in a near-transparent band, so that its transmissivity stays above the
// cutoff -- takes up to the last level's step budget; a launch that starts
// it late idles while it finishes.  The march therefore claims the tiles
// holding such a bundle first.  The estimate of a bundle's path length is
//   L = min(d_x / |s_x|, ln(1/tol) / k_min),
// d_x the distance from its start to the x wall it moves towards, k_min the
// smallest absorption coefficient of its band and g point over the table
// rows the field's temperatures span (k_prio_kmin); a tile is listed when
// some bundle has L > thr * Lx, and in the first part of the list when
// L > kSoloPath * thr * Lx.  Such a ray decides when a short launch ends: a
// warp that has claimed its tile claims no other before its rays have
// finished, so the ray is not held up by the emission and feeding of others
// (its warp then steps it 2-3 times as often).  That holds as long as there is
// a warp for every such tile; with more of them (a near-transparent gas, a low
// threshold) warps that step one ray each would be the rule, and the tiles are
// only claimed early (grey 32^3, k 0.01 1/m: 19.3 ms with a warp held for every
// one, 10.6 so; k 0.001: 51 and 37 ms; narrow-band cases with a handful of such
// tiles, 20-30% faster by the hold, are the same).  The draws are the emission's own (Philox
// counter of the bundle, select_band_g), so the estimate sees the same
// direction, band and g point the march will trace.  Only the order in
// which tiles are claimed changes, never a result.
constexpr float kSoloPath = 16.f;

template <typename R>
__global__ void k_prio_kmin(const DSolve<R> *Sp, float *kmin) {
    const DSolve<R> &S = *Sp;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.nB * S.nQ) return;
    const double T0 = S.sc->T0, idt = S.sc->inv_dT;
    const double tmin = (double)__uint_as_float(S.sc->tmin_bits), tmax = (double)__uint_as_float(S.sc->tmax_bits);
    const int lo = max(0, min(S.nT - 1, (int)floor((tmin - T0) * idt)));
    const int hi = max(lo, min(S.nT - 1, (int)floor((tmax - T0) * idt) + 1));
    float k = 3.0e38f;
    for (int t = lo; t <= hi; ++t) k = fminf(k, (float)S.ki[(size_t)i * S.nT + t].k0);
    kmin[i] = fmaxf(k, 0.f);
}

template <typename R>
__global__ void k_prio_tiles(const DSolve<R> *Sp, float thr, const float *kmin, unsigned *prio_tiles,
                             unsigned char *tile_prio, unsigned *n_prio) {
    const DSolve<R> &S = *Sp;
    const int lane = threadIdx.x & 31;
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    const float Lx = (float)S.Lx, Lthr = thr * Lx;
    const float tau_f = logf(1.0f / fmaxf((float)S.toll, 1e-30f)), tau_w = logf(1.0f / fmaxf((float)S.tollS, 1e-30f));
    for (long long tile = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < S.n_tiles;
         tile += nw) {
        const ItemId it = decode_item(S, tile * kWarp + lane);
        bool cand = false, solo = false;
        if (it.kind >= 0) {
            const uint32_t cell = (it.kind == 0)
                                      ? (uint32_t)((it.i - 1) + S.imax * ((it.j - 1) + S.jmax * (it.k - 1)))
                                      : (uint32_t)((it.j - 1) + S.jmax * (it.k - 1));
            const float x0 = it.kind == 0 ? (float)S.xc[it.i] : (it.kind == 1 ? 0.f : Lx);
            const float tau = it.kind == 0 ? tau_f : tau_w;
            const int h1 = min(it.h0 + S.rpt, S.photmax);
            for (int h = it.h0; h < h1 && !solo; ++h) {
                const rc_u32x4 d = bundle_draws(S.key0, S.key1, h, it.v, it.kind, cell);
                const float u = rc_u01(d.y);
                // s_x as emit_bundle draws it: 1 - 2u (fluid), sqrt(1 - u) / -sqrt(u) (walls)
                const float sx = it.kind == 0 ? 1.f - 2.f * u : (it.kind == 1 ? sqrtf(1.f - u) : -sqrtf(u));
                const float dx = sx > 0.f ? Lx - x0 : x0;
                const float Lw = dx / fmaxf(fabsf(sx), 1e-10f);
                if (!(Lw > Lthr)) continue;
                int nb, g;
                select_band_g(S, S.row, it.kind, (R)rc_u01(d.z), (R)rc_u01(d.w), nb, g);
                const float k = kmin[nb * S.nQ + g];
                cand = cand || k * Lthr < tau;  // ln(1/tol) / k > Lthr
                solo = Lw > kSoloPath * Lthr && k * (kSoloPath * Lthr) < tau;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, cand), ms = __ballot_sync(0xffffffffu, solo);
        if (lane == 0) {
            tile_prio[tile] = m != 0u;
            if (ms) prio_tiles[atomicAdd(n_prio, 1u)] = (unsigned)tile;
            else if (m) prio_tiles[S.n_tiles - 1 - atomicAdd(n_prio + 1, 1u)] = (unsigned)tile;
        }
    }
}

template <typename R, bool SCAT>
struct WarpShared {
    Emitted<R> ring[kRing];
    TileBuf tile[kTileBufs];
};
// With scattering, also the free path to the first event of every ring
// entry (drawn by the emission wave), and the scattering coefficient and
// event count of every lane's bundle (read and written by that lane only,
// at placement and at events; its counter words are decoded again from its
// work item at an event).  The ring entries keep their 32 bytes.
template <typename R>
struct WarpShared<R, true> {
    Emitted<R> ring[kRing];
    TileBuf tile[kTileBufs];
    R dist[kRing];
    R ks[kWarp];
    uint32_t nev[kWarp];
};

__device__ __forceinline__ void flush_counters(DScalars *sc, unsigned long long &nsteps, unsigned long long &nbund,
                                               int lane) {
    unsigned long long st = nsteps, nb = nbund;
    for (int o = 16; o > 0; o >>= 1) {
        st += __shfl_xor_sync(0xffffffffu, st, o);
        nb += __shfl_xor_sync(0xffffffffu, nb, o);
    }
    if (lane == 0) {
        atomicAdd(&sc->steps, st);
        atomicAdd(&sc->bundles, nb);
    }
    nsteps = nbund = 0;
}

// Ring position of a running index (below 2 kRing).
__device__ __forceinline__ int ring_at(int i) { return i < kRing ? i : i - kRing; }

// SCAT: the variant for media with scattering particles.  MINB: the occupancy
// knob.  Registers of its values: 128 lets two 256-thread blocks onto an SM, 72
// seven 128-thread blocks, 64 four 256-thread blocks.  72 is the default: 28
// warps and 24 bytes of spill, 40 with SCAT (64^3, photmax 256: 22.1 ms, with
// 64 registers 24.2, with 80 and 24 warps 23.3; with scattering coefficients
// of 0.1-1 1/m 37.2 ms, with 64 registers 40.0, with 128 43.0).  FP64 fits 128
// (64 and 72 spill 550-750 bytes: 48x40x32 2.5 ms, 3.2 and 3.0).
constexpr int march_regs(int minb) { return minb >= 4 ? 64 : minb == 3 ? 72 : 128; }

template <typename R, int MINB, bool SCAT>
__global__ void __launch_bounds__(256) __maxnreg__(march_regs(MINB)) k_march(const __grid_constant__ MarchParams<R> prm) {
    const MarchArgs &a = prm.m;
    extern __shared__ __align__(16) unsigned char smem[];
    // volatile: kept in a register instead of read again at every use
    int lane, warp;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    asm volatile("mov.u32 %0, %1;" : "=r"(warp) : "r"(threadIdx.x >> 5));
    const int nwarps = blockDim.x >> 5;
    WarpShared<R, SCAT> *ws = reinterpret_cast<WarpShared<R, SCAT> *>(smem) + warp;
    const size_t wbytes = ((sizeof(WarpShared<R, SCAT>) * nwarps) + 15) & ~(size_t)15;
    const DSolve<R> &S = prm.one;
    double *slots0 = reinterpret_cast<double *>(smem + wbytes) + (size_t)warp * a.nbuf * (kWarp * S.rpt);
    const DSolve<R> &D = *reinterpret_cast<const DSolve<R> *>(a.desc);  // with the run-time values
    const unsigned lt = (1u << lane) - 1u;

    // warp-uniform state
    unsigned busy = 0u;     // bit p: buffer p holds a tile not yet reduced
    int epar = -1;          // buffer being emitted from (-1: every bundle of the busy buffers is emitted)
    int next_b = 0, head = 0, count = 0;
    bool drained = false;   // no more tiles
    // tiles claimed from the queue but not started: chunk_left from chunk_next on
    unsigned long long chunk_next = 0;
    int chunk_left = 0;
    bool hold = false;      // a tile of the priority list's first part is in flight: claim no other
    unsigned amask = 0u;    // lanes tracing a ray (warp-uniform; kept in step with the lanes' own flags)
    // lane state
    bool active = false;
    int myslot = 0;  // the lane's bundle: buffer << 12 | index in the tile
    unsigned long long nsteps = 0, nbund = 0;
    Ray<R> r = {};
    ScatState<R> qs;
    qs.dist = (R)0;

    for (;;) {
        // ---- fetch the next tile into a free buffer
        if (epar < 0 && !drained && !hold) {
            const int fpar = __ffs(~busy) - 1;
            if (fpar < a.nbuf) {
                // with the long-ray priority list, the claim space is the
                // listed tiles followed by all tiles in natural order (listed
                // ones skipped there); the counts are read here, not kept
                const volatile unsigned *np = a.n_prio;
                const unsigned nsolo = np ? np[0] : 0u, nprio = np ? nsolo + np[1] : 0u;
                const unsigned long long total = (unsigned long long)a.total_tiles + nprio;
                unsigned long long tile;
                // ends: every pass advances chunk_next or the shared
                // counter, and a claim at or past `total` ends the queue
                for (;;) {
                    if (chunk_left <= 0) {
                        // guided self-scheduling: claim up to kChunkMax
                        // consecutive tiles (neighbouring cells); claim
                        // fewer as the queue drains to keep the tail short,
                        // and the longest rays one by one
                        if (lane == 0) {
                            const unsigned long long seen = *(volatile unsigned long long *)a.tile_counter;
                            const unsigned long long rem = seen < total ? total - seen : 0ull;
                            const unsigned long long k = rem / (4ull * gridDim.x * nwarps);
                            chunk_left = seen < nsolo ? 1 : (int)max(1ull, min((unsigned long long)kChunkMax, k));
                            chunk_next = atomicAdd(a.tile_counter, (unsigned long long)chunk_left);
                        }
                        chunk_next = __shfl_sync(0xffffffffu, chunk_next, 0);
                        chunk_left = __shfl_sync(0xffffffffu, chunk_left, 0);
                    }
                    tile = chunk_next++;
                    chunk_left--;
                    if (tile >= total) {
                        tile = total;
                        break;
                    }
                    if (!np) break;
                    if (tile < nprio) {
                        const bool solo = tile < nsolo;
                        hold = solo && nsolo <= gridDim.x * nwarps;
                        tile = __ldg(a.prio_tiles + (solo ? tile : (unsigned long long)a.total_tiles - 1 - (tile - nsolo)));
                        break;
                    }
                    if (!__ldg(a.tile_prio + (tile - nprio))) {
                        tile -= nprio;
                        break;
                    }
                    // a listed tile met again in natural order: claim the next
                }
                if (tile >= (unsigned long long)a.total_tiles) {
                    drained = true;
                } else {
                    if (lane == 0) decode_tile(S, ((long long)tile + S.tile_base) * kWarp, ws->tile[fpar]);
                    double *sl = slots0 + fpar * (kWarp * S.rpt);
                    for (int b = lane; b < kWarp * S.rpt; b += kWarp) sl[b] = 0.0;
                    busy |= 1u << fpar;
                    epar = fpar;
                    next_b = 0;
                    __syncwarp();
                }
            }
        }
        const int rpt = S.rpt;
        const int lrpt = __ffs(rpt) - 1;
        const int pool = kWarp * rpt;
        // ---- converged emission wave: one bundle per lane
        if (count < kRefill && epar >= 0) {
            const int b = next_b + lane;
            Emitted<R> e;
            R dist0 = (R)kNoEvent;
            ItemId it = tile_item(S, ws->tile[epar], b >> lrpt);
            int h = it.h0 + (b & (rpt - 1));
            const bool valid = it.kind >= 0 && h < S.photmax;
            if (!valid) {  // a padding item: emit anything, and drop it
                it.kind = 0;
                it.i = it.j = it.k = 1;
                it.v = h = 0;
            }
            nbund += valid;
            // with particles, draw 1 (scatter_first_lnu, written out: the
            // call form spilled more) before the emission itself: little is
            // live then, and the variant spills 40 bytes in all
            R lnu = (R)0;
            if constexpr (SCAT) {
                if (S.nA > 0) {
                    const uint4 c0 = scatter_counter(S.imax, S.jmax, it.kind, it.i, it.j, it.k, it.v, h, 0u);
                    rc_u32x4 c;
                    c.x = c0.x;
                    c.y = c0.y;
                    c.z = c0.z;
                    c.w = 1u;
                    const rc_u32x4 d = rc_philox4x32_10(c, S.key0, S.key1);
                    lnu = -RT<R>::log_((R)rc_u01(d.x));
                }
            }
            const bool ok = emit_bundle(e, S, D.row, it.kind, it.i, it.j, it.k, it.v, h) && valid;
            e.kk |= (b << 18) | (epar << 29);
            if constexpr (SCAT) {
                const R ks = scatter_coef(S, e.nbg & 0xfffff, e.nbg >> 20);
                if (ks > (R)0) dist0 = lnu / ks;  // scatter_first_dist
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            int pos = __popc(m & lt);
            if (S.sort) {
                // band-sorted order: the wave enters the ring by ascending
                // k_{nb,g} at the table row nearest Tmax (ties by lane), so
                // bundles handed out together have similar optical path
                // lengths.  Which lane traces a bundle does not change its
                // tally (each bundle owns its slot).
                unsigned key = 0xffffffffu;
                if (ok) {
                    const int nb = e.nbg & 0xfffff, g = e.nbg >> 20;
                    key = __float_as_uint((float)S.ki[RC_IX(((size_t)nb * S.nQ + g) * S.nT + D.row,
                                                            (long long)S.nB * S.nQ * S.nT, SITE_EMIT_ROW, S)]
                                              .k0);  // k >= 0: monotone bits
                }
                int rank = 0;
                for (int q = 0; q < kWarp; ++q) {
                    const unsigned kq = __shfl_sync(0xffffffffu, key, q);
                    rank += (kq < key) || (kq == key && q < lane);
                }
                pos = rank;
            }
            if (ok) {
                const int at = ring_at(head + count + pos);
                ws->ring[at] = e;
                if constexpr (SCAT) ws->dist[at] = dist0;
            }
            count += __popc(m);
            if (lane == 0) ws->tile[epar].out += __popc(m);
            next_b += kWarp;
            if (next_b >= pool) epar = -1;
            __syncwarp();
        }
        // ---- idle lanes take emitted bundles
        {
            const int navail = min(count, kWarp - __popc(amask));
            if (navail > 0) {
                const int rank = __popc(~amask & lt);
                const bool take = !active && rank < navail;
                if (take) {
                    const int at = ring_at(head + rank);
                    const Emitted<R> &e = ws->ring[at];
                    place_bundle(r, S, D, e);
                    if constexpr (SCAT) {
                        qs.dist = ws->dist[at];
                        ws->ks[lane] = scatter_coef(S, e.nbg & 0xfffff, e.nbg >> 20);
                        ws->nev[lane] = 0u;
                    }
                    myslot = (((e.kk >> 29) & 3) << 12) | ((e.kk >> 18) & 0x7ff);
                    active = true;
                }
                head = ring_at(head + navail);
                count -= navail;
                amask |= __ballot_sync(0xffffffffu, take);
                __syncwarp();
            }
        }
        // ---- step every active ray; stay in this loop until enough lanes
        //      are idle to be worth handing out bundles (or, with nothing to
        //      hand out, a tile can be reduced, or every lane is idle)
        bool check;
        {
            const bool can_feed = count > 0 || epar >= 0 || (!drained && !hold && busy != (1u << a.nbuf) - 1u);
            // leave the loop once this few lanes move, or (nothing to hand
            // out) as soon as a ray stops
            const int enough = can_feed ? kWarp - kFeedIdle : 0;
            const unsigned on_stop = can_feed ? 0u : 0xffffffffu;
            unsigned am = amask;
            for (;;) {
                // a black wall ends the ray; other walls, a spent step
                // budget and a cell to be rebuilt take the slow path
                active = active && r.q < kBlack;
                bool go = active;
                if constexpr (SCAT) go = active && !(qs.dist < (R)0);
                if (go && (r.q >= kSpecular || r.rem <= 0)) {
                    if (r.q == kPeriodic && r.rem > 0) wrap_cell(r, S);
                    else active = enter_cell(r, S);
                }
                go = go && active && r.q < kSpecular;
                const bool above = march_step<R, SCAT>(r, qs, S, go);
                active = active && (above || !go);
                bool wait_turn = false;
                if constexpr (SCAT) wait_turn = active && qs.dist < (R)0;
                am = __ballot_sync(0xffffffffu, active);
                // lanes stopped at a scattering event wait for a turn pass,
                // which draws all their new directions at once; the pass is
                // long and runs on the waiting lanes only, so it waits until
                // kTurnGather lanes wait, or every traced ray does
                unsigned tm = 0u;
                bool turn_now = false;
                if constexpr (SCAT) {
                    tm = __ballot_sync(0xffffffffu, wait_turn);
                    turn_now = __popc(tm) >= kTurnGather || (tm && !(am & ~tm));
                }
                const unsigned moving = am & ~tm;
                if (__popc(moving) <= enough || ((am ^ amask) & on_stop) || (SCAT && turn_now && __popc(moving) <= kWarp - kFeedIdle))
                    break;
            }
            // ---- retire the rays that stopped: last deposit, tally slot
            bool last = false;
            if (am != amask) {
                if (((amask & ~am) >> lane) & 1u) {
                    retire_ray(r, S);
                    nsteps += S.steps_to[r.ln >> 20] - r.rem;
                    slots0[(myslot >> 12) * pool + (myslot & 0xfff)] = r.De;
                    last = atomicSub(&ws->tile[myslot >> 12].out, 1) == 1;
                }
                amask = am;
                __syncwarp();  // (without it ptxas keeps the warp's state in vector registers)
            }
            // a tile may be complete: its last ray has stopped, or its last
            // wave was empty
            check = __any_sync(0xffffffffu, last) || count == 0;
        }
        // ---- scattering: the new directions of every lane stopped at an
        //      event, once kTurnGather lanes wait or no traced ray is left
        //      that does not wait (waiting lanes never deadlock the warp)
        if constexpr (SCAT) {
            const unsigned tw = __ballot_sync(0xffffffffu, active && qs.dist < (R)0);
            const bool turn_now = __popc(tw) >= kTurnGather || (tw && !(amask & ~tw));
            if (turn_now && active && qs.dist < (R)0) {
                const int myb = myslot & 0xfff;
                const ItemId it = tile_item(S, ws->tile[myslot >> 12], myb >> lrpt);
                uint4 c = scatter_counter(S.imax, S.jmax, it.kind, it.i, it.j, it.k, it.v, it.h0 + (myb & (rpt - 1)),
                                          ws->nev[lane]);
                scatter_turn(r, c, ws->ks[lane], qs, S);
                ws->nev[lane] = c.w;
            }
        }
        // ---- reduce finished tiles: chunk sums in bundle order, group sums
        //      in item order
        if (check) {
            __syncwarp();
            unsigned ready = busy & (epar < 0 ? ~0u : ~(1u << epar));
            ready &= __ballot_sync(0xffffffffu, ws->tile[lane < kTileBufs ? lane : 0].out == 0);
            const int lgs = __ffs(S.gsize) - 1;  // items of a group: a power of two
            while (ready) {
                const int par = __ffs(ready) - 1;
                ready &= ready - 1u;
                const double *sl = slots0 + par * pool;
                double s = 0.0;
                for (int h = 0; h < rpt; ++h) s += sl[lane * rpt + h];
                const int base = lane >> lgs << lgs;
                double g = 0.0;
                for (int q = 0; q < S.gsize; ++q) g += __shfl_sync(0xffffffffu, s, base + q);
                const long long item = ws->tile[par].item0 + lane;
                if (lane == base && item < S.n_items) S.partial[RC_IX(item >> lgs, S.n_partial, SITE_PARTIAL, S)] = g;
                busy &= ~(1u << par);
                __syncwarp();
            }
            if (!busy) hold = false;
        }
        if (drained && !busy) break;
    }
    flush_counters(S.sc, nsteps, nbund, lane);
}

// Tiles a warp keeps in flight.  A tile's slots are held until its longest
// ray has finished, and with every buffer held the warp runs out of bundles.
constexpr int tile_bufs(int rpt) { return rpt <= 4 ? kTileBufs : 2; }

template <typename R, bool SCAT>
constexpr size_t march_smem_bytes(int block, int rpt, int nbuf) {
    return ((((size_t)sizeof(WarpShared<R, SCAT>) * (block / kWarp)) + 15) & ~(size_t)15) +
           (size_t)(block / kWarp) * nbuf * kWarp * rpt * sizeof(double);
}

}  // namespace rc
