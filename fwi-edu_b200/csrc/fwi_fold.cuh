// fwi_fold.cuh -- the time-step kernel on folded fields.
//
// A folded field pairs column x of the padded grid with column x + W, W = ceil(Nx / 2): element
// (x, z) of the left half and (x + W, z) of the right half are neighbours in memory,
//     [W + 6 columns][ld rows][2 halves],  column f at index f + 3, z fastest but for the pair.
// Both halves of a pair take the same path through the stencil, so every operand of the packed
// f32x2 arithmetic -- the column itself, its neighbours in z and in x, the previous field, the
// coefficients -- is a register pair exactly as it was loaded.  (Pairing neighbours in z instead
// makes every odd z offset a pair that straddles two loads, rebuilt with moves for each cell.)
// Three halo columns at either end continue each half across the seam: index -3..-1 holds the
// left half's last columns for the right half, W..W+2 the right half's first ones for the left;
// the thread that updates such a column writes its copy too.  What lies outside the grid is zero.
//
// A block owns a tile of TZ rows by TX folded columns (2 TX columns of the grid) and walks a chunk
// of shots that share the model window; a thread updates two rows of one or two folded columns, four
// or eight cells, per shot.  One extra producer warp moves, per shot, the tile of u(t) with its halo
// (four rows, three columns) and the tile of u(t-1) into a ring of nst shared-memory stages by two
// tensor copies (cp.async.bulk.tensor; out-of-range parts read as zero), each stage with a "full" and
// an "empty" mbarrier; consumer warps meet at no block barrier.  The thread's coefficients stay in
// registers for all shots of the chunk.  In a model with a free surface the tiles start at the
// surface row: nothing above it is ever updated.
//
// What bounds it: the FP32 pipes and shared memory about alike.  A cell update is 50 operations the
// reference rounds one by one (50 pipe cycles per 128 cells and SM) and, with the coefficients in
// registers, 9 (two columns per thread) to 11 16-byte shared loads per four cells plus the stage's
// writes (46 .. 58 cycles per 128 cells); spills, or rare parts of the epilogue in the common loop,
// cost far more than either (a spilling build of the same tile: 66 us).  Blocks of the free-surface
// tiles pace the others through the waits between launches, so what they do beside the stencil --
// receiver sampling, the injection's values -- is the producer warp's work, and the epilogue is
// compiled in four forms, chosen per tile.
// Measured, 60 shots on 221 x 601 (B200, 1.9 GHz): 34.2 us per forward step and 73.3 us per replay +
// adjoint launch, against 38.6 and 83.1 with k_tile3 of fwi_tile.cuh; 8 shots on 301 x 901: 10.5 and
// 22.1 against 13.2 and 30.4; 6 shots on 601 x 2001: 31.0 and 61.3 against 34.5 and 72.0; one shot on
// 221 x 601: 2.7 us per forward step against 3.4.
//
// Arithmetic (MATH 0): every product and sum rounded on its own in the reference's association
// order (acoustic_iso2d_fd_it_6order, propagation.c:13-74).  A packed multiply that feeds a packed
// add would be contracted by the compiler although both carry .rn, so such a product is
// fma(a, b, -0), which rounds exactly as a * b and is not fused any further; -0 is read at run time
// so that it stays.  MATH 1 contracts multiply-adds (fwi_tile.cuh).
//
// The epilogue fuses what the reference does around the stencil: point source (forward: double,
// before the free surface, propagation.c:558; replay: float, after it, :662), mirror free surface
// (:76-101), pseudo-Hessian (:579-594), imaging (:700-714), receiver sampling (:567-576) and the
// adjoint injection (:676-682), each only in the tiles that it reaches.
#pragma once
#include "fwi_tile.cuh"

namespace fwi {

constexpr int FOLD_HALO = 3;  // halo columns at either end of a folded field

// ------------------------------------------------------------ tile geometry
// A launch's tiles: TZ rows (even), NP threads of ncol folded columns each along x, a ring of nst
// stages.  The kernel takes it as a parameter, so that a window's rows and columns fill its tiles:
// fixed 64-row tiles left a fifth of the threads of a 258-row window idle.
struct FoldTile {
    int TZ, NP, nst, ncol;
    int nw;  // consumer warps, at least what NZP() * NP threads need
    __host__ __device__ int NZP() const { return TZ / 2; }    // row pairs of a column
    __host__ __device__ int TX() const { return ncol * NP; }  // folded columns
    __host__ __device__ int ZP() const { return TZ + 8; }     // rows of the u(t) tile: Z0-4 .. Z0+TZ+3
    __host__ __device__ int XP() const { return TX() + 2 * FOLD_HALO; }
    __host__ __device__ int p1_bytes() const { return ZP() * XP() * 8; }
    __host__ __device__ int p0_bytes() const { return TZ * TX() * 8; }
    __host__ __device__ int p0_off() const { return round128(p1_bytes()); }
    __host__ __device__ int stage() const { return p0_off() + round128(p0_bytes()); }
    __host__ __device__ int smem() const { return nst * stage(); }
};
constexpr int FOLD_WARPS = 7;    // most consumer warps of a block: with the producer warp, two blocks of
                                 // 128 registers a thread (two columns) or three of 80 (one column)
constexpr int FOLD_NST = 4;      // deepest ring
constexpr int FOLD_TX_MAX = 32;  // widest tile

// As mbar_wait of fwi_tile.cuh (false after two seconds) for waits that are expected to be long: each
// try may suspend the thread for up to a microsecond while the phase is open, and the clock is read
// once per 16 tries, so that a waiting warp takes few issue slots from the working ones
__device__ __forceinline__ bool mbar_try_long(unsigned bar, unsigned parity)
{
    unsigned done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}
__device__ __forceinline__ bool fold_mbar_wait(unsigned bar, unsigned parity, u64 limit_ns = 2000000000ull)
{
    if (mbar_try(bar, parity)) return true;
    const u64 t0 = global_ns();
    for (;;) {
#pragma unroll 1
        for (int q = 0; q < 16; ++q)
            if (mbar_try_long(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}
// the same by a whole warp, which goes on or gives up as one: a lane's own clock may run out just before the
// phase completes for another
__device__ __forceinline__ bool fold_warp_wait(unsigned bar, unsigned parity, u64 limit_ns = 2000000000ull)
{
    return __all_sync(0xffffffffu, fold_mbar_wait(bar, parity, limit_ns));
}

// ------------------------------------------------------------ arithmetic
struct FoldConst {
    float sx, sz, sxx, szz;  // 1/dx, 1/dz, 1/dx^2, 1/dz^2
    u64 NZ;                  // -0 as a pair
};
// One row of a folded column (two cells, one per half); as cell2 of fwi_tile.cuh
template <int MATH>
__device__ __forceinline__ u64 fold_cell(u64 zm3, u64 zm2, u64 zm1, u64 z0, u64 zp1, u64 zp2, u64 zp3, u64 xm3, u64 xm2,
                                         u64 xm1, u64 xp1, u64 xp2, u64 xp3, u64 c1, u64 c2, u64 ck, u64 irx, u64 irz,
                                         u64 ir, u64 p0, const FoldConst &k)
{
    if (MATH != 0)
        return cell2<1>(zm3, zm2, zm1, z0, zp1, zp2, zp3, xm3, xm2, xm1, xp1, xp2, xp3, c1, c2, ck, irx, irz, ir, p0,
                        make_pkconst(k.sx, k.sz, k.sxx, k.szz, 0.0f));
    auto mul = [&](u64 a, u64 b) { return fma2(a, b, k.NZ); };
    // by a stencil constant or a grid spacing: two scalar products with an immediate or constant-bank
    // operand take the pipe as long as one packed product and no registers
    auto mulk = [&](float c, u64 b) {
        const float2 y = upk(b);
        return pk(__fmul_rn(y.x, c), __fmul_rn(y.y, c));
    };
    const u64 dpdz = mulk(k.sz, add2(add2(mulk(FD_C1, sub2(zp1, zm1)), mulk(FD_C2, sub2(zp2, zm2))),
                                     mulk(FD_C3, sub2(zp3, zm3))));
    const u64 dpdx = mulk(k.sx, add2(add2(mulk(FD_C1, sub2(xp1, xm1)), mulk(FD_C2, sub2(xp2, xm2))),
                                     mulk(FD_C3, sub2(xp3, xm3))));
    const u64 d0 = mulk(FD_D0, z0);
    const u64 dzz = mulk(k.szz, add2(add2(add2(d0, mulk(FD_D1, add2(zp1, zm1))), mulk(FD_D2, add2(zp2, zm2))),
                                     mulk(FD_D3, add2(zp3, zm3))));
    const u64 dxx = mulk(k.sxx, add2(add2(add2(d0, mulk(FD_D1, add2(xp1, xm1))), mulk(FD_D2, add2(xp2, xm2))),
                                     mulk(FD_D3, add2(xp3, xm3))));
    const u64 lap = add2(add2(mul(irx, dpdx), mul(irz, dpdz)), mul(ir, add2(dxx, dzz)));
    return add2(add2(mul(c1, z0), mul(c2, p0)), mul(ck, lap));
}

// two folded elements (rows z and z + 1), each a register pair
struct Pair2 {
    u64 a, b;
};
// 16- and 8-byte shared loads straight into register pairs (volatile as lds4)
__device__ __forceinline__ Pair2 lds_pair2(unsigned addr)
{
    Pair2 v;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "r"(addr));
    return v;
}
__device__ __forceinline__ u64 lds_pair(unsigned addr)
{
    u64 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ Pair2 ldg_pair2(const float *p)
{
    Pair2 v;
    asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p));
    return v;
}

// ------------------------------------------------------------ program items
// One half of a launch's program item with what follows from it for a group: the frames read
// (i1: u(t), i0: the field before it) and written (io), the frame the imaging reads (iu, -1 none) and
// the record row that the step samples (srow, -1 none).  The same for every shot of the group.
struct FoldItem {
    int kind, it, i1, i0, io, iu, srow;
};
__host__ __device__ inline FoldItem fold_item(const ShotDesc &A, int kind, int it)
{
    FoldItem q{kind, it, 0, 0, 0, -1, -1};
    if (kind == K_NONE) return q;
    step_frames(A, kind, it, q.i1, q.i0, q.io);
    if (kind == K_ADJ && it % MST == 0) q.iu = img_idx(A, it);
    if ((kind == K_FWD0 || kind == K_FWD1) && it % A.sr == 0) q.srow = it / A.sr;
    return q;
}

// What the step needs of a group beside its items: the descriptor's fields, copied together for the
// launches of several groups, whose blocks each read their own group's from the constant bank, cold.
// With the fields packed and the groups' first blocks in an array of their own (the search read one
// word of every entry) a launch of 16 windows of 76 x 433 takes 15.4 us instead of 16.8, one of 48
// windows 15.7 instead of 19.8.  k_fold keeps the descriptor: one group stays cached there, and the
// packed form's other register assignment cost 60 shots of 221 x 601 35.1 us instead of 34.2.
struct FoldGeo {
    int Nx, Nz, ld, W, zb, pml, nz, nxx, fs, izStart, nfr, hessian, snap;
    float invdx, invdz, invdxdx, invdzdz, invdtdt, dt, negzero;
    long long frame;
    float *frames;
    const float *cf;
};
inline FoldGeo fold_geo(const ShotDesc &d)
{
    return FoldGeo{d.Nx, d.Nz, d.ld, d.W, d.zb, d.pml, d.nz, d.nxx, d.fs, d.izStart, d.nfr, d.hessian, d.snap,
                   d.invdx, d.invdz, d.invdxdx, d.invdzdz, d.invdtdt, d.dt, d.negzero, d.frame, d.frames, d.cf};
}

// ------------------------------------------------------------ waits between launches
// As wait_neighbours of fwi_tile.cuh over folded column tiles, by the whole producer warp, one flag
// per lane.  The columns close into a ring at the seam: the first tile's left halo is written by the
// tiles that hold columns W-3 .. W-1 (the last one or two), the right halo of the last two tiles by
// the first; each of these pairs waits for the other, as neighbours in the interior do.
__device__ __forceinline__ bool fold_wait(const TileSync &ts, int by, int bx, int bz, const int *err)
{
    const int lane = threadIdx.x & 31;
    const int need = ts.Lprev + 1;
    const u64 t0 = global_ns();
    bool ok = true;
    // candidates: column offsets -1, 0, +1 and the seam partners (two more), times 3 rows, times
    // the item halves: at most 30
    const int q = lane % 15, h = lane / 15;
    const int dz = q / 5 - 1, sel = q % 5;
    int nx = sel < 3 ? bx + sel - 1 : -1;
    if (sel >= 3) {
        if (bx == 0) nx = ts.ntx - 1 - (sel - 3);
        else if (bx >= ts.ntx - 2) nx = 0;
    }
    const int nz = bz + dz;
    const bool mine = h < ts.halves && nx >= 0 && nx < ts.ntx && nz >= 0 && nz < ts.zt;
    const int row = ts.halves == 2 ? ((by & ~1) | h) : by;
    const int *f = ts.flags + ((long long)row * ts.zt + nz) * ts.ntx + nx;
    for (;;) {
        const bool done = !mine || ld_relaxed(f) >= need;
        if (__all_sync(0xffffffffu, done)) break;
        const bool stop = global_ns() - t0 > 2000000000ull || ld_relaxed(err) != 0;
        if (__any_sync(0xffffffffu, stop)) {
            ok = false;
            break;
        }
        __nanosleep(32);
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("fence.proxy.async.global;" ::: "memory");
    return ok;
}

// ------------------------------------------------------------ the step
// A: the group's geometry, coefficients and frame layout (ShotDesc of its first shot, or FoldGeo).
// item: the block's half of the launch's program item; grid: bx column tile, by = 2 * chunk + item
// half, bz z tile.
template <int MATH, int NCOL, class Geo>
__device__ __forceinline__ void fold_body(const CUtensorMap &tm_p1, const CUtensorMap &tm_p0, const Geo &A,
                                          const FoldTile &T, const ShotDesc *__restrict__ shots, const FoldItem &item,
                                          int L, int shot_base, int nshot, int chunk, int *err, int bx, int by, int bz,
                                          const TileSync &ts)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long full[FOLD_NST], empty[FOLD_NST];
    __shared__ double s_srcd[TILE_CH_MAX];
    __shared__ float s_srcf[TILE_CH_MAX];
    // the source's folded column (-1: not in this tile, or no source in this kind of step) and
    // 2 * (row - first row of the tile) + half
    __shared__ int s_sf[TILE_CH_MAX], s_sz[TILE_CH_MAX];
    __shared__ float *s_tr[TILE_CH_MAX];         // trace row of this step's sample, or null
    __shared__ const float *s_adj[TILE_CH_MAX];  // adjoint-source row of this step's injection, or null
    __shared__ const int4 *s_rcol[TILE_CH_MAX];  // the shot's receivers by column of the grid
    // what an adjoint step injects into the shot of a stage, per column of the tile and half: (row -
    // first row of the tile, -1 none, -2 several: read from the receiver list; value)
    __shared__ __align__(16) float2 s_inj[FOLD_NST][2 * FOLD_TX_MAX];
    __shared__ double *s_acc[TILE_CH_MAX];  // the FP64 accumulator of an accumulating step

    grid_dep_launch();  // the next step may begin its set-up once every block of this one runs
    const int tid = threadIdx.x;
    const bool fine = ts.flags != nullptr;
    const int kind = item.kind, it = item.it;
    if (kind == K_NONE) {
        // an idle item half still completes its item in order, for the flags' readers
        if (fine && tid == 0) {
            int *own = ts.flags + ((long long)by * ts.zt + bz) * ts.ntx + bx;
            const u64 t0 = global_ns();
            while (ts.Lprev >= 0 && ld_relaxed(own) < ts.Lprev + 1 && global_ns() - t0 < 2000000000ull &&
                   ld_relaxed(err) == 0)
                __nanosleep(64);
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            st_relaxed_gpu(own, L + 1);
        }
        return;
    }
    const int cb = shot_base + (by >> 1) * chunk;
    const int n = min(chunk, shot_base + nshot - cb);
    if (n <= 0) return;
    const int TZ = T.TZ, TX = T.TX(), NZP = T.NZP(), NW = T.nw, NST = T.nst;
    const int W = A.W;
    const bool fwd = kind == K_FWD0 || kind == K_FWD1;
    const int warp = tid >> 5, lane = tid & 31;

    const int X0 = bx * TX, Z0 = A.zb + bz * TZ;  // first folded column and row of the tile
    const int p0_off = T.p0_off(), stage = T.stage(), ZP = T.ZP();
    // the copies of shot j into stage st; the stage is full once they have landed and the producer
    // warp has arrived on it
    auto issue = [&](int j, int st) {
        const unsigned b = smem_u32(&full[st]);
        mbar_expect(b, T.p1_bytes() + T.p0_bytes());
        unsigned char *stg = smem + st * stage;
        tma_load4(smem_u32(stg), &tm_p1, 2 * (Z0 - 4), X0, item.i1, cb + j - shot_base, b);
        tma_load4(smem_u32(stg + p0_off), &tm_p0, 2 * Z0, X0 + FOLD_HALO, item.i0, cb + j - shot_base, b);
    };
    const bool inject = kind == K_ADJ && it >= 1, samples = item.srow >= 0;
    bool spec_here = false;
    // consumers: thread (kp, zp) updates rows z0, z0 + 1 of the folded columns f0, f0 + 1
    const int kp = tid / NZP, zp = tid - kp * NZP;
    const int f0 = X0 + NCOL * kp, z0 = Z0 + 2 * zp;
    const bool act0 = kp < T.TX() / NCOL && f0 < W && z0 < A.Nz - 3 && !(A.fs && z0 + 1 < A.pml), act1 = NCOL > 1 && act0 && f0 + 1 < W;
    const int ld = A.ld;
    const int off = ((f0 + FOLD_HALO) * ld + z0) * 2;  // offset of (f0, z0) in a frame or coefficient plane
    Pair2 cf[NCOL][6] = {};  // coefficients c1, c2, coef3*K, irx, irz, ir of both columns
    if (warp == NW) {
        if (lane == 0) {
            for (int j = 0; j < NST; ++j) {
                mbar_init(smem_u32(&full[j]), 1);
                mbar_init(smem_u32(&empty[j]), samples ? NW + 1 : NW);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        if (fine && ts.Lprev >= 0) {
            const bool ok = fold_wait(ts, by, bx, bz, err);
            if (!ok && lane == 0) atomicExch(err, 1);
        } else {
            grid_dep_wait();
        }
        if (lane == 0)
            for (int j = 0; j < min(n, NST); ++j) issue(j, j);
    } else {
        // the coefficients are the pass's own: no step writes them
#pragma unroll
        for (int c = 0; c < NCOL; ++c)
            if (c ? act1 : act0)
#pragma unroll
                for (int q = 0; q < 6; ++q) cf[c][q] = ldg_pair2(A.cf + (long long)q * A.frame + off + c * 2 * ld);
        if (tid < n) {
            // ---- per-shot scalars of the chunk
            const ShotDesc &D = shots[cb + tid];
            s_srcd[tid] = fwd ? D.srcd[it] : 0.0;
            s_srcf[tid] = kind == K_REP ? D.srcf[it] : 0.0f;
            s_acc[tid] = kind == K_ADJ ? D.Gacc : D.H;
            s_rcol[tid] = D.rcol;
            // does this tile need the rare parts of the epilogue for this shot (its source, its
            // receiver rows)?
            const int half = D.isx >= W, fsrc = D.isx - half * W;
            const bool src_t = (fwd || kind == K_REP) && fsrc >= X0 && fsrc < X0 + TX && D.isz >= Z0 && D.isz < Z0 + TZ;
            const bool rows_t = Z0 + TZ > D.rz0 && Z0 <= D.rz1;
            s_sf[tid] = src_t ? fsrc : -1;
            s_sz[tid] = 2 * (D.isz - Z0) + half;
            s_tr[tid] = samples && rows_t ? D.traces_t + (long long)item.srow * D.ntr : nullptr;
            s_adj[tid] = inject && rows_t ? D.adj_t + (long long)(it - 1) * D.ntr : nullptr;
            spec_here = src_t || (inject && rows_t);
        }
    }
    // barriers and the per-shot scalars; no block-wide barrier follows
    const bool any_spec = __syncthreads_or(spec_here) != 0;
    // fields and accumulators: after the previous step (the producer warp waited already; with
    // TileSync the consumers touch them only after a stage that was filled after its wait)
    if ((!fine || ts.Lprev < 0) && warp < NW) grid_dep_wait();

    if (warp == NW) {
        // ---- producer warp.  A stage whose copies are issued becomes full once the warp has left
        // there what the step injects (the adjoint source is read here: the waits above are over).
        // Sampling steps: the warp reads the receivers' values from the full stage, beside the
        // consumers.  Then shot j + NST follows into the stage once everybody is done with it.
        auto fill = [&](int j, int st) {
            if (inject && s_adj[j] != nullptr) {
                for (int q = lane; q < 2 * TX; q += 32) {
                    const int fq = X0 + (q >> 1), xq = fq + (q & 1) * W;
                    float2 e = make_float2(__int_as_float(-1), 0.f);
                    if (fq < W && xq < A.Nx) {
                        const int4 r = __ldg(s_rcol[j] + xq);
                        if (r.x == -2) e.x = __int_as_float(-2);
                        else if (r.x >= Z0 && r.x < Z0 + TZ)
                            e = make_float2(__int_as_float(r.x - Z0),
                                            fm(fm(fm(fm(fm(__ldg(s_adj[j] + r.y), __int_as_float(r.z)), A.dt), A.dt),
                                                  A.invdx), A.invdz));
                    }
                    s_inj[st][q] = e;
                }
                __syncwarp();
            }
            if (lane == 0) mbar_arrive(smem_u32(&full[st]));
        };
        // the receivers of columns q = lane, lane + 32 of the tile (2 TX <= 64), fetched a shot ahead: the
        // loads' latency before each sample held back the next copies (60 shots: 36.0 -> 34.4 us a step)
        int4 rc[2] = {make_int4(-1, 0, 0, 0), make_int4(-1, 0, 0, 0)};
        auto fetch = [&](int j) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int q = lane + 32 * u, fq = X0 + (q >> 1), xq = fq + (q & 1) * W;
                if (j < n && s_tr[j] != nullptr && q < 2 * TX && fq < W && xq < A.Nx) rc[u] = __ldg(s_rcol[j] + xq);
                else rc[u].x = -1;
            }
        };
        auto sample = [&](int j, int st) {
            const float *sb = reinterpret_cast<const float *>(smem + st * stage);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int q = lane + 32 * u;
                const float *col = sb + (((q >> 1) + FOLD_HALO) * ZP + 4) * 2 + (q & 1);
                const int4 r = rc[u];
                if (r.x >= Z0 && r.x < Z0 + TZ) s_tr[j][r.y] = col[2 * (r.x - Z0)];
                else if (r.x == -2) {
                    const ShotDesc &D = shots[cb + j];
                    const int xq = X0 + (q >> 1) + (q & 1) * W;
                    for (int e = __ldg(D.colptr + xq), e1 = __ldg(D.colptr + xq + 1); e < e1; ++e) {
                        const int2 rr = __ldg(D.rec + e);
                        if (rr.x >= Z0 && rr.x < Z0 + TZ) s_tr[j][rr.y] = col[2 * (rr.x - Z0)];
                    }
                }
            }
            __syncwarp();
        };
        bool ok = true;
        for (int j = 0; j < min(n, NST); ++j) fill(j, j);
        if (samples) fetch(0);
        int issued = min(n, NST);
        for (int j = 0, st = 0, ph = 0; j < n; ++j) {
            if (samples) {
                if (s_tr[j] != nullptr) {
                    ok = fold_warp_wait(smem_u32(&full[st]), ph);
                    if (!ok) break;
                    sample(j, st);
                }
                if (lane == 0) mbar_arrive(smem_u32(&empty[st]));
                fetch(j + 1);
            }
            if (j + NST < n) {
                ok = fold_warp_wait(smem_u32(&empty[st]), ph);
                if (!ok) break;
                if (lane == 0) issue(j + NST, st);
                fill(j + NST, st);
                issued = j + NST + 1;
            }
            if (++st == NST) st = 0, ph ^= 1;
        }
        if (lane != 0) return;
        if (!ok) atomicExch(err, 1);
        // keep the block alive until every copy it issued has landed
        for (int j = max(0, issued - NST); j < issued; ++j) mbar_wait(smem_u32(&full[j % NST]), (j / NST) & 1);
        if (fine) {
            // the item is complete once everybody has released every stage: publish it
            for (int j = max(0, n - NST); j < n; ++j) mbar_wait(smem_u32(&empty[j % NST]), (j / NST) & 1);
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            st_relaxed_gpu(ts.flags + ((long long)by * ts.zt + bz) * ts.ntx + bx, L + 1);
        }
        return;
    }

    // ---- consumers
    const int pml = A.pml, zlo = A.izStart, zhi = A.Nz - 4;
    // free surface: row pml is -0 and rows pml+1 .. pml+3 are mirrored above it (nothing further
    // up is read again) -- all pml rows on the steps whose output is written out as a snapshot
    const int tout = kind == K_ADJ ? it - 1 : it + 1;
    const int fs_hi = (A.snap > 0 && tout % A.snap == 0) ? 2 * pml : min(2 * pml, pml + 3);
    const bool hess = kind == K_FWD1 && A.hessian && (it % MST == 0);
    const bool image = kind == K_ADJ && (it % MST == 0);
    const bool acc_tile = (hess || image) && Z0 < pml + A.nz && Z0 + TZ > pml;
    const bool fs_tile = A.fs && Z0 <= fs_hi;
    // the tile reaches the grid's edge or the seam: masked values, halo copies, the zero rows below
    const bool edge = X0 < 4 || X0 + TX > W - 5 || Z0 < zlo || Z0 + TZ - 1 >= zhi;
    const FoldConst K{A.invdx, A.invdz, A.invdxdx, A.invdzdz, pk(A.negzero, A.negzero)};
    const long long shot_stride = (long long)A.nfr * A.frame;
    const long long u_off = image ? (item.iu - item.io) * A.frame : 0;  // the imaging's field from the output
    float *out = A.frames + item.io * A.frame + (cb - shot_base) * shot_stride + off;
    const unsigned CS = ZP * 8;  // bytes of a staged column
    // the threads past the tile's last column pair (the last warp's rest) read the first pair's rows
    const int ks = kp < T.TX() / NCOL ? kp : 0;
    const unsigned rel = ((NCOL * ks + FOLD_HALO) * ZP + 2 * zp + 4) * 8u, rel0 = (NCOL * ks * TZ + 2 * zp) * 8u + p0_off;

    // stores rows z0, z0 + 1 of both halves of column f at o, and the copies beyond the seam
    auto store2 = [&](float *o, int f, const float4 &v) {
        *reinterpret_cast<float4 *>(o) = v;
        if (edge) {
            if (f < FOLD_HALO) *reinterpret_cast<float4 *>(o + 2 * W * ld) = make_float4(v.y, 0.f, v.w, 0.f);
            if (f >= W - FOLD_HALO) *reinterpret_cast<float4 *>(o - 2 * W * ld) = make_float4(0.f, v.x, 0.f, v.z);
        }
    };
    // one row of both halves
    auto store1 = [&](float *o, int f, float a, float b) {
        *reinterpret_cast<float2 *>(o) = make_float2(a, b);
        if (edge) {
            if (f < FOLD_HALO) *reinterpret_cast<float2 *>(o + 2 * W * ld) = make_float2(b, 0.f);
            if (f >= W - FOLD_HALO) *reinterpret_cast<float2 *>(o - 2 * W * ld) = make_float2(0.f, a);
        }
    };

    // one column (C = 0, 1) of the thread for shot i: x[C .. C+6] columns f-3 .. f+3 at rows z0, z0 + 1;
    // ca: the column's staged address at row z0, pa: of the previous field.  SPEC: the tile may hold the
    // free surface, a source or receivers; ACC: an accumulating step
    auto column = [&](int i, int st, auto cc, auto spec, auto accu, const Pair2 (&x)[NCOL + 6], unsigned ca, unsigned pa) {
        constexpr bool SPEC = decltype(spec)::value, ACC = decltype(accu)::value;
        constexpr int C = decltype(cc)::value;
        const int f = f0 + C;
        const bool active = C ? act1 : act0;
        float *o = out + C * 2 * ld;
        const Pair2 &ctr = x[3 + C];
        const u64 zm3 = lds_pair(ca - 24);
        const Pair2 zm = lds_pair2(ca - 16), zq = lds_pair2(ca + 16);
        const u64 zp4 = lds_pair(ca + 32);
        const Pair2 p0 = lds_pair2(pa);
        const Pair2(&k)[6] = cf[C];
        const u64 ra = fold_cell<MATH>(zm3, zm.a, zm.b, ctr.a, ctr.b, zq.a, zq.b, x[C].a, x[C + 1].a, x[C + 2].a,
                                       x[C + 4].a, x[C + 5].a, x[C + 6].a, k[0].a, k[1].a, k[2].a, k[3].a, k[4].a,
                                       k[5].a, p0.a, K);
        const u64 rb = fold_cell<MATH>(zm.a, zm.b, ctr.a, ctr.b, zq.a, zq.b, zp4, x[C].b, x[C + 1].b, x[C + 2].b,
                                       x[C + 4].b, x[C + 5].b, x[C + 6].b, k[0].b, k[1].b, k[2].b, k[3].b, k[4].b,
                                       k[5].b, p0.b, K);
        const float2 fa_ = upk(ra), fb_ = upk(rb);
        float4 v = make_float4(fa_.x, fa_.y, fb_.x, fb_.y);  // row z0: left, right half; row z0 + 1
        if (edge) {
            const bool va = f >= 3, vb = f + W <= A.Nx - 4;  // halves that are updated in this column
            const bool r0 = z0 >= zlo && z0 <= zhi, r1 = z0 + 1 >= zlo && z0 + 1 <= zhi;
            if (!va || !r0) v.x = 0.f;
            if (!vb || !r0) v.y = 0.f;
            if (!va || !r1) v.z = 0.f;
            if (!vb || !r1) v.w = 0.f;
            // the rows below the last updated one are zero in every frame
            if (active && z0 + 1 >= zhi) {
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                if (z0 + 2 < ld) store2(o + 4, f, zero);
                if (z0 + 4 < ld) store2(o + 8, f, zero);
            }
        }
        if (!active) return;
        if (!SPEC && !ACC) {
            store2(o, f, v);
            return;
        }
        [[maybe_unused]] const bool fs_top = SPEC && A.fs && z0 <= fs_hi;
        [[maybe_unused]] float4 mir = make_float4(0.f, 0.f, 0.f, 0.f);
        if (SPEC) {
            const int js = s_sz[i] - 4 * zp;  // component of v that holds the source's cell
            const bool src_here = f == s_sf[i] && js >= 0 && js < 4;
            // forward: the source enters before the free surface, in double (propagation.c:558-564)
            if (fwd && src_here) setc(v, js, (float)__dadd_rn((double)comp(v, js), s_srcd[i]));
            if (fs_top) {
                if (z0 == pml) v.x = v.y = -0.0f;
                if (z0 + 1 == pml) v.z = v.w = -0.0f;
                mir = make_float4(-v.x, -v.y, -v.z, -v.w);
            }
            // replay: free surface first, then the float source (propagation.c:656-662)
            if (kind == K_REP && src_here) setc(v, js, fa(comp(v, js), s_srcf[i]));
        }
        if (ACC && z0 + 1 >= pml && z0 < pml + A.nz) {
            const float4 uu = image ? ldg4(o + u_off) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float2 ca_ = upk(ctr.a), cb_ = upk(ctr.b), pa_ = upk(p0.a), pb_ = upk(p0.b);
            const float cc4[4] = {ca_.x, ca_.y, cb_.x, cb_.y}, pp[4] = {pa_.x, pa_.y, pb_.x, pb_.y};
            const bool r0 = z0 >= pml, r1 = z0 + 1 < pml + A.nz;
            double2 a[2];
            double *ap[2];
            bool ok[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int xc = f + h * W;
                ok[h] = xc >= pml && xc < pml + A.nxx;
                ap[h] = s_acc[i] + xc * ld + z0;
                if (ok[h]) a[h] = *reinterpret_cast<const double2 *>(ap[h]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!ok[h]) continue;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int q = 2 * j + h;
                    const float t = fm(fa(fs_(comp(v, q), fm(2.0f, cc4[q])), pp[q]), A.invdtdt);
                    const float w = image ? fm(t, comp(uu, q)) : fm(t, t);
                    if (j == 0 && r0) a[h].x = __dadd_rn(a[h].x, (double)w);
                    if (j == 1 && r1) a[h].y = __dadd_rn(a[h].y, (double)w);
                }
                *reinterpret_cast<double2 *>(ap[h]) = a[h];
            }
        }
        if (SPEC && inject && s_adj[i] != nullptr) {
            const float4 e4 = *reinterpret_cast<const float4 *>(&s_inj[st][2 * (NCOL * kp + C)]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = __float_as_int(h ? e4.z : e4.x);
                if (j >= 0) {  // the column's one receiver
                    const int q = 2 * (j - 2 * zp) + h;
                    if (q >= 0 && q < 4) setc(v, q, fs_(comp(v, q), h ? e4.w : e4.y));
                } else if (j == -2) {
                    // several receivers in the column: its list, in its order
                    const ShotDesc &D = shots[cb + i];
                    const int xr = f + h * W;
                    for (int e = __ldg(D.colptr + xr), e1 = __ldg(D.colptr + xr + 1); e < e1; ++e) {
                        const int2 r = __ldg(D.rec + e);
                        const int q = 2 * (r.x - z0) + h;
                        if (q < 0 || q > 3) continue;
                        const float a = fm(fm(fm(fm(fm(__ldg(s_adj[i] + r.y), __ldg(D.recK + e)), A.dt), A.dt), A.invdx),
                                           A.invdz);
                        setc(v, q, fs_(comp(v, q), a));
                    }
                }
            }
        }
        if (!SPEC || !fs_top || z0 >= pml) store2(o, f, v);
        else store1(o + 2, f, v.z, v.w);  // z0 + 1 == pml: row z0 is a mirrored row
        if (SPEC && fs_top) {
            if (z0 > pml && z0 <= fs_hi) store1(o + 4 * (pml - z0), f, mir.x, mir.y);
            if (z0 + 1 > pml && z0 + 1 <= fs_hi) store1(o + 4 * (pml - z0) - 2, f, mir.z, mir.w);
        }
    };
    auto consume = [&](int i, int st, auto spec, auto accu) {
        const unsigned sb = smem_u32(smem) + (unsigned)(st * stage);
        const unsigned ca = sb + rel, pa = sb + rel0;
        Pair2 x[NCOL + 6];  // columns f0-3 .. f0+3 (+1)
#pragma unroll
        for (int j = 0; j < 7; ++j) x[j] = lds_pair2(ca + (j - 3) * CS);
        column(i, st, std::integral_constant<int, 0>(), spec, accu, x, ca, pa);
        if constexpr (NCOL == 2) {
            x[NCOL + 5] = lds_pair2(ca + 4 * CS);
            column(i, st, std::integral_constant<int, 1>(), spec, accu, x, ca + CS, pa + TZ * 8);
        }
    };

    // the shots of the chunk in order; which parts of the epilogue the loop holds is uniform over the
    // tile
    auto walk = [&](auto spec, auto accu) {
        for (int i = 0, st = 0, ph = 0; i < n; ++i) {
            if (!fold_warp_wait(smem_u32(&full[st]), ph)) {
                if (lane == 0) atomicExch(err, 1);
                break;
            }
            consume(i, st, spec, accu);
            out += shot_stride;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&empty[st]));
            if (++st == NST) st = 0, ph ^= 1;
        }
    };
    const std::true_type yes{};
    const std::false_type no{};
    if (fs_tile || any_spec) {
        if (acc_tile) walk(yes, yes);
        else walk(yes, no);
    } else {
        if (acc_tile) walk(no, yes);
        else walk(no, no);
    }
}

// halves: 2 -- grid row y is 2 * chunk + item half; 1 -- the items' second halves are empty and row
// y is the chunk.  The tensor maps, the group's descriptor and the program item are kernel
// parameters: a block reads nothing from global memory before its copies are on their way.
template <int MATH, int NCOL>
__global__ void __launch_bounds__(32 * (FOLD_WARPS + 1), NCOL == 2 ? 2 : 3)
    k_fold(const __grid_constant__ CUtensorMap tm_p1, const __grid_constant__ CUtensorMap tm_p0,
           const __grid_constant__ ShotDesc A, const FoldTile T, const ShotDesc *__restrict__ shots, const FoldItem item0,
           const FoldItem item1, int L, int shot_base, int nshot, int chunk, int halves, int *err, const TileSync ts)
{
    const bool second = halves == 2 && (blockIdx.y & 1);
    fold_body<MATH, NCOL>(tm_p1, tm_p0, A, T, shots, second ? item1 : item0, L, shot_base, nshot, chunk, err, blockIdx.x,
                    halves == 2 ? blockIdx.y : 2 * blockIdx.y, blockIdx.z, ts);
}

// ------------------------------------------------------------ several groups in one launch
// One shot group of a launch that advances several groups at once -- the windows of a moving spread,
// or the runs of the request loop's batch: what k_fold takes as parameters.  The launch is a flat
// list of blocks, group g owning the blocks from b0[g] in the single-group kernel's order
// (column tile fastest, then chunk and item half, then the z tile: the surface tiles start first).
struct __align__(64) FoldGroup {
    CUtensorMap p1, p0;
    int ntx, rows, halves;  // rows: grid rows y of the group (halves x chunks)
    int L, shot_base, nshot, chunk;
    FoldTile T;
    FoldItem item[2];
    FoldGeo A;
    const ShotDesc *shots;
    TileSync ts;
};
// The table is a kernel parameter (the tensor maps sit in constant space as k_fold's do); a larger
// batch takes several launches.  48 groups are 24.6 of the 32.8 KB that a launch may pass: all that fit
// (62) ran as fast, and the whole table is copied with each launch.
constexpr int FOLD_GROUPS = 48;
struct __align__(64) FoldTable {
    int ngroups, b0[FOLD_GROUPS];  // first blocks
    FoldGroup g[FOLD_GROUPS];
};
static_assert(sizeof(FoldTable) <= 32764 - 16, "kernel parameter limit");

template <int MATH, int NCOL>
__global__ void __launch_bounds__(32 * (FOLD_WARPS + 1), NCOL == 2 ? 2 : 3)
    k_fold_groups(const __grid_constant__ FoldTable tab, int *err)
{
    // the block's group: the last one whose first block is at or before this one, counted 32 at a time
    const int lane = threadIdx.x & 31;
    int g = -1;
    for (int base = 0; base < tab.ngroups; base += 32) {
        const int i = base + lane;
        g += __popc(__ballot_sync(0xffffffffu, i < tab.ngroups && tab.b0[i] <= (int)blockIdx.x));
    }
    g = max(g, 0);
    const FoldGroup &G = tab.g[g];
    const int l = (int)blockIdx.x - tab.b0[g], bx = l % G.ntx, rest = l / G.ntx, row = rest % G.rows, bz = rest / G.rows;
    const int by = G.halves == 2 ? row : 2 * row;
    fold_body<MATH, NCOL>(G.p1, G.p0, G.A, G.T, G.shots, G.item[by & 1], G.L, G.shot_base, G.nshot, G.chunk, err, bx, by,
                          bz, G.ts);
}

}  // namespace fwi
