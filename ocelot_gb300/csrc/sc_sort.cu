// Deterministic NGP charge deposit: stable radix sort of cell keys followed
// by a segmented sum in particle order.
//
// The reference deposits with np.bincount(inds, Q) (ocelot/cpbd/sc.py:193),
// which adds the charges of each cell sequentially in particle order.  Here
// the keys are sorted by a stable least-significant-digit radix sort
// (ceil(key_bits/9) passes of at most 9-bit digits: two passes for a 64^3
// mesh), which puts the particles of each cell
// in a contiguous run in particle order, the charges travelling with the keys;
// each cell's run is then summed by one thread (FP64) or warp (FP32).  In FP64 the sum is
// a sequential fold and reproduces bincount's sums bit for bit; in FP32 it is
// Kahan-compensated.  The result does not
// depend on scheduling, so it is the same alone and in a batch.
//
// Each radix pass is three launches with no inter-block waiting:
//   hist     per-block digit histogram of a tile of 256, 1024 or 4096 keys -> hist[digit][block]
//   rowscan  one warp per digit: exclusive scan along the blocks, digit totals
//   scatter  per block: digit bases from the totals; each warp ranks the equal
//            digits of its 1, 4 or 16 rounds of 32 keys by __match_any_sync and
//            a count row, the warps are joined by a per-digit prefix in shared
//            memory (stable order: warp, round, lane = particle order)
#include <type_traits>

#include "sc_common.cuh"

namespace ocsc {

constexpr int RT = 256;
constexpr int RITEMS = 16;  // rounds of RT keys per block at most (large sorts)
constexpr int RWARPS = RT / 32;
constexpr int RMAXBITS = 9;
constexpr int RBINS = 1 << RMAXBITS;  // 512 digits at most
constexpr unsigned FULLM = 0xffffffffu;

__global__ void __launch_bounds__(RT) k_rhist(const uint32_t* __restrict__ keys, int64_t n, int shift, int bins,
                                              uint32_t* __restrict__ hist, int items) {
    pdl_wait();
    __shared__ uint32_t h[RBINS];
    for (int d = threadIdx.x; d < RBINS; d += RT) h[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * RT * items;
    const uint32_t mask = (uint32_t)bins - 1;
#pragma unroll 4
    for (int it = 0; it < items; ++it) {
        const int64_t i = base + it * RT + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & mask], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < bins; d += RT) hist[(size_t)d * gridDim.x + blockIdx.x] = h[d];
}

__global__ void k_rrowscan(uint32_t* __restrict__ hist, int nblk, int bins, uint32_t* __restrict__ tot) {
    pdl_wait();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= bins) return;
    uint32_t* row = hist + (size_t)warp * nblk;
    uint32_t carry = 0;
    for (int b0 = 0; b0 < nblk; b0 += 32) {
        const int b = b0 + lane;
        const uint32_t v = b < nblk ? row[b] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULLM, incl, o);
            if (lane >= o) incl += t;
        }
        if (b < nblk) row[b] = carry + incl - v;
        carry += __shfl_sync(FULLM, incl, 31);
    }
    if (lane == 0) tot[warp] = carry;
}

// Stable scatter of a block's RT * ITEMS keys, warp w the ITEMS rounds of 32 keys
// from w * 32 * ITEMS on.  A warp ranks its keys alone, round after round, in
// its own row of digit counts (the lanes of one digit found by a match, one of
// them adds for all); then one scan over the warps' rows, and every key
// knows its place.  Bound by latency: three barriers a block and the loads at
// its start, all issued before the first of them.  (Rounds of RT keys with a
// clear and a scan of the 512-digit table behind four barriers each, and the digit
// bases scanned by one warp in 16 dependent steps, took 45 and 71 us for the two
// passes of 2M keys, 13 a pass of 200k and 6.3 of 10k; this 42 and 60, 8 and 4;
// with the charges travelling and STAGE 38 and 30, 7.3 and 3.2.)
//
// V: what travels with the keys -- the particle index (a sort's permutation) or, for
// the deposit, the charge itself from the first pass on, read and written in
// order (the last pass used to gather it by index: 2M random 8-byte reads).
// vin == nullptr (the first pass): the index, or the charge qsrc[i].
// STAGE: the keys and values are put in digit order in shared memory first and
// leave in runs, eight of a digit in a tile of 4096; written where each thread
// has them, every 4 bytes are a sector of their own.
template <int ITEMS, typename V>
__global__ void __launch_bounds__(RT) k_rscatter(const uint32_t* __restrict__ kin, const V* __restrict__ vin,
                                                 const double* __restrict__ qsrc, int64_t n, int shift, int bins,
                                                 const uint32_t* __restrict__ hist, const uint32_t* __restrict__ tot,
                                                 uint32_t* __restrict__ kout, V* __restrict__ vout) {
    pdl_wait();
    static_assert(RBINS == 2 * RT, "two digits per thread");
    constexpr bool STAGE = ITEMS >= 16;
    constexpr size_t WC = sizeof(uint32_t) * RWARPS * RBINS, ST = STAGE ? RT * ITEMS * sizeof(V) : 0;
    __shared__ uint32_t base[RBINS];
    __shared__ __align__(16) unsigned char raw[WC > ST ? WC : ST];
    __shared__ uint32_t wtot[RWARPS];
    uint32_t(*wc)[RBINS] = reinterpret_cast<uint32_t(*)[RBINS]>(raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * RT * ITEMS + warp * 32 * ITEMS + lane;
    const uint32_t mask = (uint32_t)bins - 1;
    uint32_t key[ITEMS], rk[ITEMS];
    V val[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int64_t i = i0 + 32 * r;
        key[r] = i < n ? kin[i] : 0u;
        if (i >= n) val[r] = V(0);
        else if (vin) val[r] = vin[i];
        else if constexpr (std::is_same<V, uint32_t>::value) val[r] = (V)i;
        else val[r] = (V)qsrc[i];
    }
    // exclusive scan of the digit totals plus this block's offset within each
    // digit -> where the block's keys of a digit go
    const int d0 = 2 * tid;
    const uint32_t t0 = d0 < bins ? tot[d0] : 0u, t1 = d0 + 1 < bins ? tot[d0 + 1] : 0u;
    const uint32_t h0 = d0 < bins ? hist[(size_t)d0 * gridDim.x + blockIdx.x] : 0u;
    const uint32_t h1 = d0 + 1 < bins ? hist[(size_t)(d0 + 1) * gridDim.x + blockIdx.x] : 0u;
#pragma unroll
    for (int w = 0; w < RWARPS; ++w) wc[w][tid] = wc[w][tid + RT] = 0u;
    uint32_t inc = t0 + t1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULLM, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wtot[warp] = inc;
    __syncthreads();
    uint32_t before = inc - t0 - t1;
    for (int w = 0; w < warp; ++w) before += wtot[w];
    base[d0] = before + h0;
    base[d0 + 1] = before + t0 + h1;
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool valid = i0 + 32 * r < n;
        const uint32_t d = valid ? ((key[r] >> shift) & mask) : (uint32_t)RBINS;
        const uint32_t peers = __match_any_sync(FULLM, d);
        const uint32_t rank = __popc(peers & lt);
        uint32_t old = 0u;
        if (valid && rank == 0) {
            old = wc[warp][d];
            wc[warp][d] = old + __popc(peers);
        }
        rk[r] = rank + __shfl_sync(FULLM, old, __ffs(peers) - 1);
        __syncwarp();
    }
    __syncthreads();
    uint32_t cnt[2];  // the block's keys of this thread's two digits
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        uint32_t run = STAGE ? 0u : base[d0 + j];
#pragma unroll
        for (int w = 0; w < RWARPS; ++w) {
            const uint32_t c = wc[w][d0 + j];
            wc[w][d0 + j] = run;
            run += c;
        }
        cnt[j] = run;
    }
    if constexpr (STAGE) {  // digit starts within the tile
        uint32_t in = cnt[0] + cnt[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULLM, in, o);
            if (lane >= o) in += t;
        }
        if (lane == 31) wtot[warp] = in;
        __syncthreads();
        uint32_t start = in - cnt[0] - cnt[1];
        for (int w = 0; w < warp; ++w) start += wtot[w];
#pragma unroll
        for (int w = 0; w < RWARPS; ++w) {
            wc[w][d0] += start;
            wc[w][d0 + 1] += start + cnt[0];
        }
        base[d0] -= start;  // + the place in the tile: the place in the output (mod 2^32)
        base[d0 + 1] -= start + cnt[0];
    }
    __syncthreads();
    if constexpr (STAGE) {
        const int64_t left = n - (int64_t)blockIdx.x * RT * ITEMS;
        const int m = left < RT * ITEMS ? (int)left : RT * ITEMS;
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) rk[r] += wc[warp][(key[r] >> shift) & mask];
        __syncthreads();  // the counts are done with
        uint32_t* sk = reinterpret_cast<uint32_t*>(raw);
        V* sv = reinterpret_cast<V*>(raw);
#pragma unroll
        for (int r = 0; r < ITEMS; ++r)
            if (i0 + 32 * r < n) sk[rk[r]] = key[r];
        __syncthreads();
        uint32_t pos[ITEMS];
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int j = r * RT + tid;
            if (j >= m) continue;
            const uint32_t kk = sk[j];
            pos[r] = base[(kk >> shift) & mask] + (uint32_t)j;
            kout[pos[r]] = kk;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r)
            if (i0 + 32 * r < n) sv[rk[r]] = val[r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r)
            if (r * RT + tid < m) vout[pos[r]] = sv[r * RT + tid];
    } else {
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            if (i0 + 32 * r >= n) continue;
            const uint32_t pos = wc[warp][(key[r] >> shift) & mask] + rk[r];
            kout[pos] = key[r];
            vout[pos] = val[r];
        }
    }
}

// Rounds of RT keys per block: small sorts take one or four (more blocks in
// parallel), large ones 16 (fewer digit-table rows for the scans, and runs that leave
// in order).  The stable order, and so the result, does not depend on the tiling.
// Both passes of a deposit's sort on 63^3 (us) with 1 / 4 / 16 rounds: 32k keys
// 17.6 / 19.8 / 34.6, 64k 21.3 / 22.1 / 36.4, 128k 27.6 / 24.1 / 38.0, 256k 41.8 /
// 27.3 / 39.6, 512k 71.8 / 41.6 / 39.1, 1M 126 / 70 / 56, 2M 233 / 114 / 86.
static int sort_items(int64_t n) { return n <= (1 << 16) ? 1 : (n <= (1 << 19) ? 4 : RITEMS); }
int sort_blocks(int64_t n) {
    const int64_t t = (int64_t)RT * sort_items(n);
    return (int)((n + t - 1) / t);
}

// the kernels of a plan's deposit (none without the sorted one)
cudaError_t prepare_sort_kernels(const Plan& p) {
    if (!p.sorted_deposit) return cudaSuccess;
    cudaError_t e;
    if ((e = prefer_shared(k_rhist))) return e;
    if ((e = prefer_shared(k_rrowscan))) return e;
    auto all = [&](auto v) -> cudaError_t {
        using V = decltype(v);
        if ((e = prefer_shared(k_rscatter<1, V>))) return e;
        if ((e = prefer_shared(k_rscatter<4, V>))) return e;
        return prefer_shared(k_rscatter<RITEMS, V>);
    };
    return p.prec == SC_FP64 ? all(0.0) : all(0.0f);
}

int sort_passes(int key_bits) { return key_bits <= 0 ? 1 : (key_bits + RMAXBITS - 1) / RMAXBITS; }

size_t sort_scratch_bytes(int64_t n, int key_bits) {
    (void)key_bits;
    const size_t nb = (size_t)(sort_blocks(n) > 0 ? sort_blocks(n) : 1);
    return align_up(4 * (size_t)n) * 2 + align_up((size_t)RBINS * nb * 4) + align_up((size_t)RBINS * 4);
}

template <typename V>
static cudaError_t sort_t(const uint32_t* keys_in, int64_t n, int key_bits, uint32_t* keys_out, V* vals_out,
                          uint32_t* tmp_k, V* tmp_v, uint32_t* hist, uint32_t* tot, cudaStream_t s, const double* q_src) {
    if (n <= 0) return cudaSuccess;
    const int nb = sort_blocks(n), items = sort_items(n);
    const int passes = sort_passes(key_bits);
    const int width = key_bits <= 0 ? 1 : (key_bits + passes - 1) / passes;  // <= RMAXBITS
    const uint32_t* sk = keys_in;
    const V* sv = nullptr;
    bool to_out = (passes % 2) == 1;
    for (int p = 0; p < passes; ++p) {
        const int shift = width * p;
        int dbits = key_bits - shift;
        dbits = dbits > width ? width : (dbits < 1 ? 1 : dbits);
        const int bins = 1 << dbits;
        uint32_t* dk = to_out ? keys_out : tmp_k;
        V* dv = to_out ? vals_out : tmp_v;
        launch(k_rhist, nb, RT, 0, s, sk, n, shift, bins, hist, items);
        launch(k_rrowscan, (bins * 32 + 255) / 256, 256, 0, s, hist, nb, bins, tot);
        auto* scatter = items == 1 ? k_rscatter<1, V> : (items == 4 ? k_rscatter<4, V> : k_rscatter<RITEMS, V>);
        launch(scatter, nb, RT, 0, s, sk, sv, q_src, n, shift, bins, hist, tot, dk, dv);
        sk = dk;
        sv = dv;
        to_out = !to_out;
    }
    return cudaGetLastError();
}

cudaError_t launch_sort(const uint32_t* keys_in, int64_t n, int key_bits, uint32_t* keys_out, uint32_t* perm_out,
                        uint32_t* tmp_k, uint32_t* tmp_v, uint32_t* hist, uint32_t* tot, cudaStream_t s) {
    return sort_t<uint32_t>(keys_in, n, key_bits, keys_out, perm_out, tmp_k, tmp_v, hist, tot, s, nullptr);
}

cudaError_t launch_charge_sort(const Plan& p, const Layout& L, char* ws, const double* q, int64_t n, cudaStream_t s) {
    auto u32 = [&](size_t o) { return reinterpret_cast<uint32_t*>(ws + o); };
    auto run = [&](auto v) {
        using V = decltype(v);
        return sort_t<V>(u32(L.keys), n, p.key_bits, u32(L.sort_keys), reinterpret_cast<V*>(ws + L.sort_q),
                         u32(L.sort_tmp_k), reinterpret_cast<V*>(ws + L.sort_tmp_q), u32(L.sort_hist), u32(L.sort_tot), s, q);
    };
    return p.prec == SC_FP64 ? run(0.0) : run(0.0f);
}

// Cell bounds of the sorted runs: start[key] and end[key] (both 0 for an
// empty cell, from a memset).
__global__ void k_cell_bounds(const uint32_t* __restrict__ sk, int64_t n, uint32_t* __restrict__ start,
                              uint32_t* __restrict__ end, const ScState* st) {
    pdl_wait();
    if (st->status) return;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t key = sk[j];
        if (j == 0 || sk[j - 1] != key) start[key] = (uint32_t)j;
        if (j == n - 1 || sk[j + 1] != key) end[key] = (uint32_t)(j + 1);
    }
}

// The cell's run of charges, which the last radix pass carried into sorted
// (cell, particle) order, summed into the cell.  FP64: one thread per cell, a
// strictly sequential left fold in particle order from 0 -- np.bincount's
// summation (sc.py:193), bit for bit.  (One warp per cell with every lane
// folding the same shuffled values spent 32 lanes of this GPU's narrow FP64
// pipe per addition: 370 us per 2M particles.)  Bound by the fullest cells, some 500
// dependent additions and their loads: 16 loads at a time instead of 4 take 56 -> 44 us
// at 2M / 64^3; loads kept ahead of the additions with predicated tails cost the
// many short cells more than that.  FP32: one warp per cell,
// lane-strided Kahan sums combined by a fixed shuffle tree with error-free
// (two-sum) additions.  Empty cells get 0, so no memset of the grid.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

template <typename R>
__global__ void __launch_bounds__(256) k_deposit_cells(const R* __restrict__ sq, const uint32_t* __restrict__ start,
                                                       const uint32_t* __restrict__ end, int64_t ncell,
                                                       R* __restrict__ qgrid, const ScState* st) {
    pdl_wait();
    if (st->status) return;
    if constexpr (sizeof(R) == 8) {
        const int64_t nt = (int64_t)gridDim.x * blockDim.x;
        for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncell; c += nt) {
            const uint32_t b = start[c], e = end[c];
            double sum = 0.0;
            uint32_t k = b;
            for (; k + 16 <= e; k += 16) {  // 16 loads in flight, the additions in order
                double v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = sq[k + u];
#pragma unroll
                for (int u = 0; u < 16; ++u) sum = __dadd_rn(sum, v[u]);
            }
            for (; k + 4 <= e; k += 4) {
                const double v0 = sq[k], v1 = sq[k + 1], v2 = sq[k + 2], v3 = sq[k + 3];
                sum = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(sum, v0), v1), v2), v3);
            }
            for (; k < e; ++k) sum = __dadd_rn(sum, (double)sq[k]);
            qgrid[c] = (R)sum;
        }
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c = w0; c < ncell; c += nw) {
        const uint32_t b = start[c], e = end[c];
        {
            float sum = 0.f, comp = 0.f;
            for (uint32_t k = b + lane; k < e; k += 32) {
                const float y = __fsub_rn((float)sq[k], comp);
                const float t = __fadd_rn(sum, y);
                comp = __fsub_rn(__fsub_rn(t, sum), y);
                sum = t;
            }
            float err = -comp;
            for (int o = 16; o; o >>= 1) {
                const float s2 = __shfl_down_sync(0xffffffffu, sum, o);
                const float e2 = __shfl_down_sync(0xffffffffu, err, o);
                float ns, ne;
                two_sum(sum, s2, ns, ne);
                sum = ns;
                err = __fadd_rn(__fadd_rn(err, e2), ne);
            }
            if (lane == 0) qgrid[c] = (R)__fadd_rn(sum, err);
        }
    }
}

cudaError_t launch_deposit(const Plan& p, const Layout& L, char* ws, const double* q, int64_t n, cudaStream_t s) {
    (void)q;
    const ScState* st = reinterpret_cast<const ScState*>(ws + L.state);
    const int64_t ncell = (int64_t)p.nx * p.ny * p.nz;
    cudaError_t e = cudaMemsetAsync(ws + L.cell_start, 0, 2 * align_up(4 * (size_t)ncell), s);
    if (e) return e;
    int64_t b = (n + 255) / 256;
    if (b > (int64_t)p.sm_count * 8) b = (int64_t)p.sm_count * 8;
    if (b < 1) b = 1;
    const uint32_t* sk = reinterpret_cast<const uint32_t*>(ws + L.sort_keys);
    uint32_t* cs = reinterpret_cast<uint32_t*>(ws + L.cell_start);
    uint32_t* ce = reinterpret_cast<uint32_t*>(ws + L.cell_end);
    launch(k_cell_bounds, (int)b, 256, 0, s, sk, n, cs, ce, st);
    const int cb = p.prec == SC_FP64 ? (int)((ncell + 255) / 256 < (int64_t)p.sm_count * 16 ? (ncell + 255) / 256
                                                                                            : (int64_t)p.sm_count * 16)
                                     : p.sm_count * 8;
    if (p.prec == SC_FP64)
        launch(k_deposit_cells<double>, cb, 256, 0, s, reinterpret_cast<const double*>(ws + L.sort_q), cs, ce, ncell,
                                                   reinterpret_cast<double*>(ws + L.qgrid), st);
    else
        launch(k_deposit_cells<float>, cb, 256, 0, s, reinterpret_cast<const float*>(ws + L.sort_q), cs, ce, ncell,
                                                  reinterpret_cast<float*>(ws + L.qgrid), st);
    return cudaGetLastError();
}

}  // namespace ocsc
