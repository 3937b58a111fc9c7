// grow.cuh -- growth of the rows that a batch's insertions overflow, on the device.
//
// k_append lists the insertions that found their row full (ovf), and with the first of them the row
// itself, cut into chunks of kGrowChunk slots.  k_update then starts with the growth.  A row makes
// room in the cheapest way that leaves an eighth of its live entries (at least one slot) free
// behind the overflow: its unsorted tail alone gives up its tombstones (links that come and go live
// there; the sorted prefix keeps its own, as after any deletion); else all live entries close up
// in place, in their order, so the prefix stays sorted; else they move to a region of
// 2 * (live + overflow) + slack_min slots from the spare region (a bump allocator).  In place goes
// through scratch slots at the free end of the spare region.  Every moved entry leaves its final
// slot in its old twin word, through which its partner and the batch's recorded slots find it.
// The phases before the last write only free slots, twin words and the work arrays: until the last
// one (grow_finish) the rows stand as k_append left them, and grow_finish may be run again.
//
// Bound: random sectors (a moved entry reads its partner's place and writes its partner's twin
// word) for many entries, a chain of dependent accesses and a barrier per phase for few.  A warp
// per chunk, not per row: rows of 10^5 entries grow in a stream on a skewed graph, and a warp that
// walked one alone took up to 2 ms.  Inside k_update, not as kernels with the host between them
// (status read, eight launches, three synchronisations).  The tail alone where that does: a batch of a
// stream on a skewed graph otherwise moved a sixteenth of the adjacency.  k_update, growth included:
// 10,000 vertices and 1,000 changes 0.28 -> 0.20 ms (the batch), 300,000 and 12,345 changes 0.36 ->
// 0.28 ms, RMAT scale 20 with 10^5 insertions 0.31 -> 0.20 (all live entries) -> 0.15 ms, RMAT scale
// 22 and 10^6 changes, of which the growth 1.16 -> 0.22 and 0.52 -> 0.17 and 0.10 ms (a batch and
// its inverse).  A handful of chunks is one CTA's work with block barriers: the grid's cost more.  Three
// grid barriers where rows are of one chunk (five with the move and the overflowed ends in phases of
// their own): 300,000 vertices k_update 0.205 -> 0.194 ms.
#pragma once

// Chunks a row of `cap` slots is cut into (at least one: a row without slots grows too).
__device__ __forceinline__ unsigned grow_chunks(int cap) {
    return cap > 0 ? ((unsigned)cap + kGrowChunk - 1) / kGrowChunk : 1u;
}

// k_append: lists row r, entry j of the grow list, with its chunks from c0 on.
__device__ __forceinline__ void grow_list_row(const UpdParams& p, unsigned j, unsigned c0, int r, unsigned chunks) {
    p.grow.row[j] = (unsigned)r;
    p.grow.chunk0[j] = c0;
    p.grow.done[j] = 0;
    p.grow.gidx[r] = (int)j + 1;
    for (unsigned q = 0; q < chunks; q++) p.grow.chunk_row[c0 + q] = j;
}

// k_append, warp-collective: lists the ends of record i (c) that found their rows (rx, ry) full
// (ovx, ovy; px, py are the positions they were given), with one atomic per warp and list, and
// the record's slots (ax, ay), -1 - k for the k-th overflowed end of its row.
__device__ __forceinline__ void list_overflow(const UpdParams& p, long long i, const int4& c, const RowDesc& rx,
                                              const RowDesc& ry, int px, int py, bool ovx, bool ovy, long long ax,
                                              long long ay) {
    const unsigned lane = lane_id(), lt = (1u << lane) - 1u;
    const unsigned mx = __ballot_sync(kFull, ovx), my = __ballot_sync(kFull, ovy);
    if ((mx | my) == 0) return;
    unsigned base = 0;
    if (lane == 0) base = (unsigned)atomicAdd(&p.g.ctl->ovf_count, __popc(mx) + __popc(my));
    base = __shfl_sync(kFull, base, 0);
    if (ovx) p.ovf[base + __popc(mx & lt)] = make_int4(c.x, c.y, c.z, (int)(2 * i));
    if (ovy) p.ovf[base + __popc(mx) + __popc(my & lt)] = make_int4(c.y, c.x, c.z, (int)(2 * i + 1));
    if (ovx || ovy) {
        p.slot[2 * i] = ovx ? -1ll - (px - rx.cap) : ax;
        p.slot[2 * i + 1] = ovy ? -1ll - (py - ry.cap) : ay;
    }
    const bool fx = ovx && px == rx.cap, fy = ovy && py == ry.cap;  // the first of its row
    if (!__any_sync(kFull, fx || fy)) return;
    const unsigned nx = fx ? grow_chunks(rx.cap) : 0u, ny = fy ? grow_chunks(ry.cap) : 0u;
    const unsigned nr = (fx ? 1u : 0u) + (fy ? 1u : 0u);
    const unsigned ir = warp_incl_scan(nr), ic = warp_incl_scan(nx + ny);
    unsigned long long at = 0;
    if (lane == 31) at = atomicAdd(&p.g.ctl->grow_list, ((unsigned long long)ic << 32) | ir);
    at = __shfl_sync(kFull, at, 31);
    unsigned j = (unsigned)at + ir - nr, ch = (unsigned)(at >> 32) + ic - (nx + ny);
    if (fx) {
        grow_list_row(p, j, ch, c.x, nx);
        j++;
        ch += nx;
    }
    if (fy) grow_list_row(p, j, ch, c.y, ny);
}

// Everything a growth phase reads may have been written in this kernel by another SM, and the
// rows it reads are written by the last one: all through the L2.
__device__ __forceinline__ RowDesc ld_row(const RowDesc* r) {
    const uint4 x = __ldcg(reinterpret_cast<const uint4*>(r));
    return RowDesc{(long long)(((unsigned long long)x.y << 32) | x.x), (int)x.z, (int)x.w};
}

// The threads that take part in a growth: the grid, or one CTA of it.
struct GrowTeam {
    unsigned thread, threads;
    __device__ __forceinline__ unsigned warp() const { return thread >> 5; }
    __device__ __forceinline__ unsigned warps() const { return threads >> 5; }
};

// The live entries of a chunk (slots [lo, hi) of the row at `start`) to dst, with a forwarding pointer
// (their place from fin on) in each one's old twin word.  Warp-collective.
__device__ __forceinline__ void grow_out_chunk(const UpdParams& p, long long start, int lo, int hi, long long dst,
                                               long long fin) {
    const unsigned lane = lane_id(), lt = (1u << lane) - 1u;
    int idx = 0;
    for (int b = lo; b < hi; b += 128) {
        int2 x[4];
        unsigned tw[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int e = b + 32 * k + (int)lane;
            x[k] = e < hi ? __ldcg(&p.g.adj[start + e]) : make_int2(0, -1);
            tw[k] = p.g.twin && e < hi ? __ldcg(&p.g.twin[start + e]) : kNoTwin;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool live = x[k].y >= 0;
            const unsigned m = __ballot_sync(kFull, live);
            if (live) {
                const int at = idx + __popc(m & lt);
                p.g.adj[dst + at] = x[k];
                if (p.g.twin) {
                    p.g.twin[dst + at] = tw[k];  // the partner's old slot, re-linked by the next phase
                    p.g.twin[start + b + 32 * k + (int)lane] = (unsigned)(fin + at);
                }
            }
            idx += __popc(m);
        }
    }
}

// Phase 1: live entries of every chunk (and those of the prefix); the warp that counts a row's last
// chunk decides what moves and where, and ranks it.  A row of one chunk moves at once, if its slots
// lie in the spare region (whether all do is known after the phase; what it writes is free until
// then).
__device__ void grow_plan(const UpdParams& p, const GrowTeam& t, unsigned chunks) {
    const DevGrow& q = p.grow;
    const unsigned lane = lane_id();
    unsigned dropped = 0;
    for (unsigned c = t.warp(); c < chunks; c += t.warps()) {
        const unsigned j = __ldcg(&q.chunk_row[c]);
        const unsigned r = __ldcg(&q.row[j]), c0 = __ldcg(&q.chunk0[j]);
        const RowDesc rd = ld_row(&p.g.rows[r]);
        const int sl = __ldcg(&p.g.sorted_len[r]);
        const int lo = (int)(c - c0) * kGrowChunk, hi = min(lo + kGrowChunk, rd.cap);
        unsigned n = 0, ns = 0;
#pragma unroll
        for (int k = 0; k < kGrowChunk / 32; k++) {
            const int e = lo + 32 * k + (int)lane;
            const bool live = e < hi && __ldcg(&p.g.adj[rd.start + e].y) >= 0;
            n += live ? 1u : 0u;
            ns += live && e < sl ? 1u : 0u;
        }
        n = __reduce_add_sync(kFull, n);
        ns = __reduce_add_sync(kFull, ns);
        const unsigned parts = grow_chunks(rd.cap);
        unsigned total = n, sorted = ns;
        if (parts > 1) {
            unsigned d = 0;
            if (lane == 0) {
                q.chunk_live[c] = (int)(n | ns << 16);
                __threadfence();
                d = atomicAdd(&q.done[j], 1u);
            }
            if (__shfl_sync(kFull, d, 0) != parts - 1) continue;
            __threadfence();
            total = sorted = 0;
            for (unsigned b = lane; b < parts; b += 32) {
                const unsigned x = (unsigned)__ldcg(&q.chunk_live[c0 + b]);
                total += x & 0xFFFFu;
                sorted += x >> 16;
            }
            total = __reduce_add_sync(kFull, total);
            sorted = __reduce_add_sync(kFull, sorted);
        }
        const long long need = rd.deg - rd.cap;
        const long long room = total / 8 > 1 ? total / 8 : 1;  // free slots left in place
        const bool tail = sl + (long long)(total - sorted) + need + room <= rd.cap;
        const long long live = tail ? total - sorted : total;  // the entries that move
        if (parts == 1) {
            if (lane == 0) {
                q.chunk_live[c] = (int)live;
                q.chunk_off[c] = 0;
            }
        } else {  // the chunks' shares of them, ranked
            unsigned before = 0;
            for (unsigned b = 0; b < parts; b += 32) {
                const bool has = b + lane < parts;
                const unsigned x = has ? (unsigned)__ldcg(&q.chunk_live[c0 + b + lane]) : 0u;
                const unsigned mine = (x & 0xFFFFu) - (tail ? x >> 16 : 0u);
                const unsigned incl = warp_incl_scan(mine);
                if (has) {
                    q.chunk_live[c0 + b + lane] = (int)mine;
                    q.chunk_off[c0 + b + lane] = (int)(before + incl - mine);
                }
                before += __shfl_sync(kFull, incl, 31);
            }
        }
        const int first = tail ? sl : 0;  // entries from here on move
        long long fin = rd.start + first, scr = -1;
        if (lane == 0) {
            q.first[j] = first;
            q.live[j] = (int)live;
            q.lsorted[j] = tail ? sl : (int)sorted;
            q.ndeg[j] = (int)(first + live + need);
            dropped += (unsigned)(rd.cap - first - live);
            long long nc = rd.cap;
            if (tail || live + need + room <= rd.cap) {
                const unsigned long long at = atomicAdd(&p.g.ctl->scr_used, (unsigned long long)live);
                scr = (long long)(__ldcg(&q.spare[1]) - at - (unsigned long long)live);  // checked by grow()
            } else {
                nc = 2 * (live + need) + q.slack_min;
                if (nc > 0x7FFFFFFFLL) atomicExch(&p.g.ctl->grow_fail, 1u);
                fin = (long long)atomicAdd(&q.spare[0], (unsigned long long)nc);
            }
            q.fin[j] = fin;
            q.scr[j] = scr;
            q.ncap[j] = (int)(nc > 0x7FFFFFFFLL ? 0x7FFFFFFFLL : nc);
        }
        if (parts > 1) continue;
        fin = __shfl_sync(kFull, fin, 0);
        scr = __shfl_sync(kFull, scr, 0);
        const long long dst = scr != -1 ? scr : fin;
        if (dst >= (long long)q.spare_from && dst + live <= (long long)__ldcg(&q.spare[1]))
            grow_out_chunk(p, rd.start, first, rd.cap, dst, fin);
    }
    if (lane == 0 && dropped) atomicAdd(&p.g.ctl->grow_dropped, (unsigned long long)dropped);
}

// Phase 2 (rows of several chunks): the live entries to where their row goes (or its scratch).
__device__ void grow_out(const UpdParams& p, const GrowTeam& t, unsigned chunks) {
    const DevGrow& q = p.grow;
    for (unsigned c = t.warp(); c < chunks; c += t.warps()) {
        const unsigned j = __ldcg(&q.chunk_row[c]);
        const RowDesc rd = ld_row(&p.g.rows[__ldcg(&q.row[j])]);
        if (grow_chunks(rd.cap) == 1) continue;  // moved by phase 1
        const int c0 = (int)(c - __ldcg(&q.chunk0[j])) * kGrowChunk, hi = min(c0 + kGrowChunk, rd.cap);
        const int lo = max(c0, __ldcg(&q.first[j]));
        const long long off = __ldcg(&q.chunk_off[c]), fin = __ldcg(&q.fin[j]) + off, scr = __ldcg(&q.scr[j]);
        grow_out_chunk(p, rd.start, lo, hi, scr >= 0 ? scr + off : fin, fin);
    }
}

// Phase 3: every moved entry takes its partner's final slot, from the partner's forwarding pointer
// when the partner moves too (its row grows, and not by its tail alone with the partner in the
// prefix); else the partner stays and gets this entry's final slot.
__device__ void grow_relink(const UpdParams& p, const GrowTeam& t, unsigned chunks) {
    const DevGrow& q = p.grow;
    const unsigned lane = lane_id();
    for (unsigned c = t.warp(); c < chunks; c += t.warps()) {
        const unsigned j = __ldcg(&q.chunk_row[c]);
        const int live = __ldcg(&q.chunk_live[c]);
        const long long off = __ldcg(&q.chunk_off[c]), fin = __ldcg(&q.fin[j]) + off, scr = __ldcg(&q.scr[j]);
        const long long at0 = scr >= 0 ? scr + off : fin;
        for (int b = 0; b < live; b += 128) {
            unsigned tw[4];
            int gi[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int e = b + 32 * k + (int)lane;
                tw[k] = e < live ? __ldcg(&p.g.twin[at0 + e]) : kNoTwin;
                gi[k] = e < live ? __ldcg(&q.gidx[__ldcg(&p.g.adj[at0 + e].x)]) : 0;
                if (gi[k] && __ldcg(&q.first[gi[k] - 1]) > 0 && (long long)tw[k] < __ldcg(&q.fin[gi[k] - 1])) gi[k] = 0;
                if (tw[k] != kNoTwin && (long long)tw[k] >= p.g.cap_total) {  // internal error: report, skip
                    set_status(p.g.ctl, -4);
                    tw[k] = kNoTwin;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int e = b + 32 * k + (int)lane;
                if (tw[k] == kNoTwin) continue;
                if (gi[k]) p.g.twin[at0 + e] = __ldcg(&p.g.twin[tw[k]]);
                else p.g.twin[tw[k]] = (unsigned)(fin + e);
            }
        }
    }
}

// Beside it: the final slots of every overflowed end and of its partner.
__device__ void grow_place(const UpdParams& p, const GrowTeam& t, unsigned novf) {
    const DevGrow& q = p.grow;
    for (unsigned o = t.thread; o < novf; o += t.threads) {
        const int4 x = __ldcg(&p.ovf[o]);  // row, column, weight, 2 * record + side
        const unsigned s = (unsigned)x.w;
        const long long raw = __ldcg(&p.slot[s]), praw = __ldcg(&p.slot[s ^ 1u]);
        const int j = __ldcg(&q.gidx[x.x]) - 1, pj = __ldcg(&q.gidx[x.y]) - 1;
        if (j < 0 || raw >= 0 || (praw < 0 && pj < 0)) {  // internal error: report, skip (the row is listed)
            set_status(p.g.ctl, -4);
            q.place[o] = make_uint2(kNoTwin, kNoTwin);
            continue;
        }
        const long long own = __ldcg(&q.fin[j]) + __ldcg(&q.live[j]) + (-1 - raw);
        if (!p.g.twin) {
            q.place[o] = make_uint2((unsigned)own, (unsigned)((unsigned long long)own >> 32));
            continue;
        }
        long long partner = praw;  // it fitted: where it is, or where its row's growth puts it
        if (praw < 0) partner = __ldcg(&q.fin[pj]) + __ldcg(&q.live[pj]) + (-1 - praw);
        else if (pj >= 0) partner = __ldcg(&p.g.twin[praw]);
        q.place[o] = make_uint2((unsigned)own, (unsigned)partner);
    }
}

// Phase 4: compacted rows back from their scratch, the overflowed ends behind the live entries with
// their partners told (whose twin words say kNoTwin until then), the new descriptors.  Reads only what the phases before it wrote, so it may run again.
__device__ void grow_finish(const UpdParams& p, const GrowTeam& t, unsigned rows, unsigned chunks, unsigned novf) {
    const DevGrow& q = p.grow;
    const unsigned lane = lane_id();
    for (unsigned c = t.warp(); c < chunks; c += t.warps()) {
        const unsigned j = __ldcg(&q.chunk_row[c]);
        const long long off = __ldcg(&q.chunk_off[c]), fin = __ldcg(&q.fin[j]) + off, scr = __ldcg(&q.scr[j]);
        if (scr < 0) continue;
        const int live = __ldcg(&q.chunk_live[c]);
        for (int e = (int)lane; e < live; e += 32) {
            p.g.adj[fin + e] = __ldcg(&p.g.adj[scr + off + e]);
            if (!p.g.twin) continue;
            const unsigned tw = __ldcg(&p.g.twin[scr + off + e]);
            if (tw != kNoTwin) p.g.twin[fin + e] = tw;  // else told below
        }
    }
    for (unsigned o = t.thread; o < novf; o += t.threads) {
        const int4 x = __ldcg(&p.ovf[o]);
        const uint2 s = __ldcg(&q.place[o]);
        const long long own = p.g.twin ? (long long)s.x : (long long)(((unsigned long long)s.y << 32) | s.x);
        if (own >= p.g.cap_total) continue;  // reported by grow_place
        p.g.adj[own] = make_int2(x.y, x.z);
        if (!p.g.twin || (long long)s.y >= p.g.cap_total) continue;
        p.g.twin[own] = s.y;
        p.g.twin[s.y] = s.x;
    }
    for (unsigned j = t.thread; j < rows; j += t.threads) {
        const unsigned r = __ldcg(&q.row[j]);
        RowDesc nr;
        nr.start = __ldcg(&q.fin[j]) - __ldcg(&q.first[j]);
        nr.deg = __ldcg(&q.ndeg[j]);
        nr.cap = __ldcg(&q.ncap[j]);
        p.g.rows[r] = nr;
        p.g.sorted_len[r] = __ldcg(&q.lsorted[j]);
        q.gidx[r] = 0;
    }
}

// If the spare region cannot take the moves and the scratch, only slots that were free before the
// batch have been written: the host repacks (which folds the overflow list in).
__device__ __forceinline__ bool grow_fits(const UpdParams& p) {
    return __ldcg(&p.g.ctl->grow_fail) == 0 &&
           __ldcg(&p.grow.spare[0]) + __ldcg(&p.g.ctl->scr_used) <= __ldcg(&p.grow.spare[1]);
}

__device__ __forceinline__ void grow_give_up(const UpdParams& p, const GrowTeam& t, unsigned rows) {
    for (unsigned j = t.thread; j < rows; j += t.threads) p.grow.gidx[__ldcg(&p.grow.row[j])] = 0;
    if (t.thread == 0) set_status(p.g.ctl, kStatusOverflowPending);
}

// The whole growth (grid-wide).  Returns false when the kernel must stop.
__device__ __noinline__ bool grow(const UpdParams& p) {
    Ctl* const ctl = p.g.ctl;
    const unsigned novf = (unsigned)__ldcg(&ctl->ovf_count);
    const unsigned long long list = __ldcg(&ctl->grow_list);
    const unsigned rows = (unsigned)list, chunks = (unsigned)(list >> 32);
    if (chunks <= blockDim.x >> 5 && novf <= blockDim.x) {  // one CTA, a chunk a warp
        if (blockIdx.x == 0) {
            const GrowTeam t{threadIdx.x, blockDim.x};
            grow_plan(p, t, chunks);
            __threadfence();
            __syncthreads();
            if (grow_fits(p)) {
                if (chunks != rows) grow_out(p, t, chunks);
                __threadfence();
                __syncthreads();
                if (p.g.twin) grow_relink(p, t, chunks);
                grow_place(p, t, novf);
                __threadfence();
                __syncthreads();
                if (threadIdx.x == 0) {
                    ctl->spare_top = __ldcg(&p.grow.spare[0]);
                    ctl->grow_done = gridDim.x;
                }
                grow_finish(p, t, rows, chunks, novf);
            } else {
                grow_give_up(p, t, rows);
            }
        }
        return grid_sync(ctl);
    }
    const GrowTeam t{blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x};
    grow_plan(p, t, chunks);
    if (!grid_sync(ctl)) return false;
    if (!grow_fits(p)) {
        grow_give_up(p, t, rows);
        return false;
    }
    if (chunks != rows) {  // some row has several
        grow_out(p, t, chunks);
        if (!grid_sync(ctl)) return false;
    }
    if (p.g.twin) grow_relink(p, t, chunks);
    grow_place(p, t, novf);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (blockIdx.x == 0) ctl->spare_top = __ldcg(&p.grow.spare[0]);
        __threadfence();
        atomicAdd(&ctl->grow_done, 1u);  // every CTA's: the last phase may run (or be run again)
    }
    if (!grid_sync(ctl)) return false;
    grow_finish(p, t, rows, chunks, novf);
    return grid_sync(ctl);
}
