/*
 * xb_final.cu
 *
 * Host services of the final stage, over the kernels of the device
 * translation unit (xb_exec.cu, declared in xb_final.h):
 *
 *   xpuB200Final        kds_final in the reference layout, with GPU-Sort /
 *                       LIMIT / window rank of the groups
 *   xpuB200FinalNoAlloc the same without device allocations
 *   xpuB200MergeFinal   another kds_final merged into a session's groups
 *   xpuB200FinalParts   the groups as hash partitions for the exchange step
 *   xpuB200InnerRebuild rows appended into a KDS_FORMAT_HASH inner buffer
 */
#include <cuda_runtime.h>
#include <algorithm>
#include <mutex>
#include <vector>
#include <cstring>
#include <cstdio>
#include "xb_plan.h"
#include "xb_exec_dev.cuh"
#include "xb_sort.cuh"
#include "xpu_b200.h"
#include "xb_host.h"
#include "xb_final.h"

/* the fixed tuple of the session's groups as a program of 4-byte units
 * (xb_write_group_tuple's layout with every key present), and the bytes of
 * such an item; no units when a key's size or place depends on its value */
static void xb_final_program(const xb_plan *plan, bool row_fmt, XbFinalProg *pg)
{
    pg->nunits = 0;
    pg->item = 0;
    /* test hook, inert unless set: every tuple by the general writer */
    const char *off = getenv("XPU_B200_TEST_NO_FINAL_PROGRAM");
    if (off && off[0] == '1')
        return;
    uint8_t img[XB_FINAL_UNITS * 4] = {0};
    uint16_t op[XB_FINAL_UNITS] = {0}, src[XB_FINAL_UNITS] = {0};
    const uint32_t n = plan->naggs;
    const uint32_t hoff = (uint32_t)PGSTROM_MAXALIGN(15 + (n + 7) / 8);
    uint32_t t = hoff;
    uint16_t infomask = HEAP_HASNULL;
    auto put32 = [&](uint32_t at, uint32_t v) { memcpy(img + at, &v, 4); };
    auto unit = [&](uint32_t at, uint16_t o, uint32_t s, uint32_t imm = 0) {
        op[at / 4] = o;
        src[at / 4] = (uint16_t)s;
        put32(at, imm);
    };
    for (uint32_t j = 0; j < n; j++) {
        const xb_agg &a = plan->aggs[j];
        t = (uint32_t)PGSTROM_TYPEALIGN(a.attalign, t);
        if ((t & 3) || t + 64 + ROWID_SIZE > sizeof(img))
            return;
        uint32_t nb = 0;
        const uint32_t s = a.state_off;
        switch (a.action) {
        case KAGG_ACTION__VREF: {
            if (a.key_index < 0)
                break;
            const uint32_t k = plan->gent_keys_off + sizeof(xb_keyimg) * a.key_index + offsetof(xb_keyimg, val);
            switch (plan->keys[a.key_index].ld) {
            case XB_LD_INT4: case XB_LD_DATE: nb = 4; unit(t, XB_FU_COPY, k); break;
            case XB_LD_FLT4: nb = 4; unit(t, XB_FU_FLT4, k); break;
            case XB_LD_INT8: case XB_LD_FLT8:
                nb = 8;
                unit(t, XB_FU_COPY, k);
                unit(t + 4, XB_FU_COPY, k + 4);
                break;
            default: return;            /* varlena, or below 4 bytes */
            }
            break;
        }
        case KAGG_ACTION__NROWS_ANY: case KAGG_ACTION__NROWS_COND:
            nb = 8;
            unit(t, XB_FU_COPY, s);
            unit(t + 4, XB_FU_COPY, s + 4);
            break;
        case KAGG_ACTION__PMIN_INT32: case KAGG_ACTION__PMIN_INT64:
        case KAGG_ACTION__PMAX_INT32: case KAGG_ACTION__PMAX_INT64:
        case KAGG_ACTION__PMIN_FP64: case KAGG_ACTION__PMAX_FP64: {
            const bool fp = a.action == KAGG_ACTION__PMIN_FP64 || a.action == KAGG_ACTION__PMAX_FP64;
            const uint32_t mx = a.action == KAGG_ACTION__PMAX_FP64 ? 1 : 0;
            nb = 16;
            put32(t, nb << 2);
            unit(t + 4, XB_FU_MM_ATTRS, s);
            unit(t + 8, fp ? XB_FU_MMFP_LO : XB_FU_COPY, s, mx);
            unit(t + 12, fp ? XB_FU_MMFP_HI : XB_FU_COPY, fp ? s : s + 4, mx);
            break;
        }
        case KAGG_ACTION__PSUM_INT: case KAGG_ACTION__PAVG_INT:
        case KAGG_ACTION__PSUM_INT64: case KAGG_ACTION__PAVG_INT64:
        case KAGG_ACTION__PSUM_NUMERIC: case KAGG_ACTION__PAVG_NUMERIC: {
            const bool num = a.action == KAGG_ACTION__PSUM_NUMERIC || a.action == KAGG_ACTION__PAVG_NUMERIC;
            const bool wide = num || a.action == KAGG_ACTION__PSUM_INT64 || a.action == KAGG_ACTION__PAVG_INT64;
            nb = wide ? sizeof(kagg_state__psum_numeric_packed) : sizeof(kagg_state__psum_int_packed);
            put32(t, nb << 2);
            if (num)
                unit(t + 4, XB_FU_NUM_ATTRS, s + 24, (uint32_t)a.weight & PAGG_NUMERIC_ATTRS__WEIGHT);
            for (uint32_t k = 8; k < nb; k += 4)
                unit(t + k, XB_FU_COPY, s + k - 8);
            break;
        }
        case KAGG_ACTION__PSUM_FP: case KAGG_ACTION__PAVG_FP:
        case KAGG_ACTION__STDDEV: case KAGG_ACTION__COVAR:
            nb = a.action == KAGG_ACTION__STDDEV ? sizeof(kagg_state__stddev_packed)
               : a.action == KAGG_ACTION__COVAR ? sizeof(kagg_state__covar_packed) : sizeof(kagg_state__psum_fp_packed);
            put32(t, nb << 2);
            unit(t + 8, XB_FU_COPY, s);
            unit(t + 12, XB_FU_COPY, s + 4);
            for (uint32_t k = 16; k < nb; k += 8) {
                unit(t + k, XB_FU_SUM_LO, s + 2 * k - 24);
                unit(t + k + 4, XB_FU_SUM_HI, s + 2 * k - 24);
            }
            break;
        default:
            break;
        }
        if (a.action != KAGG_ACTION__VREF && nb != 8)
            infomask |= HEAP_HASVARWIDTH;
        if (nb)
            img[offsetof(kern_tupitem, t_bits) + (j >> 3)] |= (uint8_t)(1u << (j & 7));
        t += nb;
    }
    if (t & 3)
        return;
    unit(t, XB_FU_ROWID, 0);
    t += ROWID_SIZE;
    const uint16_t im2 = (uint16_t)(n & HEAP_NATTS_MASK);
    put32(0, t);
    unit(offsetof(kern_tupitem, hash), XB_FU_COPY, offsetof(xb_gent_head, hash));
    memcpy(img + offsetof(kern_tupitem, t_infomask2), &im2, 2);
    memcpy(img + offsetof(kern_tupitem, t_infomask), &infomask, 2);
    img[offsetof(kern_tupitem, t_hoff)] = (uint8_t)(hoff + MINIMAL_TUPLE_OFFSET);
    pg->nunits = (uint32_t)PGSTROM_MAXALIGN(t) / 4;
    for (uint32_t u = 0; u < pg->nunits; u++) {
        pg->unit[u].op = op[u];
        pg->unit[u].src = src[u];
        memcpy(&pg->unit[u].imm, img + 4 * u, 4);
    }
    pg->item = (uint32_t)PGSTROM_MAXALIGN((row_fmt ? 0 : offsetof(kern_hashitem, t)) + t);
}

/* for tests: the item bytes of the session's program (0: none) */
extern "C" uint32_t xb_final_program_item(const xb_plan *plan)
{
    XbFinalProg pg;
    xb_final_program(plan, false, &pg);
    return pg.nunits ? pg.item : 0;
}

/* The groups of a session as nparts kds_finals, in two steps: plan() counts
 * the groups and item bytes of every part, write() puts the parts where the
 * caller wants them.  Session lock held; work memory is the caller's to
 * free (tmp). */
struct XbFinalRun {
    xpuB200Session *s;
    const kern_data_store *fh;      /* the session's kds_final definition */
    uint64_t        head_len = 0;
    bool            row_fmt = false;
    std::vector<void *> tmp;
    char           *scratch = nullptr;      /* work memory of the caller's, instead of the pool's */
    uint64_t        scratch_left = 0;
    XbTileArgs      ta;
    uint64_t       *d_totals = nullptr;
    void           *d_temp = nullptr;
    uint32_t        set0 = UINT32_MAX;      /* the part set counted last */
    std::vector<uint64_t> totals;           /* groups, item bytes of every part */

    explicit XbFinalRun(xpuB200Session *sess) : s(sess)
    {
        const kern_session_info *session = (const kern_session_info *)s->h_session.data();
        fh = (const kern_data_store *)(s->h_session.data() + session->groupby_kds_final);
        head_len = KDS_HEAD_LENGTH(fh);
        row_fmt = fh->format == KDS_FORMAT_ROW;
    }
    ~XbFinalRun()
    {
        for (void *p : tmp) cudaFreeAsync(p, s->stream);
    }
    bool alloc(size_t sz, void **p)
    {
        if (scratch) {
            sz = xb_align256(sz);
            if (sz > scratch_left) return false;
            *p = scratch;
            scratch += sz;
            scratch_left -= sz;
            return true;
        }
        if (cudaMallocAsync(p, sz < 256 ? 256 : sz, s->stream) != cudaSuccess) { cudaGetLastError(); return false; }
        tmp.push_back(*p);
        return true;
    }
    int grid() const { return (int)std::min<uint64_t>(ta.ntiles, (uint64_t)s->dev->nsm * 8); }

    /* counts and prefixes of the parts from part0 on */
    bool count(uint32_t part0)
    {
        cudaStream_t st = s->stream;
        ta.part0 = part0;
        ta.pset = std::min<uint32_t>(ta.nparts - part0, XB_FINAL_PARTS);
        const uint64_t n = (uint64_t)ta.pset * ta.ntiles;
        xb_final_tiles<<<grid(), XB_FINAL_TILE, 12 * ta.pset, st>>>(ta);
        if (n <= 4096) {
            xb_final_scan_small<<<1, XB_FINAL_TILE, 0, st>>>(ta, (uint32_t *)ta.count_scan, (uint64_t *)ta.bytes_scan,
                                                              (uint32_t)n);
        } else if (xb_scan<uint32_t, XbOpSum, true>(ta.count, (uint32_t *)ta.count_scan, n, d_temp, st) != cudaSuccess ||
                   xb_scan<uint64_t, XbOpSum, true>(ta.bytes, (uint64_t *)ta.bytes_scan, n, d_temp, st) != cudaSuccess) {
            return false;
        }
        xb_final_totals<<<(ta.pset + 255) / 256, 256, 0, st>>>(ta, d_totals + 2 * part0);
        set0 = part0;
        return cudaGetLastError() == cudaSuccess;
    }
    /* tiles small enough to spread the table over the GPU, and few enough
     * that the counters of a launch's parts stay small */
    int plan(uint32_t nparts, kern_errorbuf *err, const uint32_t *list = nullptr, uint32_t nlist = 0)
    {
        cudaStream_t st = s->stream;
        memset(&ta, 0, sizeof(ta));
        ta.plan = s->d_plan;
        ta.gt = s->d_gt;
        ta.list = list;
        ta.cap = list ? nlist : s->h_gt.cap_mask + 1;
        ta.nparts = nparts;
        ta.row_format = row_fmt ? 1 : 0;
        xb_final_program(s->h_plan, row_fmt, &ta.prog);
        const uint64_t pset = std::min<uint32_t>(nparts, XB_FINAL_PARTS);
        uint64_t slots = XB_FINAL_TILE;
        while (pset * ((ta.cap + slots - 1) / slots) > (4ULL << 20))
            slots *= 2;
        ta.tile_slots = (uint32_t)slots;
        ta.ntiles = (uint32_t)((ta.cap + slots - 1) / slots);
        const uint64_t n = pset * ta.ntiles;
        /* the work arrays in one piece */
        const uint64_t tb = 16ULL * nparts;
        char *w = nullptr;
        if (!alloc(24 * n + tb + xb_scan_temp_bytes<uint64_t>(n) + 256, (void **)&w))
            return XB_ERR(err, ERRCODE_DEVICE_FATAL, "out of device memory in Final");
        ta.bytes = (uint64_t *)w;
        ta.bytes_scan = ta.bytes + n;
        d_totals = ta.bytes + 2 * n;
        ta.count = (uint32_t *)(w + 16 * n + tb);
        ta.count_scan = ta.count + n;
        d_temp = (void *)(((uintptr_t)(ta.count + 2 * n) + 255) & ~(uintptr_t)255);
        totals.assign(2 * (size_t)nparts, 0);
        if (nparts == 1 && ta.cap <= XB_FINAL_SMALL) {
            ta.pset = 1;
            xb_final_count_small<<<1, 1024, 0, st>>>(ta, s->pinned->totals);
            cudaError_t rc = cudaGetLastError();
            if (rc != cudaSuccess || (rc = cudaStreamSynchronize(st)) != cudaSuccess)
                return XB_ERR(err, ERRCODE_DEVICE_FATAL, "Final: %s", cudaGetErrorString(rc));
            totals[0] = s->pinned->totals[0];
            totals[1] = s->pinned->totals[1];
            set0 = 0;
            return 0;
        }
        for (uint32_t p = 0; p < nparts; p += XB_FINAL_PARTS)
            if (!count(p))
                return XB_ERR(err, ERRCODE_DEVICE_FATAL, "Final: %s", cudaGetErrorString(cudaGetLastError()));
        XB_CUDA(cudaMemcpyAsync(totals.data(), d_totals, 16ULL * nparts, cudaMemcpyDeviceToHost, st), err);
        XB_CUDA(cudaStreamSynchronize(st), err);
        return 0;
    }
    /* the kds_final of part p, at out of the output buffer */
    XbFinalPart part(uint32_t p, uint64_t out) const
    {
        XbFinalPart P;
        P.out = out;
        P.nitems = (uint32_t)totals[2 * p];
        P.nslots = (uint32_t)(row_fmt ? 0 : KDS_GET_HASHSLOT_WIDTH(totals[2 * p]));
        P.items_base = head_len + 8ULL * P.nslots + 8ULL * P.nitems;
        P.length = P.items_base + totals[2 * p + 1];
        return P;
    }
    int write(char *out, const std::vector<XbFinalPart> &parts, kern_errorbuf *err)
    {
        cudaStream_t st = s->stream;
        const kern_session_info *session = (const kern_session_info *)s->h_session.data();
        XbFinalPart *d_parts = nullptr;
        const char *head = s->d_session + session->groupby_kds_final;
        if (((uintptr_t)head & 7) != 0) {
            char *copy = nullptr;
            if (!alloc(head_len, (void **)&copy))
                return XB_ERR(err, ERRCODE_DEVICE_FATAL, "out of device memory in Final");
            XB_CUDA(cudaMemcpyAsync(copy, head, head_len, cudaMemcpyDeviceToDevice, st), err);
            head = copy;
        }
        if (ta.nparts > 1) {
            if (!alloc(sizeof(XbFinalPart) * parts.size(), (void **)&d_parts))
                return XB_ERR(err, ERRCODE_DEVICE_FATAL, "out of device memory in Final");
            XB_CUDA(cudaMemcpyAsync(d_parts, parts.data(), sizeof(XbFinalPart) * parts.size(),
                                    cudaMemcpyHostToDevice, st), err);
        }
        ta.head = (const uint64_t *)head;
        ta.head_len = (uint32_t)head_len;
        ta.only = parts[0];
        ta.out = out;
        for (uint32_t p0 = 0; p0 < ta.nparts; p0 += XB_FINAL_PARTS) {
            if (set0 != p0 && !count(p0))
                return XB_ERR(err, ERRCODE_DEVICE_FATAL, "Final: %s", cudaGetErrorString(cudaGetLastError()));
            ta.part = d_parts ? d_parts + p0 : nullptr;
            uint64_t most = 0;
            for (uint32_t p = p0; p < p0 + ta.pset; p++)
                most = std::max<uint64_t>(most, parts[p].nslots);
            const unsigned gx = (unsigned)std::min<uint64_t>((head_len / 8 + most + 255) / 256, 1024);
            xb_final_heads<<<dim3(gx, ta.pset), 256, 0, st>>>(ta);
            xb_final_fill<<<grid(), XB_FINAL_TILE, ta.nparts > 1 ? 16 * ta.pset : 0, st>>>(ta);
        }
        cudaError_t rc = cudaGetLastError();
        if (rc != cudaSuccess)
            return XB_ERR(err, ERRCODE_DEVICE_FATAL, "Final: %s", cudaGetErrorString(rc));
        return 0;
    }
};

/* what is wrong with a caller's output buffer at addr, memory of the given
 * kind (and device, and device address) for a call on GPU dindex: it must be
 * memory that this GPU's kernels can write, 8-byte aligned (kds_final is
 * written in words).  own: no other GPU's memory either.  nullptr: nothing */
static const char *xb_out_buffer_fault(const cudaPointerAttributes &pa, uint64_t addr, int dindex, bool own)
{
    if (pa.type == cudaMemoryTypeUnregistered)
        return "is not CUDA memory";
    if (own && !((pa.type == cudaMemoryTypeDevice && pa.device == dindex) || pa.type == cudaMemoryTypeManaged ||
                 (pa.type == cudaMemoryTypeHost && (uint64_t)pa.devicePointer == addr)))
        return "must be memory of the session's GPU (or mapped host memory)";
    if ((addr & 7) != 0)
        return "is not 8-byte aligned";
    return nullptr;
}

/* the same decision for tests, without a GPU */
extern "C" const char *xb_out_buffer_fault_of(int type, int device, uint64_t devptr, uint64_t addr, int dindex, int own)
{
    cudaPointerAttributes pa;
    memset(&pa, 0, sizeof(pa));
    pa.type = (cudaMemoryType)type;
    pa.device = device;
    pa.devicePointer = (void *)devptr;
    return xb_out_buffer_fault(pa, addr, dindex, own != 0);
}

static int xb_check_out_buffer(const char *func, const char *name, const void *p, int dindex, bool own, kern_errorbuf *err)
{
    cudaPointerAttributes pa;
    const char *why = "is not CUDA memory";
    if (cudaPointerGetAttributes(&pa, p) == cudaSuccess)
        why = xb_out_buffer_fault(pa, (uint64_t)p, dindex, own);
    else
        cudaGetLastError();
    return why ? XB_ERR(err, ERRCODE_DEVICE_ERROR, "%s: %s %s (GPU %d)", func, name, why, dindex) : 0;
}

/* GPU-Sort of the session's groups: the entries of those kept by LIMIT or
 * the window rank, in order, in *p_list (work memory of run; *p_n of them).
 * run has counted the groups of the whole table.  Returns 0, or -1. */
static int xb_final_sort(XbFinalRun &run, uint32_t **p_list, uint32_t *p_n)
{
    xpuB200Session *s = run.s;
    const xb_plan *plan = s->h_plan;
    cudaStream_t st = s->stream;
    const int grid = s->dev->nsm * 8;
    const uint32_t n = (uint32_t)run.totals[0];
    *p_n = 0;
    if (n == 0)
        return 0;
    const uint32_t nk = plan->nsort;
    uint32_t *ents, *idx, *list;
    uint64_t *keyw;
    uint8_t *nul;
    if (!run.alloc((size_t)n * 4, (void **)&ents) || !run.alloc((size_t)n * 4, (void **)&idx) ||
        !run.alloc((size_t)n * 4, (void **)&list) || !run.alloc((size_t)n * 16 * nk, (void **)&keyw) ||
        !run.alloc((size_t)n * nk, (void **)&nul))
        return -1;
    *p_list = list;
    XbSortArgs sa;
    sa.plan = s->d_plan;
    sa.gt = s->d_gt;
    sa.ents = ents;
    sa.keyw = keyw;
    sa.nul = nul;
    sa.n = n;
    const int g2 = std::min((int)((n + XB_BLOCK - 1) / XB_BLOCK), grid);
    xb_final_ents<<<run.grid(), XB_FINAL_TILE, 0, st>>>(run.ta, ents);
    xb_sort_keys<<<g2, XB_BLOCK, 0, st>>>(sa);
    uint32_t m = n;                 /* groups in idx, in sort order */
    bool sorted = false;
    if (n <= XB_SORT_SMALL) {
        xb_sort_small<<<1, 1024, 0, st>>>(sa, nullptr, n, idx);
        sorted = true;
    } else if (plan->sort_limit > 0 && !plan->sort_window && plan->sort_limit <= XB_SORT_SMALL) {
        /* the candidates, unless more than one CTA sorts share the last
         * one's leading bits */
        XbTopArgs ta;
        char *mem;
        const size_t hb = sizeof(uint32_t) * XB_TOP_DIGITS * XB_TOP_BINS;
        if (!run.alloc(hb + 32 + 4 * XB_SORT_SMALL, (void **)&mem))
            return -1;
        cudaMemsetAsync(mem, 0, hb + 32, st);
        ta.hi = keyw;
        ta.nul = nul;
        ta.n = n;
        ta.hist = (uint32_t *)mem;
        ta.prefix = (uint64_t *)(mem + hb);
        ta.ncand = (uint32_t *)(mem + hb + 16);
        ta.cand = (uint32_t *)(mem + hb + 32);
        const uint64_t want = (uint64_t)plan->sort_limit;
        cudaMemcpyAsync(&ta.prefix[1], &want, 8, cudaMemcpyHostToDevice, st);
        const int g3 = std::min(g2, s->dev->nsm * 4);
        for (uint32_t d = 0; d < XB_TOP_DIGITS; d++) {
            xb_top_hist<<<g3, XB_BLOCK, 0, st>>>(ta, d);
            xb_top_select<<<1, XB_SCAN_BLOCK, 0, st>>>(ta, d);
        }
        xb_top_gather<<<g3, XB_BLOCK, 0, st>>>(ta);
        uint32_t nc = 0;
        cudaMemcpyAsync(&nc, ta.ncand, 4, cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
        if (nc <= XB_SORT_SMALL) {
            xb_sort_small<<<1, 1024, 0, st>>>(sa, ta.cand, nc, idx);
            m = nc;
            sorted = true;
        }
    }
    const size_t tt = std::max(xb_radix_temp_bytes(n), xb_scan_temp_bytes<uint32_t>(n));
    void *d_tt = nullptr;
    if (!run.alloc(tt, &d_tt)) return -1;
    if (!sorted) {
        /* stable passes, least significant first: for each key from the
         * last, its low word, its high word, then its NULL flag (each a
         * stable radix sort of the word gathered in the current order,
         * carrying the group indexes along) */
        uint32_t *idx2;
        uint64_t *k64a, *k64b;
        uint8_t *k8a, *k8b;
        if (!run.alloc((size_t)n * 4, (void **)&idx2) || !run.alloc((size_t)n * 8, (void **)&k64a) ||
            !run.alloc((size_t)n * 8, (void **)&k64b) || !run.alloc((size_t)n, (void **)&k8a) ||
            !run.alloc((size_t)n, (void **)&k8b))
            return -1;
        xb_iota_u32<<<g2, XB_BLOCK, 0, st>>>(idx, n);
        for (int k = (int)nk - 1; k >= 0; k--) {
            for (int w = 1; w >= 0; w--) {
                if (w == 1 && plan->sort[k].words < 2)
                    continue;
                xb_sort_pass_key64<<<g2, XB_BLOCK, 0, st>>>(keyw + (2ULL * k + w) * n, idx, k64a, n);
                if (xb_radix_sort<uint64_t>(k64a, k64b, idx, idx2, n, 64, d_tt, st) != cudaSuccess) return -1;
            }
            xb_sort_pass_key8<<<g2, XB_BLOCK, 0, st>>>(nul + (uint64_t)k * n, idx, k8a, n);
            if (xb_radix_sort<uint8_t>(k8a, k8b, idx, idx2, n, 8, d_tt, st) != cudaSuccess) return -1;
        }
    }
    XbKeepArgs ka;
    memset(&ka, 0, sizeof(ka));
    uint32_t *kflag, *kscan;
    if (!run.alloc((size_t)m * 4, (void **)&kflag) || !run.alloc((size_t)m * 4, (void **)&kscan))
        return -1;
    if (plan->sort_window) {
        uint32_t *part, *peer, *pflag, *pcnt;
        if (!run.alloc((size_t)m * 4, (void **)&part) || !run.alloc((size_t)m * 4, (void **)&peer) ||
            !run.alloc((size_t)m * 4, (void **)&pflag) || !run.alloc((size_t)m * 4, (void **)&pcnt))
            return -1;
        XbRankArgs ra;
        ra.plan = s->d_plan;
        ra.idx = idx;
        ra.keyw = keyw;
        ra.nul = nul;
        ra.n = n;
        ra.part_start = part;
        ra.peer_start = peer;
        ra.peer_flag = pflag;
        xb_sort_bounds<<<g2, XB_BLOCK, 0, st>>>(ra);
        if (xb_scan<uint32_t, XbOpMax, false>(part, part, n, d_tt, st) != cudaSuccess ||
            xb_scan<uint32_t, XbOpMax, false>(peer, peer, n, d_tt, st) != cudaSuccess ||
            xb_scan<uint32_t, XbOpSum, false>(pflag, pcnt, n, d_tt, st) != cudaSuccess)
            return -1;
        ka.part_start = part;
        ka.peer_start = peer;
        ka.peer_cnt = pcnt;
    }
    ka.plan = s->d_plan;
    ka.idx = idx;
    ka.ents = ents;
    ka.n = m;
    ka.keep_flag = kflag;
    xb_sort_keepflag<<<g2, XB_BLOCK, 0, st>>>(ka);
    if (xb_scan<uint32_t, XbOpSum, true>(kflag, kscan, m, d_tt, st) != cudaSuccess) return -1;
    xb_sort_keep<<<g2, XB_BLOCK, 0, st>>>(ka, kscan, list);
    uint32_t lf = 0, ls = 0;
    cudaMemcpyAsync(&lf, kflag + m - 1, 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&ls, kscan + m - 1, 4, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    *p_n = lf + ls;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

/* ----------------------------------------------------------------
 * Final without device allocations
 *
 * xpuB200Final allocates its work arrays (the tiles' counts and their
 * prefix sums, scan storage) and a device copy of kds_final from the
 * device's memory pool on every call.  Some callers cannot do that: a
 * service that has reserved the GPU's memory up front and hands out pieces
 * of its own pool (as PG-Strom's GPU service does with its device memory),
 * or one that must not allocate device memory while other sessions'
 * kernels run (a plain cudaFree waits for the whole device).  This variant writes
 * kds_final into memory the caller already owns and keeps its work arrays
 * in the fixed array below, which lives in the library's module on every
 * GPU that loads it until the process exits.
 * ---------------------------------------------------------------- */
#define XB_FINAL_SCRATCH_BYTES  (8ULL << 20)        /* 8 MiB per GPU */
#define XB_FINAL_SCRATCH_SLOTS  262144ULL
#define XB_FINAL_SCRATCH_DEVS   64

static __device__ __align__(256) char xb_final_scratch[XB_FINAL_SCRATCH_BYTES];

/* device address of xb_final_scratch on each GPU, looked up once per device
 * (the host-side symbol is not a device address) */
static void *xb_final_scratch_dptr[XB_FINAL_SCRATCH_DEVS];
/* every session on one GPU shares that GPU's array: one call at a time
 * per GPU (calls for different GPUs use different arrays and run freely) */
static std::mutex xb_final_scratch_lock[XB_FINAL_SCRATCH_DEVS];


extern "C" int
xpuB200FinalNoAlloc(xpuB200Session *s, void *kds_final_dev, uint64_t buf_sz, uint64_t *p_required,
                    kern_exec_results *results, kern_errorbuf *err)
{
    xb_clear_error(err);
    if (!s)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "invalid FinalNoAlloc arguments");
    xb_table_hold hold(s);
    std::lock_guard<std::mutex> g(s->lock);
    const int dindex = s->dev->dindex;
    if (dindex < 0 || dindex >= XB_FINAL_SCRATCH_DEVS)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "FinalNoAlloc supports GPUs 0..%d", XB_FINAL_SCRATCH_DEVS - 1);
    std::lock_guard<std::mutex> gs(xb_final_scratch_lock[dindex]);
    XB_CUDA(cudaSetDevice(dindex), err);
    if (!xb_final_scratch_dptr[dindex]) {
        void *ptr = nullptr;
        cudaError_t rc = cudaGetSymbolAddress(&ptr, xb_final_scratch);
        if (rc != cudaSuccess || !ptr) {
            cudaGetLastError();
            return XB_ERR(err, ERRCODE_DEVICE_FATAL, "FinalNoAlloc: scratch address on GPU %d: %s",
                          dindex, cudaGetErrorString(rc));
        }
        xb_final_scratch_dptr[dindex] = ptr;
    }
    char *scratch = (char *)xb_final_scratch_dptr[dindex];
    const xb_plan *plan = s->h_plan;
    if (results) {
        uint32_t cap = results->num_rels;
        results->nitems_raw = (uint32_t)s->total_raw;
        results->nitems_in = (uint32_t)s->total_in;
        results->nitems_out = (uint32_t)s->total_out;
        results->num_rels = plan->nrels;
        for (uint32_t d = 1; d <= plan->nrels && d <= cap; d++)
            results->stats[d - 1].nitems_out = (uint32_t)s->total_depth[d];
        results->final_plan_task = true;
    }
    if (plan->nsort)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "a session with GPU-Sort keys needs xpuB200Final");
    if (!plan->has_groupby) {
        if (p_required) *p_required = 0;
        return 0;
    }
    if (s->h_gt.dump) {
        /* groups in the dump region join the table only when it grows,
         * which allocates: that is xpuB200Final's work */
        xb_gtable gh;
        int grc = xb_gt_read(s, &gh, err);
        if (grc) return grc;
        if (gh.dump_used)
            return XB_ERR(err, ERRCODE_DEVICE_ERROR,
                          "FinalNoAlloc: %llu groups wait for the group table to grow; use xpuB200Final",
                          (unsigned long long)gh.dump_used);
    }
    /* larger tables are xpuB200Final's, as they were when the work arrays
     * had an element per slot */
    const uint64_t cap = s->h_gt.cap_mask + 1;
    if (cap > XB_FINAL_SCRATCH_SLOTS)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR,
                      "FinalNoAlloc: the session's group table has %llu slots, above the %llu that this entry "
                      "point's fixed work space of %llu bytes serves; use xpuB200Final",
                      (unsigned long long)cap, (unsigned long long)XB_FINAL_SCRATCH_SLOTS,
                      (unsigned long long)XB_FINAL_SCRATCH_BYTES);
    int rc = kds_final_dev ? xb_check_out_buffer("FinalNoAlloc", "kds_final_dev", kds_final_dev, dindex, true, err) : 0;
    if (rc) return rc;
    XbFinalRun run(s);
    run.scratch = scratch;
    run.scratch_left = XB_FINAL_SCRATCH_BYTES;
    rc = run.plan(1, err);
    if (rc) return rc;
    const XbFinalPart P = run.part(0, 0);
    if (p_required) *p_required = P.length;
    if (results) {
        results->final_nitems = P.nitems;
        results->final_usage = P.length - P.items_base;
        results->final_total = P.length;
    }
    if (!kds_final_dev || buf_sz < P.length) {
        if (!kds_final_dev && buf_sz == 0)
            return 0;           /* size query only */
        return XB_ERR(err, ERRCODE_SUSPEND_NO_SPACE, "kds_final needs %llu bytes (buffer %llu)",
                      (unsigned long long)P.length, (unsigned long long)buf_sz);
    }
    rc = run.write((char *)kds_final_dev, std::vector<XbFinalPart>(1, P), err);
    if (rc) return rc;
    if (cudaStreamSynchronize(s->stream) != cudaSuccess)
        return XB_ERR(err, ERRCODE_DEVICE_FATAL, "FinalNoAlloc: %s", cudaGetErrorString(cudaGetLastError()));
    return 0;
}

extern "C" int
xpuB200Final(xpuB200Session *s, void *kds_final_buf, uint64_t buf_sz, uint64_t *p_required,
             kern_exec_results *results, kern_errorbuf *err)
{
    xb_clear_error(err);
    if (!s)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "invalid Final arguments");
    xb_table_hold hold(s);
    std::lock_guard<std::mutex> g(s->lock);
    XB_CUDA(cudaSetDevice(s->dev->dindex), err);
    cudaStream_t st = s->stream;
    const xb_plan *plan = s->h_plan;
    if (results) {
        uint32_t cap = results->num_rels;
        results->nitems_raw = (uint32_t)s->total_raw;
        results->nitems_in = (uint32_t)s->total_in;
        results->nitems_out = (uint32_t)s->total_out;
        results->num_rels = plan->nrels;
        for (uint32_t d = 1; d <= plan->nrels && d <= cap; d++)
            results->stats[d - 1].nitems_out = (uint32_t)s->total_depth[d];
        results->final_plan_task = true;
    }
    if (!plan->has_groupby) {
        if (p_required) *p_required = 0;
        return 0;
    }
    /* groups waiting in the dump region join the table first */
    int src = xb_gt_settle(s, err);
    if (src) return src;
    XbFinalRun run(s);
    int rc = run.plan(1, err);
    if (rc) return rc;
    if (plan->nsort) {
        uint32_t *list = nullptr, n = 0;
        if (xb_final_sort(run, &list, &n) != 0)
            return XB_ERR(err, ERRCODE_DEVICE_FATAL, "GPU-Sort of the groups failed (%s)",
                          cudaGetErrorString(cudaGetLastError()));
        if (n > 0 && (rc = run.plan(1, err, list, n)) != 0)
            return rc;
        if (n == 0) {
            run.totals.assign(2, 0);
            run.ta.cap = 0;
        }
    }
    const XbFinalPart P = run.part(0, 0);
    if (p_required) *p_required = P.length;
    if (results) {
        results->final_nitems = P.nitems;
        results->final_usage = P.length - P.items_base;
        results->final_total = P.length;
    }
    if (!kds_final_buf || buf_sz < P.length) {
        if (!kds_final_buf && buf_sz == 0)
            return 0;           /* size query only */
        return XB_ERR(err, ERRCODE_SUSPEND_NO_SPACE, "kds_final needs %llu bytes (buffer %llu)",
                      (unsigned long long)P.length, (unsigned long long)buf_sz);
    }
    char *d_out = nullptr;
    if (!run.alloc(P.length, (void **)&d_out))
        return XB_ERR(err, ERRCODE_DEVICE_FATAL, "out of device memory for kds_final (%llu bytes)",
                      (unsigned long long)P.length);
    rc = run.write(d_out, std::vector<XbFinalPart>(1, P), err);
    if (rc) return rc;
    cudaMemcpyAsync(kds_final_buf, d_out, P.length, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess)
        return XB_ERR(err, ERRCODE_DEVICE_FATAL, "Final: %s", cudaGetErrorString(cudaGetLastError()));
    return 0;
}

extern "C" int
xpuB200MergeFinal(xpuB200Session *s, const kern_data_store *kds_final, int kds_final_on_device,
                  kern_errorbuf *err)
{
    xb_clear_error(err);
    if (!s || !kds_final)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "invalid MergeFinal arguments");
    xb_table_hold hold(s);
    std::lock_guard<std::mutex> g(s->lock);
    const xb_plan *plan = s->h_plan;
    if (!plan->has_groupby)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "the session has no GROUP BY");
    XB_CUDA(cudaSetDevice(s->dev->dindex), err);
    cudaStream_t st = s->stream;
    /* the header, checked on the host */
    kern_data_store head;
    std::vector<char> hb;
    if (kds_final_on_device) {
        XB_CUDA(cudaMemcpy(&head, kds_final, offsetof(kern_data_store, colmeta), cudaMemcpyDeviceToHost), err);
        hb.resize(KDS_HEAD_LENGTH(&head));
        XB_CUDA(cudaMemcpy(hb.data(), kds_final, hb.size(), cudaMemcpyDeviceToHost), err);
    } else {
        hb.assign((const char *)kds_final, (const char *)kds_final + KDS_HEAD_LENGTH(kds_final));
    }
    const kern_data_store *h = (const kern_data_store *)hb.data();
    const kern_session_info *session = (const kern_session_info *)s->h_session.data();
    const char fmt = ((const kern_data_store *)(s->h_session.data() + session->groupby_kds_final))->format;
    if (h->format != fmt || h->ncols != plan->naggs || (fmt == KDS_FORMAT_ROW && h->hash_nslots != 0) ||
        KDS_HEAD_LENGTH(h) + 8 * ((uint64_t)h->hash_nslots + h->nitems) > h->length)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "kds_final to merge is not this session's KDS_FORMAT_%s",
                      fmt == KDS_FORMAT_ROW ? "ROW" : "HASH");
    if (h->nitems == 0)
        return 0;
    if (plan->gent_size > XB_GENT_MAX)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "group entries of %u bytes cannot be merged", plan->gent_size);
    const kern_data_store *d_kds = kds_final;
    char *d_copy = nullptr;
    if (!kds_final_on_device) {
        XB_CUDA(cudaMallocAsync((void **)&d_copy, h->length, st), err);
        XB_CUDA(cudaMemcpyAsync(d_copy, kds_final, h->length, cudaMemcpyHostToDevice, st), err);
        d_kds = (const kern_data_store *)d_copy;
    }
    /* room for every incoming group before the merge (the table grows as
     * for chunk launches when it would pass half of its slots) */
    {
        xb_gtable gh;
        int rc = xb_gt_read(s, &gh, err);
        if (!rc && (gh.dump_used || gh.nused + h->nitems > gh.soft_cap))
            rc = xb_gt_grow(s, gh.nused + h->nitems, err);
        if (rc) {
            if (d_copy) cudaFreeAsync(d_copy, st);
            return rc;
        }
    }
    XB_CUDA(cudaMemsetAsync(s->d_status, 0, sizeof(xb_status), st), err);
    XbMergeArgs ma;
    ma.plan = s->d_plan;
    ma.kds = d_kds;
    ma.gt = s->d_gt;
    ma.st = s->d_status;
    int grid = (int)((h->nitems + XB_BLOCK - 1) / XB_BLOCK);
    if (grid > s->dev->nsm * 8) grid = s->dev->nsm * 8;
    xb_merge_final<<<grid, XB_BLOCK, 0, st>>>(ma);
    if (d_copy)
        cudaFreeAsync(d_copy, st);
    int mrc = xb_wait_status(s, err);
    if (mrc) return mrc;
    return xb_gt_settle(s, err);
}

/* ----------------------------------------------------------------
 * the session's groups as hash partitions, for the exchange step of a
 * multi-GPU pre-aggregation: part p holds the groups whose hash % nparts
 * is p, as a KDS_FORMAT_HASH kds_final of its own (the same layout as
 * xpuB200Final's).  The parts lie back to back in one device buffer the
 * caller owns, each at a 256-byte aligned offset, so that the buffer can
 * be handed to the other GPUs whole (CUDA IPC, or NCCL all-to-all); each
 * GPU then merges the parts destined for it with xpuB200MergeFinal,
 * reading them in place from the peer's memory.
 * ---------------------------------------------------------------- */
extern "C" int
xpuB200FinalParts(xpuB200Session *s, uint32_t nparts, void *parts_dev, uint64_t buf_sz,
                  uint64_t *part_offsets, uint64_t *p_required, kern_errorbuf *err)
{
    xb_clear_error(err);
    if (!s || nparts < 1 || nparts > 4096 || !part_offsets)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "invalid FinalParts arguments");
    xb_table_hold hold(s);
    std::lock_guard<std::mutex> g(s->lock);
    XB_CUDA(cudaSetDevice(s->dev->dindex), err);
    const xb_plan *plan = s->h_plan;
    if (plan->has_groupby != 1)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "FinalParts needs a session with GROUP BY keys");
    if (plan->nsort)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "GPU-Sort applies to the merged groups, not to their parts");
    /* (another GPU's memory will do where the caller made it accessible) */
    int rc = parts_dev ? xb_check_out_buffer("FinalParts", "parts_dev", parts_dev, s->dev->dindex, false, err) : 0;
    if (rc) return rc;
    rc = xb_gt_settle(s, err);
    if (rc) return rc;
    XbFinalRun run(s);
    rc = run.plan(nparts, err);
    if (rc) return rc;
    std::vector<XbFinalPart> parts;
    uint64_t total = 0;
    for (uint32_t p = 0; p < nparts; p++) {
        parts.push_back(run.part(p, total));
        part_offsets[p] = total;
        total += xb_align256(parts[p].length);
    }
    part_offsets[nparts] = total;
    if (p_required) *p_required = total;
    if (!parts_dev || buf_sz < total) {
        if (!parts_dev && buf_sz == 0)
            return 0;           /* size query only */
        return XB_ERR(err, ERRCODE_SUSPEND_NO_SPACE, "the parts need %llu bytes (buffer %llu)",
                      (unsigned long long)total, (unsigned long long)buf_sz);
    }
    rc = run.write((char *)parts_dev, parts, err);
    if (rc) return rc;
    if (cudaStreamSynchronize(s->stream) != cudaSuccess)
        return XB_ERR(err, ERRCODE_DEVICE_FATAL, "FinalParts: %s", cudaGetErrorString(cudaGetLastError()));
    return 0;
}

extern "C" int
xpuB200InnerRebuild(xpuB200Device *dev, kern_data_store *kds_dst, const kern_data_store *kds_src,
                    uint32_t hash_divisor, uint32_t hash_remainder, uint64_t *p_required, kern_errorbuf *err)
{
    xb_clear_error(err);
    if (!dev || !kds_dst || !kds_src || (hash_divisor >= 2 && hash_remainder >= hash_divisor))
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "invalid InnerRebuild arguments");
    if (((uintptr_t)kds_dst & 7) != 0 || ((uintptr_t)kds_src & 7) != 0)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "InnerRebuild buffers must be 8-byte aligned");
    XB_CUDA(cudaSetDevice(dev->dindex), err);
    kern_data_store hd, hs;
    XB_CUDA(cudaMemcpy(&hd, kds_dst, offsetof(kern_data_store, colmeta), cudaMemcpyDeviceToHost), err);
    XB_CUDA(cudaMemcpy(&hs, kds_src, offsetof(kern_data_store, colmeta), cudaMemcpyDeviceToHost), err);
    if (hd.format != KDS_FORMAT_HASH || hd.hash_nslots == 0 || hd.nr_colmeta > 4096 ||
        (hd.length & 7) != 0 || (hd.usage & 7) != 0 ||
        KDS_HEAD_LENGTH(&hd) + 8ULL * ((uint64_t)hd.hash_nslots + hd.nitems) + hd.usage > hd.length)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "InnerRebuild destination is not a KDS_FORMAT_HASH buffer");
    if ((hs.format != KDS_FORMAT_HASH && hs.format != KDS_FORMAT_ROW) || hs.nr_colmeta > 4096 ||
        (hs.length & 7) != 0)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "InnerRebuild source must be KDS_FORMAT_HASH or _ROW");
    if (hd.ncols != hs.ncols)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "InnerRebuild source has %u columns, destination %u",
                      hs.ncols, hd.ncols);
    const uint64_t src_rowidx = KDS_HEAD_LENGTH(&hs) + (hs.format == KDS_FORMAT_HASH ? 8ULL * hs.hash_nslots : 0);
    if (src_rowidx + 8ULL * hs.nitems > hs.length)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "InnerRebuild source row index is out of the buffer");
    if (hs.nitems == 0) {
        if (p_required)
            *p_required = KDS_HEAD_LENGTH(&hd) + 8ULL * (hd.hash_nslots + hd.nitems) + hd.usage;
        return 0;
    }
    cudaStream_t st = xb_get_stream(dev);
    if (!st)
        return XB_ERR(err, ERRCODE_DEVICE_FATAL, "no stream");
    uint32_t *d_flag = nullptr;
    int rc = 0;
    if (cudaMallocAsync((void **)&d_flag, sizeof(uint32_t), st) != cudaSuccess) {
        xb_put_stream(dev, st);
        return XB_ERR(err, ERRCODE_DEVICE_FATAL, "out of device memory");
    }
    cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), st);
    XbRebuildArgs ra;
    ra.dst = kds_dst;
    ra.src = kds_src;
    ra.dst_head = KDS_HEAD_LENGTH(&hd);
    ra.src_rowidx = src_rowidx;
    ra.divisor = hash_divisor;
    ra.remainder = hash_remainder;
    ra.overflow = d_flag;
    int grid = (int)((hs.nitems + XB_BLOCK - 1) / XB_BLOCK);
    if (grid > dev->nsm * 8) grid = dev->nsm * 8;
    xb_inner_rebuild<<<grid, XB_BLOCK, 0, st>>>(ra);
    uint32_t flag = 0;
    cudaMemcpyAsync(&flag, d_flag, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&hd, kds_dst, offsetof(kern_data_store, colmeta), cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(d_flag, st);
    if (cudaStreamSynchronize(st) != cudaSuccess)
        rc = XB_ERR(err, ERRCODE_DEVICE_FATAL, "InnerRebuild: %s", cudaGetErrorString(cudaGetLastError()));
    xb_put_stream(dev, st);
    if (rc)
        return rc;
    const uint64_t required = KDS_HEAD_LENGTH(&hd) + 8ULL * (hd.hash_nslots + hd.nitems) + hd.usage;
    if (p_required)
        *p_required = required;
    if (flag & 2u)
        return XB_ERR(err, ERRCODE_DEVICE_ERROR, "InnerRebuild source has a broken row");
    /* rows claimed concurrently fit only when all of them do */
    if ((flag & 1u) || required > hd.length)
        return XB_ERR(err, ERRCODE_SUSPEND_NO_SPACE, "InnerRebuild destination needs %llu bytes (buffer %llu)",
                      (unsigned long long)required, (unsigned long long)hd.length);
    return 0;
}

