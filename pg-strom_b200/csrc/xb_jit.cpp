/*
 * xb_jit.cpp
 *
 * Session-specialised executor kernels.
 *
 * The interpreting kernel (xb_exec.cu) runs any translated session, but
 * pays for its generality on every 32-row batch: plan fields are re-read,
 * each bytecode op is fetched and dispatched, registers live in shared
 * memory.  For the sessions it accepts, this file prints a CUDA
 * translation unit in which the plan is a set of constants (register
 * numbers, loaders, join depths, uniqueness and NULL-ness of inner
 * columns, group-entry layout, aggregate actions) and every bytecode
 * program is straight-line code over per-lane registers, then compiles it
 * with NVRTC for sm_100a and loads it through the driver API.
 *
 * This is how PG-Strom itself built its GPU code before the xPU bytecode
 * (per-query CUDA C generated by codegen.c and compiled by NVRTC in
 * cuda_program.c); here the generated code reuses the same device
 * functions as the interpreter (xb_ops.cuh, xb_device.cuh,
 * xb_exec_dev.cuh) so both paths share one definition of every
 * operation's semantics.
 *
 * NVRTC and the driver are bound at run time (dlopen /
 * cudaGetDriverEntryPoint), so the library still loads on hosts without
 * them; a session whose kernel cannot be built runs on the interpreter.
 */
#include <cuda.h>
#include <cuda_runtime.h>
#include <nvrtc.h>
#include <dlfcn.h>
#include <cstdio>
#include <cstring>
#include <cstdint>
#include <cstdlib>
#include <chrono>
#include <functional>
#include <map>
#include <mutex>
#include <thread>
#include <atomic>
#include <memory>
#include <sstream>
#include <string>
#include <algorithm>
#include <vector>
#include "xb_plan.h"
#include "xb_jit.h"

/* sources of the device headers, generated by build.py */
#include "xb_jit_headers.inc"

namespace {

/* ----------------------------------------------------------------
 * run-time bindings
 * ---------------------------------------------------------------- */
struct NvrtcApi {
    bool ok = false;
    std::string why;
    decltype(&nvrtcCreateProgram) create = nullptr;
    decltype(&nvrtcCompileProgram) compile = nullptr;
    decltype(&nvrtcGetProgramLogSize) log_size = nullptr;
    decltype(&nvrtcGetProgramLog) log = nullptr;
    decltype(&nvrtcGetCUBINSize) cubin_size = nullptr;
    decltype(&nvrtcGetCUBIN) cubin = nullptr;
    decltype(&nvrtcDestroyProgram) destroy = nullptr;
    decltype(&nvrtcGetErrorString) errstr = nullptr;
};

struct DriverApi {
    bool ok = false;
    std::string why;
    decltype(&cuModuleLoadData) load = nullptr;
    decltype(&cuModuleGetFunction) getfn = nullptr;
    decltype(&cuFuncSetAttribute) setattr = nullptr;
    decltype(&cuFuncGetAttribute) getattr = nullptr;
    decltype(&cuLaunchKernel) launch = nullptr;
    decltype(&cuOccupancyMaxActiveBlocksPerMultiprocessor) occupancy = nullptr;
};

std::mutex g_lock;
NvrtcApi g_nvrtc;
DriverApi g_drv;
bool g_bound = false;

template <typename T>
bool dsym(void *h, const char *name, T *fp)
{
    *fp = (T)dlsym(h, name);
    return *fp != nullptr;
}

template <typename T>
bool drvsym(const char *name, T *fp)
{
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p)
        return false;
    *fp = (T)p;
    return true;
}

void bind_locked()
{
    if (g_bound)
        return;
    g_bound = true;
    const char *libs[] = {"libnvrtc.so.12", "libnvrtc.so", "/usr/local/cuda/lib64/libnvrtc.so.12"};
    void *h = nullptr;
    for (const char *l : libs)
        if ((h = dlopen(l, RTLD_NOW | RTLD_LOCAL)) != nullptr)
            break;
    if (!h) {
        g_nvrtc.why = "libnvrtc is not available";
    } else if (dsym(h, "nvrtcCreateProgram", &g_nvrtc.create) &&
               dsym(h, "nvrtcCompileProgram", &g_nvrtc.compile) &&
               dsym(h, "nvrtcGetProgramLogSize", &g_nvrtc.log_size) &&
               dsym(h, "nvrtcGetProgramLog", &g_nvrtc.log) &&
               dsym(h, "nvrtcGetCUBINSize", &g_nvrtc.cubin_size) &&
               dsym(h, "nvrtcGetCUBIN", &g_nvrtc.cubin) &&
               dsym(h, "nvrtcDestroyProgram", &g_nvrtc.destroy) &&
               dsym(h, "nvrtcGetErrorString", &g_nvrtc.errstr)) {
        g_nvrtc.ok = true;
    } else {
        g_nvrtc.why = "libnvrtc lacks an expected symbol";
    }
    if (drvsym("cuModuleLoadData", &g_drv.load) &&
        drvsym("cuModuleGetFunction", &g_drv.getfn) &&
        drvsym("cuFuncSetAttribute", &g_drv.setattr) &&
        drvsym("cuFuncGetAttribute", &g_drv.getattr) &&
        drvsym("cuLaunchKernel", &g_drv.launch) &&
        drvsym("cuOccupancyMaxActiveBlocksPerMultiprocessor", &g_drv.occupancy))
        g_drv.ok = true;
    else
        g_drv.why = "driver entry points are not available";
}

/* ----------------------------------------------------------------
 * code generation
 * ---------------------------------------------------------------- */
struct Gen {
    const xb_plan *p;
    uint32_t format;
    int minb = 0;               /* resident CTAs per SM the kernel is built for (0: default) */
    std::ostringstream o;
    int nlabel = 0;

    static std::string V(int r) { return "R.v[" + std::to_string(r) + "]"; }
    static std::string A(int r) { return "R.a[" + std::to_string(r) + "]"; }
    static std::string H(int r) { return "R.h[" + std::to_string(r) + "]"; }
    static std::string N(int r) { return "R.n[" + std::to_string(r) + "]"; }
    /* direct-addressed depth d's key range, loaded from the device plan
     * (the build's data decides it; sessions of one plan shape share the
     * kernel) */
    static std::string DMIN(uint32_t d)
    {
        return "((int64_t)__ldg(&E.plan->inner[" + std::to_string(d) + "].dkey_min))";
    }
    static std::string DRANGE(uint32_t d)
    {
        return "((uint64_t)__ldg(&E.plan->inner[" + std::to_string(d) + "].drange))";
    }

    /* instruction i's immediate / aux, loaded from the device plan */
    static std::string IMM(uint32_t i)
    {
        return "((uint64_t)__ldg((const unsigned long long *)&E.plan->insns[" + std::to_string(i) + "].imm))";
    }
    static std::string AUX(uint32_t i)
    {
        return "((uint32_t)__ldg(&E.plan->insns[" + std::to_string(i) + "].aux))";
    }

    static std::string U64(uint64_t v)
    {
        char b[40];
        snprintf(b, sizeof(b), "0x%016llxULL", (unsigned long long)v);
        return b;
    }

    /* one bytecode program over the registers; failures set 'failed' */
    void program(const xb_prog &pg, const std::string &ind)
    {
        if (!pg.count)
            return;
        /* mask-stack depth needed */
        int depth = 0, maxd = 0;
        for (uint32_t i = pg.start; i < (uint32_t)pg.start + pg.count; i++) {
            if (p->insns[i].op == XB_OP_MASK_PUSH) { depth++; if (depth > maxd) maxd = depth; }
            if (p->insns[i].op == XB_OP_MASK_POP && depth > 0) depth--;
        }
        const int lab = nlabel++;
        o << ind << "{\n";
        const std::string in2 = ind + "    ";
        o << in2 << "bool act = true;\n";
        for (int k = 0; k < maxd; k++)
            o << in2 << "bool ms" << k << " = true;\n";
        o << in2 << "(void)act;\n";
        depth = 0;
        bool used_end = false;
        for (uint32_t i = pg.start; i < (uint32_t)pg.start + pg.count; i++) {
            const xb_insn &x = p->insns[i];
            const int d = x.dst, a = x.a, b = x.b;
            std::ostringstream l;
            switch (x.op) {
            case XB_OP_END:
                l << "goto xbj_end_" << lab << ";";
                used_end = true;
                break;
            case XB_OP_CONST:
                /* constants are read from the plan at run time, so that
                 * sessions differing only in their constants share one
                 * compiled kernel */
                l << V(d) << " = " << IMM(i) << "; " << A(d) << " = " << AUX(i) << "; "
                  << N(d) << " = " << (x.kind != XB_RK_TEXT ? "(" + AUX(i) + " == 1u)" : std::string("false")) << ";";
                break;
            case XB_OP_MOVE:
                l << "{ const uint64_t v_ = " << V(a) << "; const uint32_t a_ = " << A(a)
                  << "; const bool n_ = " << N(a) << "; " << V(d) << " = v_; " << A(d) << " = a_; "
                  << N(d) << " = n_; }";
                break;
            case XB_OP_CMPI:
                l << "{ const bool n_ = " << N(a) << "; bool r_ = false; if (!n_) r_ = xb_cmp_sub(" << (int)x.sub
                  << ", " << (x.kind == XB_RK_INT
                              ? "xb_cmp3_int((int64_t)" + V(a) + ", (int64_t)" + IMM(i) + ")"
                              : "xb_cmp3_flt(__longlong_as_double(" + V(a) + "), __longlong_as_double(" +
                                IMM(i) + "))")
                  << "); " << V(d) << " = r_ ? 1 : 0; " << N(d) << " = n_; }";
                break;
            case XB_OP_HASH1:
            case XB_OP_HASH_ADD: {
                std::string hv = x.sub == XB_HK_CACHED
                    ? H(a)
                    : "xb_hash_reg(" + std::to_string(x.sub) + ", " + V(a) + ", " + A(a) + ", act, &bad_)";
                l << "{ uint32_t h_ = " << (x.op == XB_OP_HASH1 ? std::string("0xffffffffU") : "(uint32_t)" + V(d))
                  << "; if (!" << N(a) << ") { bool bad_ = false; const uint32_t hv_ = " << hv
                  << "; if (bad_) { XB_RAISE(E.st, ERRCODE_DEVICE_ERROR, XB_MSG_NUMERIC_CORRUPT); failed = true; }"
                  << " (void)bad_; h_ = xb_hash_merge(h_, hv_); } ";
                if (x.op == XB_OP_HASH1)
                    l << V(d) << " = h_ ^ 0xffffffffU; " << N(d) << " = false; }";
                else
                    l << V(d) << " = h_; }";
                break;
            }
            case XB_OP_CMP:
                l << "{ const bool n_ = " << N(a) << " || " << N(b) << "; bool r_ = false; if (!n_) r_ = xb_cmp_sub("
                  << (int)x.sub << ", xb_cmp3(" << (int)x.kind << ", " << V(a) << ", " << A(a) << ", " << V(b)
                  << ", " << A(b) << ", act, E.st, &failed)); " << V(d) << " = r_ ? 1 : 0; " << N(d) << " = n_; }";
                break;
            case XB_OP_ARITH:
                l << "{ const bool n_ = " << N(a) << " || " << N(b) << "; uint64_t o_ = 0; if (!n_) o_ = "
                  << (x.kind == XB_RK_INT ? "xb_arith_int(" : "xb_arith_flt(") << (int)x.sub << ", " << V(a)
                  << ", " << V(b) << ", act, E.st, &failed); " << V(d) << " = o_; " << N(d) << " = n_; }";
                break;
            case XB_OP_CAST:
                l << "{ const bool n_ = " << N(a) << "; uint64_t o_ = 0; if (!n_) o_ = xb_cast_op(" << (int)x.sub
                  << ", " << V(a) << ", act, E.st, &failed); " << V(d) << " = o_; " << N(d) << " = n_; }";
                break;
            case XB_OP_NOT:
                l << "{ const bool n_ = " << N(a) << "; const uint64_t v_ = " << V(a) << " ? 0 : 1; " << V(d)
                  << " = v_; " << N(d) << " = n_; }";
                break;
            case XB_OP_NULLTEST:
                l << "{ const bool n_ = " << N(a) << "; " << V(d) << " = " << (x.sub == 0 ? "n_" : "!n_")
                  << " ? 1 : 0; " << N(d) << " = false; }";
                break;
            case XB_OP_BOOLTEST:
                l << "{ const bool r_ = xb_booltest(" << (int)x.sub << ", " << N(a) << ", " << V(a) << " != 0); "
                  << V(d) << " = r_ ? 1 : 0; " << N(d) << " = false; }";
                break;
            case XB_OP_BOOL_INIT:
                l << V(d) << " = " << (x.sub == 0 ? 1 : 0) << "; " << N(d) << " = false;";
                break;
            case XB_OP_AND_ACC:
            case XB_OP_OR_ACC:
                l << "{ bool rn_, rv_; " << (x.op == XB_OP_AND_ACC ? "xb_and3(" : "xb_or3(") << N(d) << ", " << V(d)
                  << " != 0, " << N(a) << ", " << V(a) << " != 0, &rn_, &rv_); " << V(d) << " = rv_ ? 1 : 0; "
                  << N(d) << " = rn_; }";
                break;
            case XB_OP_MASK_PUSH:
                l << "ms" << depth << " = act;";
                depth++;
                break;
            case XB_OP_MASK_NARROW:
                l << "{ const bool an_ = " << N(a) << ", av_ = " << V(a) << " != 0; act = act && !("
                  << (x.sub == 0 ? "!an_ && !av_" : "!an_ && av_") << "); }";
                break;
            case XB_OP_MASK_POP:
                if (depth > 0) {
                    depth--;
                    l << "act = ms" << depth << ";";
                } else {
                    l << "act = true;";
                }
                break;
            case XB_OP_HASH_INIT:
                l << V(d) << " = 0xffffffffULL; " << N(d) << " = false;";
                break;
            case XB_OP_HASH_FINI:
                l << V(d) << " = (uint64_t)((uint32_t)" << V(d) << " ^ 0xffffffffU);";
                break;
            case XB_OP_DISTINCT:
                l << "{ const bool r_ = xb_distinct(" << (int)x.kind << ", " << N(a) << ", " << V(a) << ", " << A(a)
                  << ", " << N(b) << ", " << V(b) << ", " << A(b) << ", act); " << V(d) << " = r_ ? 1 : 0; "
                  << N(d) << " = false; }";
                break;
            default:
                l << "{ XB_RAISE(E.st, ERRCODE_DEVICE_FATAL, XB_MSG_NONE); failed = true; }";
                break;
            }
            o << in2 << l.str() << "\n";
        }
        if (used_end)
            o << in2 << "xbj_end_" << lab << ": ;\n";
        o << ind << "}\n";
    }

    /* lanes pass a program when its result is TRUE */
    static std::string pass_expr(const xb_prog &pg)
    {
        if (!pg.count)
            return "true";
        return "(!" + N(pg.result) + " && " + V(pg.result) + " != 0)";
    }

    /* ---- decode ------------------------------------------------- */
    void decode_general_copy(const std::string &ind)
    {
        for (uint32_t i = 0; i < p->nload0; i++) {
            const int r = p->load0[i].reg;
            o << ind << V(r) << " = tv_[" << i << "]; " << A(r) << " = ta_[" << i << "]; " << N(r)
              << " = ((nb_ >> " << i << ") & 1u) != 0;\n";
        }
    }

    /* an aligned load of a fixed-width datum (ld) at address expression p */
    static std::string typed_load(int ld, const std::string &p)
    {
        switch (ld) {
        case XB_LD_BOOL: return "(uint64_t)(*(const uint8_t *)(" + p + ") ? 1u : 0u)";
        case XB_LD_INT2: return "(uint64_t)(int64_t)*(const int16_t *)(" + p + ")";
        case XB_LD_INT4:
        case XB_LD_DATE: return "(uint64_t)(int64_t)*(const int32_t *)(" + p + ")";
        case XB_LD_FLT4: return "(uint64_t)__double_as_longlong((double)*(const float *)(" + p + "))";
        default:         return "*(const uint64_t *)(" + p + ")";
        }
    }

    /* fast path without a known layout: the header word and every
     * fixed-offset column (offsets from the launch's column layout in
     * shared memory) loaded together, before the header is checked */
    void speculative_fast_path()
    {
        const uint32_t nl = p->nload0;
        o << "        if (meta->fixed && (((uintptr_t)htup) & 7) == 0 &&\n"
             "            off + 24u + meta->fixed_end <= PGSTROM_BLCKSZ) {\n"
             "            const uint8_t *pay_ = htup + 24;\n"
             "            const uint64_t w_ = *(const uint64_t *)(htup + 16);\n";
        for (uint32_t i = 0; i < nl; i++)
            o << "            const uint64_t s" << i << "_ = "
              << typed_load((int)p->load0[i].ld, "pay_ + meta->fix[" + std::to_string(i) + "].off") << ";\n";
        o << "            if (((w_ >> 48) & 0xff) == 24 && !((w_ >> 32) & HEAP_HASNULL) &&\n"
             "                ((w_ >> 16) & HEAP_NATTS_MASK) >= " << p->max_resno0 << " && len >= 24u + meta->fixed_end) {\n";
        for (uint32_t i = 0; i < nl; i++) {
            const int r = p->load0[i].reg;
            o << "                " << V(r) << " = s" << i << "_; " << A(r) << " = 0; " << N(r) << " = false;\n";
        }
        o << "                return true;\n"
             "            }\n"
             "        }\n";
    }

    /* fast path for the heap layout the kernel is built for (the launch's
     * layout is checked once per CTA: lay_ok): the tuple's bytes from the
     * header word on are read as a few 8- or 16-byte words and every
     * column is cut out of them at a constant position */
    void layout_fast_path()
    {
        const uint32_t nl = p->nload0;
        const uint32_t nw = (8 + p->lay_end + 7) / 8;      /* 8-byte words from htup + 16 */
        const uint32_t nv = (nw + 1) / 2;                   /* 16-byte words */
        o << "        if (lay_ok && (((uintptr_t)htup) & 7) == 0 && off + " << 16 + 16 * nv << "u <= PGSTROM_BLCKSZ) {\n";
        for (uint32_t k = 0; k < 2 * nv; k++)
            o << "            uint64_t w" << k << "_;\n";
        o << "            if ((((uintptr_t)htup) & 15) == 0) {\n";
        for (uint32_t v = 0; v < nv; v++)
            o << "                const uint4 q" << v << "_ = *(const uint4 *)(htup + " << 16 + 16 * v << ");\n"
                 "                w" << 2 * v << "_ = ((uint64_t)q" << v << "_.y << 32) | q" << v << "_.x;\n"
                 "                w" << 2 * v + 1 << "_ = ((uint64_t)q" << v << "_.w << 32) | q" << v << "_.z;\n";
        o << "            } else {\n";
        for (uint32_t k = 0; k < 2 * nv; k++)
            o << "                w" << k << "_ = *(const uint64_t *)(htup + " << 16 + 8 * k << ");\n";
        o << "            }\n"
             "            if (((w0_ >> 48) & 0xff) == 24 && !((w0_ >> 32) & HEAP_HASNULL) &&\n"
             "                ((w0_ >> 16) & HEAP_NATTS_MASK) >= " << p->max_resno0 << " && len >= " << 24 + p->lay_end << "u) {\n";
        for (uint32_t i = 0; i < nl; i++) {
            const xb_load &l = p->load0[i];
            const uint32_t rel = 8 + (uint32_t)p->lay_off[i];     /* from htup + 16 */
            const std::string w = "w" + std::to_string(rel / 8) + "_";
            const uint32_t sh = (rel % 8) * 8;
            std::string e;
            switch (l.ld) {
            case XB_LD_BOOL: e = "(uint64_t)(((" + w + " >> " + std::to_string(sh) + ") & 0xffu) ? 1u : 0u)"; break;
            case XB_LD_INT2: e = "(uint64_t)(int64_t)(int16_t)(" + w + " >> " + std::to_string(sh) + ")"; break;
            case XB_LD_INT4:
            case XB_LD_DATE: e = "(uint64_t)(int64_t)(int32_t)(" + w + " >> " + std::to_string(sh) + ")"; break;
            case XB_LD_FLT4: e = "(uint64_t)__double_as_longlong((double)__int_as_float((int)(" + w + " >> " +
                                 std::to_string(sh) + ")))"; break;
            default:         e = w; break;
            }
            o << "                " << V(l.reg) << " = " << e << "; " << A(l.reg) << " = 0; " << N(l.reg) << " = false;\n";
        }
        o << "                return true;\n"
             "            }\n"
             "        }\n";
    }

    /* the launch's heap layout is the one the kernel is built for: the
     * cached offsets of the fixed-offset fast path, and the column
     * descriptors of the generated walk */
    void layout_check()
    {
        o << "__device__ __forceinline__ bool xbj_layout_ok(const XbSrcMeta *meta)\n{\n"
             "    return true";
        if (p->lay_valid) {
            o << " && meta->fixed != 0 && meta->fixed_end == " << p->lay_end << "u";
            for (uint32_t i = 0; i < p->nload0; i++)
                o << " && meta->fix[" << i << "].off == " << p->lay_off[i];
        }
        if (p->walk_ncols) {
            o << " && meta->ncols >= " << p->walk_ncols;
            for (uint32_t j = 0; j < p->walk_ncols; j++)
                o << "\n        && meta->cols[" << j << "].attlen == " << p->walk_len[j]
                  << " && meta->cols[" << j << "].attalign == " << (int)p->walk_align[j];
        }
        o << ";\n}\n\n";
    }

    /* straight-line walk over columns 1..walk_ncols of a tuple payload with
     * the column descriptors as constants (the launch's columns are checked
     * once per CTA: lay_ok): the sequential walk of the general decode,
     * alignment before fixed-width columns and before varlenas that start
     * with a pad byte, a column skipped where the tuple's NULL bitmap says
     * so.  Tuples without a bitmap take the same code with every bit set: a
     * walk of their own with constant offsets was a second pass for most
     * warps (5% of NULLs leave a NULL in four of five 32-row batches).
     * Queries over 4M rows 541 -> 494 us, every statistic over 2M 1046 ->
     * 1008 us (with the dump region no longer cleared). */
    void walk()
    {
        o << "__device__ __forceinline__ bool\n"
             "xbj_walk(XbjRegs &R, const uint8_t *pay, const uint32_t plen, const uint8_t *nullmap)\n{\n"
             "    uint32_t o = 0;\n";
        for (uint32_t j = 0; j < p->walk_ncols; j++) {
            const int len = p->walk_len[j], al = p->walk_align[j];
            std::vector<uint32_t> ls;
            for (uint32_t i = 0; i < p->nload0; i++)
                if (p->load0[i].resno == (int)j + 1)
                    ls.push_back(i);
            const std::string in = "        ";
            o << "    /* column " << j + 1 << ": attlen " << len << ", attalign " << al << " */\n"
                 "    if (!nullmap || ((nullmap[" << j / 8 << "] >> " << j % 8 << ") & 1)) {\n";
            if (len > 0) {
                if (al > 1)
                    o << in << "o = (o + " << al - 1 << "u) & ~" << al - 1 << "u;\n";
                o << in << "if (o + " << len << "u > plen) return false;\n";
                for (uint32_t i : ls) {
                    const int r = p->load0[i].reg;
                    o << in << V(r) << " = " << typed_load((int)p->load0[i].ld, "pay + o") << "; " << A(r)
                      << " = 0; " << N(r) << " = false;\n";
                }
                o << in << "o += " << len << "u;\n";
            } else {
                o << in << "if (o >= plen) return false;\n";
                if (al > 1)
                    o << in << "if (pay[o] == 0) {\n"
                      << in << "    o = (o + " << al - 1 << "u) & ~" << al - 1 << "u;\n"
                      << in << "    if (o >= plen) return false;\n"
                      << in << "}\n";
                o << in << "{\n"
                  << in << "    const uint32_t sz_ = xb_att_size(-1, pay + o, plen - o);\n"
                  << in << "    if (sz_ == 0 || sz_ > plen - o) return false;\n";
                for (uint32_t i : ls) {
                    const int r = p->load0[i].reg;
                    o << in << "    if (!xb_load_datum(" << (int)p->load0[i].ld << ", pay + o, &" << V(r) << ", &" << A(r)
                      << ")) return false;\n"
                      << in << "    " << N(r) << " = false;\n";
                }
                o << in << "    o += sz_;\n"
                  << in << "}\n";
            }
            o << "    }";
            if (!ls.empty()) {
                o << " else {\n";
                for (uint32_t i : ls)
                    o << in << N(p->load0[i].reg) << " = true;\n";
                o << "    }";
            }
            o << "\n";
        }
        o << "    (void)o;\n"
             "    return true;\n}\n\n";
    }

    void decode()
    {
        const uint32_t nl = p->nload0;
        o << "__device__ __forceinline__ bool\n"
             "xbj_decode(XbjRegs &R, const XbExecArgs &args, const uint8_t *page, const kern_data_store *kds_,\n"
             "           uint32_t row0, const XbSrcMeta *meta, uint32_t idx, uint32_t lp, bool lay_ok, bool &exists,\n"
             "           xb_status *st, const XbArrowCol *acol)\n{\n"
             "    (void)lp; (void)page; (void)kds_; (void)row0; (void)lay_ok; (void)acol;\n";
        if (format == KDS_FORMAT_BLOCK) {
            o << "    if (ITEMID_FLAGS(lp) != LP_NORMAL)\n        return false;\n"
                 "    exists = true;\n"
                 "    const uint32_t off = ITEMID_OFF(lp), len = ITEMID_LEN(lp);\n"
                 "    bool ok = false;\n"
                 "    if (off >= SizeOfPageHeaderData && len >= SizeofHeapTupleHeader && off + len <= PGSTROM_BLCKSZ) {\n"
                 "        const uint8_t *htup = page + off;\n";
            /* fast path: an 8-byte aligned tuple with the plain 24-byte
             * header (no NULL bitmap): the header word and every
             * fixed-offset column are loaded together, before the header
             * is checked, instead of one after the other (the loads stay
             * inside the page) */
            if (p->lay_valid)
                layout_fast_path();
            else
                speculative_fast_path();
            o << "        uint16_t infomask2, infomask;\n"
                 "        uint32_t t_hoff;\n"
                 "        if ((((uintptr_t)htup) & 7) == 0) {\n"
                 "            const uint64_t w_ = *(const uint64_t *)(htup + 16);   /* t_ctid tail, masks, t_hoff */\n"
                 "            infomask2 = (uint16_t)(w_ >> 16);\n"
                 "            infomask = (uint16_t)(w_ >> 32);\n"
                 "            t_hoff = (uint32_t)(w_ >> 48) & 0xff;\n"
                 "        } else {\n"
                 "            infomask2 = (uint16_t)xb_fetch_le(htup + 18, 2);\n"
                 "            infomask = (uint16_t)xb_fetch_le(htup + 20, 2);\n"
                 "            t_hoff = htup[22];\n"
                 "        }\n"
                 "        const int natts_raw = infomask2 & HEAP_NATTS_MASK;\n"
                 "        if (t_hoff >= SizeofHeapTupleHeader && t_hoff <= len) {\n"
                 "            if (meta->fixed && !(infomask & HEAP_HASNULL) && natts_raw >= " << p->max_resno0 << " &&\n"
                 "                len - t_hoff >= meta->fixed_end) {\n"
                 "                const uint8_t *payload = htup + t_hoff;\n";
            for (uint32_t i = 0; i < nl; i++) {
                const int r = p->load0[i].reg;
                o << "                xb_load_datum(" << (int)p->load0[i].ld << ", payload + meta->fix[" << i << "].off, &"
                  << V(r) << ", &" << A(r) << "); " << N(r) << " = false;\n";
            }
            o << "                ok = true;\n";
            if (p->walk_ncols)
                o << "            } else if (lay_ok && (((uintptr_t)htup) & 7) == 0 && (t_hoff & 7) == 0 &&\n"
                     "                       natts_raw >= " << p->walk_ncols << " &&\n"
                     "                       (!(infomask & HEAP_HASNULL) || SizeofHeapTupleHeader + (natts_raw + 7) / 8 <= t_hoff)) {\n"
                     "                ok = xbj_walk(R, htup + t_hoff, len - t_hoff,\n"
                     "                              (infomask & HEAP_HASNULL) ? htup + SizeofHeapTupleHeader : nullptr);\n";
            o << "            } else {\n"
                 "                const int natts = natts_raw < meta->ncols ? natts_raw : meta->ncols;\n"
                 "                const uint8_t *nullmap = (infomask & HEAP_HASNULL) ? htup + SizeofHeapTupleHeader : nullptr;\n"
                 "                if (!nullmap || SizeofHeapTupleHeader + (natts + 7) / 8 <= t_hoff) {\n"
                 "                    uint64_t tv_[" << nl + 1 << "]; uint32_t ta_[" << nl + 1 << "]; uint32_t nb_ = 0;\n"
                 "                    ok = xb_decode_tuple(meta->cols, natts, nullmap, htup + t_hoff, len - t_hoff,\n"
                 "                                         args.plan->load0, " << nl << ", tv_, ta_, 1, true, &nb_);\n"
                 "                    if (ok) {\n";
            decode_general_copy("                        ");
            o << "                    }\n"
                 "                }\n"
                 "            }\n"
                 "        }\n"
                 "    }\n"
                 "    if (!ok)\n        XB_RAISE(st, ERRCODE_DEVICE_ERROR, XB_MSG_BAD_TUPLE);\n"
                 "    return ok;\n}\n\n";
        } else if (format == KDS_FORMAT_ARROW) {
            o << "    exists = true;\n    const uint32_t row = row0 + idx;\n    bool ok = true;\n";
            for (uint32_t i = 0; i < nl; i++) {
                const xb_load &l = p->load0[i];
                /* fixed-width columns: the unit's resolved column (one bound
                 * check, the NULL bit if any, one load) */
                const char *ct = nullptr;
                const char *conv = "";
                switch (l.ld) {
                case XB_LD_INT2: ct = "int16_t"; conv = "(uint64_t)(int64_t)"; break;
                case XB_LD_INT4: ct = "int32_t"; conv = "(uint64_t)(int64_t)"; break;
                case XB_LD_INT8: ct = "int64_t"; conv = "(uint64_t)"; break;
                case XB_LD_FLT8: ct = "uint64_t"; conv = ""; break;
                case XB_LD_DATE: ct = "uint32_t"; conv = "DATE"; break;
                default: break;
                }
                if (ct) {
                    const std::string v = std::string("__ldg((const ") + ct + " *)c_->values + idx)";
                    const std::string val = std::string(conv) == "DATE"
                        ? "(uint64_t)(int64_t)(int32_t)(" + v + " - 10957u)" : std::string(conv) + v;
                    o << "    {\n"
                         "        const XbArrowCol *c_ = &acol[" << i << "];\n"
                         "        if (c_->ok) {\n"
                         "            bool nul_ = idx >= c_->nvalid;\n"
                         "            if (!nul_ && c_->nullmap)\n"
                         "                nul_ = !((__ldg(c_->nullmap + (row >> 3)) >> (row & 7)) & 1);\n"
                         "            " << V(l.reg) << " = nul_ ? 0 : " << val << ";\n"
                         "            " << A(l.reg) << " = 0;\n"
                         "            " << N(l.reg) << " = nul_;\n"
                         "        } else {\n";
                } else {
                    o << "    {\n        {\n";
                }
                o << "    {\n        bool isnull_ = true;\n"
                     "        if (" << l.resno << " >= 1 && " << l.resno << " <= (int)kds_->ncols) {\n"
                     "            const kern_colmeta *cm = &kds_->colmeta[" << l.resno - 1 << "];\n"
                     "            if (!xb_arrow_load(kds_, cm, row, " << (int)l.ld << ", &" << V(l.reg) << ", &" << A(l.reg)
                  << ", &isnull_)) {\n"
                     "                ok = false;\n"
                     "                XB_RAISE(st, ERRCODE_DEVICE_ERROR, XB_MSG_ARROW_TYPE);\n"
                     "            }\n        }\n"
                     "        " << N(l.reg) << " = isnull_;\n    }\n"
                     "        }\n    }\n";
            }
            o << "    (void)meta;\n    return ok;\n}\n\n";
        } else {
            o << "    const kern_data_store *kds = kds_;\n"
                 "    const uint64_t *rowindex = (const uint64_t *)((const char *)kds + KDS_HEAD_LENGTH(kds)) + kds->hash_nslots;\n"
                 "    const uint64_t off = rowindex[row0 + idx];\n"
                 "    if (off == 0)\n        return false;\n"
                 "    exists = true;\n"
                 "    bool ok = false;\n"
                 "    if (off <= kds->length && ((kds->length - off) & 7) == 0) {\n"
                 "        const uint8_t *t = (const uint8_t *)kds + kds->length - off;\n"
                 "        const kern_tupitem *ti = (const kern_tupitem *)t;\n"
                 "        const uint32_t pay = (uint32_t)ti->t_hoff - MINIMAL_TUPLE_OFFSET;\n"
                 "        int natts = ti->t_infomask2 & HEAP_NATTS_MASK;\n"
                 "        if (natts > meta->ncols) natts = meta->ncols;\n"
                 "        const bool hasnull = (ti->t_infomask & HEAP_HASNULL) != 0;\n"
                 "        if (!ti->has_xact_attrs && ti->t_hoff >= MINIMAL_TUPLE_OFFSET + 15 &&\n"
                 "            pay <= ti->t_len && off >= ti->t_len &&\n"
                 "            (!hasnull || 15u + (natts + 7) / 8 <= pay)) {\n"
                 "            uint64_t tv_[" << nl + 1 << "]; uint32_t ta_[" << nl + 1 << "]; uint32_t nb_ = 0;\n"
                 "            ok = xb_decode_tuple(meta->cols, natts, hasnull ? ti->t_bits : nullptr,\n"
                 "                                 t + pay, ti->t_len - pay, args.plan->load0, " << nl
              << ", tv_, ta_, 1, true, &nb_);\n"
                 "            if (ok) {\n";
            decode_general_copy("                ");
            o << "            }\n"
                 "        }\n"
                 "    }\n"
                 "    if (!ok)\n        XB_RAISE(st, ERRCODE_DEVICE_ERROR, XB_MSG_BAD_TUPLE);\n"
                 "    return ok;\n}\n\n";
        }
    }

    /* ---- group-by ------------------------------------------------ */
    void group_helpers()
    {
        /* key match against the lane's registers */
        o << "__device__ __forceinline__ bool xbj_key_match(const char *e, const XbjRegs &R)\n{\n"
             "    const xb_keyimg *img = (const xb_keyimg *)(e + XBJ_KEYS_OFF);\n    (void)img;\n";
        for (uint32_t k = 0; k < p->nkeys; k++) {
            const xb_key &key = p->keys[k];
            const int r = key.reg;
            o << "    {\n        const xb_keyimg x_ = img[" << k << "];\n        const bool rn_ = " << N(r) << ";\n"
                 "        if (x_.isnull || rn_) {\n            if (!(x_.isnull && rn_)) return false;\n        } else {\n";
            if (key.rk == XB_RK_TEXT)
                o << "            if (x_.len != " << A(r) << ") return false;\n"
                     "            if (x_.val != " << V(r) << " && !xb_bytes_eq_ool((const uint8_t *)x_.val, (const uint8_t *)"
                  << V(r) << ", x_.len)) return false;\n";
            else if (key.rk == XB_RK_NUM)
                o << "            if (x_.val != " << V(r) << ") { int err_ = 0;\n"
                     "                if (xb_numeric_cmp((const uint8_t *)x_.val, (const uint8_t *)" << V(r)
                  << ", &err_) != 0 || err_) return false; }\n";
            else
                o << "            if (x_.val != " << V(r) << ") return false;\n";
            o << "        }\n    }\n";
        }
        o << "    return true;\n}\n\n";

        /* claim: key values by value so the register set stays in registers.
         * Every table is zero-filled, so only the states that start at
         * another value are written.  New global entries are counted in
         * the shared counter newg (per warp, per CTA in the replay) and
         * added to the table's own count by xbj_count_flush: an atomic of
         * every new group on that one word took 1.9 ns, one after another
         * (20M Arrow rows into 1.7M groups: 7.29 ms a query, 4.52 ms now). */
        o << "__device__ __noinline__ int\nxbj_group_claim(char *e, uint32_t hash, xb_gtable *gt, xb_status *st, "
             "uint32_t *newg";
        for (uint32_t k = 0; k < p->nkeys; k++)
            o << ",\n                uint64_t v" << k << ", uint32_t a" << k << ", bool n" << k;
        o << ")\n{\n"
             "    xb_gent_head *h = (xb_gent_head *)e;\n"
             "    if (atomicCAS(&h->state, XB_GSTATE_EMPTY, XB_GSTATE_BUSY) != XB_GSTATE_EMPTY)\n        return 0;\n"
             "    h->hash = hash;\n"
             "    xb_keyimg *img = (xb_keyimg *)(e + XBJ_KEYS_OFF);\n    (void)img; (void)st;\n"
             "    bool ok = true;\n";
        for (uint32_t k = 0; k < p->nkeys; k++) {
            const int rk = p->keys[k].rk;
            o << "    { xb_keyimg s_; s_.val = v" << k << "; s_.len = a" << k << "; s_.isnull = n" << k << "; ";
            if (rk == XB_RK_TEXT || rk == XB_RK_NUM)
                o << "xb_key k_; k_.rk = " << rk << "; ok &= xb_key_store(k_, s_, &img[" << k << "], gt, st); }\n";
            else
                o << "img[" << k << "] = s_; }\n";
        }
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0)
                continue;
            switch (a.action) {
            case KAGG_ACTION__PMIN_INT32: case KAGG_ACTION__PMIN_INT64: case KAGG_ACTION__PMIN_FP64:
                o << "    *(int64_t *)(e + " << a.state_off << ") = INT64_MAX;\n";
                break;
            case KAGG_ACTION__PMAX_INT32: case KAGG_ACTION__PMAX_INT64: case KAGG_ACTION__PMAX_FP64:
                o << "    *(int64_t *)(e + " << a.state_off << ") = INT64_MIN;\n";
                break;
            default:
                break;
            }
        }
        o << "    if (gt) {\n        xb_red_shared_add_u32(newg, 1u);\n"
             "        xb_st_release(&h->state, XB_GSTATE_READY);\n"
             "    } else {\n        xb_st_release_cta(&h->state, XB_GSTATE_READY);\n    }\n"
             "    return ok ? 1 : 2;\n}\n\n";

        /* find or create */
        o << "template <bool SMEM>\n__device__ __forceinline__ char *\n"
             "xbj_group_get(const XbjRegs &R, const XbjEnv &E, char *entries, uint64_t cap_mask, uint32_t hash, bool *full)\n{\n"
             "    const uint32_t mask = (uint32_t)cap_mask;   /* (tables have below 2^31 slots) */\n"
             "    uint32_t pos = hash & mask;\n"
             "    const uint32_t bound = SMEM ? XB_SM_PROBES - 1 : XB_PROBE_LIMIT;\n"
             "    const uint32_t limit = mask < bound ? mask : bound;\n"
             "    for (uint32_t probe = 0; probe <= limit; probe++) {\n"
             "        char *e = SMEM ? entries + pos * XBJ_SM_STRIDE : entries + (uint64_t)pos * XBJ_GENT_SIZE;\n"
             "        xb_gent_head *h = (xb_gent_head *)e;\n"
             "        uint32_t s = SMEM ? xb_ld_acquire_cta(&h->state) : xb_ld_acquire(&h->state);\n"
             "        if (s == XB_GSTATE_EMPTY) {\n"
             "            const int rc = xbj_group_claim(e, hash, SMEM ? nullptr : E.gt, E.st, xbj_counter(E)";
        for (uint32_t k = 0; k < p->nkeys; k++) {
            const int r = p->keys[k].reg;
            o << ", " << V(r) << ", " << A(r) << ", " << N(r);
        }
        o << ");\n"
             "            if (rc == 1) return e;\n"
             "            if (rc == 2) return nullptr;\n"
             "            s = SMEM ? xb_ld_acquire_cta(&h->state) : xb_ld_acquire(&h->state);\n"
             "        }\n"
             "        uint32_t spins = 0;\n"
             "        while (s == XB_GSTATE_BUSY) {\n"
             "            if (++spins > E.plan->wait_limit) {\n"
             "                XB_RAISE(E.st, ERRCODE_DEVICE_ERROR, XB_MSG_WAIT_TIMEOUT);\n"
             "                return nullptr;\n            }\n"
             "            __nanosleep(20);\n"
             "            s = SMEM ? xb_ld_acquire_cta(&h->state) : xb_ld_acquire(&h->state);\n"
             "        }\n"
             "        if (h->hash == hash && xbj_key_match(e, R))\n            return e;\n"
             "        pos = (pos + 1) & mask;\n"
             "    }\n"
             "    *full = true;\n    return nullptr;\n}\n\n";

        if (p->has_groupby == 2) {
            accumulators();
            shared_form();
            return;
        }
        /* state updates of the global table's entries: the lanes are spread
         * over many entries (combining them per entry would run once per
         * distinct entry with the other lanes idle), so each lane updates
         * its entry directly.  The sums whose old value is needed are all
         * added before the first of these values is looked at: a lane waits
         * for the table once, not once a sum (2M rows, every statistic, 3000
         * groups: 972 -> 958 us a query, 933 with the minima and maxima below) */
        std::ostringstream late;
        o << "__device__ __forceinline__ void xbj_update(char *e, const XbjRegs &R, const XbjEnv &E)\n{\n"
             "    (void)E;\n" << numeric_args();
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0)
                continue;
            const AggExpr x = agg_expr(a);
            const std::string S = "(e + " + std::to_string(a.state_off) + ")";
            if (returning_update(a, i, S, x.c, x.xd, x.yd, late))
                continue;
            o << "    { /* aggregate " << i << ": action " << a.action << " */\n";
            direct_update(a, S, x.f, x.c);
            o << "    }\n";
        }
        o << late.str() << "}\n\n";
        shared_form();
    }

    /* per-lane update of an action whose sums need the value that the
     * addition found (the rounding error of a float sum, the carry of a
     * 128-bit one): the additions to o, what follows from the old values to
     * late; false for other actions */
    bool returning_update(const xb_agg &a, uint32_t i, const std::string &S, std::string c, const std::string &xd,
                          const std::string &yd, std::ostringstream &late)
    {
        const std::string I = std::to_string(i);
        std::vector<std::string> sums;      /* float sums, 16 bytes apart from byte 8 */
        switch (a.action) {
        case KAGG_ACTION__PMIN_INT32: case KAGG_ACTION__PMIN_INT64: case KAGG_ACTION__PMIN_FP64:
        case KAGG_ACTION__PMAX_INT32: case KAGG_ACTION__PMAX_INT64: case KAGG_ACTION__PMAX_FP64: {
            /* a relaxed read of the value, and a reduction only where the
             * row changes it (a value read too early only costs one).  The
             * flag belongs to the first row: as long as the value is what a
             * group starts with */
            const bool is_min = a.action == KAGG_ACTION__PMIN_INT32 || a.action == KAGG_ACTION__PMIN_INT64 ||
                                a.action == KAGG_ACTION__PMIN_FP64;
            const bool fp = a.action == KAGG_ACTION__PMIN_FP64 || a.action == KAGG_ACTION__PMAX_FP64;
            const std::string val = fp ? "(long long)xb_f64_ordered(" + xd + ")" : "(long long)" + V(a.arg0);
            o << "    long long o" << I << " = 0; /* aggregate " << i << ": action " << a.action << " */\n"
              << "    if (" << c << ") o" << I << " = (long long)xb_ld_relaxed_u64(" << S << ");\n";
            late << "    if (" << c << ") {\n"
                    "        if (o" << I << " == " << (is_min ? "INT64_MAX" : "INT64_MIN") << ") xb_red_g_or_u32(" << S << " + 8, 1u);\n"
                    "        if (" << val << (is_min ? " < o" : " > o") << I << ") "
                 << (is_min ? "xb_red_g_min_s64" : "xb_red_g_max_s64") << "(" << S << ", " << val << ");\n"
                    "    }\n";
            return true;
        }
        case KAGG_ACTION__PSUM_FP: case KAGG_ACTION__PAVG_FP:
            sums = {xd};
            break;
        case KAGG_ACTION__STDDEV:
            sums = {xd, xd + " * " + xd};
            break;
        case KAGG_ACTION__COVAR:
            sums = {xd, xd + " * " + xd, yd, yd + " * " + yd, xd + " * " + yd};
            c += " && !" + N(a.arg1);
            break;
        case KAGG_ACTION__PSUM_INT64: case KAGG_ACTION__PAVG_INT64:
        case KAGG_ACTION__PSUM_NUMERIC: case KAGG_ACTION__PAVG_NUMERIC: {
            const bool num = is_numeric_sum(a);
            const std::string v = num ? "x" + num_id(a) : "(xb_i128)(int64_t)" + V(a.arg0);
            const std::string put = num ? "k" + num_id(a) + " == XB_NUM_VALID" : "true";
            o << "    uint64_t o" << I << " = 0; /* aggregate " << i << ": action " << a.action << " */\n"
              << "    if (" << c << ") {\n"
              << "        if (" << put << ") {\n"
              << "            xb_red_g_add_u64(" << S << ", 1ULL);\n"
              << "            o" << I << " = xb_atom_g_add_u64(" << S << " + 8, (uint64_t)(" << v << "));\n"
              << "        }";
            if (num)
                o << " else {\n            xb_red_g_or_u32(" << S << " + 24, xb_numeric_special(k" << num_id(a) << "));\n"
                     "        }";
            o << "\n    }\n";
            late << "    if (" << c << " && " << put << ") xb_i128_carry_g(" << S << " + 16, o" << I << ", " << v << ");\n";
            return true;
        }
        default:
            return false;
        }
        o << "    double";
        for (size_t k = 0; k < sums.size(); k++)
            o << (k ? ", o" : " o") << I << "_" << k << " = 0.0";
        o << "; /* aggregate " << i << ": action " << a.action << " */\n"
          << "    if (" << c << ") {\n"
          << "        xb_red_g_add_u64(" << S << ", 1ULL);\n";
        late << "    if (" << c << ") {\n";
        for (size_t k = 0; k < sums.size(); k++) {
            o << "        o" << I << "_" << k << " = xb_atom_g_add_f64(" << S << " + " << 8 + 16 * k << ", " << sums[k] << ");\n";
            late << "        xb_f64c_err_g(" << S << " + " << 16 + 16 * k << ", o" << I << "_" << k << ", " << sums[k] << ");\n";
        }
        o << "    }\n";
        late << "    }\n";
        return true;
    }

    /* an update's numeric arguments, each decoded once per scale however
     * many sums and averages take it (k<r>_<w>: its kind, x<r>_<w>: its
     * value) */
    static bool is_numeric_sum(const xb_agg &a)
    {
        return a.action == KAGG_ACTION__PSUM_NUMERIC || a.action == KAGG_ACTION__PAVG_NUMERIC;
    }
    static std::string num_id(const xb_agg &a)
    {
        return std::to_string(a.arg0) + (a.weight < 0 ? "_m" : "_") + std::to_string(a.weight < 0 ? -a.weight : a.weight);
    }
    std::string numeric_args() const
    {
        std::ostringstream r;
        std::vector<std::string> seen;
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0 || !is_numeric_sum(a) ||
                std::find(seen.begin(), seen.end(), num_id(a)) != seen.end())
                continue;
            const std::string id = num_id(a);
            seen.push_back(id);
            /* for the rows that any of them counts */
            std::string any;
            for (uint32_t k = i; k < p->naggs; k++)
                if (p->aggs[k].state_sz && is_numeric_sum(p->aggs[k]) && num_id(p->aggs[k]) == id)
                    any += (any.empty() ? "" : " || ") + agg_expr(p->aggs[k]).c;
            r << "    uint8_t k" << id << " = XB_NUM_VALID; xb_i128 x" << id << " = 0;\n"
                 "    if ((" << any << ") && xb_numeric_sum_value((const uint8_t *)" << V(a.arg0) << ", " << a.weight
              << ", &k" << id << ", &x" << id << ")) {\n"
                 "        XB_RAISE(E.st, ERRCODE_DEVICE_ERROR, XB_MSG_NUMERIC_CORRUPT);\n"
                 "        return;\n    }\n";
        }
        return r.str();
    }

    /* C++ expressions of an aggregate: its filter (f), the condition under
     * which a row counts (c), its arguments as double (xd, yd) */
    struct AggExpr { std::string f, c, xd, yd; };
    AggExpr agg_expr(const xb_agg &a) const
    {
        auto dbl = [&](int r) {
            return p->rk[r] == XB_RK_FLT ? "__longlong_as_double(" + V(r) + ")" : "(double)(int64_t)" + V(r);
        };
        AggExpr x;
        x.f = a.filter >= 0 ? "(!" + N(a.filter) + " && " + V(a.filter) + " != 0)" : "true";
        x.c = a.arg0 >= 0 ? "(" + x.f + " && !" + N(a.arg0) + ")" : x.f;
        x.xd = a.arg0 >= 0 ? dbl(a.arg0) : "0.0";
        x.yd = a.action == KAGG_ACTION__COVAR ? dbl(a.arg1) : "0.0";
        return x;
    }

    /* ---- no GROUP BY keys: every row belongs to the one group, so a lane
     * keeps its rows' aggregate in registers over the whole launch; at its
     * end the lanes of a warp are combined and one lane adds the warp's
     * aggregate to the group's entry.  (Combining the lanes of every
     * 32-row batch took 31 shuffles per aggregate: 20M rows, 7 aggregates,
     * 3.42 ms a query, 2.50 ms now.)  Floating sums keep a
     * compensation per lane (TwoSum), added up with the others'. */
    void accumulators()
    {
        std::ostringstream decl, init, row, put, sums, carry;
        /* the rows that satisfy a condition, counted once however many
         * aggregates take the count.  Scans count in 32 bits and carry into
         * 64 (in local memory) where the lane's statistics are flushed, at
         * 2^31 rows (20M rows, 7 aggregates: 847 us a query; 867 with 64-bit
         * counters, 887 with one for each aggregate).  A join yields any
         * number of rows between two such looks: 64 bits.  Returns the name
         * of the warp's sum */
        std::vector<std::string> conds;
        auto counter = [&](const std::string &cond) {
            const size_t k = std::find(conds.begin(), conds.end(), cond) - conds.begin();
            const std::string K = std::to_string(k), n = "n" + K;
            if (k == conds.size()) {
                conds.push_back(cond);
                decl << (p->nrels ? "    unsigned long long " : "    uint32_t ") << n << ";\n";
                init << "    A." << n << " = 0; carried[" << K << "] = 0;\n";
                row << "    if (" << cond << ") A." << n << "++;\n";
                carry << "    carried[" << K << "] += A." << n << "; A." << n << " = 0;\n";
                sums << "    const unsigned long long " << n << "_ = xbj_warp_sum(carried[" << K << "] + A." << n << ");\n";
            }
            return n + "_";
        };
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0)
                continue;
            const AggExpr x = agg_expr(a);
            const std::string I = std::to_string(i), s = "A.s" + I, c2 = "A.c" + I;
            const std::string S = "(e + " + std::to_string(a.state_off) + ")";
            const bool is_min = a.action == KAGG_ACTION__PMIN_INT32 || a.action == KAGG_ACTION__PMIN_INT64 ||
                                a.action == KAGG_ACTION__PMIN_FP64;
            switch (a.action) {
            case KAGG_ACTION__NROWS_ANY: case KAGG_ACTION__NROWS_COND: {
                const std::string n = counter(a.action == KAGG_ACTION__NROWS_ANY ? x.f : x.c);
                put << "    if (leader && " << n << ") atomicAdd((unsigned long long *)" << S << ", " << n << ");\n";
                break;
            }
            case KAGG_ACTION__PMIN_INT32: case KAGG_ACTION__PMIN_INT64: case KAGG_ACTION__PMIN_FP64:
            case KAGG_ACTION__PMAX_INT32: case KAGG_ACTION__PMAX_INT64: case KAGG_ACTION__PMAX_FP64: {
                const bool fp = a.action == KAGG_ACTION__PMIN_FP64 || a.action == KAGG_ACTION__PMAX_FP64;
                const std::string mm = is_min ? "min" : "max";
                decl << "    long long s" << I << ";\n";
                init << "    " << s << " = " << (is_min ? "INT64_MAX" : "INT64_MIN") << ";\n";
                const std::string n = counter(x.c);
                row << "    if (" << x.c << ") " << s << " = " << mm << "(" << s << ", "
                    << (fp ? "(long long)xb_f64_ordered(" + x.xd + ")" : "(long long)" + V(a.arg0)) << ");\n";
                put << "    {\n"
                       "        for (int o_ = 16; o_ > 0; o_ >>= 1)\n"
                       "            " << s << " = " << mm << "(" << s << ", __shfl_xor_sync(XB_FULL, " << s << ", o_));\n"
                       "        if (leader && " << n << ") {\n"
                       "            atomicOr((unsigned int *)(" << S << " + 8), 1u);\n"
                       "            " << (is_min ? "atomicMin" : "atomicMax") << "((long long *)" << S << ", " << s << ");\n"
                       "        }\n    }\n";
                break;
            }
            case KAGG_ACTION__PSUM_INT: case KAGG_ACTION__PAVG_INT: {
                const std::string n = counter(x.c);
                decl << "    unsigned long long s" << I << ";\n";
                init << "    " << s << " = 0;\n";
                row << "    if (" << x.c << ") " << s << " += (unsigned long long)" << V(a.arg0) << ";\n";
                put << "    {\n"
                       "        const unsigned long long s_ = xbj_warp_sum(" << s << ");\n"
                       "        if (leader && " << n << ") {\n"
                       "            atomicAdd((unsigned long long *)" << S << ", " << n << ");\n"
                       "            atomicAdd((unsigned long long *)(" << S << " + 8), s_);\n"
                       "        }\n    }\n";
                break;
            }
            case KAGG_ACTION__PSUM_INT64: case KAGG_ACTION__PAVG_INT64:
            case KAGG_ACTION__PSUM_NUMERIC: case KAGG_ACTION__PAVG_NUMERIC: {
                const bool num = a.action == KAGG_ACTION__PSUM_NUMERIC || a.action == KAGG_ACTION__PAVG_NUMERIC;
                const std::string n = counter(num ? x.c + " && k" + num_id(a) + " == XB_NUM_VALID" : x.c);
                decl << "    xb_i128 s" << I << ";\n";
                init << "    " << s << " = 0;\n";
                if (num) {
                    decl << "    uint32_t c" << I << ";\n";
                    init << "    " << c2 << " = 0;\n";
                    const std::string id = num_id(a);
                    row << "    if (" << x.c << ") {\n"
                           "        if (k" << id << " == XB_NUM_VALID) " << s << " += x" << id << ";\n"
                           "        else " << c2 << " |= xb_numeric_special(k" << id << ");\n    }\n";
                } else {
                    row << "    if (" << x.c << ") " << s << " += (xb_i128)(int64_t)" << V(a.arg0) << ";\n";
                }
                put << "    {\n"
                       "        for (int o_ = 16; o_ > 0; o_ >>= 1) {\n"
                       "            const unsigned long long l_ = __shfl_xor_sync(XB_FULL, (unsigned long long)" << s << ", o_);\n"
                       "            const unsigned long long h_ = __shfl_xor_sync(XB_FULL, "
                       "(unsigned long long)((unsigned __int128)" << s << " >> 64), o_);\n"
                       "            " << s << " += (xb_i128)(((unsigned __int128)h_ << 64) | l_);\n"
                       "        }\n"
                       "        if (leader && " << n << ") {\n"
                       "            atomicAdd((unsigned long long *)" << S << ", " << n << ");\n"
                       "            xb_atomic_add_i128((uint64_t *)(" << S << " + 8), " << s << ");\n"
                       "        }\n";
                if (num)
                    put << "        const uint32_t sp_ = __reduce_or_sync(XB_FULL, " << c2 << ");\n"
                           "        if (leader && sp_) atomicOr((unsigned int *)(" << S << " + 24), sp_);\n";
                put << "    }\n";
                break;
            }
            case KAGG_ACTION__PSUM_FP: case KAGG_ACTION__PAVG_FP:
            case KAGG_ACTION__STDDEV: case KAGG_ACTION__COVAR: {
                std::string cond = x.c;
                std::vector<std::string> val = {"x_"};
                if (a.action == KAGG_ACTION__STDDEV)
                    val = {"x_", "x_ * x_"};
                if (a.action == KAGG_ACTION__COVAR) {
                    val = {"x_", "x_ * x_", "y_", "y_ * y_", "x_ * y_"};
                    cond += " && !" + N(a.arg1);
                }
                const std::string n = counter(cond);
                row << "    if (" << cond << ") {\n        const double x_ = " << x.xd << ";\n";
                if (a.action == KAGG_ACTION__COVAR)
                    row << "        const double y_ = " << x.yd << ";\n";
                put << "    {\n"
                       "        if (leader && " << n << ") atomicAdd((unsigned long long *)" << S << ", " << n << ");\n";
                for (size_t k = 0; k < val.size(); k++) {
                    const std::string K = I + "_" + std::to_string(k);
                    decl << "    double s" << K << ", c" << K << ";\n";
                    init << "    A.s" << K << " = A.c" << K << " = 0.0;\n";
                    row << "        xbj_two_sum(A.s" << K << ", A.c" << K << ", " << val[k] << ");\n";
                    put << "        xbj_warp_two_sum(A.s" << K << ", A.c" << K << ");\n"
                           "        if (leader && " << n << ") {\n"
                           "            xb_atomic_add_f64c((double *)(" << S << " + " << 8 + 16 * k << "), (double *)(" << S
                        << " + " << 16 + 16 * k << "), A.s" << K << ");\n"
                           "            if (fabs(A.c" << K << ") > 0.0) atomicAdd((double *)(" << S << " + " << 16 + 16 * k
                        << "), A.c" << K << ");\n"
                           "        }\n";
                }
                row << "    }\n";
                put << "    }\n";
                break;
            }
            default:
                break;
            }
        }
        acc_decl = decl.str();
        acc_counters = conds.size();
        o << "__device__ __forceinline__ void xbj_acc_init(XbjAcc &A, volatile unsigned long long *carried)\n{\n"
             "    (void)carried;\n    A.rows = 0;\n" << init.str() << "}\n\n"
             "__device__ __forceinline__ void xbj_acc_carry(XbjAcc &A, volatile unsigned long long *carried)\n{\n"
             "    (void)carried;\n" << carry.str() << "}\n\n"
             "__device__ __forceinline__ void xbj_acc_row(XbjAcc &A, const XbjRegs &R, const XbjEnv &E)\n{\n"
             "    (void)E;\n    A.rows = 1;\n" << numeric_args() << row.str() << "}\n\n"
             "__device__ __forceinline__ void xbj_acc_put(XbjAcc &A, volatile unsigned long long *carried, char *e, "
             "const bool leader)\n{\n    (void)carried;\n" << sums.str() << put.str() << "}\n\n"
             /* all lanes of the warp */
             "__device__ __forceinline__ void xbj_acc_flush(XbjAcc &A, volatile unsigned long long *carried, const XbjEnv &E)\n{\n"
             "    if (!__any_sync(XB_FULL, A.rows != 0)) return;\n"
             "    unsigned long long ep_ = 0;\n"
             "    if (E.lane == 0) {\n"
             "        XbjRegs R;\n"
             "        bool full = false;\n"
             "        char *e = E.sm_tab ? xbj_group_get<true>(R, E, E.sm_tab, E.sm_mask, 0, &full) : nullptr;\n"
             "        if (!e) e = xbj_group_get<false>(R, E, E.gt_entries, E.gt_mask, 0, &full);\n"
             "        ep_ = (unsigned long long)e;\n"
             "    }\n"
             "    ep_ = __shfl_sync(XB_FULL, ep_, 0);\n"
             "    if (ep_) xbj_acc_put(A, carried, (char *)ep_, E.lane == 0);\n"
             "}\n\n";
    }
    std::string acc_decl;
    size_t acc_counters = 0;

    /* ---- the shared-memory table's state form ------------------------
     * Entries of the CTA's shared table (group ids, or keyed groups that
     * fit) keep their states in a cheaper form than the global table's,
     * converted when the CTA merges them (xbj_merge_sm):
     *   - one unconditional count(*) of the entry is the row counter;
     *     every other count holds the rows it did NOT count (NULL argument,
     *     false filter, special numeric), so it is touched only for those;
     *   - counters are 32-bit native shared atomics (64-bit shared atomics
     *     are not native); integer and numeric sums are added word by word
     *     with them (a small positive value costs one atomic), except that
     *     a 64-bit sum of int8 values keeps the sum of the low 32 bits and
     *     the sum of the high halves apart.
     * Word-added sums are the two's complement words of the standard sum,
     * so they merge as they are.  Without keys (one entry, a warp's rows
     * added at once) the standard form is kept. */
    int rows_agg() const
    {
        if (p->has_groupby != 1)
            return -1;
        for (uint32_t i = 0; i < p->naggs; i++)
            if (p->aggs[i].action == KAGG_ACTION__NROWS_ANY && p->aggs[i].filter < 0 && p->aggs[i].state_sz > 0)
                return (int)i;
        return -1;
    }
    /* agg i keeps "rows not counted" in its count field */
    bool nc_form(uint32_t i) const
    {
        const int r = rows_agg();
        if (r < 0 || (int)i == r)
            return false;
        switch (p->aggs[i].action) {
        case KAGG_ACTION__NROWS_ANY: case KAGG_ACTION__NROWS_COND:
        case KAGG_ACTION__PSUM_INT: case KAGG_ACTION__PAVG_INT:
        case KAGG_ACTION__PSUM_INT64: case KAGG_ACTION__PAVG_INT64:
        case KAGG_ACTION__PSUM_FP: case KAGG_ACTION__PAVG_FP:
        case KAGG_ACTION__PSUM_NUMERIC: case KAGG_ACTION__PAVG_NUMERIC:
            return true;
        default:
            return false;
        }
    }

    void shared_form()
    {
        const int R = rows_agg();
        if (p->has_groupby == 1)
            update_shared(R);
        merge_shared(R);
    }

    void update_shared(const int R)
    {
        o << "__device__ __forceinline__ void xbj_update_sm(char *e, const XbjRegs &R, const XbjEnv &E)\n{\n"
             "    (void)E;\n" << numeric_args();
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0)
                continue;
            const std::string S = "(e + " + std::to_string(a.state_off) + ")";
            const AggExpr x = agg_expr(a);
            const std::string &f = x.f, &c = x.c, &xd = x.xd;
            const bool nc = nc_form(i);
            const std::string cond = a.action == KAGG_ACTION__NROWS_ANY ? f : c;
            /* the count: rows not counted (nc), or rows counted */
            const std::string cnt = nc ? "if (!(" + cond + ")) xb_red_shared_add_u32(" + S + ", 1u);\n"
                                       : "if (" + cond + ") xb_red_shared_add_u32(" + S + ", 1u);\n";
            o << "    { /* aggregate " << i << ": action " << a.action << " (shared form) */\n";
            if ((int)i == R) {
                o << "        xb_red_shared_add_u32(" << S << ", 1u);\n    }\n";
                continue;
            }
            switch (a.action) {
            case KAGG_ACTION__NROWS_ANY: case KAGG_ACTION__NROWS_COND:
                o << "        " << cnt;
                break;
            case KAGG_ACTION__PSUM_INT: case KAGG_ACTION__PAVG_INT:
                o << "        " << cnt
                  << "        if (" << c << ") xb_shared_add_u64w(" << S << " + 8, (uint64_t)" << V(a.arg0) << ");\n";
                break;
            case KAGG_ACTION__PSUM_INT64: case KAGG_ACTION__PAVG_INT64:
                /* the 64-bit sum kept as the sum of the values' low 32 bits
                 * plus the sum of their high halves: additions that need no
                 * returned value, the second only for values beyond 32 bits
                 * (measured faster than word atomics with carries here) */
                o << "        " << cnt
                  << "        if (" << c << ") {\n"
                     "            const long long v_ = (long long)" << V(a.arg0) << ";\n"
                     "            atomicAdd((unsigned long long *)(" << S << " + 8), (unsigned long long)(uint32_t)v_);\n"
                     "            const long long h_ = v_ >> 32;\n"
                     "            if (h_) atomicAdd((unsigned long long *)(" << S << " + 16), (unsigned long long)h_);\n"
                     "        }\n";
                break;
            case KAGG_ACTION__PSUM_FP: case KAGG_ACTION__PAVG_FP:
                o << "        " << cnt
                  << "        if (" << c << ") xb_atomic_add_f64c((double *)(" << S << " + 8), (double *)(" << S
                  << " + 16), " << xd << ");\n";
                break;
            case KAGG_ACTION__PSUM_NUMERIC: case KAGG_ACTION__PAVG_NUMERIC:
                /* the helper counts valid values (or, with nc, special ones) */
                if (nc)
                    o << "        if (!(" << c << ")) xb_red_shared_add_u32(" << S << ", 1u);\n";
                o << "        if (" << c << ") xb_agg_numeric_put_sm(" << S << ", k" << num_id(a) << ", x" << num_id(a)
                  << ", " << (nc ? "true" : "false") << ");\n";
                break;
            case KAGG_ACTION__PMIN_INT32: case KAGG_ACTION__PMIN_INT64: case KAGG_ACTION__PMIN_FP64:
            case KAGG_ACTION__PMAX_INT32: case KAGG_ACTION__PMAX_INT64: case KAGG_ACTION__PMAX_FP64: {
                /* the entry is shared memory: atomics through the generic
                 * address (the global-memory reductions of direct_update
                 * would be given an address outside their state space) */
                const bool is_min = a.action == KAGG_ACTION__PMIN_INT32 || a.action == KAGG_ACTION__PMIN_INT64 ||
                                    a.action == KAGG_ACTION__PMIN_FP64;
                const bool fp = a.action == KAGG_ACTION__PMIN_FP64 || a.action == KAGG_ACTION__PMAX_FP64;
                const std::string val = fp ? "(long long)xb_f64_ordered(" + xd + ")" : "(long long)" + V(a.arg0);
                o << "        if (" << c << ") {\n"
                     "            atomicOr((unsigned int *)(" << S << " + 8), 1u);\n"
                     "            " << (is_min ? "atomicMin" : "atomicMax") << "((long long *)" << S << ", " << val << ");\n"
                     "        }\n";
                break;
            }
            default:
                /* stddev, covariance: the helpers, which use generic atomics */
                helper_update(a, S, c, xd, agg_expr(a).yd);
                break;
            }
            o << "    }\n";
        }
        o << "}\n\n";
    }

    /* merge of a shared entry e into global entry g */
    void merge_shared(const int R)
    {
        o << "__device__ __noinline__ void xbj_merge_sm(char *g, const char *e)\n{\n";
        if (R >= 0)
            o << "    const unsigned long long rows_ = *(const unsigned long long *)(e + " << p->aggs[R].state_off << ");\n";
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0)
                continue;
            const std::string off = std::to_string(a.state_off);
            const std::string D = "(g + " + off + ")", S = "(e + " + off + ")";
            o << "    { /* aggregate " << i << " */\n"
                 "        const unsigned long long *su = (const unsigned long long *)" << S << ";\n"
                 "        const unsigned long long cnt = " << (nc_form(i) ? "rows_ - su[0]" : "su[0]") << ";\n"
                 "        (void)cnt;\n";
            switch (a.action) {
            case KAGG_ACTION__NROWS_ANY: case KAGG_ACTION__NROWS_COND:
                o << "        if (cnt) xb_red_g_add_u64(" << D << ", cnt);\n";
                break;
            case KAGG_ACTION__PSUM_INT: case KAGG_ACTION__PAVG_INT:
                o << "        if (cnt) {\n"
                     "            xb_red_g_add_u64(" << D << ", cnt);\n"
                     "            xb_red_g_add_u64(" << D << " + 8, su[1]);\n"
                     "        }\n";
                break;
            case KAGG_ACTION__PMIN_INT32: case KAGG_ACTION__PMIN_INT64: case KAGG_ACTION__PMIN_FP64:
            case KAGG_ACTION__PMAX_INT32: case KAGG_ACTION__PMAX_INT64: case KAGG_ACTION__PMAX_FP64: {
                const bool is_min = a.action == KAGG_ACTION__PMIN_INT32 || a.action == KAGG_ACTION__PMIN_INT64 ||
                                    a.action == KAGG_ACTION__PMIN_FP64;
                o << "        if (*(const uint32_t *)(" << S << " + 8)) {\n"
                     "            xb_red_g_or_u32(" << D << " + 8, 1u);\n"
                     "            " << (is_min ? "xb_red_g_min_s64" : "xb_red_g_max_s64") << "(" << D << ", (long long)su[0]);\n"
                     "        }\n";
                break;
            }
            case KAGG_ACTION__PSUM_INT64: case KAGG_ACTION__PAVG_INT64:
                o << "        if (cnt) {\n"
                     "            xb_red_g_add_u64(" << D << ", cnt);\n"
                  << (p->has_groupby == 1
                      ? "            const xb_i128 t_ = ((xb_i128)(long long)su[2] << 32) + (xb_i128)su[1];\n"
                      : "            const xb_i128 t_ = (xb_i128)(((unsigned __int128)su[2] << 64) | su[1]);\n")
                  <<                     "            xb_atomic_add_i128_g((uint64_t *)(" << D << " + 8), t_);\n"
                     "        }\n";
                break;
            case KAGG_ACTION__PSUM_NUMERIC: case KAGG_ACTION__PAVG_NUMERIC:
                o << "        if (cnt) {\n"
                     "            xb_red_g_add_u64(" << D << ", cnt);\n"
                     "            xb_atomic_add_i128_g((uint64_t *)(" << D << " + 8), "
                     "(xb_i128)(((unsigned __int128)su[2] << 64) | su[1]));\n"
                     "        }\n";
                if (a.state_sz >= 32)
                    o << "        if (*(const uint32_t *)(" << S << " + 24)) xb_red_g_or_u32(" << D
                      << " + 24, *(const uint32_t *)(" << S << " + 24));\n";
                break;
            case KAGG_ACTION__PSUM_FP: case KAGG_ACTION__PAVG_FP:
            case KAGG_ACTION__STDDEV: case KAGG_ACTION__COVAR:
                /* count, then (sum, compensation) pairs */
                o << "        if (cnt) {\n"
                     "            xb_red_g_add_u64(" << D << ", cnt);\n";
                for (uint32_t k = 8; k + 16 <= a.state_sz; k += 16)
                    o << "            xb_atomic_add_f64c_g((double *)(" << D << " + " << k << "), (double *)(" << D << " + "
                      << k + 8 << "), *(const double *)(" << S << " + " << k << "));\n"
                         "            if (fabs(*(const double *)(" << S << " + " << k + 8 << ")) > 0.0) xb_red_g_add_f64("
                      << D << " + " << k + 8 << ", *(const double *)(" << S << " + " << k + 8 << "));\n";
                o << "        }\n";
                break;
            default:
                break;
            }
            o << "    }\n";
        }
        o << "}\n\n";
    }

    /* per-lane update of the actions kept in helpers (stddev, covariance):
     * the standard form */
    void helper_update(const xb_agg &a, const std::string &S, const std::string &c, const std::string &xd,
                       const std::string &yd)
    {
        switch (a.action) {
        case KAGG_ACTION__STDDEV:
            o << "        if (" << c << ") xb_agg_stddev_add(" << S << ", " << xd << ");\n";
            break;
        case KAGG_ACTION__COVAR:
            o << "        if (" << c << " && !" << N(a.arg1) << ") xb_agg_covar_add(" << S << ", " << xd << ", "
              << yd << ");\n";
            break;
        default:
            break;
        }
    }

    /* per-lane update of a count or an integer sum of an entry of the global
     * table (keyed groups: e is global memory, the updates are
     * fire-and-forget reductions) */
    void direct_update(const xb_agg &a, const std::string &S, const std::string &f, const std::string &c)
    {
        switch (a.action) {
        case KAGG_ACTION__NROWS_ANY:
            o << "        if (" << f << ") xb_red_g_add_u64(" << S << ", 1ULL);\n";
            break;
        case KAGG_ACTION__NROWS_COND:
            o << "        if (" << c << ") xb_red_g_add_u64(" << S << ", 1ULL);\n";
            break;
        case KAGG_ACTION__PSUM_INT: case KAGG_ACTION__PAVG_INT:
            o << "        if (" << c << ") {\n"
                 "            xb_red_g_add_u64(" << S << ", 1ULL);\n"
                 "            xb_red_g_add_u64(" << S << " + 8, (unsigned long long)" << V(a.arg0) << ");\n"
                 "        }\n";
            break;
        default:
            break;
        }
    }

    /* ---- joins and the leaf --------------------------------------- */
    /* the group key tuple of every row is numbered by the inner build */
    bool gid_mode() const
    {
        return p->has_groupby == 1 && p->gid_depth >= 1 && p->gid_depth <= p->nrels &&
               p->inner[p->gid_depth].gid_on;
    }

    /* partitioned aggregation: a keyed GROUP BY into the global table can
     * defer each row's group update as a record (the registers the update
     * reads) bucketed by the high bits of its table slot, replayed bucket
     * after bucket by xbj_replay */
    bool part_mode() const
    {
        /* not with heap pages staged in shared memory: text and numeric
         * registers then point into the warp's page buffer, which is
         * overwritten (or gone with the CTA) before the replay reads them */
        return p->has_groupby == 1 && !gid_mode() && !p->has_proj && p->nkeys > 0 &&
               part_regs().size() <= 31 && xb_jit_stage_bytes(format) == 0;
    }

    std::vector<int> part_regs() const
    {
        std::vector<int> r;
        auto add = [&](int x) {
            if (x >= 0 && std::find(r.begin(), r.end(), x) == r.end())
                r.push_back(x);
        };
        for (uint32_t k = 0; k < p->nkeys; k++)
            add(p->keys[k].reg);
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0)
                continue;
            add(a.arg0);
            add(a.arg1);
            add(a.filter);
        }
        return r;
    }

    /* keys whose aux word (text length) the group lookup reads */
    std::vector<int> part_aux_keys() const
    {
        std::vector<int> r;
        for (uint32_t k = 0; k < p->nkeys; k++)
            if (p->keys[k].rk == XB_RK_TEXT || p->keys[k].rk == XB_RK_NUM)
                r.push_back(p->keys[k].reg);
        return r;
    }

    /* record: hash (4) + NULL mask (4; bit 31 marks a record a replay left
     * for after the table grows) + values (8 each) + the aux words of text /
     * numeric keys (4 each); the key hash is in the record already, so
     * cached datum hashes are not.  Written and read as 16-byte words: every
     * store of a lane is a request to L2 of its own. */
    uint32_t part_rec_size() const
    {
        const size_t n = part_regs().size();
        return (uint32_t)((8 + 8 * n + 4 * part_aux_keys().size() + 15) & ~(size_t)15);
    }

    void part_helpers()
    {
        const std::vector<int> rr = part_regs(), ax = part_aux_keys();
        /* the record's 8-byte words */
        std::vector<std::string> w = {"((uint64_t)nm << 32) | ghash"};
        for (int r : rr)
            w.push_back(V(r));
        for (size_t k = 0; k < ax.size(); k += 2)
            w.push_back("(uint64_t)" + A(ax[k]) + (k + 1 < ax.size() ? " | ((uint64_t)" + A(ax[k + 1]) + " << 32)" : ""));
        if (w.size() & 1)
            w.push_back("0");
        o << "__device__ __forceinline__ void xbj_rec_store(char *rec, const XbjRegs &R, uint32_t ghash)\n{\n"
             "    uint32_t nm = 0;\n";
        for (size_t i = 0; i < rr.size(); i++)
            o << "    nm |= (" << N(rr[i]) << " ? 1u : 0u) << " << i << ";\n";
        for (size_t i = 0; i < w.size(); i += 2)
            o << "    ((ulonglong2 *)rec)[" << i / 2 << "] = make_ulonglong2(" << w[i] << ", " << w[i + 1] << ");\n";
        o << "}\n\n"
             "__device__ __forceinline__ void xbj_rec_load(const char *rec, XbjRegs &R, uint32_t &ghash)\n{\n";
        for (size_t i = 0; i < w.size(); i += 2)
            o << "    const ulonglong2 q" << i / 2 << " = ((const ulonglong2 *)rec)[" << i / 2 << "];\n";
        auto word = [&](size_t i) { return "q" + std::to_string(i / 2) + (i & 1 ? ".y" : ".x"); };
        o << "    const uint32_t nm = (uint32_t)(q0.x >> 32); (void)nm;\n"
             "    ghash = (uint32_t)q0.x;\n";
        for (size_t i = 0; i < rr.size(); i++)
            o << "    " << V(rr[i]) << " = " << word(1 + i) << "; " << A(rr[i]) << " = 0; " << N(rr[i]) << " = (nm >> " << i
              << ") & 1u;\n";
        for (size_t k = 0; k < ax.size(); k++)
            o << "    " << A(ax[k]) << " = (uint32_t)(" << word(1 + rr.size() + k / 2) << (k & 1 ? " >> 32" : "") << ");\n";
        o << "}\n\n";
    }

    /* the lookup in and update of a slice of the global table in shared
     * memory (global-form states): counts and integer sums by native 32-bit
     * atomics with carries, min and max only where they change something */
    void slice_helpers()
    {
        o << "__device__ __forceinline__ char *\n"
             "xbj_slice_get(const XbjRegs &R, const XbjEnv &E, char *slice, uint32_t pos, uint32_t nslots, uint32_t hash, "
             "bool &failed)\n{\n"
             "    for (uint32_t probe = 0; pos < nslots && probe <= XB_PROBE_LIMIT; probe++, pos++) {\n"
             "        char *e = slice + (size_t)pos * XBJ_GENT_SIZE;\n"
             "        xb_gent_head *h = (xb_gent_head *)e;\n"
             "        uint32_t s = xb_ld_acquire_cta(&h->state);\n"
             "        if (s == XB_GSTATE_EMPTY) {\n"
             "            const int rc = xbj_group_claim(e, hash, E.gt, E.st, E.newg";
        for (uint32_t k = 0; k < p->nkeys; k++) {
            const int r = p->keys[k].reg;
            o << ", " << V(r) << ", " << A(r) << ", " << N(r);
        }
        o << ");\n"
             "            if (rc == 1) return e;\n"
             "            if (rc == 2) { failed = true; return nullptr; }\n"
             "            s = xb_ld_acquire_cta(&h->state);\n"
             "        }\n"
             "        uint32_t spins = 0;\n"
             "        while (s == XB_GSTATE_BUSY) {\n"
             "            if (++spins > E.plan->wait_limit) {\n"
             "                XB_RAISE(E.st, ERRCODE_DEVICE_ERROR, XB_MSG_WAIT_TIMEOUT);\n"
             "                failed = true;\n"
             "                return nullptr;\n            }\n"
             "            __nanosleep(20);\n"
             "            s = xb_ld_acquire_cta(&h->state);\n"
             "        }\n"
             "        if (h->hash == hash && xbj_key_match(e, R))\n            return e;\n"
             "    }\n"
             "    return nullptr;\n}\n\n"
             "__device__ __forceinline__ void xbj_update_slice(char *e, const XbjRegs &R, const XbjEnv &E)\n{\n"
             "    (void)E;\n" << numeric_args();
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            if (a.state_sz == 0)
                continue;
            const AggExpr x = agg_expr(a);
            const std::string S = "(e + " + std::to_string(a.state_off) + ")";
            o << "    { /* aggregate " << i << ": action " << a.action << " */\n";
            switch (a.action) {
            case KAGG_ACTION__NROWS_ANY: case KAGG_ACTION__NROWS_COND:
                o << "        if (" << (a.action == KAGG_ACTION__NROWS_ANY ? x.f : x.c) << ") xb_shared_add_u64w(" << S << ", 1);\n";
                break;
            case KAGG_ACTION__PMIN_INT32: case KAGG_ACTION__PMIN_INT64: case KAGG_ACTION__PMIN_FP64:
            case KAGG_ACTION__PMAX_INT32: case KAGG_ACTION__PMAX_INT64: case KAGG_ACTION__PMAX_FP64: {
                const bool is_min = a.action == KAGG_ACTION__PMIN_INT32 || a.action == KAGG_ACTION__PMIN_INT64 ||
                                    a.action == KAGG_ACTION__PMIN_FP64;
                const bool fp = a.action == KAGG_ACTION__PMIN_FP64 || a.action == KAGG_ACTION__PMAX_FP64;
                o << "        if (" << x.c << ") {\n"
                     "            const long long v_ = " << (fp ? "(long long)xb_f64_ordered(" + x.xd + ")" : "(long long)" + V(a.arg0))
                  << ";\n"
                     "            if (!*(volatile uint32_t *)(" << S << " + 8)) atomicOr((unsigned int *)(" << S << " + 8), 1u);\n"
                     "            if (v_ " << (is_min ? "<" : ">") << " *(volatile long long *)" << S << ") "
                  << (is_min ? "atomicMin" : "atomicMax") << "((long long *)" << S << ", v_);\n"
                     "        }\n";
                break;
            }
            case KAGG_ACTION__PSUM_INT: case KAGG_ACTION__PAVG_INT:
                o << "        if (" << x.c << ") {\n"
                     "            xb_shared_add_u64w(" << S << ", 1);\n"
                     "            xb_shared_add_u64w(" << S << " + 8, (uint64_t)" << V(a.arg0) << ");\n        }\n";
                break;
            case KAGG_ACTION__PSUM_INT64: case KAGG_ACTION__PAVG_INT64:
                o << "        if (" << x.c << ") {\n"
                     "            xb_shared_add_u64w(" << S << ", 1);\n"
                     "            xb_shared_add_i128w(" << S << " + 8, (xb_i128)(int64_t)" << V(a.arg0) << ");\n        }\n";
                break;
            case KAGG_ACTION__PSUM_NUMERIC: case KAGG_ACTION__PAVG_NUMERIC:
                o << "        if (" << x.c << ") {\n"
                     "            if (k" << num_id(a) << " == XB_NUM_VALID) {\n"
                     "                xb_shared_add_u64w(" << S << ", 1);\n"
                     "                xb_shared_add_i128w(" << S << " + 8, x" << num_id(a) << ");\n"
                     "            } else {\n"
                     "                atomicOr((unsigned int *)(" << S << " + 24), xb_numeric_special(k" << num_id(a) << "));\n"
                     "            }\n        }\n";
                break;
            case KAGG_ACTION__PSUM_FP: case KAGG_ACTION__PAVG_FP:
                o << "        if (" << x.c << ") {\n"
                     "            xb_shared_add_u64w(" << S << ", 1);\n"
                     "            xb_atomic_add_f64c((double *)(" << S << " + 8), (double *)(" << S << " + 16), " << x.xd
                  << ");\n        }\n";
                break;
            default:
                helper_update(a, S, x.c, x.xd, x.yd);
                break;
            }
            o << "    }\n";
        }
        o << "}\n\n";
    }

    /* the group lookup and state update of one row */
    void group_row()
    {
        /* a group the global table has no room for takes an entry of the
         * dump region (merged into the grown table after the launch); a
         * replay, which cannot stop, leaves the row for after the growth
         * instead once the dump is used up (returns true) */
        o << "__device__ __forceinline__ bool\n"
             "xbj_group_row(XbjRegs &R, const XbjEnv &E, const uint32_t ghash, bool &failed)\n{\n"
             "    char *e = nullptr;\n"
             "    bool full = false;\n"
             "    if (E.sm_tab && *(volatile uint32_t *)E.sm_on) {\n"
             "        e = xbj_group_get<true>(R, E, E.sm_tab, E.sm_mask, ghash, &full);\n"
             "        if (!e && E.sm_trial) *(volatile uint32_t *)E.sm_on = 0;\n"
             "    }\n"
             "    const bool in_sm = e != nullptr;\n"
             "    if (!e) {\n"
             "        full = false;\n"
             "        e = xbj_group_get<false>(R, E, E.gt_entries, E.gt_mask, ghash, &full);\n"
             "        if (!e && full) {\n"
             "            char *slot_ = xb_dump_slot(E.gt, XBJ_GENT_SIZE);\n"
             "            if (slot_) {\n"
             "                full = false;\n"
             "                e = xbj_group_claim(slot_, ghash, E.gt, E.st, xbj_counter(E)";
        for (uint32_t k = 0; k < p->nkeys; k++) {
            const int r = p->keys[k].reg;
            o << ", " << V(r) << ", " << A(r) << ", " << N(r);
        }
        o << ") == 1 ? slot_ : nullptr;\n"
             "            }\n"
             "        }\n"
             "        if (!e && full) {\n"
             "            if (E.replay) { failed = true; return true; }\n"
             "            XB_RAISE(E.st, ERRCODE_SUSPEND_NO_SPACE, XB_MSG_GTABLE_FULL);\n"
             "            atomicOr(&E.gt->overflow, 1u);\n"
             "        }\n"
             "    }\n"
             "    if (!e) { failed = true; return false; }\n";
        o << "    if (in_sm) xbj_update_sm(e, R, E); else xbj_update(e, R, E);\n"
             "    return false;\n}\n\n";
    }

    /* device projection: form this row's kern_tupitem into kds_dst, with
     * the attribute layout resolved here (constant ld / attalign) */
    void projection_leaf(const std::string &ind)
    {
        program(p->proj_args, ind);
        o << ind << "if (failed) return;\n"
          << ind << "{ /* projection */\n";
        const std::string i2 = ind + "    ";
        const uint32_t n = p->proj_nattrs;
        o << i2 << "const uint32_t pn = 0u";
        for (uint32_t j = 0; j < n; j++)
            o << " | (" << N(p->proj[j].reg) << " ? " << (1u << j) << "u : 0u)";
        o << ";\n"
          << i2 << "const uint32_t hoff = xb_proj_hoff(" << n << "u, pn != 0);\n"
          << i2 << "uint16_t im = pn ? HEAP_HASNULL : 0;\n"
          << i2 << "uint32_t t = hoff;\n";
        auto attrs = [&](const char *base) {
            for (uint32_t j = 0; j < n; j++) {
                const xb_projcol &pc = p->proj[j];
                o << i2 << "if (!" << N(pc.reg) << ") t = xb_proj_attr(" << base << ", t, " << (int)pc.attalign
                  << ", " << (int)pc.ld << ", " << V(pc.reg) << ", " << A(pc.reg) << ", im);\n";
            }
        };
        attrs("nullptr");
        o << i2 << "const uint32_t tl = t + ROWID_SIZE;\n"
          << i2 << "uint32_t rowid;\n"
          << i2 << "char *tp = xb_proj_claim(E.dst, E.dst_len, " << p->proj_head_len << "ULL, xb_proj_rowsz(tl, "
          << p->proj_margin << "u), E.st, &rowid);\n"
          << i2 << "if (tp) {\n"
          << i2 << "    xb_proj_head(tp, " << n << "u, hoff, pn, tl, 0, im);\n"
          << i2 << "    t = hoff;\n";
        attrs("tp");
        o << i2 << "    xb_proj_tail(tp, tl, rowid);\n"
          << i2 << "    xb_proj_index(E.dst, E.dst_len, " << p->proj_head_len << "ULL, rowid, tp);\n"
          << i2 << "}\n"
          << ind << "}\n";
    }

    void leaf(const std::string &ind)
    {
        o << ind << "C.out++;\n";
        if (p->has_proj) {
            projection_leaf(ind);
            return;
        }
        if (!p->has_groupby)
            return;
        if (gid_mode()) {
            /* entry = shared table slot of the row's group id; the key hash
             * is computed only to create the entry */
            program(p->gb_args, ind);
            o << ind << "if (failed) return;\n"
              << ind << "char *e = xb_generic_ptr(E.sm_tab + (size_t)gid * XBJ_SM_STRIDE);\n"
              << ind << "xb_gent_head *gh = (xb_gent_head *)e;\n";
            /* with at most 64 groups every lane remembers which entries it
             * has seen ready (they stay ready) and skips their state load */
            const bool mask = p->inner[p->gid_depth].ngids <= 64;
            const std::string ind0 = ind;
            std::string ind1 = ind;
            if (mask) {
                o << ind << "const uint64_t gbit_ = 1ULL << gid;\n"
                  << ind << "if (!(C.gready & gbit_)) {\n";
                ind1 = ind + "    ";
            }
            o << ind1 << "uint32_t gs = xb_ld_acquire_cta(&gh->state);\n"
              << ind1 << "if (gs != XB_GSTATE_READY) {\n";
            const std::string i2 = ind1 + "    ";
            if (lazy_record(p->gid_depth)) {
                const uint32_t gd = p->gid_depth;
                const xb_inner &gin = p->inner[gd];
                const std::string G = std::to_string(gd);
                o << i2 << "const uint4 *grec_ = (const uint4 *)(E.plan->inner[" << gd << "].dpay + poff" << G << " * "
                  << gin.drec_size << "u);\n";
                for (uint32_t w = 0; w < gin.drec_size / 16; w++)
                    o << i2 << "const uint4 q" << G << "_" << w << " = __ldg(&grec_[" << w << "]);\n";
                record_regs(gd, gin, i2);
            }
            program(p->gb_keyhash, i2);
            o << i2 << "if (failed) return;\n"
              << i2 << "const uint32_t ghash = (uint32_t)" << V(p->gb_keyhash.result) << ";\n"
              << i2 << "if (gs == XB_GSTATE_EMPTY && xbj_group_claim(e, ghash, nullptr, E.st, nullptr";
            for (uint32_t k = 0; k < p->nkeys; k++) {
                const int r = p->keys[k].reg;
                o << ", " << V(r) << ", " << A(r) << ", " << N(r);
            }
            o << ") == 2) { failed = true; return; }\n"
              << i2 << "uint32_t spins = 0;\n"
              << i2 << "while ((gs = xb_ld_acquire_cta(&gh->state)) != XB_GSTATE_READY) {\n"
              << i2 << "    if (++spins > E.plan->wait_limit) {\n"
              << i2 << "        XB_RAISE(E.st, ERRCODE_DEVICE_ERROR, XB_MSG_WAIT_TIMEOUT);\n"
              << i2 << "        failed = true;\n"
              << i2 << "        return;\n"
              << i2 << "    }\n"
              << i2 << "    __nanosleep(20);\n"
              << i2 << "}\n"
              << ind1 << "}\n";
            if (mask)
                o << ind1 << "C.gready |= gbit_;\n" << ind0 << "}\n";
            o << ind0 << "xbj_update_sm(e, R, E);\n";
            return;
        }
        program(p->gb_all, ind);
        o << ind << "if (failed) return;\n";
        if (p->has_groupby == 2) {
            o << ind << "xbj_acc_row(C.acc, R, E);\n";
            return;
        }
        o << ind << "const uint32_t ghash = (uint32_t)" << V(p->gb_keyhash.result) << ";\n";
        if (part_mode()) {
            /* deferred: the row's record into the bucket of its slot, while
             * the bucket has room */
            o << ind << "bool deferred_ = false;\n"
              << ind << "if (E.part_buf) {\n"
              << ind << "    const uint32_t pp_ = (uint32_t)((ghash & E.gt_mask) >> E.part_shift);\n"
              << ind << "    const uint32_t slot_ = atomicAdd(&E.part_cnt[pp_ * XB_PART_CNT_STRIDE], 1u);\n"
              << ind << "    if (slot_ < E.part_cap) {\n"
              << ind << "        xbj_rec_store(E.part_buf + ((uint64_t)pp_ * E.part_cap + slot_) * XBJ_REC_SIZE, R, ghash);\n"
              << ind << "        deferred_ = true;\n"
              << ind << "    }\n"
              << ind << "}\n";
            o << ind << "if (!deferred_) xbj_group_row(R, E, ghash, failed);\n";
        } else {
            o << ind << "xbj_group_row(R, E, ghash, failed);\n";
        }
        o << ind << "if (failed) return;\n";
    }

    /* per matching inner row: load its live columns, run the join quals,
     * descend to the next depth */
    void inner_body(uint32_t d, const xb_inner &in, const std::string &i4)
    {
        const std::string D = std::to_string(d);
        const std::string W = "((n" + D + " + 31) / 32)";
        if (gid_mode() && d == p->gid_depth)
            o << i4 << "const uint32_t gid = __ldg(&in" << D << "->gids[row" << D << "]);\n";
        for (uint32_t k = 0; k < in.nloads; k++) {
            if (!((in.live >> k) & 1u))
                continue;
            const int r = in.load[k].reg;
            const std::string at = "(size_t)" + std::to_string(k) + " * n" + D + " + row" + D;
            o << i4 << V(r) << " = __ldg(&vals" << D << "[" << at << "]);\n";
            if (p->rk[r] == XB_RK_TEXT)
                o << i4 << A(r) << " = __ldg(&auxs" << D << "[" << at << "]);\n";
            if ((in.hashed >> k) & 1u)
                o << i4 << H(r) << " = __ldg(&hashes" << D << "[" << at << "]);\n";
            if ((in.hasnull >> k) & 1u)
                o << i4 << N(r) << " = ((__ldg(&nulls" << D << "[(size_t)" << k << " * " << W << " + row" << D
                  << " / 32]) >> (row" << D << " % 32)) & 1u) != 0;\n";
            else
                o << i4 << N(r) << " = false;\n";
        }
        inner_quals_and_descend(d, i4);
    }

    void inner_quals_and_descend(uint32_t d, const std::string &i4)
    {
        program(p->join_quals[d], i4);
        o << i4 << "if (failed) return;\n"
          << i4 << "if (" << pass_expr(p->join_quals[d]) << ") {\n"
          << i4 << "    C.depth[" << d << "]++;\n";
        depth(d + 1, i4 + "    ");
        o << i4 << "}\n";
    }

    void depth(uint32_t d, const std::string &ind)
    {
        if (d > p->nrels) {
            leaf(ind);
            return;
        }
        const xb_inner &in = p->inner[d];
        const std::string D = std::to_string(d);
        o << ind << "{ /* depth " << d << " */\n";
        const std::string i2 = ind + "    ";
        o << i2 << "const xb_inner *in" << D << " = &E.plan->inner[" << d << "];\n"
          << i2 << "const uint32_t n" << D << " = in" << D << "->nitems;\n"
          << i2 << "const uint32_t cap" << D << " = in" << D << "->cap_mask;\n"
          << i2 << "const unsigned long long *idx" << D << " = (const unsigned long long *)in" << D << "->index;\n"
          << i2 << "const unsigned long long *vals" << D << " = (const unsigned long long *)in" << D << "->vals;\n"
          << i2 << "const uint32_t *auxs" << D << " = in" << D << "->auxs;\n"
          << i2 << "const uint32_t *nulls" << D << " = in" << D << "->nulls;\n"
          << i2 << "const uint32_t *hashes" << D << " = in" << D << "->hashes;\n"
          << i2 << "(void)vals" << D << "; (void)auxs" << D << "; (void)nulls" << D << "; (void)hashes" << D << ";\n";
        const bool fused = in.fast_key >= 0;
        if (fused) {
            const int ox = in.fast_outer;
            o << i2 << "const uint64_t okey" << D << " = " << V(ox) << ";\n"
              << i2 << "bool live" << D << " = !" << N(ox) << ";\n";
            std::string hv;
            switch (in.fast_hk) {
            case XB_HK_W1: hv = "xb_hash_u32((uint32_t)okey" + D + ", 1)"; break;
            case XB_HK_W2: hv = "xb_hash_u32((uint32_t)okey" + D + ", 2)"; break;
            case XB_HK_W4: hv = "xb_hash_u32((uint32_t)okey" + D + ", 4)"; break;
            default:       hv = "xb_hash_u64(okey" + D + ")"; break;
            }
            o << i2 << "const uint32_t hash" << D << " = xb_hash_merge(0xffffffffU, " << hv << ") ^ 0xffffffffU;\n";
            if (in.key32)
                o << i2 << "const uint32_t tag" << D << " = (uint32_t)okey" << D << ";\n"
                  << i2 << "if ((int64_t)okey" << D << " != (int64_t)(int32_t)okey" << D << ") live" << D << " = false;\n";
            else
                o << i2 << "const uint32_t tag" << D << " = hash" << D << ";\n";
        } else {
            program(p->hash_value[d], i2);
            o << i2 << "if (failed) return;\n"
              << i2 << "const uint32_t hash" << D << " = (uint32_t)" << V(p->hash_value[d].result) << ";\n"
              << i2 << "const uint32_t tag" << D << " = hash" << D << ";\n"
              << i2 << "bool live" << D << " = true;\n";
        }
        if (fused && in.key32 && in.direct && in.unique_hash) {
            /* direct addressing: one 4-byte load, no hash, no probe loop */
            const bool pre = preloadable(d);
            o << i2 << "const uint32_t *dtab" << D << " = in" << D << "->dtab;\n"
              << i2 << "const uint64_t doff" << D << " = (uint64_t)((int64_t)okey" << D << " - " << DMIN(d) << ");\n"
              << i2 << "(void)tag" << D << "; (void)hash" << D << "; (void)cap" << D << "; (void)idx" << D << "; (void)dtab" << D << ";\n";
            if (pre)
                o << i2 << "if (plive" << D << ") {\n";
            else
                o << i2 << "if (live" << D << " && doff" << D << " < " << DRANGE(d) << ") {\n";
            const std::string j3 = i2 + "    ";
            if (lazy_record(d)) {
                /* present bit and group id only; the columns are read if
                 * this row creates its group (the leaf's claim path) */
                o << j3 << "if (ph" << D << ".x & 0x80000000u) {\n";
                const std::string j4 = j3 + "    ";
                o << j4 << "const uint32_t gid = ph" << D << ".y;\n";
                inner_quals_and_descend(d, j4);
                o << j3 << "}\n" << i2 << "}\n" << ind << "}\n";
                return;
            }
            if (in.dpay) {
                /* the row's live columns come with the probe: one record load */
                const uint32_t rs = in.drec_size;
                if (pre) {
                    for (uint32_t w = 0; w < rs / 16; w++)
                        o << j3 << "const uint4 q" << D << "_" << w << " = pq" << D << "_" << w << ";\n";
                } else {
                    o << j3 << "const uint4 *rec" << D << " = (const uint4 *)(in" << D << "->dpay + doff" << D << " * "
                      << rs << "u);\n";
                    for (uint32_t w = 0; w < rs / 16; w++)
                        o << j3 << "const uint4 q" << D << "_" << w << " = __ldg(&rec" << D << "[" << w << "]);\n";
                }
                o << j3 << "if (q" << D << "_0.x & 0x80000000u) {\n";
                const std::string j4 = j3 + "    ";
                auto word = [&](int off) {
                    const char *f[] = {"x", "y", "z", "w"};
                    return "q" + D + "_" + std::to_string(off / 16) + "." + f[(off % 16) / 4];
                };
                if (gid_mode() && d == p->gid_depth)
                    o << j4 << "const uint32_t gid = " << word(4) << ";\n";
                record_regs(d, in, j4);
                inner_quals_and_descend(d, j4);
                o << j3 << "}\n" << i2 << "}\n" << ind << "}\n";
                return;
            }
            if (pre)
                o << j3 << "const uint32_t r1_ = pr1" << D << ";\n";
            else
                o << j3 << "const uint32_t r1_ = __ldg(&dtab" << D << "[doff" << D << "]);\n";
            o << j3 << "if (r1_) {\n";
            const std::string j4 = j3 + "    ";
            o << j4 << "const uint32_t row" << D << " = r1_ - 1;\n";
            inner_body(d, in, j4);
            o << j3 << "}\n" << i2 << "}\n" << ind << "}\n";
            return;
        }
        /* the index is walked to the next row of the tag, two slots a load,
         * and the rest of the row's work comes after the walk: in its loop,
         * lanes that matched at different slots went through the depths
         * below one after another (10M rows joined to 100,000 keys of two
         * rows each, found through the index: 1466 us a query, 1234 us so
         * and with the live columns in one record per row) */
        o << i2 << "if (live" << D << " && n" << D << " > 0) {\n";
        const std::string i3 = i2 + "    ";
        o << i3 << "uint32_t pos" << D << " = hash" << D << " & cap" << D << ", steps" << D << " = 0;\n"
          << i3 << (in.unique_hash ? "{" : "for (;;) {") << "\n";
        const std::string i4 = i3 + "    ", i5 = i4 + "    ";
        const std::string W = "((n" + D + " + 31) / 32)";
        o << i4 << "uint32_t r1_" << D << " = 0;\n"
          << i4 << "bool end" << D << " = false;\n"
          << i4 << "do {\n"
          << i5 << "const ulonglong2 pr_ = __ldg((const ulonglong2 *)idx" << D << " + (pos" << D << " >> 1));\n"
          << i5 << "const bool even_ = !(pos" << D << " & 1u);\n"
          << i5 << "const bool hit0_ = even_ && pr_.x != 0 && (uint32_t)(pr_.x >> 32) == tag" << D << ";\n"
          << i5 << "const bool hit1_ = pr_.y != 0 && (uint32_t)(pr_.y >> 32) == tag" << D << ";\n"
          << i5 << "end" << D << " = (even_ && pr_.x == 0) || (!hit0_ && pr_.y == 0);\n"
          << i5 << "r1_" << D << " = hit0_ ? (uint32_t)pr_.x : (hit1_ && !end" << D << ") ? (uint32_t)pr_.y : 0u;\n"
          << i5 << "pos" << D << " = hit0_ ? pos" << D << " + 1 : ((pos" << D << " | 1u) + 1) & cap" << D << ";\n";
        if (fused && !in.key32) {
            /* the tag is the key's hash: compare the key */
            const int fk = in.fast_key;
            o << i5 << "if (r1_" << D << ") {\n"
              << i5 << "    const uint32_t row_ = r1_" << D << " - 1;\n"
              << i5 << "    const unsigned long long kv_ = __ldg(&vals" << D << "[(size_t)" << fk << " * n" << D << " + row_]);\n";
            if ((in.hasnull >> fk) & 1u)
                o << i5 << "    const bool kn_ = (__ldg(&nulls" << D << "[(size_t)" << fk << " * " << W
                  << " + row_ / 32]) >> (row_ % 32)) & 1u;\n";
            else
                o << i5 << "    const bool kn_ = false;\n";
            o << i5 << "    if (kn_ || kv_ != okey" << D << ") {\n"
              << i5 << "        r1_" << D << " = 0;\n";
            if (in.unique_hash)
                o << i5 << "        end" << D << " = true;   /* no other inner row has this tag */\n";
            o << i5 << "    }\n" << i5 << "}\n";
        }
        o << i4 << "} while (!r1_" << D << " && !end" << D << " && ++steps" << D << " <= cap" << D << ");\n"
          << i4 << (in.unique_hash ? "if (r1_" + D + ") {" : "if (!r1_" + D + ") break;\n" + i4 + "{") << "\n"
          << i5 << "const uint32_t row" << D << " = r1_" << D << " - 1;\n";
        if (in.dpay) {
            /* the row's live columns in one record */
            const uint32_t rs = in.drec_size;
            o << i5 << "const uint4 *rec" << D << " = (const uint4 *)(in" << D << "->dpay + (size_t)row" << D << " * "
              << rs << "u);\n";
            for (uint32_t w = 0; w < rs / 16; w++)
                o << i5 << "const uint4 q" << D << "_" << w << " = __ldg(&rec" << D << "[" << w << "]);\n";
            if (gid_mode() && d == p->gid_depth)
                o << i5 << "const uint32_t gid = q" << D << "_0.y;\n";
            record_regs(d, in, i5);
            inner_quals_and_descend(d, i5);
        } else {
            inner_body(d, in, i5);
        }
        o << i4 << "}\n" << i3 << "}\n" << i2 << "}\n" << ind << "}\n";
    }

    /* a direct-addressed depth probed with a key read from the source row:
     * its table entry can be loaded as soon as the row is decoded */
    /* does any program run after depth d's probe, or any aggregate's
     * argument, read one of depth d's live columns */
    bool regs_used_after(uint32_t d) const
    {
        const xb_inner &in = p->inner[d];
        uint64_t regs = 0;
        for (uint32_t k = 0; k < in.nloads; k++)
            if ((in.live >> k) & 1u)
                regs |= 1ULL << in.load[k].reg;
        auto uses = [&](const xb_prog &pg) {
            for (uint32_t i = pg.start; i < (uint32_t)pg.start + pg.count; i++) {
                const xb_insn &x = p->insns[i];
                if (((regs >> x.a) & 1u) || ((regs >> x.b) & 1u) || ((regs >> x.dst) & 1u))
                    return true;
            }
            return false;
        };
        for (uint32_t e = d; e <= p->nrels; e++)
            if (uses(p->join_quals[e]) || (e > d && uses(p->hash_value[e])))
                return true;
        if (uses(p->gb_args))
            return true;
        for (uint32_t i = 0; i < p->naggs; i++) {
            const xb_agg &a = p->aggs[i];
            /* grouping keys are read only when a row creates its group, and
             * the group-id depth reloads its record for that */
            if (a.action == KAGG_ACTION__VREF)
                continue;
            for (int r : {(int)a.arg0, (int)a.arg1, (int)a.filter})
                if (r >= 0 && ((regs >> r) & 1u))
                    return true;
        }
        return false;
    }

    /* the group-id depth's record: only its present bit and group id are
     * read per row; the key columns are read when a group is created */
    bool lazy_record(uint32_t d) const
    {
        return gid_mode() && d == p->gid_depth && p->inner[d].dpay && preloadable(d) && !regs_used_after(d);
    }

    /* assign depth d's live columns from record words q<d>_<w> */
    void record_regs(uint32_t d, const xb_inner &in, const std::string &ind)
    {
        const std::string D = std::to_string(d);
        auto word = [&](int off) {
            const char *f[] = {"x", "y", "z", "w"};
            return "q" + D + "_" + std::to_string(off / 16) + "." + f[(off % 16) / 4];
        };
        for (uint32_t k = 0; k < in.nloads; k++) {
            if (!((in.live >> k) & 1u))
                continue;
            const int r = in.load[k].reg;
            int ov, oa, oh;
            xb_drec_layout(&in, p->rk, (int)k, &ov, &oa, &oh);
            o << ind << V(r) << " = ((uint64_t)" << word(ov + 4) << " << 32) | " << word(ov) << ";\n";
            if (oa >= 0 && p->rk[r] == XB_RK_TEXT)
                o << ind << A(r) << " = " << word(oa) << ";\n";
            if (oh >= 0)
                o << ind << H(r) << " = " << word(oh) << ";\n";
            o << ind << N(r) << " = ((q" << D << "_0.x >> " << k << ") & 1u) != 0;\n";
        }
    }

    /* a filter-only direct depth probed through its existence bitmap in
     * shared memory */
    bool bits_depth(uint32_t d) const
    {
        const xb_inner &in = p->inner[d];
        return format == KDS_FORMAT_BLOCK && preloadable(d) && !in.dpay && in.live == 0 && in.dbits_words > 0;
    }
    bool any_bits() const
    {
        for (uint32_t d = 1; d <= p->nrels; d++)
            if (bits_depth(d))
                return true;
        return false;
    }

    /* the bitmaps go to shared memory one after another (sizes from the
     * plan at run time, so sessions of one plan shape share the kernel) */
    void bits_helpers()
    {
        o << "__device__ __forceinline__ uint32_t xbj_stage_bits(uint32_t *sb, const xb_plan *plan)\n{\n"
             "    uint32_t off = 0;\n";
        for (uint32_t d = 1; d <= p->nrels; d++) {
            if (!bits_depth(d))
                continue;
            o << "    {\n"
                 "        const uint32_t n_ = plan->inner[" << d << "].dbits_words;\n"
                 "        const uint32_t *g_ = plan->inner[" << d << "].dbits;\n"
                 "        for (uint32_t i = threadIdx.x; i < n_; i += blockDim.x)\n"
                 "            sb[off + i] = g_[i];\n"
                 "        off += n_;\n"
                 "    }\n";
        }
        o << "    return off * 4u;\n}\n\n";
        for (uint32_t d = 1; d <= p->nrels; d++) {
            if (!bits_depth(d))
                continue;
            o << "__device__ __forceinline__ uint32_t xbj_bits_off_" << d << "(const xb_plan *plan)\n{\n"
                 "    (void)plan;\n    return 0u";
            for (uint32_t e = 1; e < d; e++)
                if (bits_depth(e))
                    o << " + __ldg(&plan->inner[" << e << "].dbits_words)";
            o << ";\n}\n\n";
        }
    }

    bool preloadable(uint32_t d) const
    {
        const xb_inner &in = p->inner[d];
        if (in.fast_key < 0 || !in.key32 || !in.direct || !in.unique_hash)
            return false;
        for (uint32_t i = 0; i < p->nload0; i++)
            if (p->load0[i].reg == in.fast_outer)
                return true;
        return false;
    }

    /* issue the table loads of every preloadable depth together, so their
     * latencies overlap instead of adding up depth after depth */
    void preload_probes(const std::string &ind)
    {
        for (uint32_t d = 1; d <= p->nrels; d++) {
            if (!preloadable(d))
                continue;
            const xb_inner &in = p->inner[d];
            const std::string D = std::to_string(d);
            const int ox = in.fast_outer;
            o << ind << "const uint64_t poff" << D << " = (uint64_t)((int64_t)" << V(ox) << " - " << DMIN(d) << ");\n"
              << ind << "const bool plive" << D << " = !" << N(ox) << " && poff" << D << " < " << DRANGE(d) << ";\n";
            if (lazy_record(d)) {
                o << ind << "uint2 ph" << D << " = make_uint2(0u, 0u);\n"
                  << ind << "if (plive" << D << ")\n"
                  << ind << "    ph" << D << " = __ldg((const uint2 *)(E.plan->inner[" << d << "].dpay + poff" << D
                  << " * " << in.drec_size << "u));\n";
            } else if (in.dpay) {
                const uint32_t rs = in.drec_size;
                for (uint32_t w = 0; w < rs / 16; w++)
                    o << ind << "uint4 pq" << D << "_" << w << " = make_uint4(0u, 0u, 0u, 0u);\n";
                o << ind << "if (plive" << D << ") {\n"
                  << ind << "    const uint4 *prec = (const uint4 *)(E.plan->inner[" << d << "].dpay + poff" << D << " * " << rs << "u);\n";
                for (uint32_t w = 0; w < rs / 16; w++)
                    o << ind << "    pq" << D << "_" << w << " = __ldg(&prec[" << w << "]);\n";
                o << ind << "}\n";
            } else if (bits_depth(d)) {
                o << ind << "const uint32_t pr1" << D << " = plive" << D << " ? ((E.sbits[xbj_bits_off_" << d
                  << "(E.plan) + (uint32_t)(poff" << D << " >> 5)] >> (poff" << D << " & 31)) & 1u) : 0u;\n";
            } else {
                o << ind << "const uint32_t pr1" << D << " = plive" << D << " ? __ldg(&E.plan->inner[" << d << "].dtab[poff" << D << "]) : 0u;\n";
            }
        }
    }

    /* ---- Arrow rows: compaction between the scan quals and the rest ----
     * The numbers of the rows that pass wait in a queue of the warp in
     * shared memory until 32 are there, so that the group lookup and the
     * updates run with every lane, and the columns that the quals do not
     * read are loaded for rows that passed only.  20M rows into
     * 1.7M groups 2314 -> 1772 us a query, 500M rows into 10M groups 23.8 ->
     * 22.2 ms.  Heap rows, which would be decoded twice, lost 3 to 14% by
     * it, and an aggregate without keys has too little to do per row.  Not
     * where the quals save a value into a slot (SaveExpr), which later
     * programs may read: a row taken from the queue is decoded again, the
     * quals are not evaluated again. */
    bool compact() const
    {
        if (format != KDS_FORMAT_ARROW || !p->scan_quals.count || p->has_groupby != 1)
            return false;
        for (uint32_t i = 0; i < p->scan_quals.count; i++) {
            const xb_insn &in = p->insns[p->scan_quals.start + i];
            const bool writes = in.op != XB_OP_MASK_PUSH && in.op != XB_OP_MASK_NARROW && in.op != XB_OP_MASK_POP;
            if (writes && in.dst < p->nslots)
                return false;
        }
        return true;
    }

    void pipeline()
    {
        o << "__device__ __forceinline__ bool xbj_quals(XbjRegs &R, const XbjEnv &E, bool &failed)\n{\n    (void)E;\n";
        program(p->scan_quals, "    ");
        o << "    return !failed && " << pass_expr(p->scan_quals) << ";\n}\n\n"
             "__device__ __forceinline__ void\n"
             "xbj_after_quals(XbjRegs &R, const XbjEnv &E, XbjCnt &C, bool &failed)\n{\n";
        preload_probes("    ");
        depth(1, "    ");
        o << "}\n";
    }

    /* resident CTAs per SM the kernel's register budget is built for;
     * XPU_B200_JIT_MINB (1..8) overrides the default for launch tuning */
    /* rows of a heap page left when the warp prefetches its next page
     * (XPU_B200_JIT_PFLEAD overrides for tuning) */
    static int pf_lead()
    {
        const char *e = getenv("XPU_B200_JIT_PFLEAD");
        const int v = e ? atoi(e) : -1;
        return (v == 0 || (v >= 32 && v <= 1024)) ? v : 32;
    }

    static int min_blocks()
    {
        const char *e = getenv("XPU_B200_JIT_MINB");
        const int v = e ? atoi(e) : 0;
        return (v >= 1 && v <= 8) ? v : XBJ_MIN_BLOCKS_DEFAULT;
    }

    std::string run()
    {
        const uint32_t nregs = p->nregs > 0 ? p->nregs : 1;
        o << "/* generated: session-specialised executor (format " << format << ") */\n";
        /* the generator's choices per join depth, for whoever reads the source */
        for (uint32_t d = 1; d <= p->nrels; d++)
            o << "/* depth " << d << ": preloaded " << preloadable(d) << ", group ids " << (gid_mode() && d == p->gid_depth)
              << ", lazy record " << lazy_record(d) << ", columns used later " << regs_used_after(d) << " */\n";
        o << "#include \"xb_exec_dev.cuh\"\n"
             "#define XBJ_MIN_BLOCKS " << (minb > 0 ? minb : min_blocks()) << "\n"
             "#define XBJ_PF_LEAD " << pf_lead() << "\n"
             "#define XBJ_NRELS " << p->nrels << "\n"
             "#define XBJ_GENT_SIZE " << (p->gent_size ? p->gent_size : 16) << "\n"
             "#define XBJ_SM_STRIDE " << xb_jit_sm_stride(p->gent_size ? p->gent_size : 16) << "\n"
             "#define XBJ_KEYS_OFF " << p->gent_keys_off << "\n"
          << (p->has_groupby ? "#define XBJ_MERGE_SM 1\n" : "")
          << (xb_jit_stage_bytes(format) ? "#define XBJ_STAGE 1\n" : "")
          << (format == KDS_FORMAT_BLOCK && (p->lay_valid || p->walk_ncols) ? "#define XBJ_LAYOUT 1\n" : "")
          << "#define XBJ_LAY_FIXED " << (format == KDS_FORMAT_BLOCK && p->lay_valid ? 1 : 0) << "\n"
          << (any_bits() ? "#define XBJ_BITS 1\n" : "");
        if (part_mode())
            o << "#define XBJ_PART 1\n#define XBJ_REC_SIZE " << part_rec_size() << "\n";
        if (compact())
            o << "#define XBJ_COMPACT 1\n";
        /* rows create groups in the global table (or the one group there
         * is): the warp counts them.  Where the groups are numbered they
         * come with the merge at the end, and the count, its reset and its
         * look after every batch are left out (100M rows joined, a pass:
         * 1270 us with them, 1245 without) */
        if (p->has_groupby == 1 && !gid_mode())
            o << "#define XBJ_KEYED 1\n";
        if ((p->has_groupby == 1 && !gid_mode()) || p->has_groupby == 2)
            o << "#define XBJ_NEWG 1\n";
        if (format == KDS_FORMAT_ARROW && p->nload0 > 0)
            o << "#define XBJ_ACOLS " << p->nload0 << "\n";
        o << "struct XbjRegs {\n"
             "    uint64_t v[" << nregs << "];\n"
             "    uint32_t a[" << nregs << "];\n"
             "    uint32_t h[" << nregs << "];\n"
             "    bool     n[" << nregs << "];\n"
             "};\n";
        if (p->has_groupby == 2) {
            /* the accumulators' fields, known once their code is printed */
            std::ostringstream keep;
            keep.swap(o);
            accumulators();
            o.swap(keep);
            o << "#define XBJ_ACC " << acc_counters + 1 << "\nstruct XbjAcc {\n    uint32_t rows;\n" << acc_decl << "};\n";
        }
        o << "#include \"xb_jit_rt.cuh\"\n\n";
        if (format == KDS_FORMAT_BLOCK && (p->lay_valid || p->walk_ncols))
            layout_check();
        if (format == KDS_FORMAT_BLOCK && p->walk_ncols)
            walk();
        if (any_bits())
            bits_helpers();
        decode();
        if (p->has_groupby) {
            group_helpers();
            if (p->has_groupby == 1)
                group_row();
            if (part_mode()) {
                part_helpers();
                slice_helpers();
            }
        }
        pipeline();
        /* the kernels that call generated functions defined above */
        o << "\n#define XBJ_RT_TAIL 1\n#include \"xb_jit_rt.cuh\"\n";
        return o.str();
    }
};

/* stand-ins for the C headers the device headers include */
const char *k_stdint =
    "#pragma once\n"
    "typedef signed char int8_t; typedef short int16_t; typedef int int32_t; typedef long int64_t;\n"
    "typedef unsigned char uint8_t; typedef unsigned short uint16_t; typedef unsigned int uint32_t;\n"
    "typedef unsigned long uint64_t; typedef long intptr_t; typedef unsigned long uintptr_t;\n"
    "#define INT8_MIN (-128)\n#define INT8_MAX 127\n#define INT16_MIN (-32768)\n#define INT16_MAX 32767\n"
    "#define INT32_MIN (-2147483647-1)\n#define INT32_MAX 2147483647\n"
    "#define INT64_MIN (-9223372036854775807L-1)\n#define INT64_MAX 9223372036854775807L\n"
    "#define UINT8_MAX 255\n#define UINT16_MAX 65535\n#define UINT32_MAX 4294967295U\n"
    "#define UINT64_MAX 18446744073709551615UL\n";
const char *k_stddef =
    "#pragma once\n"
    "typedef unsigned long size_t;\ntypedef long ptrdiff_t;\n"
    "#define offsetof(t, m) ((size_t)&(((t *)0)->m))\n"
    "#ifndef NULL\n#define NULL 0\n#endif\n";

struct CacheEntry {
    CUmodule mod = nullptr;
    CUfunction fn = nullptr;
    CUfunction fn_mix = nullptr;
    CUfunction fn_replay = nullptr;     /* partitioned aggregation's replay, if built */
    CUfunction fn_slice = nullptr;      /* and its form on slices in shared memory */
    double compile_ms = 0.0;
};
std::map<std::pair<int, std::string>, CacheEntry> g_cache;

}   /* namespace */

extern "C" uint32_t
xb_jit_sm_stride(uint32_t gent_size)
{
    /* entries of the shared group table sit 8 bytes further apart than
     * their size: with a size of a multiple of 64 bytes, the same field of
     * different entries would fall into two of the 32 banks, and the lanes
     * updating different groups would serialise on them */
    return gent_size + 8;
}

extern "C" size_t
xb_jit_stage_bytes(uint32_t format)
{
    if (format != KDS_FORMAT_BLOCK)
        return 0;
    /* staging is opt-in (XPU_B200_JIT_STAGE=1): with one buffer per warp
     * the copy of a page cannot overlap the decoding of the previous one,
     * which measured slower than reading pages in place */
    const char *e = getenv("XPU_B200_JIT_STAGE");
    if (!e || strcmp(e, "1") != 0)
        return 0;
    /* alignment slack + one 8 KB page buffer and one mbarrier per warp */
    return 128 + (size_t)XBJ_WARPS_PER_CTA * (PGSTROM_BLCKSZ + 8);
}

extern "C" int
xb_jit_source(const xb_plan *plan, uint32_t format, char *buf, size_t bufsz, size_t *p_len)
{
    Gen g;
    g.p = plan;
    g.format = format;
    const std::string s = g.run();
    if (p_len)
        *p_len = s.size();
    if (buf && bufsz > 0) {
        size_t n = s.size() < bufsz - 1 ? s.size() : bufsz - 1;
        memcpy(buf, s.data(), n);
        buf[n] = '\0';
    }
    return 0;
}

/* NVRTC: source -> sm_100a cubin; the APIs are bound (NVRTC builds distinct
 * programs concurrently, so no lock is needed here) */
static int compile_cubin(const std::string &src, std::vector<char> *cubin, double *p_ms, std::string *err)
{
    std::vector<const char *> names, texts;
    names.push_back("stdint.h");  texts.push_back(k_stdint);
    names.push_back("stddef.h");  texts.push_back(k_stddef);
    names.push_back("stdbool.h"); texts.push_back("#pragma once\n");
    for (size_t i = 0; i < sizeof(xbj_header_names) / sizeof(xbj_header_names[0]); i++) {
        names.push_back(xbj_header_names[i]);
        texts.push_back(xbj_header_texts[i]);
    }
    const auto t0 = std::chrono::steady_clock::now();
    nvrtcProgram prog;
    nvrtcResult r = g_nvrtc.create(&prog, src.c_str(), "xbj_session.cu", (int)names.size(),
                                   texts.data(), names.data());
    if (r != NVRTC_SUCCESS) {
        *err = std::string("nvrtcCreateProgram: ") + g_nvrtc.errstr(r);
        return -1;
    }
    const char *opts[] = {"--gpu-architecture=sm_100a", "-std=c++17", "-default-device",
                          "--device-int128", "-lineinfo", "-DXB_JIT=1", "--diag-suppress=550,177"};
    r = g_nvrtc.compile(prog, (int)(sizeof(opts) / sizeof(opts[0])), opts);
    if (r != NVRTC_SUCCESS) {
        size_t ls = 0;
        g_nvrtc.log_size(prog, &ls);
        std::string log(ls, '\0');
        if (ls)
            g_nvrtc.log(prog, &log[0]);
        g_nvrtc.destroy(&prog);
        if (log.size() > 900)
            log.resize(900);
        *err = std::string("nvrtc: ") + g_nvrtc.errstr(r) + ": " + log;
        return -1;
    }
    size_t cs = 0;
    g_nvrtc.cubin_size(prog, &cs);
    cubin->resize(cs);
    g_nvrtc.cubin(prog, cubin->data());
    g_nvrtc.destroy(&prog);
    *p_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return 0;
}

extern "C" int
xb_jit_check(const xb_plan *plan, uint32_t format, uint64_t *p_cubin_bytes, double *p_compile_ms,
             char *errbuf, size_t errlen)
{
    Gen g;
    g.p = plan;
    g.format = format;
    const std::string src = g.run();
    std::lock_guard<std::mutex> guard(g_lock);
    bind_locked();
    std::string err;
    if (!g_nvrtc.ok)
        err = g_nvrtc.why;
    std::vector<char> cubin;
    double ms = 0.0;
    if (err.empty() && compile_cubin(src, &cubin, &ms, &err) == 0) {
        if (p_cubin_bytes) *p_cubin_bytes = cubin.size();
        if (p_compile_ms) *p_compile_ms = ms;
        return 0;
    }
    if (errbuf && errlen)
        snprintf(errbuf, errlen, "%s", err.c_str());
    return -1;
}

extern "C" uint64_t
xb_jit_shape_key(const xb_plan *plan, uint32_t format)
{
    Gen g;
    g.p = plan;
    g.format = format;
    g.minb = 1;                 /* one fixed value: the key names the plan shape only */
    const std::string src = g.run();
    uint64_t h = 1469598103934665603ULL;        /* FNV-1a, 64-bit */
    for (unsigned char c : src) {
        h ^= c;
        h *= 1099511628211ULL;
    }
    return h ^ ((uint64_t)format << 56);
}

extern "C" int
xb_jit_compile(const xb_plan *plan, uint32_t format, int dindex,
               void **p_func, void **p_mixfn, double *p_compile_ms, char *errbuf, size_t errlen)
{
    return xb_jit_compile_minb(plan, format, dindex, 0, p_func, p_mixfn, nullptr, p_compile_ms, errbuf, errlen);
}

extern "C" uint32_t
xb_jit_part_rec_size(const xb_plan *plan, uint32_t format)
{
    Gen g;
    g.p = plan;
    g.format = format;
    return g.part_mode() ? g.part_rec_size() : 0;
}

/* find the kernels of plan + format in the process-wide cache, or (unless
 * lookup_only) build them: the NVRTC compilation runs without the cache
 * lock held, so that launches and lookups of other sessions go on while a
 * new plan shape compiles.  Returns 0 (found or built), 1 (lookup_only and
 * not cached) or -1 (errbuf says why). */
static int
jit_build(const xb_plan *plan, uint32_t format, int dindex, int min_blocks, bool lookup_only,
          void **p_func, void **p_mixfn, void **p_replay, double *p_compile_ms,
          char *errbuf, size_t errlen)
{
    if (p_replay)
        *p_replay = nullptr;
    auto fail = [&](const std::string &m) {
        if (errbuf && errlen)
            snprintf(errbuf, errlen, "%s", m.c_str());
        return -1;
    };
    if (plan->has_proj && plan->proj_hashed)
        return fail("projection into a hashed kds_dst runs on the interpreter");
    Gen g;
    g.p = plan;
    g.format = format;
    g.minb = (min_blocks >= 1 && min_blocks <= 8) ? min_blocks : 0;
    const std::string src = g.run();
    const bool want_replay = g.part_mode();
    auto key = std::make_pair(dindex, src);
    auto give = [&](const CacheEntry &ce, double ms) {
        *p_func = (void *)ce.fn;
        if (p_mixfn)
            *p_mixfn = (void *)ce.fn_mix;
        if (p_replay)
            *p_replay = (void *)ce.fn_replay;
        if (p_compile_ms)
            *p_compile_ms = ms;
        return 0;
    };
    {
        std::lock_guard<std::mutex> guard(g_lock);
        bind_locked();
        /* diagnostics: XPU_B200_JIT_SAVE=<dir> keeps every generated source */
        if (const char *dir = getenv("XPU_B200_JIT_SAVE")) {
            char path[4096];
            snprintf(path, sizeof(path), "%s/xbj_%c_%016llx.cu", dir, (int)format,
                     (unsigned long long)std::hash<std::string>()(src));
            if (FILE *f = fopen(path, "w")) {
                fwrite(src.data(), 1, src.size(), f);
                fclose(f);
            }
        }
        if (!g_nvrtc.ok)
            return fail(g_nvrtc.why);
        if (!g_drv.ok)
            return fail(g_drv.why);
        auto it = g_cache.find(key);
        if (it != g_cache.end())
            return give(it->second, 0.0);
        if (lookup_only)
            return 1;
    }
    std::vector<char> cubin;
    std::string err;
    CacheEntry ce;
    if (compile_cubin(src, &cubin, &ce.compile_ms, &err) != 0)
        return fail(err);
    std::lock_guard<std::mutex> guard(g_lock);
    auto it = g_cache.find(key);
    if (it != g_cache.end())                 /* built meanwhile by another thread */
        return give(it->second, ce.compile_ms);
    if (g_drv.load(&ce.mod, cubin.data()) != CUDA_SUCCESS)
        return fail("cuModuleLoadData failed");
    if (g_drv.getfn(&ce.fn, ce.mod, "xbj_kernel") != CUDA_SUCCESS ||
        g_drv.getfn(&ce.fn_mix, ce.mod, "xbj_mixed_kernel") != CUDA_SUCCESS)
        return fail("cuModuleGetFunction(xbj_kernel) failed");
    if (want_replay && (g_drv.getfn(&ce.fn_replay, ce.mod, "xbj_replay") != CUDA_SUCCESS ||
                        g_drv.getfn(&ce.fn_slice, ce.mod, "xbj_replay_slice") != CUDA_SUCCESS))
        ce.fn_replay = ce.fn_slice = nullptr;
    g_cache[key] = ce;
    return give(ce, ce.compile_ms);
}

extern "C" int
xb_jit_compile_minb(const xb_plan *plan, uint32_t format, int dindex, int min_blocks,
                    void **p_func, void **p_mixfn, void **p_replay, double *p_compile_ms,
                    char *errbuf, size_t errlen)
{
    return jit_build(plan, format, dindex, min_blocks, false, p_func, p_mixfn, p_replay, p_compile_ms,
                     errbuf, errlen);
}

extern "C" int
xb_jit_lookup_minb(const xb_plan *plan, uint32_t format, int dindex, int min_blocks,
                   void **p_func, void **p_mixfn, void **p_replay)
{
    char msg[16];
    return jit_build(plan, format, dindex, min_blocks, true, p_func, p_mixfn, p_replay, nullptr,
                     msg, sizeof(msg));
}

/* ---- background builds ------------------------------------------------
 * A served request whose plan shape has no kernel yet runs on the
 * interpreter while its kernel is built on a thread of its own; later
 * launches of the shape adopt the kernel once it is there. */
namespace {
struct JitJob {
    std::atomic<int> state{0};          /* 0 building, 1 built, -1 failed */
    xb_plan plan;
    uint32_t format = 0;
    int dindex = 0, minb = 0;
    void *fn = nullptr, *mixfn = nullptr, *replay = nullptr;
    double ms = 0.0;
    char msg[1024] = {0};
};
std::atomic<int> g_jobs_running{0};
std::atomic<bool> g_exiting{false};
/* the builds under way, by GPU and source: sessions of one plan shape that
 * open meanwhile wait for the same one (a build each was hundreds of threads
 * compiling the same source when clients opened sessions quickly) */
std::mutex g_jobs_lock;
std::map<std::pair<int, std::string>, std::shared_ptr<JitJob>> g_jobs;

void wait_for_jobs()
{
    for (int i = 0; i < 3000 && g_jobs_running.load() > 0; i++)
        std::this_thread::sleep_for(std::chrono::milliseconds(10));
}

void jobs_at_exit()
{
    /* builds still running may not outlive the objects they use */
    g_exiting = true;
    wait_for_jobs();
}
}   /* namespace */

extern "C" void
xb_jit_wait_builds(int exiting)
{
    if (exiting)
        g_exiting = true;
    wait_for_jobs();
}

extern "C" void *
xb_jit_build_async(const xb_plan *plan, uint32_t format, int dindex, int min_blocks)
{
    static std::once_flag once;
    std::call_once(once, [] { std::atexit(jobs_at_exit); });
    Gen g;
    g.p = plan;
    g.format = format;
    g.minb = (min_blocks >= 1 && min_blocks <= 8) ? min_blocks : 0;
    const auto key = std::make_pair(dindex, g.run());
    std::lock_guard<std::mutex> jobs(g_jobs_lock);
    auto it = g_jobs.find(key);
    if (it != g_jobs.end())
        return new std::shared_ptr<JitJob>(it->second);
    auto job = std::make_shared<JitJob>();
    memcpy(&job->plan, plan, sizeof(xb_plan));
    job->format = format;
    job->dindex = dindex;
    job->minb = min_blocks;
    g_jobs[key] = job;
    g_jobs_running++;
    try {
        std::thread([job, key]() {
            if (!g_exiting) {
                cudaSetDevice(job->dindex);
                const int rc = jit_build(&job->plan, job->format, job->dindex, job->minb, false, &job->fn,
                                         &job->mixfn, &job->replay, &job->ms, job->msg, sizeof(job->msg));
                job->state = rc == 0 ? 1 : -1;
            } else {
                snprintf(job->msg, sizeof(job->msg), "process exiting");
                job->state = -1;
            }
            {
                std::lock_guard<std::mutex> done(g_jobs_lock);
                g_jobs.erase(key);
            }
            g_jobs_running--;
        }).detach();
    } catch (...) {
        g_jobs.erase(key);
        g_jobs_running--;
        return nullptr;
    }
    return new std::shared_ptr<JitJob>(job);
}

/* for tests: builds under way */
extern "C" int xb_jit_jobs_running(void)
{
    return g_jobs_running.load();
}

extern "C" int
xb_jit_job_poll(void *h, void **p_func, void **p_mixfn, void **p_replay, double *p_compile_ms,
                char *errbuf, size_t errlen)
{
    const std::shared_ptr<JitJob> &job = *(std::shared_ptr<JitJob> *)h;
    const int st = job->state.load();
    if (st == 0)
        return 1;
    if (st < 0) {
        if (errbuf && errlen)
            snprintf(errbuf, errlen, "%s", job->msg);
        return -1;
    }
    *p_func = job->fn;
    if (p_mixfn) *p_mixfn = job->mixfn;
    if (p_replay) *p_replay = job->replay;
    if (p_compile_ms) *p_compile_ms = job->ms;
    return 0;
}

extern "C" void
xb_jit_job_release(void *h)
{
    delete (std::shared_ptr<JitJob> *)h;
}

extern "C" void *
xb_jit_slice_of(void *replay)
{
    std::lock_guard<std::mutex> guard(g_lock);
    for (const auto &kv : g_cache)
        if (replay && (void *)kv.second.fn_replay == replay)
            return (void *)kv.second.fn_slice;
    return nullptr;
}

extern "C" int
xb_jit_prepare(void *func, int block, size_t smem, int *p_per_sm)
{
    std::lock_guard<std::mutex> guard(g_lock);
    if (!g_drv.ok)
        return -1;
    /* the limit is the function's, which sessions of one plan shape share
     * with shared tables of their own sizes: it is only ever raised */
    int cur = 0;
    if (g_drv.getattr(&cur, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (CUfunction)func) != CUDA_SUCCESS)
        cur = 0;
    if ((size_t)cur < smem &&
        g_drv.setattr((CUfunction)func, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem) != CUDA_SUCCESS)
        return -1;
    int per_sm = 0;
    if (g_drv.occupancy(&per_sm, (CUfunction)func, block, smem) != CUDA_SUCCESS || per_sm < 1)
        return -1;
    *p_per_sm = per_sm;
    return 0;
}

extern "C" size_t
xb_jit_static_smem(void *func)
{
    std::lock_guard<std::mutex> guard(g_lock);
    int sz = 0;
    if (!g_drv.ok || g_drv.getattr(&sz, CU_FUNC_ATTRIBUTE_SHARED_SIZE_BYTES, (CUfunction)func) != CUDA_SUCCESS)
        return 0;
    return (size_t)sz;
}

extern "C" int
xb_jit_occupancy(void *func, int block, size_t smem, int *p_per_sm)
{
    std::lock_guard<std::mutex> guard(g_lock);
    int per_sm = 0;
    if (!g_drv.ok || g_drv.occupancy(&per_sm, (CUfunction)func, block, smem) != CUDA_SUCCESS || per_sm < 1)
        return -1;
    *p_per_sm = per_sm;
    return 0;
}

extern "C" int
xb_jit_launch(void *func, int grid, int block, size_t smem, void *stream, void *args)
{
    void *params[] = {args};
    return g_drv.launch((CUfunction)func, grid, 1, 1, block, 1, 1, (unsigned int)smem,
                        (CUstream)stream, params, nullptr) == CUDA_SUCCESS ? 0 : -1;
}
