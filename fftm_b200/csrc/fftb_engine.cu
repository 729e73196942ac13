// fftb_engine.cu -- kernel registry, twiddle tables, program builder / executor.
#include "fftb_engine.h"
#include "fftb_bluestein.h"
#include "fftb_longline.h"

#include <algorithm>
#include <cstring>
#include <cstdio>
#include <map>
#include <mutex>
#include <set>
#include <tuple>

#include "../../include/fftb.h"
#include "fftb_device.cuh"
#include "fftb_line.cuh"

// Kernel tables exported by the fftb_pass_inst.cu and fftb_line_inst.cu objects.
#define FFTB_DECL_PASS(k) extern "C" int fftb_pass_table_float_part##k(fftb::PassKernelInfo *, int);
#define FFTB_DECL_LINE(k)                                                                                             \
    extern "C" int fftb_line_table_float_part##k(fftb::LineKernelInfo *, int);                                        \
    extern "C" int fftb_line_table_double_part##k(fftb::LineKernelInfo *, int);
#define FFTB_PARTS8(X) X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7)
#define FFTB_PARTS64(X)                                                                                               \
    FFTB_PARTS8(X) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) X(21) X(22) X(23)      \
    X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31) X(32) X(33) X(34) X(35) X(36) X(37) X(38) X(39) X(40) X(41)       \
    X(42) X(43) X(44) X(45) X(46) X(47) X(48) X(49) X(50) X(51) X(52) X(53) X(54) X(55) X(56) X(57) X(58) X(59)       \
    X(60) X(61) X(62) X(63)
FFTB_PARTS8(FFTB_DECL_PASS)
FFTB_PARTS64(FFTB_DECL_LINE)

namespace fftb {

namespace {

thread_local std::string g_last_error;

struct Registry {
    std::vector<PassKernelInfo> pass = std::vector<PassKernelInfo>(4097, PassKernelInfo{});  // f32 pass kernels by length
    std::vector<LineKernelInfo> line[2];  // [2 length + row mapping], nf = 0 where there is none
    std::set<std::pair<int, const void *>> smem_configured;  // (device, kernel): the limit is per device
    std::map<std::tuple<int, int, int>, void *> roots;  // (device, dtype, ntw) -> device table
    std::map<std::tuple<int, int, int, int>, void *> stages;  // (device, dtype, nf, row) -> stage tables
    std::mutex mu;

    Registry()
    {
#define FFTB_FN_PASS(k) fftb_pass_table_float_part##k,
#define FFTB_FN_LINE32(k) fftb_line_table_float_part##k,
#define FFTB_FN_LINE64(k) fftb_line_table_double_part##k,
        int (*const fp[])(PassKernelInfo *, int) = {FFTB_PARTS8(FFTB_FN_PASS)};
        int (*const fl[2][64])(LineKernelInfo *, int) = {{FFTB_PARTS64(FFTB_FN_LINE32)}, {FFTB_PARTS64(FFTB_FN_LINE64)}};
        PassKernelInfo pb[256];
        for (auto f : fp) {
            const int n = f(pb, 256);
            for (int i = 0; i < n && i < 256; ++i)
                if (pb[i].nf <= 4096) pass[pb[i].nf] = pb[i];
        }
        std::vector<LineKernelInfo> lb(256);
        for (int d = 0; d < 2; ++d) {
            line[d].resize(2 * 4097);
            for (auto f : fl[d]) {
                const int n = f(lb.data(), 256);
                for (int i = 0; i < n && i < 256; ++i)
                    if (lb[i].nf <= 4096) line[d][2 * lb[i].nf + lb[i].row] = lb[i];
            }
        }
    }
    const LineKernelInfo *find_line(int dtype, int nf, int row) const
    {
        if (nf < 1 || nf > 4096 || line[dtype][2 * nf + row].nf != nf) return nullptr;
        return &line[dtype][2 * nf + row];
    }
};

Registry &reg()
{
    static Registry r;
    return r;
}

template <typename R> __global__ void make_roots_kernel(cpx<R> *w, int n)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < n) {
        double s, c;
        // exp(-2 pi i m / n) evaluated in FP64, then rounded to R
        sincospi(-2.0 * (double)m / (double)n, &s, &c);
        w[m] = mk<R>((R)c, (R)s);
    }
}

int get_roots(int dtype, int ntw, void **out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_status_from_cuda(e);
    Registry &r = reg();
    std::lock_guard<std::mutex> lk(r.mu);
    auto key = std::make_tuple(dev, dtype, ntw);
    auto it = r.roots.find(key);
    if (it != r.roots.end()) {
        *out = it->second;
        return FFTB_SUCCESS;
    }
    void *p = nullptr;
    e = cudaMalloc(&p, complex_bytes(dtype) * (size_t)ntw);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_last_error("cudaMalloc of a twiddle table failed");
        return FFTB_ERROR_ALLOC;
    }
    const int bs = 256, gs = (ntw + bs - 1) / bs;
    if (dtype == FFTB_F32) make_roots_kernel<float><<<gs, bs>>>((float2 *)p, ntw);
    else make_roots_kernel<double><<<gs, bs>>>((double2 *)p, ntw);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaFree(p);
        return set_status_from_cuda(e);
    }
    r.roots[key] = p;
    *out = p;
    return FFTB_SUCCESS;
}

// table w[(q - 1) ns + j] = exp(-2 pi i q j / (ns rad)), q = 1 .. rad - 1, j < ns
template <typename R> __global__ void make_stage_kernel(cpx<R> *w, int ns, int rad)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < (rad - 1) * ns) {
        double s, c;
        sincospi(-2.0 * (double)((m / ns + 1) * (m % ns)) / (double)(ns * rad), &s, &c);
        w[m] = mk<R>((R)c, (R)s);
    }
}

// The line kernel's stage tables (of its plan, then of the reversed plan), made once per device.
int get_stages(int dtype, const LineKernelInfo &k, void **out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_status_from_cuda(e);
    Registry &r = reg();
    std::lock_guard<std::mutex> lk(r.mu);
    auto key = std::make_tuple(dev, dtype, k.nf, k.row);
    auto it = r.stages.find(key);
    if (it != r.stages.end()) {
        *out = it->second;
        return FFTB_SUCCESS;
    }
    const LinePlan rev = line_reverse(k.plan);
    const size_t n = (size_t)line_table_size(k.plan) + (size_t)line_table_size(rev);
    if (n == 0) {
        *out = nullptr;
        return FFTB_SUCCESS;
    }
    char *p = nullptr;
    e = cudaMalloc(&p, complex_bytes(dtype) * n);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_last_error("cudaMalloc of a stage table failed");
        return FFTB_ERROR_ALLOC;
    }
    size_t base = 0;
    for (const LinePlan &pl : {k.plan, rev}) {
        int ns = 1;
        for (int i = 0; i < pl.S; ++i) {
            const int rad = pl.r[i], cnt = (rad - 1) * ns;
            if (i > 0) {
                char *w = p + complex_bytes(dtype) * (base + (size_t)line_tab_off(pl, i));
                if (dtype == FFTB_F32) make_stage_kernel<float><<<(cnt + 255) / 256, 256>>>((float2 *)w, ns, rad);
                else make_stage_kernel<double><<<(cnt + 255) / 256, 256>>>((double2 *)w, ns, rad);
            }
            ns *= rad;
        }
        base += (size_t)line_table_size(pl);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaFree(p);
        return set_status_from_cuda(e);
    }
    r.stages[key] = p;
    *out = p;
    return FFTB_SUCCESS;
}

long long labs_ll(long long v) { return v < 0 ? -v : v; }

int floor_pow2(int v)
{
    int p = 1;
    while (p * 2 <= v) p *= 2;
    return p;
}

} // namespace

void set_last_error(const std::string &msg) { g_last_error = msg; }
const char *last_error() { return g_last_error.c_str(); }

int set_status_from_cuda(cudaError_t e)
{
    if (e == cudaSuccess) return FFTB_SUCCESS;
    set_last_error(std::string("CUDA: ") + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? FFTB_ERROR_ALLOC : FFTB_ERROR_CUDA;
}

bool has_kernel(int dtype, int nf) { return reg().find_line(dtype, nf, 1) != nullptr; }

int engine_roots(int dtype, int ntw, void **out) { return get_roots(dtype, ntw, out); }

bool lookup_kernel(int nf, PassKernelInfo *out)
{
    Registry &r = reg();
    if (nf < 1 || nf > 4096 || r.pass[nf].nf != nf) return false;
    *out = r.pass[nf];
    return true;
}

// Division by d of l < 2^31 as (l m) >> (31 + s): s = ceil(log2 d), m = ceil(2^(31+s) / d) < 2^32; the
// product's excess l (m d - 2^(31+s)) is below 2^31 2^s, so the quotient is exact.
void line_divisors(PassArgs &a)
{
    a.c_shift = -1;
    if (a.nlines > 0x7fffffffLL) return;
    auto magic = [](long long d, unsigned *m) {
        int s = 0;
        while ((1LL << s) < d) ++s;
        *m = (unsigned)((((unsigned long long)1 << (31 + s)) + (unsigned long long)d - 1) / (unsigned long long)d);
        return 31 + s;
    };
    const int s0 = magic(a.c0, &a.c0_mul), s1 = magic(a.c1, &a.c1_mul);
    a.c_shift = s0 | (s1 << 6);
}

// Whether a pass from rows to columns runs the column mapping with its input staged, instead of the
// row mapping k with its output staged.  Double lines that the row mapping splits do while they are
// short: a thread of a column tile holds most of a line, where the row tile exchanges and often needs
// the whole block's barriers for it (2^22 points as C2C of 4, 8 and 35 points 32 -> 26, 31 -> 25 and
// 51 -> 43 us, R2C of 8 and 16 points 20 -> 15 and 19 -> 14, C2R of 35 points 43 -> 30).  Lines of one
// stage, odd R2C lines, C2C from 64 and real lines from 48 complex points on are as fast or
// faster as rows (C2C of 2 points 27 us against 29, R2C of 25 points 23 against 25, of 112 points 15.5
// against 17.4).  So do the longest C2R lines in float, of which a row tile holds two or one, so
// that its column segments are 8 bytes (3840 points 29 -> 20 us, 8192 points 42 -> 21; 3456
// points and below are faster as rows).
bool columns_from_rows(int dtype, int kind, bool half, const LineKernelInfo &k)
{
    if (dtype == FFTB_F32) return kind == K_C2R && k.nf >= 1792;
    if (k.plan.S < 2 || (kind == K_R2C && !half)) return false;
    return k.nf < (kind == K_R2C || kind == K_C2R ? 48 : 64);
}

int program_add(Program &prog, int dtype, const AxisPass &p)
{
    if (p.n < 1) return FFTB_ERROR_INVALID_VALUE;
    Launch L;
    memset(&L.args, 0, sizeof(L.args));
    PassArgs &a = L.args;
    const bool realk = (p.kind == K_R2C || p.kind == K_C2R);
    bool half = realk && (p.n % 2 == 0);
    int nf = half ? p.n / 2 : p.n;
    Registry &r = reg();
    bool line = r.find_line(dtype, nf, 1) != nullptr;
    if (!line && half) {
        // no half-length kernel: the real line as a full complex line
        half = false;
        nf = p.n;
        line = r.find_line(dtype, nf, 1) != nullptr;
    }
    if ((p.ep_mode & EP_DERIV) && (!line || (p.kind != K_C2R && p.kind != K_SANDWICH))) {
        set_last_error("the derivative multiply needs a line kernel");
        return FFTB_ERROR_UNSUPPORTED_SIZE;
    }
    bool chirpz = false;
    PassKernelInfo bs = {};  // the chirp-z pass; bs.nf is its convolution length
    if (!line && bluestein_kernel(dtype, p.n, &bs)) {
        chirpz = true;
        const void *ch = nullptr, *bh = nullptr;
        int st = bluestein_tables(dtype, p.n, &ch, &bh);
        if (st != FFTB_SUCCESS) return st;
        a.bs_n = p.n;
        a.bs_chirp = ch;
        a.bs_bhat = bh;
    } else if (!line) {
        // longer than one pass holds: a long-line step (four-step or chirp-z)
        if (p.in_blk || p.out_blk) {
            set_last_error("blocked point indices need a C2C line kernel (line length up to 4096)");
            return FFTB_ERROR_UNSUPPORTED_SIZE;
        }
        std::shared_ptr<LongLine> ll;
        int st = longline_create(dtype, p, ll);
        if (st != FFTB_SUCCESS) return st;
        Launch S;
        memset(&S.args, 0, sizeof(S.args));
        S.nf = 0;
        S.fn = nullptr;
        S.line = nullptr;
        S.programmatic = 0;
        S.in_buf = p.in_buf;
        S.out_buf = p.out_buf;
        S.in_off_bytes = S.out_off_bytes = 0;
        S.pair_candidate = 0;
        S.real_align = 0;
        S.real_side = 0;
        S.block = 0;
        S.smem = 0;
        S.ep_dynamic = p.ep_dynamic;
        S.alg_bytes = longline_alg_bytes(*ll);
        static const char *kn[] = {"c2c_fwd", "c2c_inv", "r2c", "c2r", "sandwich"};
        S.name = std::string("fftb_long_line<") + (dtype == 0 ? "f32" : "f64") + ">/" + kn[p.kind] + "/n" +
                 std::to_string(p.n);
        S.longline = ll;
        prog.dtype = dtype;
        prog.launches.push_back(S);
        return FFTB_SUCCESS;
    }
    L.nf = chirpz ? bs.nf : nf;
    const int ntw = half ? 2 * nf : L.nf;
    void *roots = nullptr;
    int st = get_roots(dtype, ntw, &roots);
    if (st != FFTB_SUCCESS) return st;

    // batch dims: drop trivial ones, sort by input stride so dim 0 is the most contiguous
    std::vector<Dim> b;
    for (const Dim &d : p.batch)
        if (d.count > 1) b.push_back(d);
    std::stable_sort(b.begin(), b.end(), [](const Dim &x, const Dim &y) { return labs_ll(x.is) < labs_ll(y.is); });
    if (b.size() > 3) {
        set_last_error("more than three batch dimensions");
        return FFTB_ERROR_INVALID_VALUE;
    }
    while (b.size() < 3) b.push_back(Dim{1, 0, 0, -1});
    long long nlines = b[0].count * b[1].count * b[2].count;

    a.kind = p.kind;
    a.half = half ? 1 : 0;
    a.is = p.is;
    a.os = p.os;
    a.nlines = nlines;
    a.c0 = b[0].count;
    a.c1 = b[1].count;
    a.ib0 = b[0].is; a.ib1 = b[1].is; a.ib2 = b[2].is;
    a.ob0 = b[0].os; a.ob1 = b[1].os; a.ob2 = b[2].os;
    a.in_pts_fast = (labs_ll(p.is) == 1) || (b[0].count == 1) ||
                    (labs_ll(b[0].is) != 1 && labs_ll(p.is) < labs_ll(b[0].is));
    a.out_pts_fast = (labs_ll(p.os) == 1) || (b[0].count == 1) ||
                     (labs_ll(b[0].os) != 1 && labs_ll(p.os) < labs_ll(b[0].os));
    a.tw = roots;
    a.ntw = ntw;
    a.ep_tw = p.ep_tw;
    if ((p.in_blk || p.out_blk) && (chirpz || (p.kind != K_C2C_FWD && p.kind != K_C2C_INV) ||
                                    (p.out_blk && p.n / p.out_blk > 8))) {
        set_last_error("blocked point indices need a C2C line kernel and at most 8 blocks");
        return FFTB_ERROR_UNSUPPORTED_SIZE;
    }
    a.in_blk = p.in_blk;
    a.in_hi = p.in_hi;
    a.out_blk = p.out_blk;
    a.out_hi = p.out_hi;
    const size_t cb = complex_bytes(dtype);

    // epilogue
    a.ep_mode = p.ep_mode;
    a.ep_scale = p.ep_scale;
    a.ep_sign = p.ep_sign;
    a.ep_gauss = p.ep_gauss;
    a.ep_hw = p.ep_hw;
    a.ep_naxes = (int)p.ep_axes.size();
    if (a.ep_naxes > 4) return FFTB_ERROR_INVALID_VALUE;
    for (int i = 0; i < a.ep_naxes; ++i) {
        const EpAxis &e = p.ep_axes[i];
        int src = 0;
        if (!e.from_point) {
            src = -1;
            for (int j = 0; j < 3; ++j)
                if (b[j].id == e.dim_id && b[j].count > 1) src = j + 1;
            if (src < 0) {
                // a dimension of count 1 contributes index 0; use the point slot of an
                // axis that is always zero by pointing at an unused batch slot
                for (int j = 2; j >= 0; --j)
                    if (b[j].count == 1) { src = j + 1; break; }
            }
            if (src < 0) return FFTB_ERROR_INVALID_VALUE;
        }
        a.ep_src[i] = src;
        a.ep_n[i] = e.n;
        a.ep_half[i] = e.half;
        a.ep_kscale[i] = 1.0;
    }
    L.ep_dynamic = p.ep_dynamic;

    // real side pairing: contiguous real line with even batch strides
    L.real_side = (p.kind == K_R2C) ? 1 : (p.kind == K_C2R ? 2 : 0);
    L.pair_candidate = 0;
    if (half) {
        if (p.kind == K_R2C)
            L.pair_candidate = (p.is == 1) && b[0].is % 2 == 0 && b[1].is % 2 == 0 && b[2].is % 2 == 0 &&
                               p.in_base % 2 == 0;
        else
            L.pair_candidate = (p.os == 1) && b[0].os % 2 == 0 && b[1].os % 2 == 0 && b[2].os % 2 == 0 &&
                               p.out_base % 2 == 0;
    }
    L.real_align = 2 * real_bytes(dtype);

    long long ncta = 0;
    L.line = nullptr;
    L.programmatic = line ? 1 : 0;
    if (line) {
        // the thread mapping follows the input side; a side of the other order, or with blocked
        // points, is staged through shared memory
        const bool row = a.in_pts_fast &&
                         (a.out_pts_fast || !columns_from_rows(dtype, p.kind, half, *r.find_line(dtype, nf, 1)));
        const LineKernelInfo &k = *r.find_line(dtype, nf, row ? 1 : 0);
        if ((p.ep_mode & ~(EP_SCALE | EP_HALFW | EP_TWIDDLE | EP_DERIV)) != 0 && p.kind != K_SANDWICH) return FFTB_ERROR_INVALID_VALUE;
        L.line = &k;
        a.line_in = !p.in_blk && (row ? p.is == 1 : !a.in_pts_fast);
        a.line_out = !p.out_blk && (row ? p.os == 1 : !a.out_pts_fast);
        line_divisors(a);
        void *tab = nullptr;
        if ((st = get_stages(dtype, k, &tab)) != FFTB_SUCCESS) return st;
        a.ltw = tab;
        L.fn = p.kind == K_SANDWICH ? k.fn_sand : k.fn;
        L.block = k.NT;
        L.smem = a.line_in && a.line_out ? k.smem : k.smem_t;
        ncta = (nlines + k.G - 1) / k.G;
    } else {
        // chirp-z: lines per CTA
        const int T = bs.threads_per_line;
        a.tw_smem = ((size_t)ntw * cb <= 16384) ? 1 : 0;
        int G = std::max(1, 256 / T);
        if (!a.in_pts_fast || !a.out_pts_fast) G = std::max(G, 16);
        G = floor_pow2(std::min(G, std::max(1, 512 / T)));
        while (G > 1 && G / 2 >= nlines) G /= 2;
        auto smem_of = [&](int g) -> size_t {
            return (a.tw_smem ? (size_t)ntw * cb : 0) + (size_t)g * 32 + (size_t)g * (size_t)bs.line_pitch * cb;
        };
        while (G > 1 && smem_of(G) > 160 * 1024) G /= 2;
        if (smem_of(G) > 227 * 1024) {
            set_last_error("line too long for shared memory");
            return FFTB_ERROR_UNSUPPORTED_SIZE;
        }
        a.G = G;
        while ((1 << a.gshift) < G) ++a.gshift;
        L.fn = bs.fn;
        L.block = G * T;
        L.smem = smem_of(G);
        ncta = (nlines + G - 1) / G;
    }
    if (ncta > 0x7fffffffLL) return FFTB_ERROR_INVALID_VALUE;
    L.grid = dim3((unsigned)ncta, 1, 1);
    {
        std::lock_guard<std::mutex> lk(r.mu);
        if (L.smem > 40 * 1024) {  // beside up to 8 KB of static shared memory
            int dev = 0;
            cudaError_t e = cudaGetDevice(&dev);
            if (e != cudaSuccess) return set_status_from_cuda(e);
            if (!r.smem_configured.count({dev, L.fn})) {
                // to what the device allows beside the kernel's static shared memory
                cudaFuncAttributes fa;
                e = cudaFuncGetAttributes(&fa, L.fn);
                if (e == cudaSuccess)
                    e = cudaFuncSetAttribute(L.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             227 * 1024 - (int)fa.sharedSizeBytes);
                if (e != cudaSuccess) return set_status_from_cuda(e);
                r.smem_configured.insert({dev, L.fn});
            }
        }
    }
    L.in_buf = p.in_buf;
    L.out_buf = p.out_buf;
    const size_t in_el = (p.kind == K_R2C) ? real_bytes(dtype) : cb;
    const size_t out_el = (p.kind == K_C2R) ? real_bytes(dtype) : cb;
    L.in_off_bytes = (size_t)p.in_base * in_el;
    L.out_off_bytes = (size_t)p.out_base * out_el;
    {
        static const char *kn[] = {"c2c_fwd", "c2c_inv", "r2c", "c2r", "sandwich"};
        const long long pin = (p.kind == K_C2R) ? (long long)(p.n / 2 + 1) : (long long)p.n;
        const long long pout = (p.kind == K_R2C) ? (long long)(p.n / 2 + 1) : (long long)p.n;
        L.alg_bytes = (double)nlines * ((double)pin * (double)in_el + (double)pout * (double)out_el);
        L.name = std::string(chirpz ? "fftb_bluestein_kernel<" : "fftb_line_kernel<") + (dtype == 0 ? "f32" : "f64") +
                 "," + std::to_string(L.nf) + ">/" + kn[p.kind] + "/n" + std::to_string(p.n);
    }
    prog.dtype = dtype;
    prog.launches.push_back(L);
    return FFTB_SUCCESS;
}

int LaunchTimer::reserve(size_t n)
{
    release();
    ev.resize(n, nullptr);
    for (size_t i = 0; i < n; ++i) {
        cudaError_t e = cudaEventCreate(&ev[i]);
        if (e != cudaSuccess) {
            ev.resize(i);
            return set_status_from_cuda(e);
        }
    }
    owner.assign(n, -1);
    names.assign(n, std::string());
    bytes.assign(n, 0.0);
    used = 0;
    return FFTB_SUCCESS;
}

void LaunchTimer::release()
{
    for (cudaEvent_t e : ev)
        if (e) cudaEventDestroy(e);
    ev.clear();
    owner.clear();
    names.clear();
    bytes.clear();
    used = 0;
}

int timer_mark(LaunchTimer *t, cudaStream_t s, const std::string &name, double b)
{
    if (!t || t->used >= t->ev.size()) return FFTB_SUCCESS;
    const size_t i = t->used++;
    t->owner[i] = 1;
    t->names[i] = name;
    t->bytes[i] = b;
    return set_status_from_cuda(cudaEventRecord(t->ev[i], s));
}

int timer_end(LaunchTimer *t, cudaStream_t s)
{
    if (!t || t->used >= t->ev.size()) return FFTB_SUCCESS;
    const size_t i = t->used++;
    t->owner[i] = -1;
    return set_status_from_cuda(cudaEventRecord(t->ev[i], s));
}

int program_exec(const Program &prog, void *in, void *out, void *work, cudaStream_t stream, const EpValues *ep,
                 LaunchTimer *timer)
{
    void *bufs[3] = {in, out, work};
    for (const Launch &L : prog.launches) {
        if (timer) {
            int ts = timer_mark(timer, stream, L.name, L.alg_bytes);
            if (ts != FFTB_SUCCESS) return ts;
        }
        if (L.longline) {
            int st = longline_exec(*L.longline, bufs, stream, ep && L.ep_dynamic ? ep : nullptr);
            if (st != FFTB_SUCCESS) return st;
            continue;
        }
        PassArgs a = L.args;
        char *ib = (char *)bufs[L.in_buf];
        char *ob = (char *)bufs[L.out_buf];
        if (!ib || !ob) {
            set_last_error("missing buffer");
            return L.in_buf == B_WORK || L.out_buf == B_WORK ? FFTB_ERROR_NO_WORK_AREA : FFTB_ERROR_INVALID_VALUE;
        }
        a.in = ib + L.in_off_bytes;
        a.out = ob + L.out_off_bytes;
        a.pair_io = 0;
        if (L.pair_candidate) {
            const void *rp = L.real_side == 1 ? a.in : a.out;
            a.pair_io = ((uintptr_t)rp % L.real_align) == 0;
        }
        if (ep && L.ep_dynamic) {
            a.ep_scale = ep->scale;
            a.ep_sign = ep->sign;
            a.ep_gauss = ep->gauss;
            if (ep->mode >= 0) a.ep_mode = ep->mode;
        }
        void *args[] = {&a};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = L.grid;
        cfg.blockDim = dim3(L.block);
        cfg.dynamicSmemBytes = L.smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = L.programmatic ? 1 : 0;
        cudaError_t e = cudaLaunchKernelExC(&cfg, L.fn, args);
        if (e != cudaSuccess) return set_status_from_cuda(e);
    }
    if (timer) return timer_end(timer, stream);
    return FFTB_SUCCESS;
}

} // namespace fftb
