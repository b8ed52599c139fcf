// Host check of the device tables' uploads against fake_cudart.h: complete when the call returns, whatever
// stream their readers run on, and made again after a failure; buffers that cannot be had.
#include "fake_cudart.h"

#include <chrono>
#include <cmath>
#include <cstdio>
#include <ctime>
#include <thread>

#include "host_math.h"

using namespace cf;

static cudaStream_t const kStream = reinterpret_cast<cudaStream_t>(0x1000);

static int check(const char* what, bool ok)
{
    std::printf("%s %s\n", ok ? "ok" : "BAD", what);
    return !ok;
}

static bool sobolRight(const McParams& p, int dim)
{
    const std::vector<uint32_t> d = sobol_dirs(dim);
    if (std::memcmp(p.sobolDir, d.data(), size_t(32) * dim * 4)) return false;
    for (int k = 0; k < dim; ++k)
        for (int l = 0; l < 32; ++l)
        {
            const unsigned g = unsigned(l) ^ (unsigned(l) >> 1);
            unsigned s = 0;
            for (int b = 0; b < 5; ++b)
                if (g >> b & 1) s ^= d[size_t(b) * dim + k];
            if (p.sobolLow[k * 32 + l] != s) return false;
        }
    return true;
}

static int sobol()
{
    int bad = 0;
    for (int dim : {1, 13, 520})
    {
        Context c;
        c.stream = kStream;
        McParams p{};
        bad += check("sobol tables: call", c.sobolTables(dim, p) == CF_OK);
        bad += check("sobol tables: complete on return", !fake::inFlight() && sobolRight(p, dim));
        fake::arrive(nullptr);
    }
    for (int kind = 0; kind < 2; ++kind)
    {
        Context c;
        c.stream = kStream;
        McParams p{};
        (kind ? fake::failCopies : fake::failAllocs) = 1;
        const size_t held = fake::device.size();
        bad += check("sobol tables: failure reported", c.sobolTables(13, p) != CF_OK);
        bad += check("sobol tables: nothing kept after a failure", fake::device.size() == held);
        bad += check("sobol tables: made again", c.sobolTables(13, p) == CF_OK && !fake::inFlight() && sobolRight(p, 13));
        fake::arrive(nullptr);
    }
    return bad;
}

static int gauss()
{
    Context c;
    c.stream = kStream;
    int bad = check("inverse normal tables: call", c.initGauss() == CF_OK);
    McParams p{};
    std::vector<FxgPiece> t(FXG_PIECES);
    bool ok = !fake::inFlight();
    for (int sobol = 0; sobol < 2; ++sobol)
    {
        c.setGenerator(p, sobol != 0);
        for (int h = 0; h < 2; ++h)
        {
            const int g = !sobol ? FXG_MRG : h ? FXG_SOBOL_UPPER : FXG_SOBOL_LOWER;
            ok = ok && inv_normal_table64(g, t.data()) == p.fx.brk[h] &&
                 !std::memcmp(t.data(), p.fx.g[h], t.size() * sizeof(t[0]));
        }
    }
    long long e[1 << FX_EXP_BITS];
    exp_table64(e);
    ok = ok && !std::memcmp(e, p.fx.expTab, sizeof(e));
    bad += check("inverse normal and exponential tables: complete on return", ok);
    fake::arrive(nullptr);
    return bad;
}

// A buffer that cannot be had: a status, nothing held, and no error left for the next launch's check.
static int allocations()
{
    int bad = 0;
    for (int kind = 0; kind < 3; ++kind)
    {
        DevBuf d;
        PinnedBuf h;
        auto get = [&](size_t n) { return kind == 2 ? h.ensure(n) : d.ensure(n, kind ? kStream : nullptr); };
        bad += check("buffer: small", get(1000) == CF_OK);
        fake::failAllocs = 1;
        bad += check("buffer: out of memory", get(size_t(100) << 20) == CF_E_NOMEM);
        bad += check("buffer: no error left behind", cudaGetLastError() == cudaSuccess);
        bad += check("buffer: nothing held", !d.ptr && !d.bytes && !h.ptr && !h.bytes);
        bad += check("buffer: smaller form", get(2000) == CF_OK);
    }
    return bad;
}

// The fixed-point tables of a plan: a failed upload sends that run to the generic kernel, not all later ones.
static int fixedPoint()
{
    int bad = 0;
    for (int kind = 0; kind < 3; ++kind)
    {
        Context c;
        c.stream = kStream;
        Plan plan;
        plan.fxState = 0;
        FxInput& in = plan.fxIn;
        in.nSteps = 2;
        in.x0 = std::log(100.0);
        in.X = {-0.5, 0.0, 0.7};
        in.Y = {0.05, 0.06, 0.07, 0.04, 0.05, 0.06};
        in.sq = {0.25, 0.25};
        in.tw = {0.0, 0.5};
        in.colA = {0, 0};
        in.colB = {0, 1};
        FxHost h;
        bad += check("fixed point: lowered", fx_lower(in, h));
        if (kind) (kind == 1 ? fake::failAllocs : fake::failCopies) = 1;
        if (kind) bad += check("fixed point: failure reported", !c.fxReady(plan) && plan.fxState == 0);
        bad += check("fixed point: built", c.fxReady(plan) && plan.fxState == 1 && !fake::inFlight());
        bad += check("fixed point: tables", plan.fx.vol && !std::memcmp(plan.fx.vol, h.vol.data(), h.vol.size() * sizeof(h.vol[0])) &&
                                                !std::memcmp(plan.fx.bucket, h.bucket.data(), h.bucket.size() * 8));
        bad += check("fixed point: kept", c.fxReady(plan));
    }
    Context c;
    Plan plan;
    plan.fxState = 0;
    plan.fxIn.nSteps = 1;
    plan.fxIn.X = {0.0, 1e-12};  // knots too close
    plan.fxIn.Y = {0.05, 0.06};
    plan.fxIn.sq = {0.25};
    plan.fxIn.tw = {0.0};
    plan.fxIn.colA = plan.fxIn.colB = {0};
    bad += check("fixed point: refused for good", !c.fxReady(plan) && plan.fxState == -1 && !c.fxReady(plan));
    return bad;
}

// The first context of a process makes the inverse normal tables: on several cores, not one after the other.
static int firstContext()
{
    if (std::thread::hardware_concurrency() < 4) return check("first context: too few cores to tell", true);
    const auto t0 = std::chrono::steady_clock::now();
    const std::clock_t c0 = std::clock();  // of all threads
    Context c;
    c.stream = kStream;
    const int bad = check("first context: call", c.initGauss() == CF_OK);
    const double wall = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() * 1e3;
    const double cpu = double(std::clock() - c0) / CLOCKS_PER_SEC * 1e3;
    std::printf("%s first context: %.1f ms for %.1f ms of work\n", wall < 0.6 * cpu ? "ok" : "BAD", wall, cpu);
    return bad + !(wall < 0.6 * cpu);
}

int main()
{
    const int bad = firstContext();
    return bad + sobol() + gauss() + allocations() + fixedPoint() != 0;
}
