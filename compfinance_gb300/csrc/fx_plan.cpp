// Device tables of the generators (inverse normals, Sobol), and of the FP64 Dupire kernel's fixed-point form
// (fx_tables.h, mc_dupire_fx64.cuh), built on the first FP64 value or risk run of a (model, product) pair.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <future>
#include <vector>

#include "engine.h"
#include "host_math.h"

namespace cf {

// The generators' inverse normal tables and the exponential's, made once per process (20 ms of host work for
// each of the former, on several cores).
namespace {
struct Tables
{
    std::vector<FxgPiece> g;
    unsigned brk[3];
    long long e[1 << FX_EXP_BITS];
    Tables() : g(size_t(3) * FXG_PIECES)
    {
        auto make = [this](int k) { brk[k] = inv_normal_table64(k, &g[size_t(k) * FXG_PIECES]); };
        auto a = std::async(make, 0), b = std::async(make, 1);  // in this thread where no other can be had
        make(2);
        exp_table64(e);
        a.get();
        b.get();
    }
};
}  // namespace

int Context::initGauss()
{
    static const Tables t;
    std::copy(t.brk, t.brk + 3, fxgBrk);
    const size_t n = t.g.size() * sizeof(FxgPiece);
    int rc = fxg.ensure(n + sizeof(t.e));
    if (rc) return rc;
    rc = fxg.upload(t.g.data(), n, stream);
    return rc ? rc : fxg.upload(t.e, sizeof(t.e), stream, n);
}

int Context::sobolTables(int dim, McParams& p)
{
    DevBuf& b = sobolTabs[dim];
    if (!b.ptr)
    {
        std::vector<uint32_t> t = sobol_dirs(dim);
        t.resize(size_t(64) * dim, 0u);
        uint32_t* low = t.data() + size_t(32) * dim;
        for (int d = 0; d < dim; ++d)
            for (int l = 1; l < 32; ++l) low[d * 32 + l] = low[d * 32 + l - 1] ^ t[size_t(__builtin_ctz(l)) * dim + d];
        int rc = b.ensure(t.size() * 4);
        if (!rc) rc = b.upload(t.data(), t.size() * 4, stream);
        if (rc)
        {
            sobolTabs.erase(dim);  // the next plan of this size starts afresh
            return rc;
        }
        h2d += t.size() * 4;
    }
    p.sobolDir = static_cast<const unsigned*>(b.ptr);
    p.sobolLow = p.sobolDir + size_t(32) * dim;
    return CF_OK;
}

void Context::setGenerator(McParams& p, bool sobol) const
{
    p.mrgJumpA = jumpA;
    p.mrgJumpB = jumpB;
    p.invnF = sobol ? invnSobol : invnMrg;
    const FxgPiece* g = static_cast<const FxgPiece*>(fxg.ptr);
    p.fx.g[0] = g + size_t(sobol ? FXG_SOBOL_LOWER : FXG_MRG) * FXG_PIECES;
    p.fx.g[1] = g + size_t(sobol ? FXG_SOBOL_UPPER : FXG_MRG) * FXG_PIECES;
    p.fx.expTab = reinterpret_cast<const long long*>(g + size_t(3) * FXG_PIECES);
    p.fx.brk[0] = fxgBrk[sobol ? FXG_SOBOL_LOWER : FXG_MRG];
    p.fx.brk[1] = fxgBrk[sobol ? FXG_SOBOL_UPPER : FXG_MRG];
}

bool Context::fxReady(Plan& plan)
{
    if (plan.fxState != 0) return plan.fxState > 0;
    FxHost h;
    const bool ok = fx_lower(plan.fxIn, h);
    if (ok)
    {
        std::vector<unsigned char> buf;
        auto put = [&](const void* src, size_t n) {
            const size_t off = (buf.size() + 255) & ~size_t(255);
            buf.resize(off + n);
            std::memcpy(buf.data() + off, src, n);
            return off;
        };
        auto vec = [&](const auto& v) { return put(v.data(), v.size() * sizeof(v[0])); };
        const size_t oB = vec(h.bucket), oI = vec(h.interval), oN = vec(h.inv), oV = vec(h.vol), oS = vec(h.slope),
                     oT = vec(h.step);
        // without memory for them this run is the generic kernel's, and the next one tries again
        if (plan.fxTables.ensure(buf.size()) || plan.fxTables.upload(buf.data(), buf.size(), stream)) return false;
        h2d += buf.size();
        const char* d = static_cast<const char*>(plan.fxTables.ptr);
        FxParams& f = plan.fx;
        std::memset(&f, 0, sizeof(f));
        f.r = h.r;
        f.sh = h.sh;
        f.center = h.center;
        f.grid = h.grid;
        f.half = h.grid << 31;
        f.nBuckets = int(h.bucket.size());
        f.shift = h.shift;
        f.x0h = h.x0h;
        f.bucket = reinterpret_cast<const long long*>(d + oB);
        f.interval = reinterpret_cast<const FxInterval*>(d + oI);
        f.inv = reinterpret_cast<const long long*>(d + oN);
        f.vol = reinterpret_cast<const FxVol*>(d + oV);
        f.slope = reinterpret_cast<const double*>(d + oS);
        f.step = reinterpret_cast<const FxStep*>(d + oT);
        f.node = plan.fxIn.node;
        const double x0 = plan.base.x0d, spot = std::exp(x0);
        f.yTop = fx_today(plan.base.barSmooth, spot, fx_state(plan.base.barSmooth, x0, h.r));
        f.yBand = fx_today(plan.base.minusSmooth, spot, fx_state(plan.base.minusSmooth, x0, h.r));
        const double w = plan.fxTop - plan.fxBand, top = plan.base.barSmooth / plan.base.twoSmooth;
        if (w >= 0.0 && w < std::ldexp(0.99, -FX_SMOOTH_BITS)) f.bandScale = top * std::ldexp(1.0, -3 - 62);
    }
    plan.fxState = ok ? 1 : -1;
    plan.fxIn = FxInput();
    return ok;
}

// Range of a risk launch's vol adjoints: a slab word of 96 bits takes at most `block` paths x (steps that
// share its time column) of them, each below 2^53 units of 2^-(60 - nodeShift).  It must not depend on the
// run's size: larger adjoints are split in doubles, and round differently.
int fx_node_shift(const Plan& plan, int block)
{
    int s = 30;
    while (s > 0 && std::ldexp(1.0, 95 - 53 - s) <= double(block) * std::max(1, plan.fxTouch)) --s;
    return s;
}

}  // namespace cf
