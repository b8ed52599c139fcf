// Tables of the FP64 Dupire kernel's fixed-point form (fixed64.h), made on the host.
#pragma once
#include <vector>

#include "fixed64.h"

namespace cf {

// A Dupire plan's steps in doubles.
struct FxInput
{
    int nSteps = 0;
    NodeStride node = {1, 1};     // of the reverse's slab
    double x0 = 0;                // log S0
    std::vector<double> X;        // knots, log S - log S0
    std::vector<double> Y;        // [nSteps][X.size()] sqrt(dt) sigma
    std::vector<double> sq, tw;   // sqrt(dt) and the weight of column colB per step
    std::vector<int> colA, colB;
};

struct FxHost
{
    int nSteps = 0, nS = 0;
    int r = 0, sh = 0, shift = 0, x0h = 0;
    long long center = 0, grid = 1;
    std::vector<long long> bucket, inv;
    std::vector<FxInterval> interval;
    std::vector<FxVol> vol;
    std::vector<double> slope;
    std::vector<FxStep> step;
};

// False when a magnitude does not fit with up to four bits of range (the generic kernel then runs):
// states that could pass 2^8, vols of 16 or slopes of that order, knots closer than 2^-24 or needing
// more than 4096 buckets, values that are not numbers.
bool fx_lower(const FxInput& in, FxHost& h);

// The last state with r bits of range whose spot exp(logSpot + y) is not above level (at the ends of the
// type where none or every state is).  The logarithm is taken to twice a double's precision: a
// barrier's survival factor multiplies an error of its level by barrier / band width, the same on all paths
// (60x30 weekly barrier, 2^18 paths: a double's logarithm cost the mean price up to 3.7e-15).
long long fx_state(double level, double logSpot, int r);

// The same with today's state (0), which all paths share at a product's first date and every state of a model
// without vol is, above the level when today's spot as a double is: on a level that is today's spot, a
// payoff's or barrier's slope is one side's or the other's for all of them.
inline long long fx_today(double level, double spot, long long state)
{
    return spot > level ? (state < 0 ? state : -1) : (state > 0 ? state : 0);
}

}  // namespace cf
