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

}  // namespace cf
