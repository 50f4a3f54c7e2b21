// Length of the evaluator's wall-flux buffer (EvalD::fluxWall): the integral [8], then one row of up to 6
// partial sums per block of the boundary-face reduction.
#pragma once
namespace dndsb
{
constexpr int kWallFluxBlocks = 148;
constexpr int kWallFluxLen = 8 + kWallFluxBlocks * 6;
} // namespace dndsb
