// Planes per CTA of the kernels that march in z.  Plain C++, so the host tests
// can check the rule.
#pragma once

namespace ekc
{

// What a march costs, in units of one plane's work of one CTA.  A CTA that
// finishes kc planes does (kc + over) planes' work: the extra half planes and
// halo planes at its ends, its start-up and its share of the launch.  Alone on
// its SM it takes that time; of it, `share` is time in which the SM can do
// nothing else, the rest overlaps with other CTAs.
struct ChunkModel
{
  double share, over;
  int    fit; // up to this many CTAs per SM the number counts in whole CTAs
};
// Fitted on GB300 (planes per CTA from 1 to 32 on five to seven grids of 24^3
// to 200 x 180 x 160 each): the kernels then take 0.3 to 2.1 % longer on
// average than with each grid's best value, 6.4 % at most.
constexpr ChunkModel kChunkHydro64 = { 0.60, 3.0, 4 }, kChunkHydro32 = { 0.25, 2.0, 1 };
constexpr ChunkModel kChunkTrace64 = { 0.25, 2.0, 1 }, kChunkTrace32 = { 0.25, 2.5, 2 };
constexpr ChunkModel kChunkUpdate64 = { 0.35, 3.0, 5 }, kChunkUpdate32 = { 0.25, 2.5, 1 };

// Planes per CTA for `columns` tiles of `planes` planes on `sms` SMs: short
// chunks repeat the work at their ends, long ones leave SMs idle (16 planes put
// 8 CTAs on the 152 SMs for a 32^3 grid).  Of equal values the longest.
inline int
choose_chunk(long long columns, int planes, int sms, ChunkModel m)
{
  int    best = 1;
  double cost = 0.0;
  for (int kc = 1; kc <= planes && kc <= 64; ++kc)
  {
    const long long chunks = (planes + kc - 1) / kc;
    const double    n = (double)(columns * chunks) / sms; // CTAs per SM
    // work of the busiest SM: whole CTAs while they are few, else the mean
    const double work = n <= m.fit ? (kc + m.over) * (double)((columns * chunks + sms - 1) / sms)
                                   : (double)columns * (planes + m.over * chunks) / sms;
    const double c = (1.0 - m.share) * (kc + m.over) + m.share * work;
    if (kc == 1 || c <= cost)
    {
      cost = c;
      best = kc;
    }
  }
  return best;
}

} // namespace ekc
