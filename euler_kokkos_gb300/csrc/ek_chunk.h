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

// Cost of `ctas` CTAs that finish kc planes each, `planes` CTA planes in all.
inline double
chunk_cost(int kc, long long ctas, double planes, int sms, const ChunkModel & m)
{
  const double n = (double)ctas / sms; // CTAs per SM
  // work of the busiest SM: whole CTAs while they are few, else the mean
  const double work = n <= m.fit ? (kc + m.over) * (double)((ctas + sms - 1) / sms) : (planes + m.over * ctas) / sms;
  return (1.0 - m.share) * (kc + m.over) + m.share * work;
}

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
    const long long ctas = columns * ((planes + kc - 1) / kc);
    const double    c = chunk_cost(kc, ctas, (double)columns * planes, sms, m);
    if (kc == 1 || c <= cost)
    {
      cost = c;
      best = kc;
    }
  }
  return best;
}

// The 2D hydro marches: strips of kRowCols columns, CTAs of kRowWarps warps on
// consecutive runs of rows (a "plane" above is a row of each warp).  Fitted on
// runs of 1 to 32 rows; us per step, mixed, with 1 / 2 / 4 / 8 / 16 / 32 rows and by
// the rule: 64^2 7.9 / 8.4 / 9.6 / 11.1 / 16.1 / 24.3, 7.9; 512^2 21.7 / 15.7 / 13.1 /
// 13.3 / 16.0 / 24.4, 13.2; 1022 x 518 36.8 / 25.7 / 20.2 / 18.7 / 21.4 / 29.5, 19.4;
// 1024^2 67 / 45 / 33 / 27.6 / 25.5 / 35.5, 27.6; 2048^2 258 / 160 / 114 / 91.9 /
// 84.1 / 80.5, 84.1.
constexpr int kRowCols = 28, kRowWarps = 4;
constexpr ChunkModel kChunkRows64 = { 0.60, 2.0, 8 }, kChunkRows32 = { 0.35, 2.0, 2 };
inline int
row_strips(int nx)
{
  return (nx + kRowCols - 1) / kRowCols;
}
inline int
row_groups(int ny, int rows)
{
  return (ny + kRowWarps * rows - 1) / (kRowWarps * rows);
}
// rows of a warp's run for the n grids of nx[i] x ny[i] cells of one launch
inline int
choose_rows(const int * nx, const int * ny, int n, int sms, ChunkModel m)
{
  double planes = 0.0, cost = 0.0;
  int    most = 1, best = 1;
  for (int i = 0; i < n; ++i)
  {
    planes += (double)row_strips(nx[i]) * ny[i] / kRowWarps;
    most = ny[i] > most ? ny[i] : most;
  }
  for (int rows = 1; rows <= most && rows <= 64; ++rows)
  {
    long long ctas = 0;
    for (int i = 0; i < n; ++i)
      ctas += (long long)row_strips(nx[i]) * row_groups(ny[i], rows);
    const double c = chunk_cost(rows, ctas, planes, sms, m);
    if (rows == 1 || c <= cost)
    {
      cost = c;
      best = rows;
    }
  }
  return best;
}

} // namespace ekc
