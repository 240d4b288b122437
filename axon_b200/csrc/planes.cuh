// Host/device interface of the bit-plane batched readout (planes.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace axon {

// Transposed W3 ("W3P"): per (column, branch, word of the presynaptic group) a block of
// kPlaneBlk words: 32 masks, mask j = the postsynaptic neurons (bit = lane) whose synapse
// with presynaptic neuron j is functional; then the six bit planes of the row counts (plane
// i = the neurons whose number of functional synapses in the word has bit i set); then two
// zero words, which padding entries of a record's position list point at.
constexpr uint32_t kPlaneBlk = 40;
// one (column, branch): the eight blocks and four words more, so that the row-count planes of
// different branches and words spread over all shared-memory banks
constexpr uint32_t kPlaneTile = 8u * kPlaneBlk + 4u;
constexpr uint32_t kPlaneCol = 32u * kPlaneTile;    // one column
constexpr uint32_t kPlanes = 14;                    // bit planes of a per-neuron drive (below 2^14)
constexpr uint32_t kPlanesMaxB = 512;               // trajectories per launch (the host splits larger batches)
constexpr uint32_t kPlanesVals = 1024;              // candidates a phase-2 group keeps in shared memory
constexpr uint32_t kPlanesList = 384;               // gated columns it lists there
// 640 threads leave 96 registers; tiles read through L2 want more warps (at most 28: a phase-2
// group keeps two words per warp beside its counters)
constexpr int planes_threads(bool direct) { return direct ? 896 : 640; }

constexpr uint32_t kPlanesDirectB = 160;            // most trajectories whose tiles are read through L2
// up to this width every column with a drive is a candidate: storing their planes costs less than
// recomputing gated columns after a threshold below the floor, which small networks meet often
// (us of a 30-step call, floor / all: 40 trajectories of whole cues 256 columns 800 / 726, 512: 806 /
// 671, 1,024: 740 / 772; of three quarters of a cue 544: 725 / 575, 576: 710 / 601; 300
// trajectories 544: 924 / 913, 576 with partial cues 1,093 / 993, 640: 913 / 1,055)
constexpr uint32_t kPlanesAllCols = 576;
constexpr uint32_t kNoSlot = 0xFFFFFFFFu;

// A network and the team's words for it.
struct PlanesNet {
  const uint32_t* W3P;    // [ncol][kPlaneCol]
  const uint32_t* conn;   // [ncol*32]
  uint32_t* act;          // [2][ngrp][astr] by step parity: bit j of word (g, k) = trajectory 32k + j spikes in group g
  uint32_t* bar;          // grid barrier counter (zeroed before the launch)
  const uint32_t* lanes;  // server: entry of each trajectory, or kNoSlot
  uint32_t astr, par;     // words per group of act; its parity that the launch's first step reads
};

// The server's tables: the CTAs and trajectories of one network, and one trajectory.
struct PlanesTeam {
  PlanesNet net;
  uint32_t cta0, ncta, B;
  uint32_t moved;  // lanes differ from those of the launch before: the first step's activity words are permuted
};
struct PlanesEntry {
  uint32_t slot;             // state slot
  uint32_t t0, clamp, steps;  // its step at the launch's first, clamped steps, all steps
  uint32_t ncue, cueOff;     // clamped input columns, in the launch's cue area
  uint32_t done;             // row of its final spikes when it ends in this launch
  uint32_t from;             // its lane in the launch before (a new trajectory's: one that no other has)
};

struct PlanesDev {
  PlanesNet net;            // (the server takes the team's)
  const uint32_t* biasP;    // [ncol][16] planes of min(bias >> shift, 2^14 - 1), or null (no bias)
  const uint32_t* multM;    // [ncol] neurons with multiplicity > 1 (with refBall)
  const uint32_t* stims;    // [B][ncol] clamp patterns
  const uint32_t* refBall;  // [B][ncol] logged reference assemblies, or null
  uint4* rec;               // [B][ngrp + ncol] per group the record of its first nonzero spike word, then per
                            // column the records of the further ones
  uint32_t* candB;          // [B][ncol/32] candidates of the step, a bit per column (zeroed before the launch)
  uint4* candP;             // [B][ncol][4] their drive planes (words 0..13); word 15: the ballot, in a step with more
                            // than kPlanesList gated columns
  uint4* aff;               // [ncol][32 * blocks][4] planes of the input groups' share of the drives, or null
  uint32_t* drv;            // column drives of the step, trajectory b's column c at b * drvB + c * drvC
  uint32_t* thPrev;         // [2][thStride] the last two thresholds, by step parity
  uint32_t* finalOut;       // [B][ncol] spikes of the last step (zeroed before the launch), or null
  uint32_t* hist;           // [B][T][ncol] spikes of every step (zeroed before the launch), or null
  uint32_t* stats;          // [B][1024] counters (zeroed before the launch), or null
  uint32_t* driveLog;       // [B][256] member-drive log (accumulated), or null
  uint32_t* err;            // device error word
  uint32_t drvB, drvC, thStride;
  // server (B counts state slots above): finalOut holds the rows of the trajectories that end
  const PlanesTeam* teams;  // by cta0, covering the grid
  const PlanesEntry* entries;
  const uint32_t* cues;
  uint32_t* teamNs;         // [nteams] duration of the launch on each team's first CTA
  uint32_t nteams;
};

struct PlanesCfg {
  uint32_t ncol, incols, B, T, clampSteps, k, dthr, mode, targetCols, topkPar;
  uint32_t bst;          // dendritic bonus per branch at or above dthr: boost (mode 1), 0 (mode 0)
  uint32_t allCand;      // 1: every column with a positive drive is a candidate
  uint32_t storeAll;     // 1: every column with a positive drive keeps its planes, candidate or not
  uint32_t slabAlways;   // 1: the first step after the clamp takes no floor of its own
  uint32_t ns, nl, ng;   // tile slots, list slots (0 when direct), phase-2 groups
  uint32_t nsl, nll;     // log2 of ns and nl
  uint32_t ls;           // log2 of the lanes per trajectory in phase 1
  uint32_t aff;          // 1: the afferent cache pays
  uint64_t waitNs;
};

struct PlanesShape {
  int grid;
  uint32_t direct;  // 1: tiles read through L2 as needed (few trajectories), 0: column tiles staged in shared memory
  size_t smem;
};

// Launch shape for B trajectories: fills the last fields of c.
PlanesShape planes_shape(uint32_t ncol, uint32_t B, int sms, PlanesCfg* c);
cudaError_t planes_max_blocks_per_sm(const PlanesCfg& c, const PlanesShape& s, int* out);
cudaError_t launch_recall_planes(const PlanesDev& d, const PlanesCfg& c, const PlanesShape& s, cudaStream_t st);
// The server's form: at most B trajectories in a team and `cols` columns in a CTA, `want`
// phase-2 groups; fills the last fields of c.
PlanesShape planes_serve_shape(uint32_t ncol, uint32_t B, int grid, uint32_t cols, uint32_t want, PlanesCfg* c);
cudaError_t planes_serve_prepare(const PlanesCfg& c);
cudaError_t launch_serve_planes(const PlanesDev& d, const PlanesCfg& c, const PlanesShape& s, cudaStream_t st);
// W3 [col][s][j][lane][comp] -> W3P
cudaError_t launch_make_w3p(const uint4* W3, uint32_t* W3P, uint32_t ncol, cudaStream_t st);
// bias planes and multiplicity masks (either output may be null)
cudaError_t launch_planes_aux(const uint32_t* bias, uint32_t biasShift, const uint32_t* mult, uint32_t* biasP,
                              uint32_t* multM, uint32_t ncol, cudaStream_t st);
// checks plane_kwta on columns that k_kwtatest has answered (see there)
cudaError_t launch_kwtatest_planes(const uint32_t* v, const uint32_t* k, uint32_t* out, uint32_t n, cudaStream_t st);

}  // namespace axon
