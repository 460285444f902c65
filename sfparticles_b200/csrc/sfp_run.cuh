// sfp_run.cuh -- device-side layout of a fused-step run, shared by the host
// C-ABI (nvcc) and the NVRTC-compiled step modules.
//
// A step runs up to three kernels:
//   massive -- warp tiles over the e+- (massive) segments, streamed through
//              a ring of asynchronous copies: QED photon emission at t; an
//              emitter is marked (pruned = 2) with its delta stored and is
//              left unpushed, every other particle is pushed to t+dt;
//              per-tile emission counts, summed per super-tile of 64;
//   photon  -- warp tiles over the photon segments: pair creation (the
//              converted photon is marked and its delta stored), photon
//              push; per-tile event counts, summed per super-tile.  Its last
//              block scans both groups' super-tile counts (segmented by
//              instance, per append channel) into the step's append counts
//              and checks the room of every destination exactly;
//   appends -- photon children of the marked emitters (then their recoil
//              and push) and e-/e+ children of the marked photons (pushed),
//              each written at the slot the reference's find_event_index +
//              create_* gives it.
// The last block of the step's last event launch folds the step's appends and
// prepares the next step; a bookkeeping kernel prepares the first of a call.
// Both groups' segments start at multiples of 64 tiles, so a super-tile
// never spans two segments.  No block of these launches waits for another.
// Small populations take several steps in one cooperative launch instead
// (sfp_steps_body), whose blocks meet at three grid barriers a step, each wait
// with a time limit.
#pragma once
#include "sfp_types.h"

// Tile length.  Each step of three launches the bookkeeping gives each group the
// shortest power-of-two tile from SFP_TILE_MIN to SFP_TILE_MAX particles that cuts
// its population into at most SFP_TILE_TARGET tiles (massive group:
// SFP_TILE_TARGET_M): a large population keeps 1024-particle tiles (32
// sub-steps of the copy ring per ticket), a small one is spread over every
// warp of the grid instead of running a few long tiles serially.  An e+-
// takes ten times a photon's work, so its tiles are shorter: 1e6 e- as 3900
// tiles of 256 gave 3552 resident warps one or two each, half of the last
// round idle; as 15600 tiles of 64, 64 -> 50 us (float32 form, rejection
// sampling), 183 -> 122 us (spin, learned sampler).  Results do not depend on
// the tile: draws are keyed by particle index and children are written in
// index order.  The tile counters hold SFP_TILE_TARGET_M tiles plus the
// segments' padding at least, so the rule always fits.  The one-launch kernel's
// tiles are shares of the work, any multiple of 32 (sfp_small_tile).
#define SFP_TILE_MIN 32
#define SFP_TILE_MAX 1024
#define SFP_TILE_TARGET 4096
#define SFP_TILE_TARGET_M 16384

// what a step is planned with: its time and number, and each group's tiles
struct sfp_step_plan {
    double t;
    long long step;
    long long n_mtiles;         // massive-group tiles
    long long n_ptiles;         // photon-group tiles
    int mtile;                  // particles per massive-group tile
    int ptile;                  // particles per photon-group tile
};

struct sfp_step_state {
    double t;                   // time of the next step
    long long step;             // steps completed
    sfp_step_plan plan[2];      // the next step's plan in slot `cur`, the last one's in the other
    int cur;
    int mticket;                // next massive tile to hand out
    int pticket;                // next photon tile to hand out
    int skip;                   // 1: the prepared step must not run
    int halted;                 // sticky: a destination lacked room (host regrows, resumes)
    int error;                  // sticky device error (SFP_DEV_*)
    int blocks_done;            // blocks of the running launch that are done (sfp_last_block)
    int hot_ok;                 // the running call's store of hot photons holds all of them
    unsigned int barrier;       // arrivals at the grid barriers of the running launch (sfp_steps_body)
    int append_wait;            // the step in slot `cur` stopped before writing its children (no room)
    long long particle_steps;   // sum over executed steps of all N_buffered
    // Photons fly straight: a photon segment stores each position as of the
    // start of step pos_epoch, and the photon at the start of step `step`
    // is at stored + (step - pos_epoch) * (its one-step displacement).  The
    // step kernels advance positions in registers only; sfp_sync_positions
    // writes them out and moves pos_epoch to step.
    long long pos_epoch;
};

// a segment as the end of a step walks it (sfp_step_end)
struct sfp_end_seg {
    int super0;                 // first super-tile in the sequence of both groups'
    int chain;                  // instance and group
    int channel;
    int dest0, dest1;           // segments that its events append to, or -1
};

// segments whose data sfp_step_end holds in shared memory; runs of more keep
// them in the run's own scratch (end_seg, end_app, end_nb)
#define SFP_END_SEGS 768
// shared memory of sfp_step_end: the launch's dynamic shared memory, whose
// tables and rings the block no longer needs (every launch that ends a step,
// and sfp_book_kernel, has this much)
struct sfp_end_smem {
    uint4 wv[8];
    unsigned int wh[8];
    long long tiles[2], ps[8];
    int tile[2];
    int lacks, pad;
    sfp_end_seg seg[SFP_END_SEGS];
    unsigned long long app[SFP_END_SEGS];
    long long nb[SFP_END_SEGS];
};

// one group of tiles (massive or photon): the tile map of its segments and
// its per-tile / per-super-tile event counts
struct sfp_group_dev {
    const int* seg;             // [n_seg] segment indices, in segment order
    long long* tile_start;      // [2][n_seg + 1] per plan slot: first tile of each segment (multiples of 64)
    unsigned int* tile_cnt;     // [max_tiles] events per tile
    unsigned int* super_cnt;    // [max_tiles / 64 + 2] events per super-tile
    long long* super_pre;       // [max_tiles / 64 + 2] exclusive prefix in its instance, per channel
    long long max_tiles;
    int n_seg;
    int pad;
};

// The photons whose pair test can pass somewhere in the field (sfp_step.cuh,
// "hot photons"), copied out of their segments for one sfp_run_steps call:
// entries start[s] .. start[s] + count[s] - 1 are segment s's, each its
// photon's index, stored position and momentum (float32 form: as float32,
// all that its tests read).  A converted photon's entry gets index SFP_HOT_DEAD.
#define SFP_HOT_DEAD 0xFFFFFFFFu
struct sfp_hot_dev {
    double *x, *y, *z;
    void *ux, *uy, *uz;           // float or double
    unsigned int* idx;
    const long long* start;       // [n_seg]
    const long long* cap;         // [n_seg] room of a segment's entries
    unsigned long long* count;    // [n_seg]
};

struct sfp_run_dev {
    const sfp_segment* seg;
    const sfp_instance* inst;
    int n_seg;
    int n_inst;
    double dt;
    double photon_threshold;
    int qed;                    // SFP_QED_*
    int pad_tile;
    int any_rad;                // some massive segment radiates
    int any_bw;                 // some photon segment creates pairs
    int n_dseg;                 // segments receiving children (photons or pairs)
    int m_ring_off;             // massive kernel: byte offset of its copy ring in dynamic smem
    int m_stage_bytes;          // massive kernel: bytes per ring stage (the run's widest segment layout)
    int ring_off;               // photon kernel: byte offset of its copy ring in dynamic smem
    int mlp_off;                // massive kernel: byte offset of the network weights in dynamic smem
    int small_ring;             // one-launch kernel: bytes of a warp's ring (at m_ring_off)
    int small_end_off;          // one-launch kernel: byte offset of sfp_end_smem in dynamic smem
    int pad1;
    const int* dseg;            // [n_dseg]
    sfp_group_dev mg;           // massive group
    sfp_group_dev pg;           // photon group
    sfp_rs_table rs;
    sfp_od_table od_photon;
    sfp_od_table od_pair;
    long long* n_buffered;        // [n_seg] authoritative buffered counts
    unsigned long long* appended; // [n_seg] children appended by the running step
    long long* n_buf_step;        // [2][n_seg] per plan slot: counts at the start of the step
    sfp_end_seg* end_seg;         // [n_seg] scratch of sfp_step_end for runs of many segments
    unsigned long long* end_app;  // [n_seg]
    long long* end_nb;            // [n_seg]
    const float* mlp_params;      // learned photon-energy sampler (optical depth), or NULL: the table
    sfp_step_state* st;
    // rejection sampling: per chi bin an upper bound of the pair rate over
    // every delta (SFP_PAIR_BOUND_BINS floats, the bins of sfp_pair_bin), so
    // photons whose pair test no draw can pass skip the draw; then its prefix
    // maximum (as many floats)
    const float* pair_bound;
    sfp_hot_dev hot;              // x NULL: no store
};

// chi bins of the pair-rate bound: the float's exponent and 3 mantissa bits
// from chi = 2^-16 up; bin 0 also holds every smaller chi, the last bin
// (bound +inf) every larger one
#define SFP_PAIR_BOUND_BINS 256
#define SFP_PAIR_BOUND_BASE ((127 - 16) << 3)
SFP_DEVICE_INLINE int sfp_pair_bin(float chi) {
    int k = (int)(__float_as_uint(chi) >> 20) - SFP_PAIR_BOUND_BASE;
    return k < 0 ? 0 : (k > SFP_PAIR_BOUND_BINS - 1 ? SFP_PAIR_BOUND_BINS - 1 : k);
}
