// hydro.cuh — P4 (hydro), P8 (floors) and P1/P9 (Δt) kernel entry points.
#pragma once

#include "common.cuh"

enum { kHydroUpdate = 0, kHydroPredict = 1, kHydroStep = 2 };

// The Δt record kept on the device (crates/sr-engine/src/step/dt.rs:51-61): steps never wait on the host for it.
struct DtRecord {
    double dt;        // Δt_n of the last step
    double dt_next;   // Δt_{n+1}
    double sim_time;  // Σ Δt, f64
    unsigned long long steps;
    int non_finite;
    int nf_channel;
    long long nf_cell;
    unsigned long long nf_step;
};

// P9's rule for the next Δt, and where the step's Δt record lives.
struct DtRule {
    double cfl, eta_g, dt_fixed, dt_cap;
    DtRecord* rec;
    int advance;  // 1: a step ends here (its Δt, the sim time and the step count are booked)
};

struct HydroArgs {
    HydroConst H;
    const double* dt;          // device Δt_n
    const float* U;            // state in: 4 planes
    float* Uout;               // state out: 4 planes
    const float* gx;           // P2's field of the start state (nullptr: no gravity)
    const float* gy;
    float* src;                // kHydroPredict: out; hydro_gravity: in (Σ_src,mid; -0 where the cell is empty)
    float* mid;                // likewise: the half-step Σ, Σu, Σv (3 planes)
    float* mfx;                // likewise: the mass flux through each cell's +x and +y face
    float* mfy;
    const float* phim;         // the half step's φ, g (hydro_gravity)
    const float* gxm;
    const float* gym;
    void* part;                // partials of the grid's sums (hydro_part_count x kHydroPartBytes)
    unsigned* tickets;         // hydro_ticket_count counters, 0 between launches
    DtRule rule;               // kHydroStep
    int* err;                  // set to 1 when a bounded wait of the kernel gave up (its TMA box never landed)
};

size_t hydro_smem_bytes();
constexpr size_t kHydroPartBytes = 24;
size_t hydro_part_count(int w, int h);
size_t hydro_ticket_count(int h);
void hydro_launch(int mode, const HydroArgs& A, cudaStream_t s);
// After kHydroPredict and the half step's solve: gravity's kick and work on Uout, the net kick taken back.
void hydro_gravity_launch(const HydroArgs& A, cudaStream_t s);

int floors_dt_blocks(int w, int h);
void floors_dt_launch(const HydroConst& H, float* U, const float* gx, const float* gy, int do_floors, float* part_rate,
                      float* part_g, long long* part_nf, unsigned* ticket, const DtRule& rule, cudaStream_t s);
// Δt_{n+1} and the guard from per-CTA partials (the guard's codes are cell * channels + channel).
void dt_finalize_launch(int nblocks, int channels, const float* part_rate, const float* part_g,
                        const long long* part_nf, const DtRule& rule, cudaStream_t s);
