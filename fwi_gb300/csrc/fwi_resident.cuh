// Launch parameters of the resident kernel (fwi_resident.cu).
#pragma once
#include <cuda_runtime.h>

#include "fwi_items.h"
#include "fwi_resident.h"

namespace fwi {

struct ResShot {
    const float* model;      // velocity or lambda, column-major with leading dimension ldv
    const float* srcv;       // injected values [vidx][nt]
    float* rec;              // Rec_point(nt, nrec)
    float* snaps;            // FP32 snapshots [s][ny][pitch]
    float* k32;              // imaging accumulator [ny][pitch], FP32 or FP64
    double* k64;
    int ldv, x0;             // leading dimension; first model column of the window
    int ny, nx, dn;
    int off, pitch;          // physical column of logical column 0; row pitch of snaps and the accumulator
    int pad_;
};

struct ResParams {
    const ResTile* tiles;
    const ResShot* shots;
    const ResSrc* src;
    const ResRec* rec;
    const int* rows;
    uint2* out;              // outboxes: words of a value and its step, zero before the launch
    size_t plane;            // words of one parity: even steps, then odd steps
    float* c2g;              // c2 of all tiles, filled by the launch
    int* err;                // set when a wait for a neighbour ran out
    const float* fA;         // CPML factors (dn entries)
    const float* fB;
    int nt;                  // stride of rec and srcv
    int steps;               // last time step k (2..steps)
    int store_snap, nt_store;
    int store;               // forward: store snapshots
    int record;              // forward: record receivers
    int from_lambda;
    int grad_form;
    float dt, rdt, ss;
    float dt2, d2;           // dt**2, d**2 of c2 = c**2*dt**2/d**2
    float c1[MAXR + 1], c2[MAXR + 1];
};

cudaError_t launch_resident(int acc, int mode, const ResParams& p, int tiles, size_t smem, cudaStream_t st);
// Resident blocks per SM of both modes' kernels.
cudaError_t resident_blocks(int acc, size_t smem, int* blocks);
cudaError_t configure_resident();

}  // namespace fwi
