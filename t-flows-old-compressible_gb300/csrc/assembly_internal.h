// Device-resident mesh data shared by the pressure-correction assembly
// (assembly.cu) and the momentum assembly (momentum.cu).
#pragma once

#include <cuda_runtime.h>

#include <string>

constexpr int kAsmBlock = 256;

// Library/allp_mod.f90:16-24
enum : int {
    kInflow = 1,
    kWall = 2,
    kOutflow = 3,
    kConvect = 5,
    kWallfl = 6,
    kBuffer = 11,
    kPressure = 12
};

// A block's sums of b volume and volume, and its largest |b| (the bits).
struct AsmPartial {
    double sum, vol;
    unsigned long long errmax;
};

// What the kernels tell the host, in mapped host memory: read after the
// stream is synchronised, without a copy.
struct AsmNote {
    volatile unsigned long long errmax_bits;  // of the last CalcPS
    volatile int blend, material;             // input errors of the last NewUVW
};

struct tflows_assembly {
    int device = 0;
    int NC = 0, NbC = 0, NS = 0, NONZ = 0;
    int nblocks = 0;
    // every entry 0..NONZ-1 is the diagonal of one cell or belongs to one side
    // of one interior face: an assembly sets each entry once
    bool single = false;
    int *c1 = nullptr, *c2 = nullptr, *sid1 = nullptr, *sid2 = nullptr;
    int *adia = nullptr, *type = nullptr, *cf_ptr = nullptr;
    // each interior cell's faces in increasing order: entry e holds the face
    // (0-based) where the cell is the face's c1, its complement ~s where it
    // is the face's c2 (entries cf_ptr[i] .. cf_ptr[i+1]-1 of cell i + 1)
    int* slot_face = nullptr;
    // the cell across that face (c at [c + NbC]), -1 across a boundary face
    // that is not BUFFER
    int* slot_cell = nullptr;
    // each boundary cell's faces in increasing order (cell c = j - NbC at
    // bnd_ptr[j] .. bnd_ptr[j+1]-1)
    int *bnd_ptr = nullptr, *bnd_face = nullptr;
    double* geom = nullptr;  // Sx Sy Sz Dx Dy Dz f SMDPN (1-f), NS each
    double* vol = nullptr;   // -NbC..NC
    double2* rec = nullptr;  // per face: A12 and the flux, and what it adds
    unsigned char* kind = nullptr;
    AsmPartial* parts = nullptr;  // one per block
    double* sums = nullptr;       // the two totals and their quotient
    unsigned* done = nullptr;     // blocks of the cell pass that have finished
    AsmNote *note = nullptr, *d_note = nullptr;
    // momentum assembly, allocated on its first call
    void* mom_rec = nullptr;        // one record per face
    double* mom_cells = nullptr;    // rhoUi, PHImax, PHImin over -NbC..NC
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

namespace tflows {
int report_status(int status, const std::string& msg);
}
