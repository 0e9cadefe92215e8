// Compact partition-function table shared by the host builder and the
// kernels: per (element, stage) up to FZ_PF_MAXV value pieces of
// src/atom_database.f90:121-1035 with 6 (zero-padded) Horner coefficients.
#pragma once
#ifndef FZ_PF_MAXV
#define FZ_PF_MAXV 3
#endif
#ifndef FZ_NELEM
#define FZ_NELEM 92
#endif

struct PFPiece {
  double c[6];
  double th, base, clamp;
  int cond, form, var, pad;
};
struct PFTable {
  PFPiece p[FZ_NELEM][3][FZ_PF_MAXV];
  int nv[FZ_NELEM][3];
};

// Derivative pieces (dlnU/dT) of src/atom_database.f90:121-1035 in the same
// padded form: the active piece is the last whose condition holds (on T, or
// on the value of the referenced value piece, ref < 0 = the stage's U);
// d = horner(c, var) * mult * (dx ? -1/T : 1) * (ub ? uref - base : 1) / (up ? uref : 1).
struct PFDPiece {
  double c[6];
  double th, base, mult;
  int cond, var, dx, ub, up, ref, pad0, pad1;
};
struct PFDTable {
  PFDPiece d[FZ_NELEM][3][3];
  int nd[FZ_NELEM][3];
};

// The pieces of one element that hold on an interval of T, for kernels that
// keep them in registers: per stage the active value piece and the active
// derivative piece (its factor in the coefficients).  An element's records run
// up in T and alternate between the open intervals between its thresholds and
// the thresholds themselves (lo = hi).
#define FZ_PF_MAXREC 13
struct PFRec {
  double c[3][6], bc[3], lo, hi;   // value coefficients; base, clamp or a limit that never holds; the interval
  int flags, dflags;               // bits 2s: variable of stage s; 6 + s: exponential form; as below
  double d[3][6], db[3], c5[3];    // derivative coefficients, base, condition 5's value
};
// dflags of stage s, from bit 10 s: 0-1 variable, 2 dx, 3 ub, 4 up, 5 condition
// 5, 6-7 the value piece of the factors + 1 where it is not the active one
struct PFRecTable {
  PFRec r[FZ_NELEM][FZ_PF_MAXREC];
  int n[FZ_NELEM];
};

// Fill t from the generated piece table (host).
void fzh_pf_table(PFTable* t);
// Fill t from the generated derivative pieces (host); returns 0, or -1 if a
// piece needs more than the padded form holds.
int fzh_pfd_table(PFDTable* t);
// Fill t from both (host); returns 0, or -1 if an element has more thresholds
// than the records hold or a piece needs what they do not.
int fzh_pf_records(const PFTable* v, const PFDTable* d, PFRecTable* t);
