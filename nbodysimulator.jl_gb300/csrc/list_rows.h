// list_rows.h - the capacity of a Verlet-list row (host only).
//
// A row is a whole number of 32-byte units (8 entries): the force kernels'
// tensor map wants a row stride that is a multiple of 16 bytes, and the
// replica loop reads its rows as 16-byte vectors from byte 4 * capacity *
// atom on. At least 32 entries: the replica loop spreads a row of c 16-bit
// entries over whole blocks of 8 entries per lane (64 with 8 lanes), which
// the row's 2 * capacity halves have to hold.
#pragma once

inline int list_row_capacity(int entries)
{
    const int whole = (entries + 7) / 8 * 8;
    return whole < 32 ? 32 : whole;
}

// after rows overflowed: half as much again and 32
inline int list_grown_capacity(int cap) { return list_row_capacity(cap + cap / 2 + 32); }
