// Where aligned accesses may go: copies of whole words and 16-byte vectors from arrays that start or end between two
// boundaries stay inside the array.  Plain arithmetic on addresses, usable on the host too.
#pragma once
#include <stddef.h>

#ifdef __CUDACC__
#define FTB_HD __host__ __device__ __forceinline__
#else
#define FTB_HD inline
#endif

namespace ftb200 {

// A row of `cols` 16-bit columns, as vectors counted from the 16-byte boundary at or before its first column.
struct RowSpan {
    size_t base;  // address of vector 0
    int    mis;   // columns between it and the row's first
    int    nv;    // vectors that hold columns of the row
};
FTB_HD RowSpan row_span(size_t row, int cols)
{
    RowSpan   S;
    const int off = (int)(row & 15);
    S.base        = row - (size_t)off;
    S.mis         = off / 2;
    S.nv          = (S.mis + cols + 7) / 8;
    return S;
}

// Which vectors of row r of a [rows, stride] tensor lie inside the tensor and can be copied whole: its first row may reach
// back over its start with vector 0, its last one over its end with the last vector.  The columns of those two are loaded
// one by one.  (Rows are counted up to eight: that many hold a vector's columns however short a row is.)
struct VecRange {
    int first, last;
};
FTB_HD VecRange whole_vectors(int rows, int stride, int r, int mis, int nv)
{
    const int before = r < 8 ? r : 8, after = rows - r < 8 ? rows - r : 8;
    VecRange  V;
    V.first = before * stride < mis ? 1 : 0;
    V.last  = 8 * nv - mis > after * stride ? nv - 1 : nv;
    V.last  = V.last < V.first ? V.first : V.last;
    return V;
}

// The aligned 32-bit word around byte `at` of an array of n bytes: it starts at byte `from`, and `bytes` of it, counted from
// there, may be read; none where the array starts inside the word (that byte is then loaded by itself).
struct WordSpan {
    int from, bytes;
};
FTB_HD WordSpan word_span(size_t array, int n, int at)
{
    WordSpan W;
    W.from  = at - (int)((array + (size_t)at) & 3);
    W.bytes = W.from < 0 ? 0 : (n - W.from < 4 ? n - W.from : 4);
    return W;
}

// Whether the aligned 32-bit words around the entries of arrays of n bytes lie inside their arrays (null: no array).
FTB_HD bool whole_words(int n, size_t a, size_t b, size_t c)
{
    return n % 4 == 0 && ((a | b | c) & 3) == 0;
}

}  // namespace ftb200
