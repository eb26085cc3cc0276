// Whole numbers out of a Python list or tuple: what a step's tokens and wanted places come as.  The interpreter's own conversions
// go through an iterator and a checked store per entry (2,048 of them: 34 us by array.array); this reads the entries in place.
// The interpreter's functions are declared here (they are part of its stable ABI), so that no header of it is needed, and are
// found in the process that loads this library.  The caller holds the interpreter's lock (ctypes.PyDLL).
#include <cstddef>
#include <cstdint>

extern "C" {
struct _object;
_object* PyList_GetItem(_object* list, ptrdiff_t i);
_object* PyTuple_GetItem(_object* tuple, ptrdiff_t i);
long long PyLong_AsLongLongAndOverflow(_object* v, int* overflow);
_object* PyErr_Occurred();
void PyErr_Clear();

// seq (a list, or a tuple) has n entries; out [n].  0, or -1 where an entry is no whole number of 64 bits (or the sequence shrank
// while an entry converted itself): out is then not to be used, and no exception is left behind.
int imparo_int_sequence(_object* seq, int tuple, long long n, int64_t* out) {
    for (long long i = 0; i < n; ++i) {
        _object* item = tuple ? PyTuple_GetItem(seq, (ptrdiff_t)i) : PyList_GetItem(seq, (ptrdiff_t)i);
        int overflow = 0;
        const long long v = item ? PyLong_AsLongLongAndOverflow(item, &overflow) : -1;
        if (!item || overflow != 0 || (v == -1 && PyErr_Occurred())) {
            PyErr_Clear();
            return -1;
        }
        out[i] = v;
    }
    return 0;
}
}
