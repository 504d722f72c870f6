"""The chain kernels' index arithmetic (csrc/qf_chain_index.cuh) as a host library."""
import ctypes
import functools
import os
import subprocess
import tempfile

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quantforge_b200", "csrc")
SOURCE = """
#include "qf_chain_index.cuh"
using namespace qf;
static StreamPhase phase(int pieces, int q, int r, int streams, int home, int flip) { return {0, pieces, q, r, streams, home, flip, 0, {-1, -1}}; }
extern "C" {
int range_first(int id, int q, int r) { int u; stream_range(phase(0, q, r, 0, 0, 0), id, &u); return u; }
int range_units(int id, int q, int r) { int u; return stream_range(phase(0, q, r, 0, 0, 0), id, &u); }
int of(int u, int q, int r) { return stream_of(phase(0, q, r, 0, 0, 0), u); }
int piece(int pieces, int streams, int home, int flip, int id, int round) { return stream_piece(phase(pieces, 0, 0, streams, home, flip), id, round); }
int number(int n_sm, int home, int per_sm, int first_sm, int place) { return (int)sc_number(n_sm, home, per_sm, first_sm, place); }
int place(int n_sm, int sm, int sms, unsigned *started, unsigned *given) {
    return (int)sc_place(n_sm, sm, sms, [&] { return started[sm]++; }, [&](unsigned i) { return given[i]++; });
}
}
"""


@functools.cache
def library():
    folder = tempfile.mkdtemp()
    path = os.path.join(folder, "chain_index.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-fPIC", "-shared", "-I", CSRC, "-x", "c++", "-", "-o", path],
                   input=SOURCE, text=True, check=True)
    return ctypes.CDLL(path)
