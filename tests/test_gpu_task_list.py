"""The task list is written whole whatever its items hold (GPU).

The list is sized by the cells' task counts and written by the items'; the host
compares the two only after a count pass may have read the list.  A program
against the engine's internal launcher writes a list that is longer than its one
item's tasks, over memory filled with ones: the rest has to be empty tasks.
"""
import os
import subprocess

import pytest

import sjoin

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(sjoin.PKG), "csrc")
INCLUDE = os.path.join(os.path.dirname(os.path.dirname(sjoin.PKG)), "include")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "sj_internal.h"
template <typename T> T *dev(const T *h, size_t n)
{
    T *d = nullptr;
    cudaMalloc((void **)&d, n * sizeof(T));
    cudaMemcpy(d, h, n * sizeof(T), cudaMemcpyHostToDevice);
    return d;
}
int main()
{
    const uint32_t cellStart[2] = {0, 10}, none[2] = {0, 0}, nt = 5;   // one cell of ten points, no neighbours
    sj_task tasks[nt];
    float pred[nt];
    memset(tasks, 0xff, sizeof(tasks));
    memset(pred, 0xff, sizeof(pred));
    sj_taskgen g{};
    g.cellStart = dev(cellStart, 2);
    g.nbrStart = dev(none, 2);
    g.nbrCell = dev(none, 1);
    g.groupBase = dev(none, 1);
    g.groupLen = dev(none, 1);
    g.nCells = 1;
    g.tile = 128;
    g.cap = 1000000;
    g.pairsPerTask = 4096;
    g.sym = 1;
    sj_task *dTasks = dev(tasks, nt);
    float *dPred = dev(pred, nt);
    const uint32_t *zero = dev(none, 2);
    cudaError_t e = sj_tg_item_write(g, zero, nullptr, zero, 1, zero, dTasks, nt, dPred, 0);
    if (e == cudaSuccess) e = cudaMemcpy(tasks, dTasks, sizeof(tasks), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(pred, dPred, sizeof(pred), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return 2;
    for (uint32_t t = 0; t < nt; t++)
        printf("%u %u %u %u %u %u %u %u %d\n", tasks[t].cell, tasks[t].qBegin, tasks[t].qCount, tasks[t].segBase,
               tasks[t].segCount, tasks[t].sBegin, tasks[t].sEnd, tasks[t].flags, pred[t] == 0.0f);
    return 0;
}
"""


def test_tasks_left_over_are_empty(tmp_path):
    sjoin.load()
    (tmp_path / "list.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, "-I", INCLUDE, "-I", os.path.join(CUDA, "include"),
                           str(tmp_path / "list.cpp"), "-o", str(tmp_path / "list"), "-L", sjoin.PKG, "-lsj",
                           f"-Wl,-rpath,{sjoin.PKG}", "-L", os.path.join(CUDA, "lib64"), "-lcudart_static", "-lpthread",
                           "-ldl", "-lrt"])
    rows = [[int(x) for x in ln.split()] for ln in subprocess.check_output([str(tmp_path / "list")], text=True).split("\n")
            if ln]
    assert rows[0][:8] == [0, 0, 10, 0, 1, 0, 10, 3]
    assert all(row == [0] * 8 + [1] for row in rows[1:]) and len(rows) == 5
