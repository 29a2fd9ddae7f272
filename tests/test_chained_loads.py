"""Loads of kernels that are launched while their predecessor still runs, by their source.

Such a kernel's lifetime begins before the predecessor's last write.  A load through ``const __restrict__`` or a
read-only load (``__ldg``, ``ld.global.nc``) is only valid for memory that nobody writes during the kernel's lifetime, and
the compiler may move the former above the wait for the predecessor.  Weights and biases are written by no
kernel of a chain; everything else has to be read by ordinary loads."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "iris_testing_b200" / "csrc"
UNWRITTEN = {"wr", "wr_kmajor", "bias"}


def functions(text, keyword):
    """(name, parameter list, body) of every function whose definition starts with ``keyword``."""
    for m in re.finditer(keyword + r"(?:void\s+)?(?:__launch_bounds__\([^()]*\)\s*)?(\w+)\(([^{};]*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(2), text[m.end():i]


def chained_kernels():
    for f in sorted(CSRC.glob("*.cu")):
        for name, params, body in functions(f.read_text(), "__global__ "):
            if "chain_wait()" in body:
                yield f.name, name, params, body


def test_chained_kernels_take_no_read_only_views_of_what_the_chain_writes():
    found = set()
    for file, name, params, body in chained_kernels():
        found.add(name)
        views = set(re.findall(r"\*\s*__restrict__\s+(\w+)", params)) - UNWRITTEN
        assert not views, (file, name, views)
        loads = [a for a in re.findall(r"(?:__ldg|ld_nc_16)\(([^()]*)", body) if not a.startswith("ra.bias")]
        assert not loads, (file, name, loads)
    assert {"plan_count_kernel", "plan_place_kernel", "route_plan_small_kernel", "grouped_gemm_kernel", "slot_reduce_kernel",
            "padded_bulk_kernel", "padded_wait_kernel", "weighted_gather_kernel"} <= found, found


def test_router_tile_reads_only_weights_through_the_read_only_path():
    text = (CSRC / "router_mma.cuh").read_text()
    assert set(re.findall(r"__ldg\((\w+)", text)) <= {"wp"}
    for name, params, body in functions(text, "__device__ __forceinline__ "):
        assert not set(re.findall(r"\*\s*__restrict__\s+(\w+)", params)) - UNWRITTEN, name
