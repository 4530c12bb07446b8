"""Rules of kernels that begin while the one before them in the stream ends
(programmatic dependent launches), and of the copies they read, checked in the
source: no GPU needed.

An overlapped kernel's fields are written by the kernel before it while it already
lives, so it must not take them through __restrict__ pointers: the compiler may
then load them through the non-coherent path, or above the wait.  Tables of
descriptors and units are written by copies that end before the launch begins."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "pysweep_b200", "csrc")
TABLES = {"BlockInst", "MarchInst", "SweptArgs", "int2"}
WAITS = ("grid_wait()", "griddepcontrol.wait", "block_stream_body", "block_tile_body", "march_body")


def _kernels(text):
    """(parameters, body) of every kernel defined in `text`."""
    for m in re.finditer(r"__global__", text):
        name = re.compile(r"(?:__launch_bounds__\s*\([^;{]*?\)\s*)?(\w+)\s*\(").search(text, m.end())
        i = text.index("(", name.start(1))
        depth, j = 1, i + 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[j], 0)
            j += 1
        k = j
        while text[k] not in "{;":
            k += 1
        if text[k] == ";":
            continue
        depth, e = 1, k + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[e], 0)
            e += 1
        yield name.group(1), text[i + 1:j - 1], text[k:e]


def test_overlapped_kernels_promise_nothing_about_their_fields():
    seen = []
    for f in sorted(os.listdir(CSRC)):
        text = re.sub(r"//.*", "", open(os.path.join(CSRC, f)).read())
        for name, params, body in _kernels(text):
            if not any(w in body for w in WAITS):
                continue
            seen.append(name)
            for p in params.split(","):
                if "__restrict__" in p:
                    kind = re.sub(r"\bconst\b", "", p).split("*")[0].strip()
                    assert kind in TABLES, f"{f}: {name}: {p.strip()}"
    assert {"heat_standard", "heat_block_stream", "heat_block_tile", "heat_block_tile_batch",
            "heatvar_tile", "heatvar_back", "euler_march", "euler_march_batch", "psh_block"} <= set(seen)


def test_device_data_is_copied_on_the_stream_that_reads_it():
    """Solvers and batches run on non-blocking streams, which the legacy stream's
    copies do not wait for and are not waited for by; one from pageable memory may
    return before it lands."""
    for f in sorted(os.listdir(CSRC)):
        text = re.sub(r"//.*", "", open(os.path.join(CSRC, f)).read())
        assert not re.search(r"\bcuda(Memcpy|Memset|Memcpy2D|MemcpyToSymbol)\s*\(", text), f
