"""The library's kernels run on streams that do not wait for the default stream. So no host data and no memset may go to
device memory through the default stream (cudaMemcpy, cudaMemset and their pitched forms): a copy from pageable memory
may return before its data is on the device, a memset always does, and a kernel launched next could overtake them. Reads
back to the host are complete when they return, and follow a synchronise of the stream that wrote."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "atsat_gb300", "csrc")
DEFAULT_STREAM = re.compile(r"\b(cudaMem(?:cpy|set)(?:2D|3D)?|cudaMemcpyToSymbol|cudaMemcpyFromSymbol)\s*\(")


def calls(text):
    """(line, name, arguments) of every default-stream copy or memset, comments and texts left out."""
    text = re.sub(r'//[^\n]*|/\*.*?\*/|"(?:\\.|[^"\\\n])*"', lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.S)
    for m in DEFAULT_STREAM.finditer(text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text.count("\n", 0, m.start()) + 1, m.group(1), text[m.end():i - 1]


def test_no_default_stream_writes_to_the_device():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")) or name == "conv_check.cu":     # its kernels run on the default stream
            continue
        for line, fn, args in calls(open(os.path.join(CSRC, name)).read()):
            if "cudaMemcpyDeviceToHost" not in args:
                found.append(f"{name}:{line} {fn}")
    assert not found, found
