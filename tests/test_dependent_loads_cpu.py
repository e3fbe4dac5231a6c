"""The kernels that are launched as programmatic dependents are resident while the kernel before
them still writes, so nothing that a kernel of the chain writes (level set, blurred fields, data
factor) may reach them through the non-coherent load (`__ldg`), which wants memory that stays
unwritten for the whole life of the kernel.  Read from the sources: which load a kernel issues does
not show in its results."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "paper-rsf-vesselseg_gb300" / "csrc"
# loads of the image, which no kernel writes
IMAGE_LOADS = {"load_img", "image_bits", "border_word"}


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _functions(text):
    """name -> body of every function defined in `text`."""
    out = {}
    for m in re.finditer(r"\b(\w+)\s*\((?:[^(){};]|\([^()]*\))*\)\s*(?:const\s*)?\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        if m.group(1) not in ("if", "for", "while", "switch"):
            out.setdefault(m.group(1), text[m.end():i])
    return out


def _argument(text, start):
    depth, i = 1, start
    while depth:
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        i += 1
    return text[start:i - 1].strip()


def test_dependent_kernels_read_the_chains_fields_coherently():
    functions = {}
    for path in sorted(CSRC.glob("*.cuh")):
        functions.update(_functions(_code(path)))
    launched = set()
    for path in sorted(CSRC.glob("*.cu")):
        code = _code(path)
        if "launch_dependent(" in code:
            launched |= {n for n in re.findall(r"\b(\w+_kernel)\s*<", code)}
    launched -= {n for n in launched if re.search(r"\bdebug\b|_debug_|adjoint|^box_", n)}  # ordinary launches
    assert {"xpass_kernel", "ypass_kernel", "ypass_chunk_kernel", "zpass_kernel", "zpass_chunk_kernel",
            "stencil_pair_kernel"} <= launched
    reached, todo = set(), sorted(launched)
    while todo:
        name = todo.pop()
        if name in reached or name not in functions:
            continue
        reached.add(name)
        todo += sorted(set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\s*\(", functions[name])) & functions.keys() - reached)
    assert {"find_sv", "zchunk", "pair_step"} <= reached
    bad = []
    for name in sorted(reached - IMAGE_LOADS):
        for m in re.finditer(r"__ldg\(", functions[name]):
            arg = _argument(functions[name], m.end())
            if not re.match(r"pre\b", arg):  # the block prefix table, written before the chain
                bad.append(f"{name}: __ldg({arg})")
    assert not bad, bad
