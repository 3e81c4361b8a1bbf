"""A kernel that raises the step's status itself and has block barriers must not
let each thread read the status and leave on its own: a block that starts while
another block raises it would lose some of its warps before the barrier, and the
others would go on with shared memory that nobody wrote.  Read from the sources
(such a kernel is not run to see it fail): the status is read by one thread, or
combined over the block by the barrier itself."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcmtop_b200", "csrc")
FUNCTION = re.compile(r"__(global|device)__[^;{}]*?\b(\w+)\s*\([^;{}]*\)\s*(?:const\s*)?\{")
OWN_EXIT = re.compile(r"^\s*if \((?!__syncthreads_or|threadIdx)[^\n]*(?:status->code|skip_step\()[^\n]*return", re.M)


def functions():
    """(file, name) -> (is a kernel, body without comments) of every device function."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        # launch bounds hold parentheses of their own
        text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
        for m in FUNCTION.finditer(text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            key = (os.path.basename(path), m.group(2))
            old = out.get(key, (False, ""))
            out[key] = (m.group(1) == "global" or old[0], old[1] + text[m.end():at])
    return out


def reaches(funcs, needle):
    """Names of the functions whose body, or that of a function they name, holds needle."""
    hit = {k for k, (_, body) in funcs.items() if needle in body}
    while True:
        names = {name for _, name in hit} - {"operator"}
        word = re.compile(r"\b(%s)\s*[<(]" % "|".join(sorted(names)))
        more = {k for k, (_, body) in funcs.items() if word.search(body)} - hit
        if not more:
            return hit
        hit |= more


def offenders(*files):
    funcs = functions()
    both = reaches(funcs, "raise_status(") & reaches(funcs, "__syncthreads")
    kernels = [k for k in both if funcs[k][0]]
    assert kernels
    return sorted(name for file, name in kernels if file in files and OWN_EXIT.search(funcs[(file, name)][1]))


def test_the_reading_finds_kernels():
    funcs = functions()
    assert funcs[("cells.cu", "k_cell_keys")][0] and not funcs[("cells.cu", "origin_of")][0]
    assert ("cells.cu", "k_ghost_count") in reaches(funcs, "raise_status(")   # through origin_of
    assert OWN_EXIT.search("    if (a.status->code) return;") and OWN_EXIT.search("    if (skip_step(a)) return;")
    assert not OWN_EXIT.search("    if (__syncthreads_or(skip_step(a))) return;")


def test_cell_and_ghost_kernels_leave_as_blocks():
    assert offenders("cells.cu") == []


def test_every_kernel_leaves_as_blocks():
    assert offenders(*os.listdir(CSRC)) == []
