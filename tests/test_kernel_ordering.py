"""Orders of memory accesses that only timing would hide if they were wrong, read from the kernels' source."""
import pathlib
import re

CSRC = pathlib.Path(__file__).parent.parent / "mycel_b200/csrc"
SRC = (CSRC / "fp32_kernels.cu").read_text()


def _body(name):
    """The function's body, comments taken out."""
    at = re.search(r"__device__ __forceinline__ \w+ " + name + r"\(", SRC).start()
    open_, depth = SRC.index("{", at), 0
    for i in range(open_, len(SRC)):
        depth += {"{": 1, "}": -1}.get(SRC[i], 0)
        if depth == 0:
            return re.sub(r"//[^\n]*", "", SRC[open_:i])


def test_cluster_waits_for_every_cta_zeros():
    """The CTAs of the cluster kernel write into one another's vectors: each has to count itself in at the cluster
    barrier after its own zeros are stored, or a slow CTA's zeros overwrite what a fast one has put there."""
    body = _body("mg_tail_smem")
    zeros = [m.start() for m in re.finditer(r"make_float4\(0\.f, 0\.f, 0\.f, 0\.f\)", body)]
    arrive, wait, put = (body.index(s) for s in ("mg_cluster_arrive()", "mg_cluster_wait()", "mg_put_all("))
    assert zeros and max(zeros) < arrive < wait < put


def test_sums_read_other_ctas_parts_after_a_warp_barrier():
    """Lane 0 alone acquires the other CTAs' partial sums; a warp barrier has to stand between that and the other
    lanes' loads of them."""
    body = _body("grid_sums")
    acquired = body.index("atom.add.acq_rel")
    read = body.index("const volatile double*", acquired)
    assert "__syncwarp()" in body[acquired:read]


def test_dependent_kernels_promise_read_only_for_fixed_data_only():
    """A kernel that waits for the one before it (dep_begin) may not declare read-only what that one writes: the
    compiler could load it before the wait. Read-only are what a solve leaves as it is (moduli, stencils, inverse
    diagonals, flags, dampings) and the descriptor tables."""
    fixed = {"E", "S", "dom", "nf", "invd", "invdf", "invdc", "om", "tab"}
    seen = 0
    for name in ("fp32_kernels.cu", "fp64_kernels.cu"):
        src = (CSRC / name).read_text()
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(([^{;]*)\)\s*\{", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            if not re.search(r"dep_begin|mg_tail_smem|mg_apply_rows", src[m.end():i]):
                continue
            seen += 1
            named = set(re.findall(r"const \w+\* __restrict__ (\w+)", m.group(2)))
            assert named <= fixed, (m.group(1), named - fixed)
    assert seen >= 20
