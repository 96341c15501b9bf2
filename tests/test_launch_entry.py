"""What a kernel launched with programmatic dependent launch may read before
its entry (griddepcontrol.wait, FE_PDL_ENTRY): nothing that a kernel of the
same stream writes.  Checked on the sources."""
import re

from conftest import ROOT

SOURCES = sorted((ROOT / "feng_gb300" / "csrc").glob("*.cu"))

# The products of an iteration, which take their operator's first entries
# ahead of the entry (constant from one factorisation to the next).
OPERATORS = {"k_down", "k_up", "k_dense", "k_bsell", "k_spmv"}
# The Gram-Schmidt passes, which take basis columns of earlier steps there.
BASIS = {"k_gs_dots_all", "k_gs_upd"}


def _close(text, i, pair):
    """Index behind the bracket that closes the one at i."""
    depth = 0
    for k in range(i, len(text)):
        depth += (text[k] == pair[0]) - (text[k] == pair[1])
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced source")


def entered_kernels():
    """(name, parameters, body) of every kernel with a dependent-launch entry."""
    for path in SOURCES:
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\b", text):
            i = text.index("(", m.end())
            head = text[m.end():i]
            if head.strip() == "__launch_bounds__":
                i = _close(text, i, "()")
                head, i = text[i:text.index("(", i)], text.index("(", i)
            end = _close(text, i, "()")
            b = text.index("{", end)
            body = text[b + 1:_close(text, b, "{}") - 1]
            if "FE_PDL_ENTRY" in body:
                yield head.split()[-1], text[i + 1:end - 1], body


def test_the_kernels_are_found():
    names = [n for n, _, _ in entered_kernels()]
    assert len(names) > 60 and OPERATORS | BASIS <= set(names)


def test_only_operators_and_older_columns_are_read_ahead_of_the_entry():
    late = [n for n, _, body in entered_kernels()
            if n not in OPERATORS | BASIS and not body.lstrip().startswith("FE_PDL_ENTRY();")]
    assert late == []
    for n, _, body in entered_kernels():
        if n in BASIS:
            # what runs there: the passes' loads (a lambda) only of columns below the step's newest
            # (the first eight where there are more), through the L2, and nothing of w
            ahead = re.sub(r"auto load = .*?\n  };", "", body[:body.index("FE_PDL_ENTRY")], flags=re.S)
            assert re.search(r"ahead = [^;]*(cb \+ 8 < ncols|ncols > 8);", ahead), n
            assert "__ldcg(" in ahead and "__ldcs(" not in ahead and "load(" not in ahead, n
            assert "w4[" not in ahead and "(w)[" not in ahead, n


# Read-only for as long as a system's set-up or factorisation stands: patterns
# and maps, and operators where an iteration's kernels read them.
CONSTANT = set("""ia ja a dinv sp sc sv ria rja ra tia tja ta trow qia qja qa qrow M steps stepStart start perm col from
lia lja ldiag val scale lvl rows srcPos diag pos upIa upPos upCol upColP dnIa dnPos dnCol slotOf dofX dofY dofC pRows
mass consts gs f g""".split())
# ... and where a kernel of the factorisation reads values that one before it wrote.
FORMED = {"k_bgather": {"a"}, "k_inv_diag": {"a"}, "k_diag_part": {"a"}, "k_gsum": {"a"}, "k_dw": {"a"},
          "k_gather_vals": {"a"}, "k_gsum_nc": {"a"}, "k_dw_nc": {"a"}, "k_fold_prep": {"g", "sc", "u"},
          "k_dot_part": {"a", "b"}, "k_copy_v": {"a"}, "k_copy": {"a"}, "k_ilu_pack": {"f"}}


def test_what_an_earlier_kernel_writes_is_read_through_plain_pointers():
    """Loads through const __restrict__ pointers are read-only to the compiler,
    which may move them ahead of the entry."""
    found = []
    for n, params, _ in entered_kernels():
        for x in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params):
            if x not in CONSTANT or x in FORMED.get(n, ()):
                found.append(f"{n}: {x}")
    assert found == []
