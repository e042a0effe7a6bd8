"""Static check that runs without a GPU: every call of a native op (``lib.<op>(...)`` / ``native.lib().<op>(...)``)
in the package, the tests and the benchmark names an op the library registers and passes a number of arguments
that op's schema accepts.  The ops themselves only run on a GPU, so a binding that drifted from its call sites
would otherwise first show on a GPU box."""
import ast
import re
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def _is_lib_call(base: ast.AST) -> bool:
    if isinstance(base, ast.Name):
        return base.id == "lib"
    if isinstance(base, ast.Call):
        f = base.func
        return (isinstance(f, ast.Attribute) and f.attr == "lib") or (isinstance(f, ast.Name) and f.id == "lib")
    return False


def test_native_op_call_sites_match_the_registered_schemas():
    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    torch.ops.load_library(str(native.lib_path()))
    ns = torch.ops.piper_c
    files = sorted((ROOT / "piper_b200").rglob("*.py")) + sorted((ROOT / "tests").glob("*.py")) \
        + [ROOT / "bench.py", ROOT / "__graft_entry__.py"]
    problems, checked = [], 0
    for path in files:
        for node in ast.walk(ast.parse(path.read_text())):
            if not (isinstance(node, ast.Call) and isinstance(node.func, ast.Attribute) and _is_lib_call(node.func.value)):
                continue
            if any(isinstance(a, ast.Starred) for a in node.args):
                continue
            name = node.func.attr
            op = getattr(ns, name, None)
            if op is None:
                problems.append(f"{path.relative_to(ROOT)}:{node.lineno}: no native op named {name}")
                continue
            args = op.default._schema.arguments
            required = sum(1 for a in args if not a.has_default_value())
            given = len(node.args) + len(node.keywords)
            checked += 1
            if not required <= given <= len(args):
                problems.append(f"{path.relative_to(ROOT)}:{node.lineno}: {name} gets {given} arguments, "
                                f"its schema takes {required}..{len(args)}")
    assert not problems, "\n".join(problems)
    assert checked > 100


def test_read_only_pointers_come_out_of_the_wait():
    """A kernel that may start before the one in front of it has ended reads nothing early: what the compiler may take for
    constant over the kernel (const __restrict__) goes through the wait."""
    waits, problems = 0, []
    for path in sorted((ROOT / "piper_b200" / "csrc").glob("*.cu")):
        text = path.read_text()
        for m in re.finditer(r"\bgrid_(?:wait|begin)\(([^)]*)\);", text):
            function = text[text.rfind("\n}\n", 0, m.start()):m.start()]
            params = re.findall(r"const [\w ]+\* __restrict__ (\w+)", function)
            missing = set(params) - {a.strip() for a in m.group(1).split(",")}
            waits += 1
            if missing:
                problems.append(f"{path.name}:{text[:m.start()].count(chr(10)) + 1}: {sorted(missing)}")
    assert waits > 20 and not problems, problems


def test_products_draw_their_first_tile_behind_the_wait():
    for name in ("gemm_sm100.cu", "grouped_gemm_sm100.cu"):
        text = (ROOT / "piper_b200" / "csrc" / name).read_text()
        lines = text[:text.index("atomicAdd(&p.sched[0], 1)")].splitlines()[-3:]
        assert any(line.strip() == "grid_wait();" for line in lines), name


@pytest.mark.parametrize("M,N,K,f32,sms,rows", [
    (2048, 4096, 4096, False, 148, 256),      # 128 big tiles in one round, 256 small ones in two
    (2048, 4096, 2048, False, 148, 128),      # the same with too short a contraction
    (1184, 6400, 64, False, 100, 128),        # 125 in two, 250 in three
    (4096, 5120, 8192, False, 148, 128),      # 320 in three, 640 in five
    (9472, 8192, 64, False, 148, 256),        # 1184 in eight, 2368 in sixteen
    (2048, 4096, 64, False, 64, 256),         # two rounds against four
    (2048, 4096, 8192, False, 256, 128),      # one round either way
    (2048, 4096, 4096, True, 148, 128), (4096, 2048, 4096, True, 148, 256),      # wide and tall fp32
    (255, 65536, 4096, False, 148, 128), (65536, 255, 4096, False, 148, 128),    # narrower than a big tile
    (65536, 256, 64, False, 148, 256),
])
def test_gemm_tile_rule(M, N, K, f32, sms, rows):
    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    assert native.lib().gemm_tile_rows(M, N, K, f32, sms) == rows


@pytest.mark.parametrize("M,N,K,b_mn,f32,sms,shape", [
    (1, 8, 8, False, False, 148, (1, 32)),                    # one tile: the narrowest
    (512, 768, 256, False, False, 148, (1, 32)),              # 96 tiles on as many SMs
    (128, 16384, 2048, False, False, 148, (1, 128)),          # 128 tiles in one round
    (200, 8192, 3072, False, False, 148, (2, 128)),           # the same with two rows of tiles: pairs
    (1000, 3072, 8192, False, False, 148, (2, 192)),          # 64 pairs of 192 columns in one round, 48 of 256 in one
    (1000, 8192, 3072, True, False, 148, (2, 224)),           # 148 pairs in two rounds exactly
    (4096, 28672, 4096, False, False, 148, (2, 256)), (28672, 4096, 4096, True, True, 148, (2, 256)),
    (4096, 28672, 4096, False, False, 1, (1, 256)),           # no pairs on a single SM
    (2048, 2048, 448, False, False, 148, (1, 256)),           # near ties, by gemm_tile_rows: 128 rows where pairs cost less
    (4096, 4096, 256, False, False, 148, (2, 256)),           # and 256 rows where they cost more
])
def test_gemm_shape_rule(M, N, K, b_mn, f32, sms, shape):
    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    assert tuple(native.lib().gemm_shape(M, N, K, b_mn, f32, sms)) == shape


@pytest.mark.parametrize("M,N,K,b_mn,f32,sms,splits", [
    (128, 2048, 128256, True, False, 148, 8), (1, 8, 32000, True, False, 148, 32),      # few tiles over a long contraction
    (128, 2048, 128256, False, False, 148, 1), (128, 2048, 128256, True, True, 148, 1),  # forward pass, fp32 buckets
    (1000, 4096, 28672, True, False, 148, 1), (4096, 4096, 28672, True, False, 148, 1),  # tiles for every SM
    (512, 768, 256, True, False, 148, 1), (128, 256, 448, True, False, 148, 1),          # short contractions
    (128, 1024, 8192, True, False, 1, 1),                                                # one SM gains nothing
])
def test_gemm_split_rule(M, N, K, b_mn, f32, sms, splits):
    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    lib = native.lib()
    ctas, width, got = lib.gemm_split_shape(M, N, K, b_mn, f32, sms)
    assert got == splits
    if got == 1:
        assert (ctas, width) == tuple(lib.gemm_shape(M, N, K, b_mn, f32, sms))


def test_gemm_split_parts_have_blocks_and_scratch_is_bounded():
    import random

    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    rng, split = random.Random(3), 0
    for _ in range(2000):
        M, N, K = (int(2 ** rng.uniform(0, top)) for top in (12, 14, 17))
        _, _, parts = native.lib().gemm_split_shape(M, N, K, True, False, rng.choice([148, 148, 64, 1]))
        blocks = -(-K // 64)
        per = -(-blocks // parts)
        assert (parts - 1) * per < blocks <= parts * per                # none is empty
        assert parts == 1 or parts * (M + 31) * (N + 7) * 4 <= (64 << 20) + parts * 4 * 31 * (M + N + 64)
        split += parts > 1
    assert split > 100


@pytest.mark.parametrize("B,S,Hq,Hkv,sms,parts", [
    (1, 4096, 32, 32, 148, 1), (1, 4096, 32, 8, 148, 1), (1, 4096, 32, 4, 148, 2), (1, 5120, 16, 2, 148, 2),
    (1, 512, 32, 4, 148, 4), (1, 2048, 16, 2, 148, 8), (8, 1024, 16, 2, 148, 1), (8, 128, 16, 4, 148, 1),
    (1, 1024, 12, 2, 148, 2), (1, 1024, 9, 3, 148, 1), (1, 5120, 16, 2, 16, 1), (0, 128, 2, 1, 148, 1),
])
def test_attention_backward_parts_rule(B, S, Hq, Hkv, sms, parts):
    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    assert native.lib().attn_bwd_parts(B, S, Hq, Hkv, sms) == parts


@pytest.mark.parametrize("B,S,Hq,sms,tiles", [
    (1, 128, 148, 148, 1), (1, 128, 149, 148, 2),         # an SM for every tile, and one too few (one block each)
    (1, 512, 44, 148, 1), (1, 512, 45, 148, 2),           # 440 of 444 block times in which the longest tile is done
    (1, 2048, 16, 148, 1), (2, 2048, 8, 148, 1), (1, 2048, 17, 148, 2),
    (1, 2048, 16, 64, 2), (8, 4096, 32, 148, 2),
])
def test_attention_tiles_per_cta_rule(B, S, Hq, sms, tiles):
    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    assert native.lib().attn_tiles_per_cta(B, S, Hq, sms) == tiles
