"""The blocks of the halo sweep program (host only): every slice's 16-byte pieces decode to the
program's columns, coefficients and rows, stay inside the block that the next slice starts after, and
the export numbers join each halo slot to the one row that its owner exports under it."""
import numpy as np
import pytest

from conftest import base_mesh
from test_halo_layout import NO_COL, dump_layout

from ufemism_gb300 import api


def block_layout(w, boundary, mixed):
    """Byte offsets (coefficients, rows, row data, end) of a slice's block."""
    coef = max(1, -(-w // 8)) * 512
    if mixed:
        row = coef + (0 if boundary else max(3, -(-w // 2)) * 512)
        return coef, row, row + 256, row + 768
    row = coef + (0 if boundary else w * 512)
    return coef, row, row + 512, row + 512 + (0 if boundary else 1536)


@pytest.mark.parametrize("name,n_patch", [("tiny", 0), ("1k", 0), ("4k", 7), ("4k", 40)])
def test_blocks_decode_to_the_program(name, n_patch):
    mesh = api.build_aaac(base_mesh(name))
    lay = dump_layout(mesh, n_patch=n_patch)
    n_patch, nP = int(lay["sizes"][0]), int(lay["sizes"][1])
    hp, e0, w = lay["hp_slice"], lay["hslice_e0"], lay["hslice_w"]
    ps = lay["patch_slice"].reshape(n_patch, 7)
    ex0, hl, hx, hd = lay["hex_ptr"], lay["hload_ptr"], lay["hload_ex"], lay["hload_dev"]
    exported = np.full(int(ex0[-1]), -1)
    for mixed in (True, False):
        prog = lay["hprog32" if mixed else "hprog64"].tobytes()
        first = lay["hslice_b32" if mixed else "hslice_b64"].astype(np.int64) * 16
        coefs = lay["hcuv32" if mixed else "hcuv"]
        for b in range(n_patch):
            p0, p1 = int(ps[b, 0]) * 32, int(ps[b, 6]) * 32
            for s in range(int(hp[7 * b]), int(hp[7 * b + 7])):
                boundary = s >= hp[7 * b + 5]
                n = int(w[s])
                coef, row, dat, end = block_layout(n, boundary, mixed)
                last = first[s + 1] if s + 1 < first.size else len(prog)
                assert first[s] + end == last
                blk = prog[first[s]:first[s] + end]
                cols = np.frombuffer(blk[:coef], np.uint16).reshape(-1, 32, 8).transpose(0, 2, 1).reshape(-1, 32)
                want = lay["hcol"][e0[s]:e0[s] + 32 * n].reshape(n, 32)
                # mixed colour slices: missing entries name the zero slot after the halo slots
                none = p1 - p0 + int(hl[b + 1] - hl[b]) if mixed and not boundary else NO_COL
                assert np.array_equal(cols[:n], np.where(want == NO_COL, none, want)) and np.all(cols[n:] == none)
                if not boundary:
                    per = 2 if mixed else 1
                    dt = np.float32 if mixed else np.float64
                    c = np.frombuffer(blk[coef:row], dt).reshape(-1, 32, per, 2).transpose(0, 2, 1, 3).reshape(-1, 32, 2)
                    used = want != NO_COL
                    assert np.array_equal(c[:n][used], coefs[e0[s]:e0[s] + 32 * n].reshape(n, 32, 2)[used])
                    assert not mixed or (np.all(c[:n][~used] == 0) and np.all(c[n:] == 0))
                words = np.frombuffer(blk[row:dat], np.uint32).reshape(32, 2 if mixed else 4)[:, 0]
                loc, ex = words & 0xFFFF, words >> 16
                rl, rg = lay["hrow_l"][32 * s:32 * s + 32], lay["hrow_g"][32 * s:32 * s + 32]
                assert np.array_equal(loc, np.where(rl < 0, NO_COL, rl))
                for lane in np.flatnonzero((rl >= 0) & (ex != NO_COL)):
                    e = int(ex0[b]) + int(ex[lane])
                    assert e < ex0[b + 1] and p0 <= rg[lane] < p1 and exported[e] in (-1, rg[lane])
                    exported[e] = rg[lane]
    assert np.all(exported >= 0)
    assert np.array_equal(exported[hx], hd)   # a halo slot polls the row it stands for
