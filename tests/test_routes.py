"""The rules that pick a kernel by sizes (csrc/it_route.h), held to their edges on the CPU.  148 SMs are a B200's."""
import ctypes as C
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "irontimber_b200", "csrc")
SM = 148


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    d = tmp_path_factory.mktemp("routes")
    src, lib = d / "routes.cpp", d / "routes.so"
    src.write_text('#include "it_route.h"\n'
                   'extern "C" int takes_tc(long rg, long cols, long ntok, int sm) { return it_mm_takes_tc(rg, cols, ntok, sm); }\n'
                   'extern "C" int tc_tile(long rg, long ntok, int sm) { return it_tc_tile(rg, ntok, sm); }\n'
                   'extern "C" int attn_tiled(int slot0, int nt, int blk, int sm) { return it_attn_takes_tiled(256, 24, 4, slot0, nt, blk, sm); }\n'
                   'extern "C" int attn_group(int hd, int nh, int nkv, int npos) { auto g = it_attn_grouping(hd, nh, nkv, npos); return 10 * g.heads + g.rows; }\n'
                   'extern "C" int mv_ring(int slots, int groups) { return it_mv_ring(slots, groups); }\n'
                   'extern "C" int gdn_rows(int sd, int nt) { return it_gdn_rows_takes(sd, nt); }\n')
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-Wno-unused-function", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


@pytest.mark.parametrize("rows,cols,ntok,tc", [
    (512, 1024, 32, 0), (512, 1024, 33, 1), (5000, 1024, 9, 0), (9000, 1024, 9, 1), (4736, 2048, 32, 0), (4737, 2048, 9, 1), (32, 3072, 9, 1)])
def test_tile_kernel_of_a_product(routes, rows, cols, ntok, tc):
    assert routes.takes_tc(C.c_long((rows + 31) // 32), C.c_long(cols), C.c_long(ntok), SM) == tc


@pytest.mark.parametrize("rows,ntok,tile", [
    (9472, 64, 2), (9473, 64, 1), (5120, 65, 1), (4736, 128, 2), (4737, 128, 1), (9472, 128, 1), (9473, 128, 0), (18944, 64, 1), (34816, 512, 0), (34816, 64, 1)])
def test_tiles_by_rounds(routes, rows, ntok, tile):
    assert routes.tc_tile(C.c_long((rows + 31) // 32), C.c_long(ntok), SM) == tile


# passes at the 27B shape measured both ways (24 heads over 4 of dimension 256), where the sides differ by more than 2 %: a prompt from
# position 0, a few new tokens far into a context, passes in several blocks of rows
@pytest.mark.parametrize("slot0,nt,tiled", [
    (0, 9, 0), (0, 128, 0), (0, 257, 0), (0, 384, 1), (0, 512, 1), (0, 777, 1),
    (500, 32, 0), (500, 96, 0), (500, 192, 1), (1024, 9, 0), (1024, 96, 0), (1024, 128, 1), (2048, 32, 0), (2048, 96, 0), (2048, 128, 1),
    (4096, 24, 0), (4096, 64, 0), (4096, 96, 0), (4096, 128, 1), (4096, 256, 1), (7000, 9, 0), (7000, 64, 0), (7000, 96, 1), (7000, 192, 1),
    (11200, 192, 0), (12400, 256, 0), (13900, 9, 0), (14000, 32, 1), (14300, 64, 1), (19500, 256, 1)])
def test_attention_of_a_prompt_pass(routes, slot0, nt, tiled):
    npad = (slot0 + nt + 127) // 128 * 128
    assert routes.attn_tiled(slot0, nt, min(nt, (32 << 20) // (24 * npad)), SM) == tiled


@pytest.mark.parametrize("hd,nh,nkv,npos,heads,rows", [
    (256, 24, 4, 6400, 3, 2), (256, 24, 4, 6402, 3, 1), (256, 24, 4, 13056, 3, 1), (256, 24, 4, 13057, 3, 0), (256, 4, 2, 100, 2, 2), (256, 4, 4, 100, 1, 2),
    (256, 4, 4, 19713, 1, 0), (64, 32, 1, 100, 2, 2), (100, 24, 4, 100, 0, 0)])
def test_grouping_of_attention_heads(routes, hd, nh, nkv, npos, heads, rows):
    """One head a CTA keeps two rows or gives way."""
    assert routes.attn_group(hd, nh, nkv, npos) == 10 * heads + rows


@pytest.mark.parametrize("sd,nt,takes", [(128, 1, 0), (128, 2, 0), (128, 3, 1), (128, 9, 1), (64, 9, 0), (256, 9, 0)])
def test_prompt_delta_rule(routes, sd, nt, takes):
    """One or two tokens are refused: one warp would store a state row that the other may not have read yet."""
    assert routes.gdn_rows(sd, nt) == takes


def overtaken_copy(slots, groups):
    """A chunk whose group can find its slot a phase behind: the chunk before it in the slot may still be landing when the group, through with
    its own chunks up to then, begins to wait.  Copies land in any order; a chunk is issued when its slot's last one has been read."""
    for q in range(slots, 4 * slots):
        own = range(q - groups, -1, -groups)                       # chunks this group has read
        read = set(own)
        for c in own:                                              # a chunk that was read had been issued, and so had all before it: their slots' last ones were read
            read |= set(range(0, c - slots + 1))
        if q - slots not in read:
            return q
    return None


@pytest.mark.parametrize("slots", range(4, 17))
def test_ring_of_several_groups(routes, slots):
    """Three groups of k_matvec_t2 on the ring that the launch gives them; sizes that are no multiple of three can be overtaken."""
    ring = routes.mv_ring(slots, 3)
    assert 3 <= ring <= slots and overtaken_copy(ring, 3) is None
    assert slots % 3 == 0 or overtaken_copy(slots, 3) is not None
    with open(os.path.join(CSRC, "it_matvec_t2.cu")) as f:
        src = f.read()
    assert re.findall(r"launch_cfg<MT, 3,[^;]*;", src) == re.findall(r"launch_cfg<MT, 3,[^;]*it_mv_ring\(slots, 3\)[^;]*;", src) != []
