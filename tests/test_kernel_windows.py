"""Shared-memory and tensor-memory layouts of the tensor-core counters and of the projection, restated
over every shape they can be given, with the constants read from the sources: every window that is
written or read stays inside its allocation."""
import os
import re

import tensorfim_b200 as tf

CSRC = os.path.join(os.path.dirname(os.path.abspath(tf.__file__)), "csrc")
SM_BYTES = 227 * 1024


def _constants(*names):
    """The integer constants of the sources, in order (later files may use earlier ones')."""
    env = {}
    for name in names:
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"//.*", "", f.read())
        for decl in re.findall(r"^constexpr (?:int|int32_t|int64_t|uint32_t) (k\w+ = [^;]*);", src, re.M):
            for part in re.split(r",\s*(?=k\w+ =)", decl):
                key, expr = part.split(" = ", 1)
                env[key] = int(eval(expr.replace("1u", "1"), {"sizeof": None}, env))
    return env


def test_wave_counter_windows():
    c = _constants("tfim_internal.h", "tcgen05.cuh", "count_f4.cu")
    K = type("K", (), c)
    assert K.kQSmem <= SM_BYTES - 20 * 1024 and K.kQWideSmem <= K.kQSmem   # 16 KiB staging of A's words and barriers beside it
    # tensor memory: the accumulator, the scales, two stages of A
    assert K.kQN <= K.kQScale and K.kQScale + 3 * K.kScaleCols <= K.kQACol and K.kQACol + 64 * K.kQWideStages <= K.kQTmemCols == 512
    for cols in range(1, K.kQM + 1):
        for nr in range(1, K.kQN + 1):
            n = (nr + 15) & ~15
            ua, ub = (cols + 7) >> 3, n >> 3
            units = ua + ub
            narrow = units <= K.kQNarrow
            # the host's side of the same line (tiles_f4)
            assert narrow == (not (cols + 7) // 8 + (nr + 15) // 16 * 2 > K.kQNarrow)
            rb = ua if narrow else 0
            kc = 4 if units <= K.kQNarrow // 2 else 2 if narrow else 1
            kb_bytes = (rb + ub) * 1024
            stage = kc * K.kQBlocks * kb_bytes
            stages = min(K.kQMaxStages, (K.kQStaged - K.kQGuard) // stage) if narrow else K.kQWideStages
            assert stages >= 2 and 64 % (kc * K.kQChunkWords) == 0   # slices are multiples of 64 words
            room = (K.kQSmem if narrow else K.kQWideSmem) - 1024     # behind the 1,024-byte alignment
            last = stages * stage - kb_bytes                         # the last K block
            assert last + (rb + ub) * 1024 <= room                   # what is written, and the B window
            if narrow:
                assert last + K.kQM * 128 <= room                    # the A window: 128 rows whatever the width
                load = kc * units
                per_warp = 1 if load <= K.kQExpWarps else 2 if load <= 2 * K.kQExpWarps else 3
                assert load <= per_warp * K.kQExpWarps and per_warp <= K.kQUnits
            else:
                assert ub <= 4 * (K.kQExpWarps - K.kQAWarps)


def test_family_counter_windows():
    c = _constants("tfim_internal.h", "tcgen05.cuh", "count_pk.cu")
    K = type("K", (), c)
    assert K.kPSmem <= SM_BYTES - 512 and 256 + 3 * K.kScaleCols <= 512 and K.kPScale == 256
    for cols in range(1, K.kPkMaxCols + 1):
        cls = max(0, (cols - 1) >> 3) if cols <= 40 else 5 if cols <= 64 else 6
        per = 16 // (cls + 1) if cls <= 3 else {4: 3, 5: 2, 6: 1}[cls]
        assert per <= K.kPkJobs and per * ((cols + 7) // 8) <= K.kPUnits   # every column has its unit
        for r0 in range(cols):
            for nr in range(1, cols - r0 + 1):
                lo, hi = r0 >> 3, (r0 + nr + 7) >> 3
                u0, u1 = (lo * per) & ~1, min(K.kPUnits, (hi * per + 1) & ~1)
                n = 8 * (u1 - u0)
                assert 16 <= n <= 128 and n % 16 == 0
                # the window holds the tail rows' units of all jobs, and ends inside the block
                assert u0 <= lo * per and hi * per <= u1 and u0 * 1024 + n * 128 <= K.kPBlockBytes


def test_projection_windows():
    c = _constants("resident.cu")
    K = type("K", (), c)
    tile, far = K.kProjTile * 32, 32 * K.kProjWarps
    assert K.kProjGroups % 2 == 1
    for gc in range(1, K.kProjGroups + 1, 2):
        assert (1024 * gc + 32) * 4 <= SM_BYTES
        assert 1023 * gc + (gc - 1) + 31 < 1024 * gc + 32            # a word of padding per 32 transactions
        assert (tile + far) * gc <= 0xFFFF                           # rows as 16-bit offsets, the zero row last
        rows = (((tile + far + 1) * gc + 3) & ~3) * 4
        assert rows + K.kProjWarps * (tile + 32) * 2 <= SM_BYTES
        assert (tile + 32) * 2 % 16 == 0                             # each warp's list starts on 16 bytes
    # a list: up to 31 entries before the tile's first whole word, the tile's, and padding to 32
    assert max(32 * ((lead + n + 31) >> 5) for lead in range(32) for n in range(tile + 1)) <= tile + 32
