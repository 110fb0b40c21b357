"""Patterns whose sweep steps fill their stage buffers: structures that get
buffers of one or two steps, four of them (tests of the ordered sweeps'
staging, on the CPU and on the GPU)."""
import numpy as np


def grid(nx, ny, nz, seed=1):
    """Seven-point pattern in its natural numbering (five-point for nz = 1)."""
    i = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    pairs = [np.stack([i[:-1].ravel(), i[1:].ravel()]), np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()]),
             np.stack([i[:, :, :-1].ravel(), i[:, :, 1:].ravel()])]
    return symmetric(nx * ny * nz, np.concatenate(pairs, axis=1), np.random.default_rng(seed))


def red_black(nx, ny, nz, hubs=0, spokes=0, seed=1):
    """Symmetric seven-point pattern, cells of one colour numbered first, and
    `hubs` of them coupled to `spokes` cells of the other colour each; values
    diagonally dominant by a tenth.  0-based ia, ja, dg, a."""
    n = nx * ny * nz
    i, j, k = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
    cell = (i + nx * (j + ny * k)).ravel()
    order = np.argsort(((i + j + k) % 2).ravel() * n + cell, kind="stable")
    number = np.empty(n, np.int64)
    number[cell[order]] = np.arange(n)
    at = lambda a, b, c: number[(a + nx * (b + ny * c)).ravel()]
    pairs = [np.stack([at(i[:-1], j[:-1], k[:-1]), at(i[1:], j[1:], k[1:])]),
             np.stack([at(i[:, :-1], j[:, :-1], k[:, :-1]), at(i[:, 1:], j[:, 1:], k[:, 1:])]),
             np.stack([at(i[:, :, :-1], j[:, :, :-1], k[:, :, :-1]), at(i[:, :, 1:], j[:, :, 1:], k[:, :, 1:])])]
    rng = np.random.default_rng(seed)
    red = (n + 1) // 2
    for h in range(hubs):
        other = red + rng.choice(n - red, spokes, replace=False)
        pairs.append(np.stack([np.full(spokes, h * (red // max(1, hubs))), other]))
    return symmetric(n, np.concatenate(pairs, axis=1), rng)


def blocks_coupled(n1, n2, between, seed=2):
    """n1 rows that do not depend on each other, each coupled to the same n2
    further rows, through a chain of `between` rows in the numbering."""
    n = n1 + between + n2
    tail = n1 + between + np.arange(n2)
    pairs = [np.stack([np.repeat(np.arange(n1), n2), np.tile(tail, n1)])]
    if between:
        chain = n1 - 1 + np.arange(between + 1)
        pairs.append(np.stack([chain[:-1], chain[1:]]))
    return symmetric(n, np.concatenate(pairs, axis=1), np.random.default_rng(seed))


def symmetric(n, pairs, rng):
    key = np.unique(np.min(pairs, axis=0).astype(np.int64) * n + np.max(pairs, axis=0))
    p = np.stack([key // n, key % n])
    v = -rng.uniform(0.5, 1.5, p.shape[1])
    diag = np.zeros(n)
    np.add.at(diag, p[0], -1.1 * v)
    np.add.at(diag, p[1], -1.1 * v)
    row = np.concatenate([p[0], p[1], np.arange(n)])
    col = np.concatenate([p[1], p[0], np.arange(n)])
    val = np.concatenate([v, v, diag])
    s = np.lexsort((col, row))
    row, col, val = row[s], col[s], val[s]
    ia = np.zeros(n + 1, np.int32)
    np.add.at(ia, row + 1, 1)
    return np.cumsum(ia).astype(np.int32), col.astype(np.int32), np.flatnonzero(row == col).astype(np.int32), val


def write_pattern(path, ia, ja, dg):
    with open(path, "wb") as f:
        f.write(np.array([len(dg), len(ja)], np.int32).tobytes())
        for v in (ia, ja, dg):
            f.write(np.ascontiguousarray(v, np.int32).tobytes())


# structures whose exchanged values leave no room for steps of 32 rows: pattern, tiles
DENSE = {
    "hubs_16": (lambda: red_black(16, 16, 16, 40, 200), 4),
    "hubs_24": (lambda: red_black(24, 24, 24, 40, 200), 12),
    "blocks": (lambda: blocks_coupled(250, 250, 0), 8),
    "most": (lambda: blocks_coupled(255, 255, 0), 3),
}

# pattern, tiles, steps of a buffer (setups and applications, Gauss-Seidel)
STAGED = {
    "red_black": (dict(nx=24, ny=24, nz=24), 12, 2, 2),
    "hubs": (dict(nx=30, ny=30, nz=30, hubs=40, spokes=200), 30, 1, 1),
    "small_hubs": (dict(nx=30, ny=30, nz=30, hubs=100, spokes=60), 30, 2, 1),
}
