"""Training calls with the tile heights (rows per warp) that the library takes for them on 148 SMs, at
ITERS sweeps in intervals of CKPT: the GPU tests run them, the route tests hold the heights."""

ITERS, CKPT = 25, 11

# one pair: (H, W, rows of the backward's tiles); each but the first of several tiles, its exchange
# in lambda's second buffer
SINGLE = [(24, 119, 2), (600, 799, 3), (437, 613, 4), (720, 1279, 4), (801, 1198, 5), (950, 1501, 6)]

# a batch: (shapes, rows of each forward launch, rows of each backward launch)
GROUPS = [([(500, 701)] * 5, [2, 6], [2, 6]),
          ([(240, 321)] * 20, [8], [2, 6]),
          ([(200, 150)] * 32, [7], [3, 4]),
          ([(300, 402)] * 14, [2, 7], [5, 5])]
