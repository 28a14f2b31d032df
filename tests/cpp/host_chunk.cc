/* prints host_chunk() of each "frames n pinned posterior" on the command line */
#include <cstdio>
#include <cstdlib>
#include "host_batch.h"

int main(int argc, char** argv)
{
    for (int i = 1; i + 3 < argc; i += 4)
        std::printf("%lu\n", wldpc::host_chunk(std::strtoul(argv[i], nullptr, 10), std::strtoul(argv[i + 1], nullptr, 10),
                                               std::atoi(argv[i + 2]) != 0, std::atoi(argv[i + 3]) != 0));
    return 0;
}
