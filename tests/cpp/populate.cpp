// populate_host with the system calls it makes counted: the page tables are looked
// at, and asked to be populated, no further than the first refusal.
#include <sys/mman.h>
#include <sys/syscall.h>
#include <unistd.h>

#include <cerrno>
#include <cstddef>
#include <cstdio>
#include <vector>

namespace fsr {
void populate_host(void* p, size_t bytes);
}

static int looks, asks, refuse;
extern "C" int mincore(void* p, size_t n, unsigned char* there)
{
    ++looks;
    return (int)syscall(SYS_mincore, p, n, there);
}
extern "C" int madvise(void* p, size_t n, int advice)
{
    ++asks;
    if (refuse) {
        errno = refuse;
        return -1;
    }
    return (int)syscall(SYS_madvise, p, n, advice);
}

int main()
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), bytes = 64 * 1024 * page;  // 64 looks of 1024 pages
    char* p = (char*)mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) return std::printf("no memory\n"), 0;
    for (int error : {EINVAL, EFAULT, ENOMEM}) {  // an older kernel, a mapping that may not be written, no memory
        refuse = error;
        looks = asks = 0;
        errno = 7;
        fsr::populate_host(p, bytes);
        if (looks != 1 || asks != 1 || errno != 7)
            return std::printf("refused with %d: %d looks, %d asks, errno %d\n", error, looks, asks, errno), 0;
    }
    refuse = 0;
    fsr::populate_host(p + 100, 3 * page);
    std::vector<unsigned char> there(bytes / page);
    syscall(SYS_mincore, p, bytes, there.data());
    for (size_t k = 0; k < there.size() && (there[0] & 1); ++k)  // (none: a kernel that refuses)
        if ((there[k] & 1) != (k < 4)) return std::printf("page %zu\n", k), 0;
    std::printf("ok\n");
    return 0;
}
